"""Markers by cell: the counting sort (no cell above 256 markers) and the
radix sort (one cell above) give the oracle's node fields bit for bit, with the
markers in shuffled order, empty cells, markers outside the box, types that are
not interpolated, and a cell at and just above the limit."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import model as M

pytestmark = pytest.mark.gpu


def _model(crowd, shape, viscmod):
    m = M.random_spheres_model(shape[0], 1, 3, (1e-2, 1e2), markers=(2, 1, 2), seed=8, shape=shape)
    m.params.viscmod = viscmod
    rng = np.random.Generator(np.random.PCG64(crowd + 1))
    keep = rng.random(m.markx.size) < 0.8
    x, y, z, t = (a[keep] for a in (m.markx, m.marky, m.markz, m.markt))
    # crowd markers in the cell (2, 3, 4), which the regular ones leave
    g = [m.gx, m.gy, m.gz]
    lo = [g[a][2 + a] for a in range(3)]
    hi = [g[a][3 + a] for a in range(3)]
    out = ~((x > lo[0]) & (x < hi[0]) & (y > lo[1]) & (y < hi[1]) & (z > lo[2]) & (z < hi[2]))
    x, y, z, t = (a[out] for a in (x, y, z, t))
    more = [(lo[a] + (hi[a] - lo[a]) * rng.uniform(0.01, 0.99, crowd)).astype(np.float32) for a in range(3)]
    away = [np.array([-0.5, 0.5, 0.5, 0.0], np.float32), np.array([0.5, 1.5, 0.5, 0.5], np.float32),
            np.array([0.5, 0.5, 0.0, 0.5], np.float32)]
    mt = np.concatenate([t, rng.integers(0, 4, crowd).astype(np.int8), np.zeros(4, np.int8)])
    mt[:3] = 60  # types from 50 on are not interpolated
    order = rng.permutation(mt.size)
    m.markx, m.marky, m.markz = (np.concatenate([a, b, c]).astype(np.float32)[order]
                                 for a, b, c in zip((x, y, z), more, away))
    m.markt = mt[order]
    return m


@pytest.mark.parametrize("crowd", [0, 256, 257, 700])
@pytest.mark.parametrize("shape,viscmod", [((17, 19, 21), 0), ((12, 9, 33), 1)])
def test_sorts_match_the_oracle(oracle_mod, crowd, shape, viscmod):
    m = _model(crowd, shape, viscmod)
    want = oracle_mod.ronurecalc(m)
    prob = P.StokesProblem(m)
    got = prob.ronurecalc()
    prob.close()
    for k in want:
        assert np.array_equal(got[k], want[k]) if viscmod == 0 else np.allclose(got[k], want[k], rtol=1e-6), k
