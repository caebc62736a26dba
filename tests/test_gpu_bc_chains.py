"""Boundary rows that copy boundary rows with coefficients whose product has no
exact float: after FP64 sweeps every row holds its own equation to FP64
rounding, whichever form the level's sweeps take."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu
KEYS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


# 49^3 takes a launch per pass, 27^3 the grid, 16^3 the cluster
@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("precision,eps", [(1, 2.0 ** -53), (0, 2.0 ** -24)])
def test_chained_rows_hold_their_equations(smoother, precision, eps):
    m = M.random_spheres_model(49, 2, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1)
    m.params.nubeg, m.params.nuend = 1e-3, 1e3
    lv, bc = m.levels, m.bc
    rng = np.random.Generator(np.random.PCG64(8))
    v1 = np.array(bc.bondv1, np.float32)
    linked = np.nonzero(bc.bondn1)[0]
    v1[linked, 1] = rng.choice(np.array([0.3, 0.7, -0.9], np.float32), linked.size)
    ctx = P.Context(0)
    ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m, precision=precision, smoother=smoother))
    ctx.set_bc(bc.bondm, v1, bc.bondn1)
    ctx.set_nodes({k: np.exp(rng.uniform(-1, 1, m.nodenum)).astype(np.float32) for k in KEYS})
    H = capi.DebugHooks(ctx)
    for l in range(3):
        n, off = lv.mgn[l], 4 * lv.mgp[l]
        mask = unknown_mask((lv.mgx[l], lv.mgy[l], lv.mgz[l]))
        row = np.where(mask, bc.bondm[off:off + 4 * n], 0)
        target = np.where((row > 0) & (bc.bondn1[row] > 0), bc.bondn1[row] - 1 - off, -1)
        chained = np.nonzero((target >= 0) & (row[target] > 0))[0]
        assert chained.size > 0
        x, b = (np.where(mask, rng.standard_normal(4 * n), 0.0).astype(np.float32).astype(np.float64) for _ in range(2))
        got = H.smooth(l, 2, b, x)
        u = np.nonzero(target >= 0)[0]
        k = v1[row[u], 1].astype(np.float64)
        t = target[u]
        size = np.abs(b[u]) + np.abs(k * got[t]) + np.abs(k * b[t])
        # two links, a few roundings each
        assert np.all(np.abs(got[u] - (b[u] + k * got[t])) <= 8 * eps * size), l
    ctx.close()
