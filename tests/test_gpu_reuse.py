"""One context set up anew: other boundary tables (a few unknowns fewer on the
coarsest level, the padded size the same), the same sides in another order,
another precision.  Every V-cycle is bit for bit a fresh context's, from a
blocked inverse that stands (flag 0), so nothing of an earlier set-up is left
in the captured graphs."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu
KEYS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


def _setup(shape, levels, precision, fixed):
    """Model, parameters and boundary tables with `fixed` more Vx rows of the coarsest level held at 0."""
    m = M.random_spheres_model(shape[0], levels, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1, shape=shape)
    m.params.nubeg, m.params.nuend = 1e-3, 1e3
    lv, c = m.levels, levels
    bondm, v1, n1 = m.bc.bondm.copy(), [m.bc.bondv1], [m.bc.bondn1]
    for q in range(fixed):
        u = lv.mgp[c] + 4 * lv.mgxy[c] + (3 + q) * lv.mgy[c] + 4
        assert bondm[4 * u + 1] == 0
        bondm[4 * u + 1] = m.bc.bondnum + 1 + q
        v1.append(np.zeros((1, 2), np.float32))
        n1.append(np.zeros(1, np.int32))
    return m, P.params_for(m, precision=precision), (bondm, np.concatenate(v1), np.concatenate(n1))


def _vcycle(ctx, m, params, tables):
    ctx.set_grid(m.gx, m.gy, m.gz, params)
    ctx.set_bc(*tables)
    rng = np.random.Generator(np.random.PCG64(2))
    ctx.set_nodes({k: np.exp(rng.uniform(-1, 1, m.nodenum)).astype(np.float32) for k in KEYS})
    free = unknown_mask(m.shape) & (m.bc.bondm[:4 * m.nodenum] == 0)
    H = capi.DebugHooks(ctx)
    x = H.vcycle(np.where(free, rng.standard_normal(4 * m.nodenum), 0.0))
    flag, _ = H.coarse()
    assert flag == 0
    assert np.all(np.isfinite(x)) and np.any(x != 0)
    return x


@pytest.mark.parametrize("steps", [
    [((9, 12, 10), 0, 1, 0), ((9, 12, 10), 0, 1, 3), ((9, 12, 10), 0, 1, 0)],
    [((9, 12, 10), 0, 1, 0), ((12, 10, 9), 0, 1, 0), ((10, 9, 12), 0, 1, 1)],
    [((11, 11, 11), 0, 1, 0), ((11, 11, 11), 0, 0, 0)],
    [((17, 19, 21), 1, 0, 0), ((17, 19, 21), 1, 0, 2), ((21, 17, 19), 1, 0, 2), ((21, 17, 19), 1, 1, 2)],
])
def test_a_context_set_up_anew_is_a_fresh_one(steps):
    ctx = capi.Context(0)
    for step in steps:
        m, params, tables = _setup(*step)
        got = _vcycle(ctx, m, params, tables)
        fresh = capi.Context(0)
        want = _vcycle(fresh, m, params, tables)
        fresh.close()
        assert np.array_equal(got, want), step
    ctx.close()


def test_pivoted_inverse_agrees():
    """The coarsest inverse by the pivoted LU on request, then the blocked one again: both ways stay usable."""
    m, params, tables = _setup((9, 12, 10), 0, 1, 0)
    ctx = capi.Context(0)
    want = _vcycle(ctx, m, params, tables)
    H = capi.DebugHooks(ctx)
    assert H.coarse(1)[0] == -1
    assert H.coarse()[0] == 0
    assert np.array_equal(_vcycle(ctx, m, params, tables), want)
    ctx.close()
