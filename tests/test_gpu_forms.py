"""Devices that cannot place a cluster of 16 blocks, or a cooperative grid of a
block per SM: the resident sweeps step down to the next form (p2_debug_forms
stands in for such a device) and the results stay."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.golden.make_golden import HEAT_COMMON
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu
KEYS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


# level 1 of 33^3 (19^3) takes the cluster, level 0 the grid; both smoothers
@pytest.mark.parametrize("smoother", [0, 1])
@pytest.mark.parametrize("precision,tol", [(0, 2e-4), (1, 1e-11)])  # as test_gpu_resident.py: rounding of the same sweeps
def test_smoother_forms_agree(smoother, precision, tol):
    m = M.random_spheres_model(33, 1, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1)
    m.params.nubeg, m.params.nuend = 1e-3, 1e3
    lv = m.levels
    rng = np.random.Generator(np.random.PCG64(4))
    f = {k: np.exp(rng.uniform(-1, 1, m.nodenum)).astype(np.float32) for k in KEYS}
    data = []
    for l in range(2):
        mask = unknown_mask((lv.mgx[l], lv.mgy[l], lv.mgz[l]))
        data.append([mask] + [np.where(mask, rng.standard_normal(4 * lv.mgn[l]), 0.0) for _ in range(2)])
    out, kernels = {}, []
    for without in (0, 1, 2):
        ctx = P.Context(0)
        H = capi.DebugHooks(ctx)
        H.forms(without)
        ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m, precision=precision, smoother=smoother, max_iter=1))
        ctx.set_bc(m.bc.bondm, m.bc.bondv1, m.bc.bondn1)
        ctx.set_nodes(f)
        out[without] = [H.smooth(l, 3, b, x)[mask] for l, (mask, x, b) in enumerate(data)]
        kernels.append(ctx.solve_resident(check=False).kernels)
        ctx.close()
    for without in (1, 2):
        for l in range(2):
            want = out[0][l]
            assert np.linalg.norm(out[without][l] - want) <= tol * np.linalg.norm(want), (without, l)
    # the grid form stands in for the cluster with the same operations
    assert np.array_equal(out[1][1], out[0][1]) and np.array_equal(out[1][0], out[0][0])
    assert kernels[0] == kernels[1] < kernels[2]  # a launch per call or per pass


# nodes of one colour: 16337 takes the cluster, 17298 the grid
@pytest.mark.parametrize("shape", [(31, 33, 31), (31, 35, 31)])
def test_heat_forms_agree(shape):
    g = [M.uniform_lines(n) for n in shape]
    lv = M.make_levels(*g, 1)
    sp = M.SolverParams()
    bc = M.build_bc_tables(lv, M.free_slip_lines(sp.pin, sp.pinit) + M.thermal_lines())
    no = np.zeros(0, np.float32)
    m = M.Model("box", *g, 1, lv, bc, no, no, no, np.zeros(0, np.int8), M.Rocks(np.ones(1), np.ones(1), np.zeros(1)), sp)
    th = M.thermal_fields(m, seed=5)
    d = dict(HEAT_COMMON, heatmin=5e-3, multinumt=1, multicyct=1, pre=[5, 0], post=[0, 5], frictyn=0, adiabyn=0,
             heatdif=0.0, max_cycles=200)
    hp = capi.heat_params(**{k: d[k] for k in ("maxtkstep", "heatmin", "t0koef", "t1koef", "heatdif", "tdeep", "zdeep",
                                               "multinumt", "multicyct", "frictyn", "adiabyn", "max_cycles", "pre", "post")})
    out, kernels = [], []
    for without in (0, 1, 2):
        ctx = P.Context(0)
        capi.DebugHooks(ctx).forms(without)
        ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m))
        ctx.heat_set_bc(bc, m.nodenum)
        tk, _, info = ctx.titerate(hp, 500.0 * (64.0 / 34) ** 2, th)
        out.append(tk)
        kernels.append(info.kernels)
        ctx.close()
    # the same operations in the same order in every form
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert kernels[0] == kernels[1] < kernels[2]
