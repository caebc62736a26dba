"""Heat smoother with a level resident in one launch: on both sides of each
limit of its forms (one block of 1024 threads, a cluster of 16, a block per SM,
a launch per colour beyond) against the oracle.

Both stop once the RMS error of the heat rows times the sub-step is below
heatmin; the bars follow from it as in test_gpu_heat.py."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.golden.make_golden import HEAT_COMMON

pytestmark = pytest.mark.gpu
TK_MAX, TK_RMS = 0.1, 0.02

# nodes of one colour: 936, 1080, 16337, 17298, 148840, 152561
SHAPES = [(9, 15, 13), (9, 15, 15), (31, 33, 31), (31, 35, 31), (61, 79, 61), (61, 81, 61)]


@pytest.mark.parametrize("levels", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_heat_sweeps_forms(oracle_mod, shape, levels):
    g = [M.uniform_lines(n) for n in shape]
    nl, n = 0, min(shape)
    while (n - 5) // 2 + 5 >= 7 and (n - 5) // 2 + 5 < n:
        nl, n = nl + 1, (n - 5) // 2 + 5
    lv = M.make_levels(*g, nl)
    sp = M.SolverParams()
    bc = M.build_bc_tables(lv, M.free_slip_lines(sp.pin, sp.pinit) + M.thermal_lines())
    no = np.zeros(0, np.float32)
    m = M.Model("box", *g, nl, lv, bc, no, no, no, np.zeros(0, np.int8), M.Rocks(np.ones(1), np.ones(1), np.zeros(1)), sp)
    th = M.thermal_fields(m, seed=5)
    if levels > nl:
        pytest.skip("one level only")
    v = dict(multinumt=levels, multicyct=1, pre=[5, 0][:levels + 1], post=[0, 5][:levels + 1], frictyn=0, adiabyn=0,
             heatdif=0.0)
    dt = 500.0 * (64.0 / (max(shape) - 1)) ** 2  # about half a cell diffusion time
    hpd = dict(HEAT_COMMON, **v, heatmin=5e-3, gx=sp.gx, gy=sp.gy, gz=sp.gz, max_cycles=200, timestep=dt)
    tko, _, oi = oracle_mod.titerate(*g, levels, bc.bondt, bc.bondv1, bc.bondn1, hpd, th)
    assert not oi["capped"]
    prob = P.StokesProblem(m)
    prob.ctx.heat_set_bc(bc, m.nodenum)
    hp = capi.heat_params(**{k: hpd[k] for k in ("maxtkstep", "heatmin", "t0koef", "t1koef", "heatdif", "tdeep", "zdeep",
                                                 "multinumt", "multicyct", "frictyn", "adiabyn", "max_cycles", "pre",
                                                 "post")})
    tk, _, info = prob.ctx.titerate(hp, dt, th)
    again, _, _ = prob.ctx.titerate(hp, dt, th)
    assert info.converged == 1 and info.substeps == oi["substeps"]
    d = tk.astype(np.float64) - tko
    assert np.abs(d).max() <= TK_MAX and np.sqrt(np.mean(d * d)) <= TK_RMS
    assert np.array_equal(tk, again)
    prob.close()
