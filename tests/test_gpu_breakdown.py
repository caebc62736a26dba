"""A solve whose V-cycle stops giving numbers in the middle of a cycle of
directions (over-relaxed sweeps that diverge, in FP32): it reports P2_ERR_NAN,
keeps the corrections up to there and reports the true residual of what it
returns."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu


def test_corrections_before_the_breakdown_count():
    m = M.random_spheres_model(17, 1, 1, (1e-2, 1e2), markers=(2, 2, 2), seed=4)
    ref = P.StokesProblem(m, precision=1, tol=1e-12)
    ref.ronurecalc()
    exact, info = ref.solve_fp64()
    assert info.status == 0
    H = capi.DebugHooks(ref.ctx)
    keys = ("pr", "vx", "vy", "vz")
    rows = unknown_mask(m.shape).reshape(-1, 4)
    pin = m.params.pin
    rows[pin[2] * m.shape[0] * m.shape[1] + pin[0] * m.shape[1] + pin[1], 0] = False
    inter = lambda s: np.stack([s[k] for k in keys], axis=1).reshape(-1)
    norm = lambda x: np.linalg.norm(H.apply(0, x).reshape(-1, 4)[rows])
    seen = 0
    for omega in np.arange(1.70, 1.84, 0.01):
        prob = P.StokesProblem(m, precision=0, omega=float(omega), npre=[32, 32], npost=[32, 32], max_iter=30, tol=1e-10,
                               restart=18)
        prob.ronurecalc()
        info = prob.ctx.solve_resident(check=False)
        got = prob.ctx.solution(m.nodenum)
        prob.close()
        if info.status != 5 or info.iterations < 2:
            continue
        seen += 1
        assert any(np.any(got[k] != 0) for k in ("vx", "vy", "vz"))
        assert info.rel_residual < info.rel_residual0 <= 1.0
        rel = norm(inter(exact) - inter(got)) / norm(inter(exact))
        assert abs(rel - info.rel_residual) <= 1e-6
    assert seen > 0
    ref.close()
