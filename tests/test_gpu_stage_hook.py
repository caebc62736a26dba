"""Timing a stage of the solve (p2_debug_time_stage) leaves the context as it
was: the next solve takes the same iterations to the same bits."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("stage", sorted(capi.DebugHooks.STAGES))
def test_a_solve_after_timing_a_stage(stage, precision):
    m = M.random_spheres_model(33, 2, 3, (1e-1, 1e1), markers=(2, 2, 2), seed=4)
    prob = P.StokesProblem(m, precision=precision)
    prob.ronurecalc()
    want, info = prob.solve_fp64()
    assert info.status == 0
    H = capi.DebugHooks(prob.ctx)
    for variant in (0, 2) if stage in ("residual", "true_residual", "operator") else (0,):
        assert H.time_stage(stage, variant=variant, reps=2) > 0
        got, again = prob.solve_fp64()
        assert again.iterations == info.iterations
        for k in want:
            assert np.array_equal(got[k], want[k]), (k, variant)
    prob.close()
