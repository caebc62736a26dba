"""In a batch the levels of the cooperative form take a launch per pass where
that gives the same bits (FP32, full cell block): more launches, the solution
of a solve alone; with the diagonal block or in FP64 the form stays."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M

pytestmark = pytest.mark.gpu


# 33^3, 43 x 45 x 41 and level 1 of 49^3 are grid levels; odd sides and doubled sweeps among them
@pytest.mark.parametrize("precision,smoother,changes", [(0, 1, True), (0, 0, False), (1, 1, False)])
def test_a_batch_gives_the_bits_of_single_solves(precision, smoother, changes):
    probs = []
    for shape, levels, per in (((33, 33, 33), 2, [4, 4, 4]), ((43, 45, 41), 2, [4, 8, 16]), ((49, 49, 49), 3, [4, 8, 16, 32])):
        m = M.random_spheres_model(shape[0], levels, 3, (1e-2, 1e2), markers=(2, 2, 2), seed=shape[1], shape=shape)
        p = P.StokesProblem(m, precision=precision, smoother=smoother, npre=per, npost=per)
        p.ronurecalc()
        probs.append((m, p))
    single = [(p.ctx.solve_resident(), p.ctx.solution(m.nodenum)) for m, p in probs]
    for threads in (0, 2, 1):
        infos, _ = capi.solve_batch([p.ctx for _, p in probs], host_threads=threads)
        for (m, p), info, (alone, want) in zip(probs, infos, single):
            assert info.iterations == alone.iterations
            assert (info.kernels > alone.kernels) == (changes and threads != 1)
            got = p.ctx.solution(m.nodenum)
            for k in want:
                assert np.array_equal(got[k], want[k]), (m.shape, k, threads)
    for m, p in probs:  # alone again: the form of a single solve
        assert p.ctx.solve_resident().kernels == single[[q for q, _ in probs].index(m)][0].kernels
        p.close()
