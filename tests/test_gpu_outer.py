"""The outer loop's vector kernels (dots, orthogonalisation, solution update)
at the edges of their dispatch: one, two and the most stored vectors, vectors
below and above the length from which a thread takes four pairs, an odd node
count.  The converged solution must not depend on the restart length."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import model as M

pytestmark = pytest.mark.gpu


def _solve(m, fields, precision, restart, tol=1e-10):
    prob = P.StokesProblem(m, precision=precision, restart=restart, tol=tol, max_iter=600)
    try:
        prob.set_nodes(fields)
        sol, info = prob.solve_fp64()
    finally:
        prob.close()
    assert info.status == 0 and info.rel_residual <= tol
    return sol


@pytest.mark.parametrize("shape,levels,restarts", [((33, 33, 33), 2, (1, 2, 18)), ((37, 33, 41), 2, (3, 17)),
                                                   ((69, 69, 69), 3, (5, 18))])
@pytest.mark.parametrize("precision", [0, 1])
def test_restart_lengths_agree(shape, levels, restarts, precision):
    m = M.random_spheres_model(shape[0], levels, 3, (1e-1, 1e1), markers=(2, 2, 2), seed=6, shape=shape)
    prob = P.StokesProblem(m)
    fields = prob.ronurecalc()
    prob.close()
    ref = _solve(m, fields, 1, 16)
    for r in restarts:
        sol = _solve(m, fields, precision, r)
        # residuals at 1e-10 of the right-hand side leave the solutions within 1e-6 of each other, the bound
        # that the parity tests derive for 1e-8
        for k in ("vx", "vy", "vz", "pr"):
            assert np.linalg.norm(sol[k] - ref[k]) <= 1e-6 * np.linalg.norm(ref[k]), (r, k)
