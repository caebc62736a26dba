"""The check of the blocked coarsest inverse does not depend on the units: the
inverse stands at any size and viscosity of the box (metres and Pa s among
them), fails where a pivot vanishes, and solves A x = b either way."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_coarse import KEYS, _check

pytestmark = pytest.mark.gpu


def _problem(shape, side, eta, contrast):
    m = M.random_spheres_model(shape[0], 0, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1, shape=shape)
    m.gx, m.gy, m.gz = (g * side for g in (m.gx, m.gy, m.gz))
    m.params.nubeg, m.params.nuend = 1e-6 * eta, 1e6 * eta
    prob = P.StokesProblem(m, precision=1)
    rng = np.random.Generator(np.random.PCG64(6))
    f = {k: (eta * contrast ** rng.uniform(-0.5, 0.5, m.nodenum)).astype(np.float32) for k in KEYS}
    prob.set_nodes(f)
    return m, prob, f


# side of the box and mean viscosity: nondimensional, stiff, a 500 km box of mantle rock, a 10 cm box of syrup
@pytest.mark.parametrize("side,eta", [(1.0, 1.0), (1.0, 1e8), (5e5, 1e21), (0.1, 1e2), (1e-3, 1e-3)])
@pytest.mark.parametrize("shape", [(9, 10, 8), (12, 12, 12)])
def test_units_do_not_matter(shape, side, eta):
    m, prob, _ = _problem(shape, side, eta, 1e4)
    assert capi.DebugHooks(prob.ctx).coarse(2)[0] == 0
    prob.close()


@pytest.mark.parametrize("side,eta", [(1.0, 1.0), (5e5, 1e21)])
def test_a_vanishing_pivot_is_seen(side, eta):
    """As test_vanishing_pivot_takes_the_pivoted_path: the six viscosities of one Vx row far below the others."""
    shape = (9, 10, 8)
    nx, ny, nz = shape
    m, prob, f = _problem(shape, side, eta, 1e1)
    prob.close()
    i, j, k = 4, 4, 3
    at = lambda a, b, c: c * nx * ny + a * ny + b
    for key, nodes in (("nxx", [(i + 1, j + 1, k + 1), (i, j + 1, k + 1)]), ("nxy", [(i, j, k), (i, j + 1, k)]),
                       ("nxz", [(i, j, k), (i, j, k + 1)])):
        for q in nodes:
            f[key][at(*q)] = 0.0
    m.params.nubeg = 1e-30 * eta
    prob = P.StokesProblem(m, precision=1)
    prob.set_nodes(f)
    assert capi.DebugHooks(prob.ctx).coarse()[0] > 0
    if side == 1.0:
        _check(m, prob, 1e-8)
    prob.close()
