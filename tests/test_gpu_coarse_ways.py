"""Which way the coarsest inverse is formed: the pivoted band LU on levels long
along z (their band is narrow), the blocked elimination on the others; either
way the one-level V-cycle solves A x = b, and a singular level is a status."""
import numpy as np
import pytest

from pardiso2_b200 import capi
from tests.test_gpu_coarse import _check, _fields, _one_level

pytestmark = pytest.mark.gpu


# on both sides of the rule's line: 8 x 8 x 50 and 8 x 8 x 70 (6 and 9 thousand unknowns, half band 160)
@pytest.mark.parametrize("shape,lu", [((8, 8, 70), True), ((8, 8, 50), False), ((50, 8, 9), False)])
@pytest.mark.parametrize("precision,tol", [(1, 1e-9), (0, 1e-1)])  # as in test_inverse
def test_the_sizes_choose(shape, lu, precision, tol):
    rng = np.random.Generator(np.random.PCG64(3))
    m, prob = _one_level(shape, precision, _fields(int(np.prod(shape)), rng))
    H = capi.DebugHooks(prob.ctx)
    assert H.coarse()[0] == (-1 if lu else 0)
    assert H.coarse(1)[0] == -1 and H.coarse(2)[0] == 0
    _check(m, prob, tol)
    prob.close()


def test_a_singular_long_level_is_a_status():
    """A cell whose six faces are held leaves its pressure without an equation; afterwards the context solves again."""
    shape = (8, 8, 70)
    nx, ny, nz = shape
    rng = np.random.Generator(np.random.PCG64(3))
    f = _fields(nx * ny * nz, rng)
    m, prob = _one_level(shape, 1, f)
    i, j, k = 4, 4, 30
    at = lambda a, b, c: 4 * (c * nx * ny + a * ny + b)
    bondm, v1, n1 = m.bc.bondm.copy(), [m.bc.bondv1], [m.bc.bondn1]
    for q, uc in enumerate((at(i - 1, j - 1, k - 1) + 1, at(i, j - 1, k - 1) + 1, at(i - 1, j - 1, k - 1) + 2,
                            at(i - 1, j, k - 1) + 2, at(i - 1, j - 1, k - 1) + 3, at(i - 1, j - 1, k) + 3)):
        assert bondm[uc] == 0
        bondm[uc] = m.bc.bondnum + 1 + q
        v1.append(np.zeros((1, 2), np.float32))
        n1.append(np.zeros(1, np.int32))
    prob.ctx.set_bc(bondm, np.concatenate(v1), np.concatenate(n1))
    prob.set_nodes(f)
    with pytest.raises(capi.P2Error) as e:
        prob.ctx.solve_resident()
    assert e.value.code == 6  # P2_ERR_SINGULAR
    prob.ctx.set_bc(m.bc.bondm, m.bc.bondv1, m.bc.bondn1)
    prob.set_nodes(f)
    _check(m, prob, 1e-9)
    prob.close()
