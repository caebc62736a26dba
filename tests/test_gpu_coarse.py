"""The coarsest level's inverse.  On a grid of one level the V-cycle is the
coarsest solve, so p2_debug_vcycle solves A x = b: blocked Gauss-Jordan on
sizes with and without padding in its last tiles, its pivoted fallback on an
operator with a vanishing pivot, and a status (no fault) where the operator
is not a number."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu
KEYS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


def _fields(n, rng):
    return {k: np.exp(rng.uniform(-1.0, 1.0, n)).astype(np.float32) for k in KEYS}


def _one_level(shape, precision, fields, nubeg=1e-3):
    m = M.random_spheres_model(shape[0], 0, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1, shape=shape)
    m.params.nubeg, m.params.nuend = nubeg, 1e3
    prob = P.StokesProblem(m, precision=precision)
    prob.set_nodes(fields)
    return m, prob


def _check(m, prob, tol):
    """A V(b) = b on the free rows for a random b (zero on the boundary rows, which the solve takes as homogeneous)"""
    rng = np.random.Generator(np.random.PCG64(5))
    free = unknown_mask(m.shape) & (m.bc.bondm[:4 * m.nodenum] == 0)
    b = np.where(free, rng.standard_normal(4 * m.nodenum), 0.0)
    H = capi.DebugHooks(prob.ctx)
    r = H.apply(0, H.vcycle(b)) - b
    err = np.linalg.norm(r[free]) / np.linalg.norm(b)
    assert err < tol, err


# the operator's condition number on these grids is about 1e5: 1e-9 leaves FP64
# four digits of slack, 1e-1 the FP32 copy of the inverse (6e-8 times it) one
@pytest.mark.parametrize("shape", [(8, 8, 8), (9, 11, 10), (12, 12, 12), (13, 9, 14)])
@pytest.mark.parametrize("precision,tol", [(1, 1e-9), (0, 1e-1)])
def test_inverse(shape, precision, tol):
    rng = np.random.Generator(np.random.PCG64(3))
    m, prob = _one_level(shape, precision, _fields(int(np.prod(shape)), rng))
    _check(m, prob, tol)
    prob.close()


def test_vanishing_pivot_takes_the_pivoted_path():
    """One interior Vx whose six stencil viscosities are 1e-30 has a diagonal
    that elimination without interchanges cannot divide by."""
    shape = (9, 10, 8)
    nx, ny, nz = shape
    rng = np.random.Generator(np.random.PCG64(4))
    f = _fields(nx * ny * nz, rng)
    i, j, k = 4, 4, 3
    at = lambda a, b, c: c * nx * ny + a * ny + b
    for key, nodes in (("nxx", [(i + 1, j + 1, k + 1), (i, j + 1, k + 1)]), ("nxy", [(i, j, k), (i, j + 1, k)]),
                       ("nxz", [(i, j, k), (i, j, k + 1)])):
        for q in nodes:
            f[key][at(*q)] = 0.0
    m, prob = _one_level(shape, 1, f, nubeg=1e-30)
    _check(m, prob, 1e-8)
    prob.close()


@pytest.mark.parametrize("levels", [0, 1, 3])
def test_not_a_number_is_a_status(levels):
    n = {0: 9, 1: 17, 3: 65}[levels]
    m = M.sphere_model(n, levels, (2, 2, 2), seed=1)
    prob = P.StokesProblem(m)
    f = prob.ronurecalc()
    bad = {k: v.copy() for k, v in f.items()}
    for k in KEYS:
        bad[k][:] = np.nan
    prob.set_nodes(bad)
    with pytest.raises(capi.P2Error) as e:
        prob.ctx.solve_resident()
    assert e.value.code in (5, 6)  # P2_ERR_NAN, P2_ERR_SINGULAR
    prob.set_nodes(f)
    assert prob.ctx.solve_resident().status == 0
    prob.close()
