"""The sweeps of a small level in one launch (k_smooth_resident): against the
same sweeps as separate colour passes and boundary-row launches (smoother 3,
the same cell solve factored on every pass), on levels that take one cluster,
a cooperative grid and the largest that still fit; and the diagonal block
against a numpy restatement of the colour passes on the assembled operator."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi
from pardiso2_b200 import model as M
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu
KEYS = ("nu", "ro", "nxx", "nxy", "nxz", "nyz")


def _problem(shape, levels, smoother, precision, seed=3):
    m = M.random_spheres_model(shape[0], levels, 1, (1.0, 1.0), markers=(1, 1, 1), seed=1, shape=shape)
    m.params.nubeg, m.params.nuend = 1e-3, 1e3
    prob = P.StokesProblem(m, precision=precision, smoother=smoother)
    rng = np.random.Generator(np.random.PCG64(seed))
    prob.set_nodes({k: np.exp(rng.uniform(-1, 1, m.nodenum)).astype(np.float32) for k in KEYS})
    return m, prob, capi.DebugHooks(prob.ctx)


# levels: (19^3) one cluster, (33^3) and (43x45x41) a grid, the last near its largest size; even and odd sides
@pytest.mark.parametrize("shape,levels", [((33, 33, 33), 1), ((43, 45, 41), 2), ((37, 33, 41), 2), ((9, 12, 20), 0)])
@pytest.mark.parametrize("precision,tol", [(0, 2e-4), (1, 1e-11)])
def test_matches_separate_passes(shape, levels, precision, tol):
    m, prob, H = _problem(shape, levels, 1, precision)
    _, ref, R = _problem(shape, levels, 3, precision)
    lv = m.levels
    rng = np.random.Generator(np.random.PCG64(9))
    for l in range(levels + 1):
        mask = unknown_mask((lv.mgx[l], lv.mgy[l], lv.mgz[l]))
        x, b = (np.where(mask, rng.standard_normal(4 * lv.mgn[l]), 0.0) for _ in range(2))
        for sweeps in (1, 3):
            got, want = H.smooth(l, sweeps, b, x), R.smooth(l, sweeps, b, x)
            # both round every operation; FP32 factors are stored rounded in one and eliminated in the other
            assert np.linalg.norm((got - want)[mask]) <= tol * np.linalg.norm(want[mask]), (l, sweeps)
    prob.close()
    ref.close()


@pytest.mark.parametrize("precision,tol", [(0, 1e-4), (1, 1e-10)])
def test_diagonal_block_matches_numpy(precision, tol):
    shape = (8, 9, 8)
    nx, ny, nz = shape
    m, prob, H = _problem(shape, 0, 0, precision)
    n = m.nodenum
    mask = unknown_mask(shape)
    row = m.bc.bondm[:4 * n].copy()
    pin = m.params.pin
    row[4 * (pin[2] * nx * ny + pin[0] * ny + pin[1])] = 0
    row = np.where(mask, row, 0)
    A = np.zeros((4 * n, 4 * n))
    for u in np.nonzero(mask)[0]:
        e = np.zeros(4 * n)
        e[u] = 1
        A[:, u] = H.apply(0, e)
    rng = np.random.Generator(np.random.PCG64(11))
    x, b = (np.where(mask, rng.standard_normal(4 * n), 0.0) for _ in range(2))

    def boundary(v):
        for _ in range(6):  # copy chains are shorter than that
            for u in np.nonzero(row)[0]:
                t = m.bc.bondn1[row[u]]
                v[u] = b[u] + (m.bc.bondv1[row[u], 1] * v[t - 1] if t else 0.0)

    ih = [1.0 / np.diff(g) for g in (m.gx, m.gy, m.gz)]
    at = lambda i, j, k: k * nx * ny + i * ny + j
    want = x.copy()
    boundary(want)
    omega = prob.params.omega
    for col in (0, 1, 0, 1):
        old = want.copy()
        res = b - A @ old
        for k in range(1, nz):
            for i in range(1, nx):
                for j in range(1, ny):
                    if (i + j + k) & 1 != col:
                        continue
                    f = np.array([4 * at(i - 1, j - 1, k - 1) + 1, 4 * at(i, j - 1, k - 1) + 1,
                                  4 * at(i - 1, j - 1, k - 1) + 2, 4 * at(i - 1, j, k - 1) + 2,
                                  4 * at(i - 1, j - 1, k - 1) + 3, 4 * at(i - 1, j - 1, k) + 3])
                    c = np.repeat([ih[0][i - 1], ih[1][j - 1], ih[2][k - 1]], 2) * np.array([-1, 1, -1, 1, -1, 1])
                    p = 4 * at(i, j, k)
                    act = row[f] == 0
                    fa, ca = f[act], c[act]
                    d, g = A[fa, fa], A[fa, p]
                    den = np.sum(ca * g / d)
                    dp = 0.0
                    if row[p] == 0 and den != 0:
                        dp = (np.sum(ca * res[fa] / d) - (b[p] - np.sum(c * old[f]))) / den
                        want[p] += omega * dp
                    want[fa] = old[fa] + omega * (res[fa] - g * dp) / d
        boundary(want)
    got = H.smooth(0, 2, b, x)
    assert np.linalg.norm((got - want)[mask]) <= tol * np.linalg.norm(want[mask])
    prob.close()
