"""A coarsest level of more unknowns than a launch grid's second dimension has
blocks (65535): the V-cycle of the one-level grid still solves A x = b."""
import numpy as np
import pytest

from tests.test_gpu_coarse import _check, _fields, _one_level
from tests.test_gpu_vcycle import unknown_mask

pytestmark = pytest.mark.gpu


def test_coarsest_level_above_65535_unknowns():
    import torch
    shape = (28, 28, 28)  # 68 thousand unknowns: three matrices of 93 GB together
    if torch.cuda.mem_get_info(0)[0] < 110e9:
        pytest.skip("needs 110 GB of free device memory")
    rng = np.random.Generator(np.random.PCG64(3))
    m, prob = _one_level(shape, 0, _fields(int(np.prod(shape)), rng))
    assert np.count_nonzero(unknown_mask(shape) & (m.bc.bondm[:4 * m.nodenum] == 0)) > 65535
    _check(m, prob, 1e-1)  # the FP32 copy's bound of test_inverse
    prob.close()
