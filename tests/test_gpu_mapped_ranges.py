"""Which host arrays p2_movemark moves in place: only those that one
page-locked range holds as a whole and that are aligned.  The decision alone
(p2_debug_mapped): nothing is copied or launched."""
import ctypes
import mmap

import pytest

import pardiso2_b200 as P
from pardiso2_b200 import capi

pytestmark = pytest.mark.gpu
PAGE = mmap.PAGESIZE


def test_one_range_has_to_hold_the_array():
    import torch
    rt = torch.cuda.cudart()
    H = capi.DebugHooks(P.Context(0))
    buf = mmap.mmap(-1, 6 * PAGE)
    base = ctypes.addressof(ctypes.c_char.from_buffer(buf))
    floats = PAGE // 4

    def registered(*pages):
        for first, count in pages:
            assert int(rt.cudaHostRegister(base + first * PAGE, count * PAGE, 0)) == 0
        try:
            # the whole first three pages; their middle; up to the last byte; one float past three pages; off by a byte
            return [H.mapped(base, 3 * floats), H.mapped(base + 4 * 7, 2 * floats), H.mapped(base + 4, 3 * floats - 1),
                    H.mapped(base + 4, 3 * floats), H.mapped(base + 1, floats)]
        finally:
            for first, _ in pages:
                assert int(rt.cudaHostUnregister(base + first * PAGE)) == 0

    assert registered() == [False] * 5                                     # pageable
    assert registered((0, 3)) == [True, True, True, False, False]           # one range
    assert registered((0, 6)) == [True, True, True, True, False]
    # both ends page-locked, the page between them not
    assert registered((0, 1), (2, 1)) == [False] * 5
    # ends inside the first and the last of two registrations of two pages with a gap
    assert registered((0, 2), (3, 2)) == [False, False, False, False, False]
    H.ctx.close()


def test_torch_pinned_memory_is_one_range():
    import torch
    H = capi.DebugHooks(P.Context(0))
    t = torch.zeros(5000).pin_memory()
    assert H.mapped(t.data_ptr(), 5000) and H.mapped(t.data_ptr() + 28, 4993)
    H.ctx.close()
