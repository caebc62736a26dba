"""p2_movemark on page-locked markers moves them in place over the bus, on
pageable ones through device buffers: the same positions bit for bit, for
counts around a block's 256 threads, arrays that start inside an allocation,
and a mix of both kinds."""
import numpy as np
import pytest

import pardiso2_b200 as P
from pardiso2_b200 import model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,offset", [(1, 0), (255, 1), (257, 3), (5000, 7)])
def test_mapped_and_pageable_markers_agree(n, offset):
    import torch
    m = M.sphere_model(12, 1, (1, 1, 1), seed=1)
    ctx = P.Context(0)
    ctx.set_grid(m.gx, m.gy, m.gz, P.params_for(m))
    rng = np.random.Generator(np.random.PCG64(n))
    vel = [(rng.random(m.nodenum) - 0.5).astype(np.float32) for _ in range(3)]
    pos = [rng.uniform(-0.05, 1.05, n).astype(np.float32) for _ in range(3)]
    typ = rng.integers(0, 110, n).astype(np.int8)
    want = ctx.movemark(0.03, *vel, *pos, typ)  # copies into pageable arrays
    pinned = [torch.zeros(n + offset, dtype=torch.float32).pin_memory() for _ in range(3)]
    ptyp = torch.zeros(n + offset, dtype=torch.int8).pin_memory()
    ptyp[offset:] = torch.from_numpy(typ)
    for kind in ("mapped", "mixed"):
        for a in range(3):
            pinned[a][offset:] = torch.from_numpy(pos[a])
        got = [p.numpy()[offset:] for p in pinned]
        if kind == "mixed":
            got[1] = pos[1].copy()
        ctx._check(ctx.L.p2_movemark(ctx.h, 0.03, 2, 0, *vel, n, *got, ptyp.numpy()[offset:]), "p2_movemark")
        for a in range(3):
            assert np.array_equal(got[a], want[a]), (kind, a)
    ctx.close()
