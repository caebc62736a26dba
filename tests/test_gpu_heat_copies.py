"""Heat step: pageable arrays in pieces through page-locked slots, page-locked
ones directly.  Marker counts on both sides of one piece (65536 floats), of the
least number of pieces that a second thread takes part in (8), and of all slots
in flight (12); without the numerical diffusion a marker's temperature depends
on itself and the node fields alone, so any count gives the same bits."""
import numpy as np
import pytest
import torch

import pardiso2_b200 as P
from pardiso2_b200 import capi
from tests.golden.make_golden import HEAT_COMMON, HEAT_VARIANTS, heat_inputs, heat_model

pytestmark = pytest.mark.gpu
PIECE = 65536


def test_pageable_and_page_locked_arrays():
    m = heat_model()
    th, vel, se, pr, _, _ = heat_inputs(m)
    v = HEAT_VARIANTS["mg"]
    d = {**HEAT_COMMON, **v, "max_cycles": 200, "heatdif": 0.0}
    hp = capi.heat_params(**{k: d[k] for k in ("maxtkstep", "heatmin", "t0koef", "t1koef", "heatdif", "tdeep", "zdeep",
                                               "multinumt", "multicyct", "frictyn", "adiabyn", "max_cycles", "pre", "post")})
    n = 13 * PIECE + 7
    rng = np.random.Generator(np.random.PCG64(3))
    mk = [rng.random(n).astype(np.float32) for _ in range(3)] + [(rng.integers(0, 60, n)).astype(np.int8)]
    tk = (800 + 400 * rng.random(n)).astype(np.float32)
    pinned = [torch.from_numpy(a).pin_memory() for a in mk]
    prob = P.StokesProblem(m)
    prob.ctx.heat_set_bc(m.bc, m.nodenum)

    def step(markers, count):
        return prob.ctx.titerate(hp, v["timestep"], th, vel=vel, pr=pr, se=se, markers=[a[:count] for a in markers],
                                 markk=tk[:count])[:2]

    nodes, want = step([p.numpy() for p in pinned], n)
    assert np.count_nonzero(want != tk) > n // 2
    for count in (1, PIECE - 1, PIECE, PIECE + 1, 2 * PIECE, 2 * PIECE + 1, 8 * PIECE, 12 * PIECE, 12 * PIECE + 1, n):
        t, k = step(mk, count)
        np.testing.assert_array_equal(t, nodes)
        np.testing.assert_array_equal(k, want[:count])
    prob.close()
