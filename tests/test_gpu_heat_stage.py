"""Heat step on a small grid: pageable lists are copied directly until one of
10.5 MB arrives, which makes the page-locked slots; every later list goes through
them in pieces.  Marker counts on both sides of that size (17 bytes a marker) and
of one piece afterwards; as in test_gpu_heat_copies.py any count gives the bits
of page-locked arrays."""
import numpy as np
import pytest
import torch

import pardiso2_b200 as P
from pardiso2_b200 import capi
from tests.golden.make_golden import HEAT_COMMON, HEAT_VARIANTS, heat_inputs, heat_model

pytestmark = pytest.mark.gpu
IN = (40 << 18) // 17  # the largest count below the size
PIECE = 1 << 16        # temperatures in one piece


@pytest.mark.parametrize("counts", [(3, IN, IN + 1, IN), (IN + 1, 1, PIECE - 1, PIECE, PIECE + 1)])
def test_both_sides_of_the_least_size(counts):
    m = heat_model()
    th, vel, se, pr, _, _ = heat_inputs(m)
    v = HEAT_VARIANTS["mg"]
    d = {**HEAT_COMMON, **v, "max_cycles": 200, "heatdif": 0.0}
    hp = capi.heat_params(**{k: d[k] for k in ("maxtkstep", "heatmin", "t0koef", "t1koef", "heatdif", "tdeep", "zdeep",
                                               "multinumt", "multicyct", "frictyn", "adiabyn", "max_cycles", "pre", "post")})
    n = max(counts)
    rng = np.random.Generator(np.random.PCG64(4))
    mk = [rng.random(n).astype(np.float32) for _ in range(3)] + [rng.integers(0, 60, n).astype(np.int8)]
    tk = (800 + 400 * rng.random(n)).astype(np.float32)
    pinned = [torch.from_numpy(a).pin_memory().numpy() for a in mk]

    def step(ctx, markers, count):
        return ctx.titerate(hp, v["timestep"], th, vel=vel, pr=pr, se=se, markers=[a[:count] for a in markers],
                            markk=tk[:count])[:2]

    probs = [P.StokesProblem(m) for _ in range(2)]
    for p in probs:
        p.ctx.heat_set_bc(m.bc, m.nodenum)
    nodes, want = step(probs[0].ctx, pinned, n)
    assert np.count_nonzero(want != tk) > n // 2
    for count in counts:
        t, k = step(probs[1].ctx, mk, count)
        np.testing.assert_array_equal(t, nodes)
        np.testing.assert_array_equal(k, want[:count])
    for p in probs:
        p.close()
