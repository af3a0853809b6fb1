"""Captured iterations of a batch follow every plan's own buffers: plans that are
reset, or given another layout, one by one between the calls keep the bits of
plans iterated alone."""
import numpy as np
import pytest

import trace_gb300 as tg
from tests._util import bits, theta_uniform

pytestmark = pytest.mark.gpu

HALF = dict(mode="fast", len_storage="u16", delta_index=True, forward_tiles=True,
            half_gathers=True, slices_per_pass=8)
# (columns, angles, slices, options) of the plans of one batch: strips (40
# slices, and angles close enough), tiles, FP32 lengths, one slice per pass
STRIPS, TILES, FP32, EXACT = ((64, 260, 40, HALF), (48, 30, 5, HALF),
                              (40, 32, 9, {**HALF, "half_gathers": False, "len_storage": "f32"}),
                              (32, 24, 3, {}))


def _plan(size, seed):
    C, P, S, kw = size
    sino = np.random.default_rng(seed).uniform(5.0, 9.0, (P, S, C)).astype(np.float32)
    plan = tg.Plan(P, S, C, theta_uniform(P), **kw)
    plan.set_sinogram(sino, apply_abs=True)
    return plan


@pytest.mark.parametrize("sizes", [(STRIPS, TILES), (TILES, STRIPS, FP32), (EXACT, FP32),
                                   (TILES, TILES)])
def test_layouts_and_resets_between_calls(sizes):
    both = [[_plan(s, i) for i, s in enumerate(sizes)] for _ in range(2)]
    batch = tg.Batch(both[0])

    def reset(alg, which):
        for plans in both:
            for i in which:
                plans[i].reset_recon(alg)

    def step(alg, n):
        prm = tg.default_params(alg, beta=0.1)
        batch.iterate(alg, n, prm)
        for i, (a, b) in enumerate(zip(*both)):
            b.iterate(alg, n, prm)
            assert np.array_equal(bits(a.get_recon(alg)), bits(b.get_recon(alg))), (alg, n, i)

    every = range(len(sizes))
    # the halo layout and back: other buffers under the same algorithm
    for alg, n in (("mlem", 2), ("apmlr", 1), ("mlem", 2), ("apmlr", 3), ("mlem", 3)):
        reset(alg, every)
        step(alg, n)
    # one plan starts again where the others have run an odd number of iterations
    reset("sirt", every)
    step("sirt", 3)
    reset("sirt", [1])
    step("sirt", 1)
    step("sirt", 3)
    # and comes back from another layout alone
    reset("apmlr", [0])
    reset("sirt", [0])
    step("sirt", 2)
    batch.close()
    for plan in both[0] + both[1]:
        plan.close()
