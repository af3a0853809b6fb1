"""The autotuner on a sample whose plans take the strip-ordered forward: it does
not refine what those plans do not read."""
import numpy as np
import pytest

import trace_gb300 as tg
from trace_gb300.autotune import autotune
from tests._util import theta_uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,strips", [(32, True), (16, False)])
def test_no_tile_sides_for_strips(S, strips):
    C, P = 96, 288
    th = theta_uniform(P)
    sino = np.random.default_rng(3).uniform(0.5, 2.0, (P, S, C)).astype(np.float32)
    best, res = autotune(th, sino, "mlem", iters=1, warmup=1,
                         space={"slices_per_pass": (8,), "forward_tiles": (True,)},
                         refine={"forward_tile_side": (32, 64, 96), "forward_block_warps": (16, 32)},
                         fixed={"half_gathers": True})
    for key in ("forward_tile_side", "forward_block_warps"):
        assert any(key in c for c, *_ in res) != strips, key
    plan = tg.Plan(P, S, C, th, len_storage="u16", mode="fast", delta_index=True,
                   half_gathers=True, **best)
    assert (plan.info()["tile_runs"] % (P * C) == 0) == strips
    plan.close()
