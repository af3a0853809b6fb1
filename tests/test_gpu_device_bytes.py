"""info()["device_bytes"] is what the plan takes from the device."""
import pytest

import trace_gb300 as tg
from tests._util import theta_uniform

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

HALF = dict(mode="fast", len_storage="u16", delta_index=True, forward_tiles=True,
            half_gathers=True, slices_per_pass=8)


# chunks of 64 MB that the plan's small buffers fill to different heights
@pytest.mark.parametrize("C,P,S,kw", [(512, 360, 8, HALF), (640, 300, 8, HALF), (768, 200, 16, HALF),
                                      (512, 400, 40, HALF), (600, 300, 4, {})])
def test_counts_what_the_device_gives(C, P, S, kw):
    th = theta_uniform(P)
    first = tg.Plan(P, S, C, th, **kw)  # kernels and their memory are loaded now
    first.reset_recon("mlem")
    first.close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan = tg.Plan(P, S, C, th, **kw)
    plan.reset_recon("mlem")
    plan.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    said = plan.info()["device_bytes"]
    plan.close()
    # the device rounds each allocation up to 2 MiB; a plan makes at most 16 of its
    # own beside its chunks
    assert said <= taken <= said + 16 * (2 << 20), (said, taken)
