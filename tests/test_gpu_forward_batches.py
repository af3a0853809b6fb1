"""Half-gather plans of fewer than 8 slices per pass take 8 slices per forward
launch: the same bits as batch by batch (a batch of plans launches them so)."""
import numpy as np
import pytest

import trace_gb300 as tg
from tests._util import bits, theta_uniform

pytestmark = pytest.mark.gpu


# whole groups of 8 slices, a rest of one slice to one batch short of a group,
# a last batch that is not full; two groups' finishes on two streams
@pytest.mark.parametrize("K,S", [(4, 8), (4, 5), (4, 13), (4, 19), (2, 8), (2, 9), (2, 15),
                                 (1, 8), (1, 11), (1, 16)])
@pytest.mark.parametrize("side", [64, 96])
def test_same_bits_as_batch_by_batch(K, S, side):
    C, P = 101, 40
    th = theta_uniform(P)
    rng = np.random.default_rng(S)
    sino = rng.uniform(20.0, 30.0, (P, S, C)).astype(np.float32)
    for alg in ("sirt", "mlem", "apmlr"):
        prm = tg.default_params(alg, beta=0.05)
        plans = []
        for _ in range(2):
            plan = tg.Plan(P, S, C, th, mode="fast", len_storage="u16", delta_index=True,
                           forward_tiles=True, half_gathers=True, slices_per_pass=K,
                           forward_tile_side=side)
            plan.set_sinogram(sino, apply_abs=alg != "sirt")
            plan.reset_recon(alg)
            plans.append(plan)
        plans[0].iterate(alg, 3, prm)
        batch = tg.Batch([plans[1]])
        batch.iterate(alg, 3, prm)
        got = [plan.get_recon(alg) for plan in plans]
        assert np.isfinite(got[0]).all()
        assert np.array_equal(bits(got[0]), bits(got[1])), alg
        # a non-finite ray stays with its batch
        bad = sino.copy()
        bad[3, S - 1, 50] = np.inf
        for plan in plans:
            plan.set_sinogram(bad, apply_abs=alg != "sirt")
            plan.reset_recon(alg)
        plans[0].iterate(alg, 1, prm)
        batch.iterate(alg, 1, prm)
        got = [plan.get_recon(alg) for plan in plans]
        assert not np.isfinite(got[0]).all()
        assert np.array_equal(bits(got[0]), bits(got[1])), alg
        batch.close()
        for plan in plans:
            plan.close()
