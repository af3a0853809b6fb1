"""Captured iterations may outlive a reset of the reconstruction: the same bits
as launches without graphs, whatever changes between the passes."""
import numpy as np
import pytest

import trace_gb300 as tg
from tests._util import bits, theta_uniform

pytestmark = pytest.mark.gpu


# both sides of the line between short passes (captured anew, one branch) and
# long ones (graphs kept, two branches)
@pytest.mark.parametrize("size", [(48, 36, 19), (320, 260, 19)])
@pytest.mark.parametrize("kw", [dict(),
                                dict(mode="fast", len_storage="u16", delta_index=True,
                                     forward_tiles=True, half_gathers=True, slices_per_pass=8),
                                dict(mode="fast", len_storage="u16", delta_index=True,
                                     forward_tiles=True, slices_per_pass=4)])
def test_resets_between_captured_passes(size, kw):
    C, P, S = size
    rng = np.random.default_rng(0)
    sinos = [rng.uniform(5.0, 9.0, (P, S, C)).astype(np.float32) for _ in range(2)]
    plans = [tg.Plan(P, S, C, theta_uniform(P), **kw) for _ in range(2)]
    plans[0].set_graphs(True)
    # another algorithm of the same layout, other parameters, an odd count of
    # iterations, another sinogram, the layout with halo slices and back
    for alg, beta, n, k in (("mlem", 0.1, 2, 0), ("mlem", 0.1, 2, 0), ("mlem", 0.1, 3, 1),
                            ("pml", 0.1, 2, 1), ("pml", 0.3, 2, 1), ("sirt", 0.1, 1, 0),
                            ("apmlr", 0.1, 2, 0), ("apmlr", 0.1, 3, 1), ("mlem", 0.1, 2, 0)):
        got = []
        for plan in plans:
            plan.set_sinogram(sinos[k], apply_abs=alg != "sirt")
            plan.reset_recon(alg)
            plan.iterate(alg, n, tg.default_params(alg, beta=beta))
            got.append(plan.get_recon(alg))
        assert np.array_equal(bits(got[0]), bits(got[1])), (alg, beta, n, k)
    for plan in plans:
        plan.close()
