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


@pytest.mark.parametrize("K,S", [(8, 19), (16, 40), (4, 21)])
def test_short_passes_before_and_after_their_capture(K, S):
    """Short iterations on two streams are launched one by one at first (16 of
    them) and captured then: every count of iterations gives the bits of plain
    launches, across parameters that change and a reset that starts again."""
    C, P = 48, 36
    kw = dict(mode="fast", len_storage="u16", delta_index=True, forward_tiles=True,
              half_gathers=True, slices_per_pass=K)
    sino = np.random.default_rng(1).uniform(5.0, 9.0, (P, S, C)).astype(np.float32)
    plans = [tg.Plan(P, S, C, theta_uniform(P), **kw) for _ in range(2)]
    plans[0].set_graphs(True)
    for plan in plans:
        plan.set_sinogram(sino, apply_abs=True)
    for again in range(2):
        for plan in plans:
            plan.reset_recon("pml")
        for n, beta in ((15, 0.1), (1, 0.1), (1, 0.1), (4, 0.1), (3, 0.3), (2, 0.1)):
            got = []
            for plan in plans:
                plan.iterate("pml", n, tg.default_params("pml", beta=beta))
                got.append(plan.get_recon("pml"))
            assert np.array_equal(bits(got[0]), bits(got[1])), (again, n, beta)
    for plan in plans:
        plan.close()
