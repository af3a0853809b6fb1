"""Plans without the tile-ordered matrix run several slice batches per launch:
the same bits as one batch at a time (a batch of plans launches them so), at
slice counts off the launch's 16 slices and off the slices per pass."""
import numpy as np
import pytest

import trace_gb300 as tg
from tests._util import bits, theta_uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(), dict(slices_per_pass=4), dict(forward_on_the_fly=True),
                                dict(mode="fast", len_storage="u16", delta_index=True,
                                     slices_per_pass=8),
                                dict(mode="fast", backward_staged=True, slices_per_pass=2)])
@pytest.mark.parametrize("S", [1, 5, 16, 17, 35])
def test_grouped_launches_keep_the_bits(kw, S):
    C, P = 40, 30
    th = theta_uniform(P)
    rng = np.random.default_rng(S)
    sino = rng.uniform(0.5, 2.0, (P, S, C)).astype(np.float32)
    for alg in ("sirt", "pml", "apmlr"):
        prm = tg.default_params(alg, beta=0.2)

        def make():
            plan = tg.Plan(P, S, C, th, **kw)
            plan.set_sinogram(sino, apply_abs=alg != "sirt")
            plan.reset_recon(alg)
            return plan

        a, b = make(), make()
        a.iterate(alg, 2, prm)
        batch = tg.Batch([b])
        batch.iterate(alg, 2, prm)
        assert np.array_equal(bits(a.get_recon(alg)), bits(b.get_recon(alg))), alg
        # the operators and the projector group the batches too
        a.reduce(alg, prm)
        rep = a.get_replica(alg)
        sim = a.forward_project(alg)
        for s in range(0, S, 7):
            one = tg.Plan(P, 1, C, th, **kw)
            if alg != "apmlr":  # its slices are coupled
                one.set_sinogram(np.ascontiguousarray(sino[:, s:s + 1]), apply_abs=alg != "sirt")
                one.set_recon(alg, a.get_recon(alg)[s:s + 1])
                one.reduce(alg, prm)
                assert np.array_equal(bits(one.get_replica(alg)[0]), bits(rep[s]))
                assert np.array_equal(bits(one.forward_project(alg)[:, 0]), bits(sim[:, s]))
            one.close()
        batch.close()
        a.close()
        b.close()
