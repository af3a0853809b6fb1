"""One slice per pass: several slices per thread (and, for several slices, a
transposed copy of the planes for the rays closer to the horizontal) give the
bits of one slice alone; plans of few slices with half gathers keep the scalar
backprojection where the grid fills the GPU."""
import numpy as np
import pytest

import trace_gb300 as tg
from oracle import oracle as O
from tests._util import bits, rel_l2, theta_uniform

pytestmark = pytest.mark.gpu


# groups of four, three, two and one slice, the last group full, early or not;
# 33 columns leave a ray group of one ray, 120 give the forward launch warps
# enough for two slices a thread, 400 for four
@pytest.mark.parametrize("C,P,S", [(33, 20, 1), (33, 20, 2), (33, 21, 7), (33, 23, 16),
                                   (120, 90, 19), (120, 90, 33), (400, 320, 15)])
@pytest.mark.parametrize("kw", [dict(), dict(delta_index=True), dict(forward_on_the_fly=True),
                                dict(mode="fast", len_storage="u16", delta_index=True),
                                dict(mode="fast", len_storage="bf16"),
                                dict(mode="fast", len_storage="f16")])
def test_every_slice_has_the_bits_it_has_alone(C, P, S, kw):
    if C == 400 and kw not in (dict(), dict(delta_index=True)):
        pytest.skip("the launch's shape does not depend on the rest")
    th = theta_uniform(P)
    rng = np.random.default_rng(S)
    sino = rng.uniform(0.5, 2.0, (P, S, C)).astype(np.float32)
    for alg in ("sirt", "mlem", "pml"):
        prm = tg.default_params(alg, beta=0.2)
        plan = tg.Plan(P, S, C, th, **kw)
        plan.set_sinogram(sino, apply_abs=alg != "sirt")
        plan.reset_recon(alg)
        plan.iterate(alg, 2, prm)
        got = plan.get_recon(alg)
        plan.close()
        for s in sorted({0, S // 2, S - 2, S - 1} & set(range(S))):
            one = tg.Plan(P, 1, C, th, **kw)
            one.set_sinogram(np.ascontiguousarray(sino[:, s:s + 1]), apply_abs=alg != "sirt")
            one.reset_recon(alg)
            one.iterate(alg, 2, prm)
            assert np.array_equal(bits(one.get_recon(alg)[0]), bits(got[s])), (alg, s)
            one.close()


@pytest.mark.parametrize("S,K", [(1, 1), (2, 2), (3, 4), (4, 4), (4, 2)])
@pytest.mark.parametrize("C", [319, 320])
def test_few_slices_against_fp64(S, K, C):
    """Both sides of the rule's line, and in a batch; the operands' rounding as
    for the other half-gather plans."""
    P, it = 60, 2
    th = theta_uniform(P)
    tabs = O.angle_table(th)
    rng = np.random.default_rng(S)
    sino = rng.uniform(50.0, 60.0, (P, S, C)).astype(np.float32)
    for alg in ("sirt", "mlem", "apmlr"):
        kw = dict(beta=0.05) if alg == "apmlr" else {}
        prm = tg.default_params(alg, **kw)
        ref = O.run(alg, sino, tables=tabs, n_iter=it, precision=O.F64, **kw)["recon"]
        plans = []
        for _ in range(2):
            plan = tg.Plan(P, S, C, th, mode="fast", len_storage="u16", delta_index=True,
                           forward_tiles=True, half_gathers=True, slices_per_pass=K)
            plan.set_sinogram(sino, apply_abs=alg != "sirt")
            plan.reset_recon(alg)
            plans.append(plan)
        plans[0].iterate(alg, it, prm)
        batch = tg.Batch([plans[1]])
        batch.iterate(alg, it, prm)
        for plan in plans:
            assert rel_l2(plan.get_recon(alg), ref) < 1e-4
        batch.close()
        for plan in plans:
            plan.close()
