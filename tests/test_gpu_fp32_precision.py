"""FP32 plans on the tensor cores are as close to 64 bits as the scalar kernels
with the same operands (whose sums are rounded, not truncated)."""
import numpy as np
import pytest

import trace_gb300 as tg
from oracle import oracle as O
from tests._util import rel_l2, theta_uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,P", [(96, 72), (160, 120), (256, 180)])
@pytest.mark.parametrize("alg,n", [("sirt", 1), ("mlem", 1), ("mlem", 10), ("pml", 1)])
def test_no_further_off_than_scalar_sums(C, P, alg, n):
    S, th = 10, theta_uniform(P)
    rng = np.random.default_rng(C)
    vol = rng.uniform(0.1, 1.0, (S, C, C)).astype(np.float32)
    tabs = O.angle_table(th)
    sino = O.forward(vol, tabs)
    kw = dict(beta=0.05) if alg == "pml" else {}
    ref = O.run(alg, sino, tables=tabs, n_iter=n, precision=O.F64, threads=8, **kw)["recon"]
    errs = []
    # ten slices at 8 per pass: tensor cores; ray-ordered plans: scalar sums
    for tiles in (True, False):
        plan = tg.Plan(P, S, C, th, slices_per_pass=8, mode="fast", len_storage="f32",
                       delta_index=True, forward_tiles=tiles)
        plan.set_sinogram(sino, apply_abs=alg != "sirt")
        plan.reset_recon(alg)
        plan.iterate(alg, n, tg.default_params(alg, **kw))
        errs.append(rel_l2(plan.get_recon(alg), ref))
        plan.close()
    # a rounded and a truncated sum of the same length differ by their bias; half as
    # much again covers the spread of two orders of summation
    assert errs[0] < 1.5 * errs[1], errs
