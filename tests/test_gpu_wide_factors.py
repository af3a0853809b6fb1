"""One huge finite value in a slice's sinogram (a hot or sentinel detector pixel):
its ray's factor stands far over all others, which keep their precision - the
pixels off that ray are as they are without it."""
import numpy as np
import pytest

import trace_gb300 as tg
from oracle import oracle as O
from tests._util import bits, rel_l2, theta_uniform

pytestmark = pytest.mark.gpu

HALF = dict(mode="fast", len_storage="u16", delta_index=True, forward_tiles=True,
            half_gathers=True, slices_per_pass=8)
KINDS = {"half": HALF,
         "u16": {**HALF, "half_gathers": False},
         "f32": {**HALF, "half_gathers": False, "len_storage": "f32"},
         "f16": {**HALF, "half_gathers": False, "len_storage": "f16"}}
# lengths of 16 bits: half an ulp of the code (2^-17 of the longest), f16 2^-12 of
# each, over at least some tens of rays per pixel; f32: rounded sums of 2^-24
TOL = {"half": 2e-4, "u16": 1e-4, "f32": 1e-5, "f16": 3e-4}
HOT = {2: (7, 12), 8: (21, 33)}  # slice: (angle, column)


def _data(C, P, S, hot):
    rng = np.random.default_rng(C)
    tabs = O.angle_table(theta_uniform(P))
    sino = O.forward(rng.uniform(0.5, 1.5, (S, C, C)).astype(np.float32), tabs)
    sino = (sino * rng.uniform(0.97, 1.03, sino.shape)).astype(np.float32)
    counts, offs, idx, *_ = O.trace(C, tabs)
    hit = np.zeros((S, C * C), bool)
    for s, (a, c) in HOT.items():
        sino[a, s, c] = hot
        r = a * C + c
        hit[s, idx[offs[r]:offs[r] + counts[r]]] = True
    return tabs, sino, hit


def _check(got, ref, hit, tol):
    for s in range(len(ref)):
        off = ~hit[s]
        assert rel_l2(got[s][off], ref[s][off]) < tol, s


# 34 columns: units of 8 slices; 261: of 32
@pytest.mark.parametrize("C,P", [(34, 40), (261, 36)])
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("hot", [1e6, 1e12, 3e38])
def test_sirt_off_the_hot_rays(C, P, kind, hot):
    S = 9
    tabs, sino, hit = _data(C, P, S, hot)
    ref = O.run("sirt", sino, tables=tabs, n_iter=1, precision=O.F64)["recon"].reshape(S, -1)
    plan = tg.Plan(P, S, C, theta_uniform(P), **KINDS[kind])
    plan.set_sinogram(sino)
    plan.reset_recon("sirt")
    plan.iterate("sirt", 1)
    _check(plan.get_recon("sirt").reshape(S, -1), ref, hit, TOL[kind])
    plan.close()


@pytest.mark.parametrize("alg", ["mlem", "pml", "apmlr"])
@pytest.mark.parametrize("kind", ["half", "f16", "f32"])
@pytest.mark.parametrize("hot", [1e6, 1e12, 3e38])
def test_reduce_off_the_hot_rays(alg, kind, hot):
    """The operator calls keep float factors on every plan."""
    C, P, S = 34, 40, 9
    tabs, sino, hit = _data(C, P, S, hot)
    kw = {} if alg == "mlem" else {"beta": 0.1}
    ref = O.run(alg, sino, tables=tabs, n_iter=1, precision=O.F64, want_replica=True, **kw)
    prm = tg.default_params(alg, **kw)
    plan = tg.Plan(P, S, C, theta_uniform(P), **KINDS[kind])
    plan.set_sinogram(sino, apply_abs=True)
    plan.reset_recon(alg)
    plan.reduce(alg, prm)
    got = plan.get_replica(alg).reshape(S, -1, 2)[..., 0]
    _check(got, ref["replica"].reshape(S, -1, 2)[..., 0], hit, TOL[kind])
    plan.close()


def test_hot_slices_leave_the_others_bits():
    C, P, S = 261, 36, 9
    outs = []
    for hot in (1.0, 1e12):
        _, sino, _ = _data(C, P, S, hot)
        plan = tg.Plan(P, S, C, theta_uniform(P), **HALF)
        plan.set_sinogram(sino)
        plan.reset_recon("sirt")
        plan.iterate("sirt", 3)
        outs.append(plan.get_recon("sirt"))
        plan.close()
    same = [s for s in range(S) if s not in HOT]
    assert np.array_equal(bits(outs[0][same]), bits(outs[1][same]))


@pytest.mark.parametrize("kind", ["u16", "f32", "f16"])
def test_finite_factors_at_the_top_of_the_range(kind):
    """Ratios from 1e38 on, which rounding up could make infinite: their slices are
    summed ray by ray as those with an infinite factor."""
    C, P, S = 34, 40, 9
    rng = np.random.default_rng(C)
    tabs = O.angle_table(theta_uniform(P))
    sino = O.forward(rng.uniform(0.5, 1.5, (S, C, C)).astype(np.float32), tabs)
    counts, offs, idx, *_ = O.trace(C, tabs)
    start = np.full((S, C, C), 0.05, np.float32)
    sim = O.forward(start[:1], tabs)[:, 0]  # of the ratio's first projection
    hit = np.zeros((S, C * C), bool)
    for s, (a, c) in HOT.items():
        c = min(c, 20)
        assert 1.05e38 < 3e38 / sim[a, c] < 3.3e38, (s, sim[a, c])
        sino[a, s, c] = 3e38
        r = a * C + c
        hit[s, idx[offs[r]:offs[r] + counts[r]]] = True
    ref = O.run("mlem", sino, tables=tabs, n_iter=1, precision=O.F64, want_replica=True,
                recon_in=start)
    plan = tg.Plan(P, S, C, theta_uniform(P), **KINDS[kind])
    plan.set_sinogram(sino, apply_abs=True)
    plan.set_recon("mlem", start)
    plan.reduce("mlem")
    got = plan.get_replica("mlem").reshape(S, -1, 2)[..., 0]
    _check(got, ref["replica"].reshape(S, -1, 2)[..., 0], hit, TOL[kind])
    plan.close()
