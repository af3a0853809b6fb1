"""The tensor-core backprojection (tile-staged plans: half gathers, or FP32
operands at 8 slices per pass) at the edges of its tiles, stages, slice units
and groups of units, with non-finite factors, and across float scales."""
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
# a float reconstruction after two iterations: a few hundred rounded sums of
# 2^-24 each, and the 2^-23 of a split factor; 16-bit lengths: half an ulp of
# the code (2^-17 of the longest), f16 2^-12 of each, with at least some tens
# of rays per pixel; a half factor 2^-12 of the factor
TOL = {"half": 2e-4, "u16": 1e-4, "f32": 1e-5, "f16": 3e-4}


def _sino(C, P, S, seed):
    """Line integrals of a smooth positive volume with noise of a few per cent."""
    rng = np.random.default_rng(seed)
    vol = rng.uniform(0.5, 1.5, (S, C, C)).astype(np.float32)
    tabs = O.angle_table(theta_uniform(P))
    sim = O.forward(vol, tabs)
    return tabs, (sim * rng.uniform(0.97, 1.03, sim.shape)).astype(np.float32)


def _run(sino, alg, it, kw, prm, center=0.0):
    P, S, C = sino.shape
    plan = tg.Plan(P, S, C, theta_uniform(P), center=center, **kw)
    plan.set_sinogram(sino)
    plan.reset_recon(alg)
    plan.iterate(alg, it, prm)
    out = plan.get_recon(alg)
    plan.close()
    return out


# 16 x 8 pixel blocks, stages of 16 (8) angles, window starts every 32 angles
@pytest.mark.parametrize("C,P", [(15, 30), (16, 32), (17, 33), (40, 61), (67, 97)])
# one to nine units of 8 slices, a second group (these grids are small)
@pytest.mark.parametrize("S", [3, 8, 9, 33, 70])
@pytest.mark.parametrize("kind", list(KINDS))
def test_against_fp64(C, P, S, kind):
    tabs, sino = _sino(C, P, S, C + S)
    for alg in ("sirt", "pml"):
        kw = {"beta": 0.1} if alg == "pml" else {}
        ref = O.run(alg, sino, tables=tabs, n_iter=2, precision=O.F64, **kw)["recon"]
        got = _run(sino, alg, 2, KINDS[kind], tg.default_params(alg, **kw))
        assert rel_l2(got, ref) < TOL[kind], alg


@pytest.mark.parametrize("kind,alg", [("half", "mlem"), ("half", "sirt"), ("u16", "pml"),
                                      ("f32", "sirt")])
def test_unit_sizes_keep_the_bits(kind, alg):
    """Units of 8, 16 and 32 slices (enough blocks for the larger ones from
    about 250 columns on) sum each slice in the same order: slabs of 8, 16
    and 17 slices give the bits of the 40-slice volume."""
    C, P, S = 260, 24, 40
    rng = np.random.default_rng(23)
    sino = rng.uniform(0.5, 1.5, (P, S, C)).astype(np.float32) * C / 2
    prm = tg.default_params(alg, beta=0.1)
    want = _run(sino, alg, 2, KINDS[kind], prm)
    for s0, s1 in ((0, 8), (8, 24), (16, 33)):
        part = _run(np.ascontiguousarray(sino[:, s0:s1]), alg, 2, KINDS[kind], prm)
        assert np.array_equal(bits(part), bits(want[s0:s1])), (s0, s1)


@pytest.mark.parametrize("alg", ["sirt", "mlem", "pml"])
def test_slices_per_pass_and_groups_keep_the_bits(alg):
    """Each slice's sums do not depend on the other slices: the slices per
    pass, and the group and place in the ring of units that a slice falls in
    (130 slices: three groups), leave its bits as they are."""
    tabs, sino = _sino(48, 40, 130, 5)
    prm = tg.default_params(alg, beta=0.1)
    want = _run(sino, alg, 3, HALF, prm)
    for K in (1, 4, 16):
        assert np.array_equal(bits(_run(sino, alg, 3, {**HALF, "slices_per_pass": K}, prm)),
                              bits(want))
    for s0, s1 in ((0, 40), (64, 128)):
        part = _run(np.ascontiguousarray(sino[:, s0:s1]), alg, 3, HALF, prm)
        assert np.array_equal(bits(part), bits(want[s0:s1]))


@pytest.mark.parametrize("kind", ["half", "u16", "f32"])
@pytest.mark.parametrize("alg", ["sirt", "mlem"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 3e38])
def test_non_finite_factors_stay_on_their_rays(kind, alg, bad):
    """A non-finite factor (also one that only a half cannot hold) reaches the
    pixels its ray crosses, as in the reference, and no others."""
    C, P, S = 34, 40, 9
    tabs, sino = _sino(C, P, S, 11)
    sino[7, 2, 12] = bad
    sino[21, 5, 33] = bad
    ref = O.run(alg, sino, tables=tabs, n_iter=1, precision=O.F64)["recon"]
    got = _run(sino, alg, 1, KINDS[kind], tg.default_params(alg))
    if bad == 3e38 and kind != "half" or bad == 3e38 and alg == "sirt":
        return  # finite as a float: nothing to hold apart
    hit = ~np.isfinite(ref) | (np.abs(ref) > 1e30)
    assert hit.any() and np.array_equal(~np.isfinite(got) | (np.abs(got) > 1e30), hit)
    assert rel_l2(got[~hit], ref[~hit]) < TOL[kind]


def test_rays_outside_the_grid():
    """A rotation centre far off the middle leaves rays that cross no pixel
    (0 / 0 factors): they reach none."""
    C, P, S = 40, 48, 8
    th = theta_uniform(P)
    tabs = O.angle_table(th)
    rng = np.random.default_rng(3)
    sino = rng.uniform(0.5, 1.5, (P, S, C)).astype(np.float32)
    center = C / 2 + 9.25
    for kind in ("half", "u16"):
        ref = O.run("mlem", sino, tables=tabs, n_iter=2, precision=O.F64, center=center)["recon"]
        got = _run(sino, "mlem", 2, KINDS[kind], tg.default_params("mlem"), center)
        nan = np.isnan(ref)
        assert np.array_equal(np.isnan(got), nan)
        assert rel_l2(got[~nan], ref[~nan]) < 1e-3


@pytest.mark.parametrize("shift", [-60, -20, 20, 60])
def test_float_factors_keep_their_scale(shift):
    """SIRT's float factors are split at their slice's own scale: a first
    iteration (from zero) of data 2^shift times as large is exactly 2^shift
    times the result, slice by slice."""
    tabs, sino = _sino(50, 45, 12, 13)
    prm = tg.default_params("sirt")
    want = _run(sino, "sirt", 1, HALF, prm)
    scaled = sino.copy()
    scaled[:, ::2] *= np.float32(2.0 ** shift)
    got = _run(scaled, "sirt", 1, HALF, prm)
    assert np.array_equal(bits(got[1::2]), bits(want[1::2]))
    assert np.array_equal(bits(got[::2]), bits(want[::2] * np.float32(2.0 ** shift)))


@pytest.mark.parametrize("alg", ["mlem", "pml", "apmlr"])
def test_reduce_matches_the_fused_iteration(alg):
    """The operator calls' replica (float factors) updates to the fused
    iteration's reconstruction within the half factors' rounding."""
    C, P, S = 45, 60, 11
    _, sino = _sino(C, P, S, 17)
    prm = tg.default_params(alg, beta=0.1)
    want = _run(sino, alg, 1, HALF, prm)
    plan = tg.Plan(P, S, C, theta_uniform(P), **HALF)
    plan.set_sinogram(sino)
    plan.reset_recon(alg)
    plan.reduce(alg, prm)
    if alg != "mlem":
        plan.calculate_fg(alg, prm)
    plan.update_recon(alg, prm)
    assert rel_l2(plan.get_recon(alg), want) < 2e-4
    plan.close()
