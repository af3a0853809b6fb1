"""The strip-ordered tensor-core forward projection (half-gather plans with
16-bit codes, 32 slices or more and angles close enough together) against
the tile-staged one and FP64."""
import numpy as np
import pytest

import trace_gb300 as tg
from oracle import oracle as O
from tests._util import rel_l2, theta_uniform

pytestmark = pytest.mark.gpu

KW = dict(mode="fast", len_storage="u16", delta_index=True, forward_tiles=True,
          half_gathers=True, slices_per_pass=8)


def _tables(theta):
    return dict(sin_tab=np.sin(theta.astype(np.float64)).astype(np.float32),
                cos_tab=np.cos(theta.astype(np.float64)).astype(np.float32))


# chunks of 32 rows and more need about 250 angles over 180 degrees; grids off
# and on the chunk, strip and stage sizes; 32- and 64-slice units, two groups
@pytest.mark.parametrize("C,P,S,center", [(64, 260, 32, 0.0), (97, 300, 33, 0.0),
                                          (200, 400, 34, 0.0), (131, 257, 70, 0.0),
                                          (96, 280, 32, 96 / 2 + 3.5), (256, 720, 40, 0.0)])
def test_projection_matches_the_tile_staged_one(C, P, S, center):
    """The same halves and codes, summed along strips instead of tile runs:
    ray sums agree to the rounding of the partial sums (two orders of FP32
    additions of at most a few thousand terms: 2e-6)."""
    th = theta_uniform(P)
    rng = np.random.default_rng(C)
    vol = rng.uniform(0.0, 2.0, (S, C, C)).astype(np.float32)
    sims = []
    for n in (S, 16):  # 16 slices: the tile-staged forward
        plan = tg.Plan(P, n, C, th, center=center, **KW)
        plan.set_recon("sirt", vol[:n])
        sims.append((plan.forward_project("sirt"), plan.info()))
        plan.close()
    assert sims[0][1]["tile_runs"] % (P * C) == 0  # chunks per ray: the strips
    assert sims[1][1]["tile_runs"] % (P * C) != 0
    assert rel_l2(sims[0][0][:, :16], sims[1][0]) < 2e-6


@pytest.mark.parametrize("alg", ["sirt", "mlem", "pml", "apmlr"])
@pytest.mark.parametrize("K", [4, 8, 16])
def test_iterations_against_fp64(alg, K):
    C, P, S, it = 96, 288, 35, 3
    th = theta_uniform(P)
    tabs = O.angle_table(th)
    from trace_gb300.phantom import ellipse_phantoms
    sino = O.forward(ellipse_phantoms(C, S, seed=5, texture_sigma=0.02), tabs)
    kw = dict(beta=0.05) if alg in ("pml", "apmlr") else {}
    ref = O.run(alg, sino, tables=tabs, n_iter=it, precision=O.F64, **kw)["recon"]
    plan = tg.Plan(P, S, C, th, **{**KW, "slices_per_pass": K})
    plan.set_graphs(True)
    plan.set_sinogram(sino, apply_abs=alg != "sirt")
    plan.reset_recon(alg)
    plan.iterate(alg, it, tg.default_params(alg, **kw))
    assert rel_l2(plan.get_recon(alg), ref) < 1e-4
    # the operators' path on the same plan
    plan.reduce(alg, tg.default_params(alg, **kw))
    assert np.isfinite(plan.get_replica(alg)).all()
    plan.close()


def test_angles_in_any_order_and_range():
    """Angles over the full circle, shuffled: blocks of angles whose rays do
    not run side by side leave the plan on the tile-staged forward; sorted
    full-circle angles take the strips. Both match the exact projection within
    the operands' rounding."""
    C, P, S = 80, 640, 33
    rng = np.random.default_rng(3)
    th = (np.arange(P, dtype=np.float64) * 2 * np.pi / P + 0.01).astype(np.float32)
    vol = rng.uniform(0.0, 2.0, (S, C, C)).astype(np.float32)
    for theta, strips in ((th, True), (rng.permutation(th), False)):
        plan = tg.Plan(P, S, C, theta, **_tables(theta), **KW)
        assert (plan.info()["tile_runs"] % (P * C) == 0) == strips
        plan.set_recon("sirt", vol)
        sim = plan.forward_project("sirt")
        plan.close()
        exact = tg.Plan(P, S, C, theta, **_tables(theta))
        exact.set_recon("sirt", vol)
        # halves of the pixels: 2^-12 each, averaged over tens of pixels
        assert rel_l2(sim, exact.forward_project("sirt")) < 2e-4
        exact.close()


def test_non_finite_pixels_stay_on_their_rays():
    """A non-finite pixel reaches the rays through it and no others, though the
    strips' products run over whole windows."""
    C, P, S = 72, 300, 36
    th = theta_uniform(P)
    rng = np.random.default_rng(7)
    vol = rng.uniform(0.5, 1.0, (S, C, C)).astype(np.float32)
    plan = tg.Plan(P, S, C, th, **KW)
    plan.set_recon("sirt", vol)
    clean = plan.forward_project("sirt")
    vol[3, 20, 31] = np.inf
    plan.set_recon("sirt", vol)
    got = plan.forward_project("sirt")
    tile = tg.Plan(P, 16, C, th, **KW)
    tile.set_recon("sirt", vol[:16])
    want = tile.forward_project("sirt")
    assert np.array_equal(np.isfinite(got[:, :16]), np.isfinite(want))
    ok = np.isfinite(got)
    assert rel_l2(got[ok], clean[ok]) < 2e-6  # walked ray by ray
    tile.close()
    plan.close()


@pytest.mark.parametrize("alg", ["sirt", "mlem", "pml"])
def test_marked_slices_leave_the_others_alone(alg):
    """One slice with a non-finite pixel, or factor, on a strip-ordered plan (40
    and 70 slices: one and two launches, 64 and 32 wide): every other slice
    keeps the bits it has without, in the projection and in the iterations
    that spread it over its slice."""
    for C, P, S in ((64, 260, 40), (97, 300, 70)):
        th = theta_uniform(P)
        rng = np.random.default_rng(S)
        vol = rng.uniform(0.5, 1.0, (S, C, C)).astype(np.float32)
        sino = rng.uniform(0.8, 1.2, (P, S, C)).astype(np.float32) * C / 2
        bad = (3, S - 1)
        other = [s for s in range(S) if s not in bad]
        plan = tg.Plan(P, S, C, th, **KW)
        got = []
        for worse in (False, True):
            if worse:
                for s in bad:
                    vol[s, 20, 31] = np.inf
                    sino[P // 3, s, C // 2] = np.nan
            plan.set_recon(alg, vol)
            sim = plan.forward_project(alg)
            plan.set_sinogram(sino, apply_abs=alg != "sirt")
            plan.reset_recon(alg)
            plan.iterate(alg, 3, tg.default_params(alg, beta=0.1))
            got.append((sim, plan.get_recon(alg)))
        plan.close()
        for a, b in ((got[0][0][:, other], got[1][0][:, other]), (got[0][1][other], got[1][1][other])):
            assert np.isfinite(a).all()
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        # the marked slices' rays off the pixel: the same terms walked in order
        sim, ref = got[1][0][:, list(bad)], got[0][0][:, list(bad)]
        ok = np.isfinite(sim)
        assert 0.9 < ok.mean() < 1 and rel_l2(sim[ok], ref[ok]) < 2e-6
