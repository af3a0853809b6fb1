"""Which backprojection FP32 plans take: the tensor cores where a unit of slices
serves several passes, or a single one on a small grid; else the scalar kernels.
Both sides of the lines against FP64, and in a batch."""
import numpy as np
import pytest

import trace_gb300 as tg
from oracle import oracle as O
from tests._util import bits, rel_l2, theta_uniform

pytestmark = pytest.mark.gpu

TILES = dict(mode="fast", delta_index=True, forward_tiles=True)
# two iterations' rounded sums of a few hundred 2^-24 each; 16-bit codes half an
# ulp of 2^-17 of the longest length, over at least some tens of rays per pixel
TOL = {"f32": 1e-5, "u16": 1e-4}


def _plan(C, P, S, K, storage, sino, alg):
    plan = tg.Plan(P, S, C, theta_uniform(P), slices_per_pass=K, len_storage=storage, **TILES)
    plan.set_sinogram(sino, apply_abs=True)
    plan.reset_recon(alg)
    return plan


def _sino(C, P, S):
    rng = np.random.default_rng(C * S)
    vol = rng.uniform(0.5, 1.5, (S, C, C)).astype(np.float32)
    sim = O.forward(vol, O.angle_table(theta_uniform(P)), threads=4)
    return (sim * rng.uniform(0.97, 1.03, sim.shape)).astype(np.float32)


# 240 columns: 450 blocks of 16 x 8 pixels; 300: 722; four per SM of 152 are 608
@pytest.mark.parametrize("C", [240, 300])
@pytest.mark.parametrize("K,S", [(8, 3), (8, 8), (4, 7), (2, 5), (1, 6), (4, 20)])
@pytest.mark.parametrize("storage", ["f32", "u16"])
def test_against_fp64(C, K, S, storage):
    P = 40
    sino = _sino(C, P, S)
    ref = O.run("mlem", sino, tables=O.angle_table(theta_uniform(P)), n_iter=2, precision=O.F64,
                threads=4)["recon"]
    plan = _plan(C, P, S, K, storage, sino, "mlem")
    plan.iterate("mlem", 2)
    assert rel_l2(plan.get_recon("mlem"), ref) < TOL[storage]
    plan.close()


def test_batch_of_both_sides():
    """u16 plans advance in the multi-plan launches, the scalar kernel's at 8
    slices per pass among them."""
    sizes = [(240, 36, 8, 8), (300, 36, 8, 8), (300, 36, 5, 4), (300, 36, 20, 8)]
    sinos = [_sino(C, P, S) for C, P, S, _ in sizes]
    both = [[_plan(C, P, S, K, "u16", y, "mlem") for (C, P, S, K), y in zip(sizes, sinos)]
            for _ in range(2)]
    batch = tg.Batch(both[0])
    batch.iterate("mlem", 3)
    assert batch.info()["multi"]
    for a, b in zip(*both):
        b.iterate("mlem", 3)
        assert np.array_equal(bits(a.get_recon("mlem")), bits(b.get_recon("mlem")))
    batch.close()
    for plan in both[0] + both[1]:
        plan.close()
