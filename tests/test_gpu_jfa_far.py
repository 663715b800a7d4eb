"""Passes of steps above the bit-set form's, whose chains start at slice 0 and end
at the last one after few positions: steps around the depth, half of it and of
the frame, depths of one slice and more, sparse and dense label volumes.  Equal
to the CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,K", [(40, 33, 2, 60), (48, 40, 16, 40), (33, 50, 31, 60), (64, 20, 45, 50)])
def test_far_steps(asv, orc, W, H, D, K):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W + D)
    rng = np.random.default_rng(W)
    with asv.Image(lloyd_iters=2, density_adjust=0) as img:
        img.init_gpu(rgb, K)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        img.Ld_first_init()
        seeds, lab = img.seeds(), img.lab()
        for step in sorted({7, 8, 11, D - 1, D, D + 1, D // 2 + 1, (D + 2) // 3, 64} - set(range(7))):
            for filled in (0.02, 0.5, 1.0):
                vol = rng.integers(0, len(seeds), (D, H, W)).astype(np.int32)
                vol[rng.random(vol.shape) >= filled] = -1
                got = img.jfa_pass(vol, step, 0.7)
                want = orc.jfa_pass(vol, lab, seeds, step, np.float32(0.7))
                assert mismatch(got, want) == 0, (step, filled)
