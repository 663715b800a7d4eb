"""A single JFA pass with a caller's ratio of any sign: a negative one makes near
seeds lose to far ones, zero leaves the colours alone.  Labels bit-exact against
the CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu

W, H, D = 72, 50, 30


@pytest.mark.parametrize("step", [1, 3, 6, 9])
@pytest.mark.parametrize("ratio", [-0.12, -3.0, 0.0])
def test_ratio(asv, orc, ratio, step):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=17)
    rng = np.random.default_rng(step)
    with asv.Image(lloyd_iters=2, jfa_zrun=32) as img:
        img.init_gpu(rgb, 200)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        img.Ld_first_init()
        kp, seeds = img.info().Kp, img.seeds()
        cell = np.arange(D)[:, None, None] // 10 * 60 + np.arange(H)[None, :, None] // 8 * 10 + np.arange(W) // 8
        labels = (cell % kp).astype(np.int32)
        labels[rng.random(labels.shape) < 0.2] = -1
        want = orc.jfa_pass(labels, img.lab(), seeds, step, ratio)
        assert mismatch(img.jfa_pass(labels, step, ratio), want) == 0
