"""The second pass where labels meet: equal distances (flat colours, a still
picture, seeds on a grid), which the order of the candidates decides, and floods
of the Lloyd loop and step by step in turn on one context.  Bit-exact against the
CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip
from test_gpu_first_passes import _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("full", [0, 1])
@pytest.mark.parametrize("W,H,D,K", [(64, 48, 24, 60), (33, 31, 17, 40), (24, 24, 8, 100)])
def test_equal_distances(asv, orc, W, H, D, K, full):
    rgb = np.full((D, H, W, 3), 90, np.uint8)
    still = np.zeros((D, H, W, 2), np.float32)
    with asv.Image(lloyd_iters=2, full_ladder=full, density_adjust=0) as img:
        img.init_gpu(rgb, K)
        img.upload_flow(still, still)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        img.Ld_first_init()
        seeds = img.seeds()
        img.flood(1)
        img.check_dead_seeds()
        assert mismatch(img.raw_labels(), _expected(orc, img, seeds, (D, H, W))) == 0


def test_loop_and_steps_in_turn(asv, orc):
    W, H, D, K = 60, 44, 20, 50
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=4)
    want = orc.run_clip(rgb, fwd, bwd, K, iters=3)[0]
    with asv.Image(lloyd_iters=3) as img:
        for leave in (0, 1, 2):
            assert mismatch(img.segment(rgb, fwd, bwd, K), want) == 0
            img.Ld_first_init()                     # left at a draw, after a flood, at the next draw
            if leave > 0:
                img.flood(1)
            if leave > 1:
                img.centroids_next_seeds(1)
                img.Ld_next_seeds_matrix(1)
        assert mismatch(img.segment(rgb, fwd, bwd, K), want) == 0
