"""Floods that don't follow the draw of the seeds they start from: what labA holds
then decides how the first pass reads it.  Bit-exact against the CPU
restatement's passes."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu


def _image(asv, W, H, D, K):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W * D)
    img = asv.Image(lloyd_iters=3, density_adjust=0)
    img.init_gpu(rgb, K)
    img.upload_flow(fwd, bwd)
    img.initialization()
    img.seed_matrix()
    img.RGB2LAB()
    return img


def _flood(orc, img, seeds, vol):
    i = img.info()
    for p in range(i.passes):
        ratio = np.float32(i.ratio) * np.float32(2.0 if p >= i.passes - 2 else 1.0)
        vol = orc.jfa_pass(vol, img.lab(), seeds, i.steps[p], ratio)
    return vol


@pytest.mark.parametrize("K", [60, 2500])                  # 2500: neighbouring seeds share voxels
def test_seeds_moved_after_their_draw(asv, orc, K):
    """Only the records that stand at their seed's position count."""
    W, H, D = 30, 28, 26
    with _image(asv, W, H, D, K) as img:
        img.Ld_first_init()
        img.flood(1)                                       # the centroid sums
        img.Ld_first_init()
        drawn = img.seeds()
        img.centroids_next_seeds(1)
        moved = img.seeds()
        at = [tuple(int(c) for c in s[2::-1]) for s in drawn]
        vol = np.full((D, H, W), -1, np.int32)
        for k, a in enumerate(at):
            vol[a] = k
        for k, s in enumerate(moved):
            if vol[at[k]] == k and at[k] != tuple(int(c) for c in s[2::-1]):
                vol[at[k]] = -1
        assert (vol >= 0).any()
        img.flood(2)
        img.check_dead_seeds()
        assert mismatch(img.raw_labels(), _flood(orc, img, drawn, vol)) == 0


def test_flood_after_a_replayed_loop(asv, orc):
    """A draw before the loop's second run, which replays the captured graph, is
    not the flood's: it gathers from the labels that the loop left."""
    W, H, D = 48, 40, 16
    with _image(asv, W, H, D, 40) as img:
        img.run_lloyd()
        img.Ld_first_init()
        img.run_lloyd()
        vol = img.raw_labels() if img.info().passes % 2 == 0 else img.labels()
        want = _flood(orc, img, img.seeds(), vol)
        img.flood(1)
        img.check_dead_seeds()
        assert mismatch(img.raw_labels(), want) == 0
