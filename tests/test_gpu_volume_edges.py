"""Density, LAB and post-processing kernels at the edges of their groups: rows
narrower than a warp, wider than a block, volumes that end inside a thread's four
or eight voxels and inside a chunk, many and few cells, dead seeds of either rule
and fills.  Bit-exact against the CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu

SIZES = [(7, 9, 5, 6), (33, 31, 7, 40), (300, 5, 9, 200), (64, 32, 2, 700), (61, 53, 11, 900)]


@pytest.mark.parametrize("W,H,D,K", SIZES)
def test_seeds_and_lab(asv, orc, W, H, D, K):
    rng = np.random.default_rng(W + H)
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W)
    noise = rng.integers(0, 256, rgb.shape, dtype=np.uint8)
    flat = np.full_like(rgb, 255)
    flat[:, ::2] = 0
    for px in (rgb, noise, flat):
        with asv.Image(lloyd_iters=1) as img:
            img.init_gpu(px, K)
            img.upload_flow(fwd, bwd)
            img.initialization()
            img.seed_matrix()
            img.RGB2LAB()
            img.Ld_first_init()
            grid, g = orc.grid_seeds(W, H, D, K)
            want, _ = orc.density_adjust(px, grid, g)
            assert mismatch(img.seeds()[:, :3], want[:, :3]) == 0
            assert mismatch(img.lab()[..., :3], orc.rgb2lab(px)[..., :3]) == 0


@pytest.mark.parametrize("W,H,D,K", SIZES)
def test_relabel_and_fill(asv, orc, W, H, D, K):
    rng = np.random.default_rng(W * H)
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W)
    with asv.Image(lloyd_iters=1) as img:
        img.init_gpu(rgb, K)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        kp = img.info().Kp
        for dead, minus, first in ((0, 0.0, 0), (0, 0.2, 0), (0, 0.2, 3), (2, 0.1, 0), (4, 0.1, 0), (5, 0.9, 9)):
            raw = rng.integers(0, max(kp - dead, 1), (D, H, W)).astype(np.int32)
            raw[rng.random(raw.shape) < minus] = -1
            raw.ravel()[:first] = -1
            counts = np.zeros((kp + 1, 7), np.int64)
            counts[:, 3] = np.bincount(np.where(raw < 0, kp, raw).ravel(), minlength=kp + 1)
            want, _ = orc.postprocess(raw, counts, kp)
            assert mismatch(img.check_dead_seeds_host(raw), want) == 0
