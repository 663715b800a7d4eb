"""Metric solves at the edges of their layout (two solves a warp, two lanes a
column, rows split between them): seeds at corners, edges and faces of the frame
in the first, middle and last frames (4 to 18 rows), still, uniform, random and
large flows (rank-deficient and badly scaled systems), odd numbers of seeds.
Equal to the CPU restatement bit for bit."""
import numpy as np
import pytest

from conftest import small_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flow", ["still", "uniform", "random", "large", "half"])
@pytest.mark.parametrize("W,H,D,K", [(40, 30, 8, 33), (24, 50, 2, 30), (64, 48, 12, 61)])
def test_metrics_everywhere(asv, orc, W, H, D, K, flow):
    rng = np.random.default_rng(W + D)
    rgb = small_clip(asv, W, H, D, seed=1)[0]
    fwd, bwd = np.zeros((2, D, H, W, 2), np.float32)
    if flow == "uniform":
        fwd[...] = (1.4, -2.6)
        bwd[...] = (-1.4, 2.6)
    elif flow == "random":
        fwd, bwd = (rng.normal(0, 3, fwd.shape).astype(np.float32) for _ in range(2))
    elif flow == "large":
        fwd, bwd = (rng.normal(0, 300, fwd.shape).astype(np.float32) for _ in range(2))
    elif flow == "half":                              # still on one side, the boundary along x
        fwd[:, :, W // 2:] = (3.0, 0.5)
        bwd[:, :, W // 2:] = (-3.0, -0.5)
    fwd, bwd = np.ascontiguousarray(fwd), np.ascontiguousarray(bwd)
    with asv.Image(lloyd_iters=2) as img:
        img.init_gpu(rgb, K)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        img.Ld_first_init()
        for part in range(4):
            s = img.seeds()
            n = np.array([W, H, D])
            at = rng.integers(0, n, (len(s), 3))
            ax = rng.integers(0, 3, len(s))
            at[np.arange(len(s)), ax] = np.where(rng.random(len(s)) < 0.5, 0, n[ax] - 1)
            if part == 1:
                at[:, :2] = rng.integers(0, 2, (len(s), 2)) * (n[:2] - 1)
            s[:, :3] = at + 0.5
            img.set_seeds(s)
            img.Ld_next_seeds_matrix(1)
            want, _ = orc.seed_metrics(fwd, bwd, s[:, :3], 1, 1)
            assert np.array_equal(img.seeds()[:, 6:12].view(np.int32), want.view(np.int32))
