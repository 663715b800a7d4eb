"""One JFA pass in bit-set form at the widths its footprint copies
distinguish: rows whose quads (four columns) are 16-byte aligned or not, quads
inside the row or cut by its edges, tiles cut by the volume, volumes narrower
than a tile or a quad.  Labels out of [-1, Kp) count as no label.  Bit-exact
against the CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu


def _seeds(rng, kp, W, H, D):
    s = np.zeros((kp, 12), np.float32)
    for k, n in enumerate((W, H, D)):
        s[:, k] = rng.integers(0, n, kp) + 0.5
    s[:, 3:6] = rng.uniform(0, 255, (kp, 3)).astype(np.float32)
    A = rng.normal(0, 0.4, (kp, 3, 3)).astype(np.float32)
    M = np.einsum("kij,kil->kjl", A, A)
    s[:, 6:12] = M[:, [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]]
    return s


@pytest.mark.parametrize("step", [1, 3, 4, 5, 6])
@pytest.mark.parametrize("W,H,D", [(64, 32, 24), (68, 35, 21), (44, 18, 33), (37, 23, 19), (50, 17, 40), (13, 11, 12),
                                   (5, 40, 18), (3, 3, 9)])
def test_pass_at_width(asv, orc, W, H, D, step):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W)
    rng = np.random.default_rng(10 * W + step)
    with asv.Image(lloyd_iters=2, jfa_zrun=16) as img:
        img.init_gpu(rgb, max(40, W * H * D // 500))
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        kp = img.info().Kp
        seeds = _seeds(rng, kp, W, H, D)
        img.set_seeds(seeds)
        cell = np.arange(D)[:, None, None] // 7 * 64 + np.arange(H)[None, :, None] // 6 * 8 + np.arange(W) // 9
        labels = ((cell * 7) % kp).astype(np.int32)
        labels[rng.random(labels.shape) < 0.05] = -1
        dirty = labels.copy()
        dirty[labels < 0] = rng.choice(np.array([-1, -2, kp, 8191, 8192, 1 << 30], np.int32), int((labels < 0).sum()))
        dirty[(dirty >= 0) & (dirty < kp) & (labels < 0)] = -1
        got = img.jfa_pass(dirty, step, 0.031)
        want = orc.jfa_pass(labels, img.lab(), seeds, step, 0.031)
        assert mismatch(got, want) == 0


@pytest.mark.parametrize("K", [8190, 8500])
def test_pass_at_seed_limit(asv, orc, K):
    """Seed counts just below and above the bit-set form's label map."""
    W, H, D = 96, 64, 40
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=3)
    rng = np.random.default_rng(K)
    with asv.Image(lloyd_iters=2) as img:
        img.init_gpu(rgb, K)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        kp = img.info().Kp
        seeds = _seeds(rng, kp, W, H, D)
        img.set_seeds(seeds)
        cell = np.arange(D)[:, None, None] // 9 * 60 + np.arange(H)[None, :, None] // 9 * 12 + np.arange(W) // 9
        labels = (kp - 1 - cell % kp).astype(np.int32)
        for step in (1, 2):
            got = img.jfa_pass(labels, step, 0.05)
            assert mismatch(got, orc.jfa_pass(labels, img.lab(), seeds, step, 0.05)) == 0
