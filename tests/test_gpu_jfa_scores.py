"""JFA passes where the score table's margin decides which voxels take the
shader's own arithmetic: seeds a last bit apart, equal colours, forms near
zero, forms and colours too large for scores, metrics that are not finite or
not positive.  Labels are bit-exact against the CPU restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu

W, H, D = 72, 50, 30


def _table(kind, kp, rng):
    s = np.zeros((kp, 12), np.float32)
    for k, n in enumerate((W, H, D)):
        s[:, k] = rng.integers(0, n, kp) + 0.5
    s[:, 3:6] = rng.uniform(0, 255, (kp, 3))
    A = rng.normal(0, 0.5, (kp, 3, 3))
    if kind == "zero_metric":
        A[:] = 0
    M = np.einsum("kij,kil->kjl", A, A)
    s[:, 6:12] = M[:, [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]]
    if kind == "last_bit":                     # pairs that differ in one bit of one entry
        s[1::2] = s[0::2][: kp // 2]
        col = rng.integers(3, 12, kp // 2)
        i = np.arange(kp // 2)
        s[1::2][i, col] = np.nextafter(s[1::2][i, col], np.float32(1e9))
    if kind == "one_colour":
        s[:, 3:6] = 100.0
    if kind == "tiny_metric":
        s[:, 6:12] *= np.float32(1e-9)
    if kind == "large_metric":
        s[:, 6:12] *= np.float32(3e5)
    if kind == "huge_metric":                  # distances around 1e8
        s[:, 6:12] *= np.float32(1e7)
    if kind == "far_colour":
        s[::3, 3:6] += 5000.0
    if kind == "not_finite":
        s[::5, 6] = np.inf
        s[1::5, 9] = np.nan
        s[2::5, 4] = np.nan
    if kind == "negative":
        s[::2, 6:12] *= -1.0
    return s


@pytest.mark.parametrize("step", [1, 3, 6])
@pytest.mark.parametrize("kind", ["plain", "last_bit", "one_colour", "zero_metric", "tiny_metric", "large_metric",
                                  "huge_metric", "far_colour", "not_finite", "negative"])
def test_scores(asv, orc, kind, step):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=17)
    rng = np.random.default_rng(step)
    with asv.Image(lloyd_iters=2, jfa_zrun=32) as img:
        img.init_gpu(rgb, 200)
        img.upload_flow(fwd, bwd)
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        kp = img.info().Kp
        seeds = _table(kind, kp, rng)
        img.set_seeds(seeds)
        cell = np.arange(D)[:, None, None] // 10 * 60 + np.arange(H)[None, :, None] // 8 * 10 + np.arange(W) // 8
        labels = ((cell * 3) % kp).astype(np.int32)
        swap = rng.random(labels.shape) < 0.3              # neighbours of a pair side by side
        labels[swap] ^= 1
        labels[labels >= kp] = -1
        got = img.jfa_pass(labels, step, 0.12)
        want = orc.jfa_pass(labels, img.lab(), seeds, step, 0.12)
        assert mismatch(got, want) == 0
