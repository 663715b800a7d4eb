"""Clips whose seeds are so dense that sub-tiles of the chosen depth hold too
many labels: halved and halved again, or left to the list form.  Also the
shallowest tiles of tiny volumes, and a batch whose clips share a pass's step
but not its place in their ladders.  Labels and sums bit-exact against the CPU
restatement."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zrun", [0, 5, 32])
@pytest.mark.parametrize("W,H,D,spacing", [(96, 64, 34, 5), (97, 61, 31, 7), (120, 72, 33, 9), (101, 80, 40, 12),
                                           (48, 40, 2, 6), (20, 18, 3, 9)])
def test_dense_clips(asv, orc, W, H, D, spacing, zrun):
    K = max(W * H * D // spacing ** 3, 4)
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W + spacing, jitter=0.5, noise=9.0)
    want, want_raw, _, _ = orc.run_clip(rgb, fwd, bwd, K, iters=3, nthreads=8)
    with asv.Image(lloyd_iters=3, jfa_zrun=zrun) as img:
        got = img.segment(rgb, fwd, bwd, K)
        assert mismatch(img.raw_labels(), want_raw) == 0
        assert mismatch(got, want) == 0
        kp = img.info().Kp
        assert mismatch(img.sums(), orc.centroid_sums(want_raw, img.lab(), kp)) == 0


def test_batch_of_other_ladders(asv, orc):
    dims = [(64, 48, 12, 60), (80, 60, 30, 40), (40, 30, 9, 300), (33, 47, 20, 25)]     # 6, 7, 4 and 7 passes or so
    clips = [small_clip(asv, W, H, D, seed=W, jitter=0.4) for W, H, D, _ in dims]
    with asv.Batch(dims, lloyd_iters=3) as img:
        for i, c in enumerate(clips):
            img.upload(i, *c)
        img.prepare()
        img.run_lloyd()
        for i, (c, d) in enumerate(zip(clips, dims)):
            want, _, _, _ = orc.run_clip(*c, d[3], iters=3, nthreads=8)
            assert mismatch(img.clip_labels(i), want) == 0
