"""A batch with more than 2^31 / 192 seed slots: the places of the last clips'
ring metrics pass 2^31 words.  Every clip has the same input, so the last clips'
labels are the first one's, and those the CPU restatement's."""
import numpy as np
import pytest

from conftest import mismatch

pytestmark = pytest.mark.gpu


def test_ring_places_past_2_31(asv, orc):
    W, H, D, K, n = 32, 32, 32, 32767, 345
    rgb, fwd, bwd = asv.synth_clip(W, H, D, n_ellipses=4, noise_sigma=5.0, vmax=3.0, jitter=1.5, seed=5)
    with asv.Batch([(W, H, D, K)] * n, lloyd_iters=2) as b:
        kp = b.clip_info(0).Kp
        assert (n - 2) * 24 * 8 * (kp + 64) > 2 ** 31
        for i in range(n):
            b.upload(i, rgb, fwd, bwd)
        b.prepare()
        b.run_lloyd()
        first = b.clip_labels(0)
        for i in (1, n // 2, n - 3, n - 2, n - 1):
            assert mismatch(b.clip_labels(i), first) == 0
    want, _, _, _ = orc.run_clip(rgb, fwd, bwd, K, iters=2, nthreads=8)
    assert mismatch(first, want) == 0
