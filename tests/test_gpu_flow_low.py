"""Low frames that go in one strip per column of pairs, and their neighbours above
the rule (more rows than three steps, too few pairs).  Bit-exact against the NumPy
restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D", [(1000, 17, 9), (1000, 24, 9), (1000, 25, 9), (1000, 8, 9), (64, 24, 4)])
def test_low_frames(asv, W, H, D):
    from oracle import flow as ofl
    rgb, _, _ = asv.synth_clip(W, H, D, n_ellipses=9, noise_sigma=3.0, vmax=2.5, seed=W * 3 + H)
    with asv.Image(lloyd_iters=1) as img:
        img.init_gpu(rgb, W * H * D // 200)
        img.compute_flow()
        got_f, got_b = img.flow()
    want_f, want_b = ofl.compute_flow(rgb)
    assert np.array_equal(got_f.view(np.uint32), want_f.view(np.uint32))
    assert np.array_equal(got_b.view(np.uint32), want_b.view(np.uint32))
