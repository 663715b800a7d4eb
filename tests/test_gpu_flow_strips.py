"""The flow iterations' strips: widths around multiples of a strip's 64 columns,
heights around multiples of a step's eight rows, frames of one and of several
blocks per pair, frames smaller than the averaging window.  Bit-exact against
the NumPy restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D", [(64, 40, 3), (65, 41, 2), (63, 39, 3), (130, 72, 3), (257, 33, 2), (193, 150, 2),
                                   (11, 9, 3), (5, 70, 2), (320, 240, 3)])
def test_strips(asv, W, H, D):
    from oracle import flow as ofl
    rgb, _, _ = asv.synth_clip(W, H, D, n_ellipses=5, noise_sigma=3.0, vmax=2.5, seed=W * 3 + H)
    with asv.Image(lloyd_iters=1) as img:
        img.init_gpu(rgb, max(W * H * D // 200, 60))
        img.compute_flow()
        got_f, got_b = img.flow()
    want_f, want_b = ofl.compute_flow(rgb)
    assert np.array_equal(got_f.view(np.uint32), want_f.view(np.uint32))
    assert np.array_equal(got_b.view(np.uint32), want_b.view(np.uint32))
