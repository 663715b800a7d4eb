"""The overlap that a stream keeps on the device, the last ten frames of the window
before, where that window has fewer than twenty: the shift then overlaps itself."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,bs", [(40, 32, 12), (41, 33, 12), (200, 160, 18), (63, 50, 24)])
def test_overlap_of_short_windows(asv, orc, W, H, bs):
    D = 5 * bs
    rgb, fwd, bwd = asv.synth_clip(W, H, D, n_ellipses=6, noise_sigma=5.0, vmax=2.0, jitter=0.3, seed=bs)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    st = asv.Stream(W, H, D, seeds_num_100=max(W * H * 100 // 1000, 100), block_size=bs, lloyd_iters=1)
    on_device = []                                            # the window's frames, by their number in the video
    for _ in range(min(st.info().blocks, 4)):
        i = st.info()
        new = list(range(i.block_end - i.frames_needed, i.block_end))
        on_device = on_device[-10:] + new if on_device else new
        st.push(*(v[new[0]:new[-1] + 1] for v in (rgb, fwd, bwd)))
        n = len(on_device)
        lab, f, b = np.empty((n, H, W, 4), np.uint8), np.empty((n, H, W, 2), np.float32), np.empty((n, H, W, 2), np.float32)
        assert st.lib.asv_get_lab(st.h, p(lab)) == 0 and st.lib.asv_get_flow(st.h, p(f), p(b)) == 0
        assert np.array_equal(f, fwd[on_device]) and np.array_equal(b, bwd[on_device])
        assert np.array_equal(lab, orc.rgb2lab(rgb[on_device]).reshape(lab.shape))
    st.close()
