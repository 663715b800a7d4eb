"""A single JFA pass on a streaming context, whose seeds are the ones kept from the
window before and the window's own.  Labels bit-exact against the CPU
restatement, also those of the seeds past the window's own."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1, 3, 8])
def test_pass_after_two_windows(asv, orc, step):
    W, H, D = 48, 40, 75
    rgb, fwd, bwd = asv.synth_clip(W, H, D, n_ellipses=6, noise_sigma=5.0, vmax=2.0, jitter=0.3, seed=9)
    st = asv.Stream(W, H, D, seeds_num_100=200, block_size=30, lloyd_iters=3)
    lib, p = st.lib, lambda a: a.ctypes.data_as(ctypes.c_void_p)
    for _ in range(2):
        i = st.info()
        st.push(*(v[i.block_end - i.frames_needed:i.block_end] for v in (rgb, fwd, bwd)))
    kp, Db = st.info().block_Kp, i.block_end - i.block_start
    own = 200 * (Db - 10) // 100                           # seeds asked for in the window
    assert kp > own
    lab, seeds = np.empty((Db, H, W, 4), np.uint8), np.empty((kp, 12), np.float32)
    assert lib.asv_get_lab(st.h, p(lab)) == 0 and lib.asv_get_seeds(st.h, p(seeds)) == 0
    assert lib.asv_set_seeds(st.h, p(seeds), kp) == 0
    labels = np.random.default_rng(step).integers(-1, kp, (Db, H, W)).astype(np.int32)
    labels[:, : H // 2] = kp - 1
    got = np.empty_like(labels)
    assert lib.asv_jfa_pass_host(st.h, step, 0.12, p(labels), p(got)) == 0
    st.close()
    assert np.array_equal(got, orc.jfa_pass(labels, lab, seeds, step, 0.12))
