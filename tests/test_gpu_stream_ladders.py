"""Streams whose windows have the same number of chunks, tiles and passes but
different ladders, so that a Lloyd loop captured for one window must not be
replayed for the other.  Labels equal to those of a stream without graphs and,
at the block size that the CPU restatement's overlap stands for, to its labels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(asv, rgb, fwd, bwd, seeds100, bs, **kw):
    D, H, W, _ = rgb.shape
    got = np.full((D, H, W), -7, np.int32)
    st = asv.Stream(W, H, D, seeds_num_100=seeds100, block_size=bs, lloyd_iters=4, **kw)
    for _ in range(st.info().blocks):
        i = st.info()
        a, e = i.block_end - i.frames_needed, i.block_end
        f0, lab = st.push(rgb[a:e], fwd[a:e], bwd[a:e])
        got[f0:f0 + lab.shape[0]] = lab
    placed = st.info().seeds_placed
    st.close()
    return got, placed


@pytest.mark.parametrize("W,H,D,seeds100,bs,kw", [
    (48, 34, 49, 90, 30, dict(jfa_zrun=16)),       # 30 and 29 frames: third steps 3 and 4
    (36, 33, 59, 62, 36, {}),                      # 36 and 35 frames, the estimated tile depth
    (25, 49, 89, 21, 30, dict(jfa_zrun=32)),       # 1 10 5 3 2 1 2 1 and 1 11 6 3 2 1 2 1
])
def test_windows_of_different_ladders(asv, orc, W, H, D, seeds100, bs, kw):
    clip = asv.synth_clip(W, H, D, n_ellipses=6, noise_sigma=5.0, vmax=2.0, jitter=0.3, drift_amp=2.0,
                          drift_period=40.0, seed=W + D)
    got, placed = _run(asv, *clip, seeds100, bs, **kw)
    plain, plain_placed = _run(asv, *clip, seeds100, bs, use_graph=0, **kw)
    assert placed == plain_placed and np.array_equal(got, plain)
    if bs == 30:
        want, info = orc.run_stream(*clip, seeds_num_100=seeds100, iters=4, block_size=bs, nthreads=8)
        assert placed == info["placed"] and np.array_equal(got, want)
