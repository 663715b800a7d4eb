"""asv_autotune's candidates hold the depth that a context has without it."""
import ctypes

import pytest


def test_the_estimate_is_timed_first(asv):
    depths = getattr(asv.load(), "_ZN3asv15autotune_depthsEiPi")     # asv::autotune_depths
    depths.argtypes, depths.restype = [ctypes.c_int, ctypes.POINTER(ctypes.c_int)], ctypes.c_int
    for estimate in range(1, 33):
        out = (ctypes.c_int * 5)()
        n = depths(estimate, out)
        got = list(out[:n])
        assert got[0] == estimate
        assert sorted(got) == sorted({estimate, 4, 8, 16, 32})


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,D,K", [(64, 48, 12, 60), (96, 80, 30, 200)])
def test_autotune_keeps_the_labels(asv, W, H, D, K):
    rgb, fwd, bwd = asv.synth_clip(W, H, D, seed=4)
    with asv.Image(lloyd_iters=4) as img:
        want = img.segment(rgb, fwd, bwd, K)
        assert img.autotune() in (4, 8, 16, 32)
        assert (img.labels() == want).all()
