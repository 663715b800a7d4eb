"""The stream on which a context's fills and its batches' second variants run has
the priority of the context's own stream, also after the server gave it another."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def test_priorities(asv):
    import torch
    lib = asv.load()
    priority = getattr(lib, "_ZN3asv13side_priorityEPK7asv_ctx")              # asv::side_priority
    set_stream = getattr(lib, "_ZN3asv10set_streamEP7asv_ctxP11CUstream_st")  # asv::set_stream
    priority.argtypes, priority.restype = [ctypes.c_void_p], ctypes.c_int
    set_stream.argtypes, set_stream.restype = [ctypes.c_void_p, ctypes.c_void_p], None
    streams = {p: torch.cuda.Stream(priority=p) for p in (0, -1)}
    assert {p: s.priority for p, s in streams.items()} == {0: 0, -1: -1}
    with asv.Image(lloyd_iters=1) as img:
        assert priority(img.h) == 0
        for p in (-1, 0, -1):
            set_stream(img.h, streams[p].cuda_stream)
            assert priority(img.h) == p
    with asv.Image(lloyd_iters=2, stream=streams[-1].cuda_stream) as img:
        assert priority(img.h) == -1
        rgb, fwd, bwd = asv.synth_clip(40, 32, 8, seed=2)
        assert img.segment(rgb, fwd, bwd, 20).min() >= 0
