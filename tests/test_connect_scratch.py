"""Scratch of the connectivity enforcement, which a budget is held against: no more
than with the groups' counts in the chunks' place."""
import ctypes

import numpy as np
import pytest


def _bytes(n):
    return 4 * n * 6 + 4 * ((n + 2047) // 2048 + 2) + 256 * 8


@pytest.mark.parametrize("n", [1, 127, 128, 2048, 2049, 320 * 240 * 85, 2 ** 31 - 1])
def test_scratch_bytes(asv, n):
    f = getattr(asv.load(), "_Z25asv_connect_scratch_bytesx")
    f.argtypes, f.restype = [ctypes.c_longlong], ctypes.c_size_t
    assert f(n) <= _bytes(n)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 200), (7, 33, 65), (20, 64, 64)])
def test_a_budget_of_those_bytes_admits_the_call(asv, orc, shape):
    n = int(np.prod(shape))
    lab = np.random.default_rng(n).integers(0, 5, shape).astype(np.int32)
    with asv.Image(lloyd_iters=1, hbm_budget=2 * ((4 * n + 255) // 256 * 256) + _bytes(n)) as img:
        got, num = img.enforce_connectivity_labels(lab, 8)
    want, m = orc.enforce_connectivity(lab, 8)
    assert num == m and np.array_equal(got, want)
