"""Evaluation at the edges of its kernels' groups: rows narrower and wider than a
warp, volumes that end inside a warp or a word of boundary flags, label -1; one
context takes them in turn, its scratch growing and staying.  Equal to the CPU
restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 7), (1, 2, 16), (3, 5, 31), (2, 33, 32), (5, 31, 33), (4, 64, 8), (9, 29, 71), (2, 40, 129), (33, 1, 100)]


def _blocky(rng, shape, k):
    D, H, W = shape
    ids = rng.integers(0, k, (D // 3 + 1, H // 4 + 1, W // 9 + 1)).astype(np.int32)
    lab = ids[np.arange(D)[:, None, None] // 3, np.arange(H)[None, :, None] // 4, np.arange(W)[None, None, :] // 9]
    noise = rng.random(shape) < 0.05
    lab[noise] = rng.integers(0, k, int(noise.sum()))
    return np.ascontiguousarray(lab)


def test_evaluation_edges(asv):
    from oracle import evaluate as ev
    rng = np.random.default_rng(77)
    with asv.Image(lloyd_iters=1) as img:
        for shape in SHAPES + SHAPES[::-1]:
            for k, g in ((1, 1), (2, 9), (40, 6), (900, 3)):
                lab, truth = _blocky(rng, shape, k), _blocky(rng, shape, g)
                lab[rng.random(shape) < 0.1] = -1
                assert img.evaluate(lab, truth) == ev.evaluate(lab, truth)
