"""Connectivity and evaluation of volumes that would leave their kernels' tiles
nearly empty (lines, thin slabs, narrow columns), on both sides of the line where
they go without tiles.  Equal to the CPU restatements."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(300, 1, 1), (1, 300, 1), (1, 1, 300), (40, 33, 1), (40, 33, 2), (2100, 2, 2), (17, 2, 3), (9, 1, 65), (9, 2, 65),
          (9, 3, 65), (5, 70, 4), (5, 70, 8), (5, 70, 9), (70, 3, 7), (64, 4, 4), (65, 5, 31)]


def _labels(rng, shape, k):
    D, H, W = shape
    ids = rng.integers(0, k, (D // 3 + 1, H // 4 + 1, W // 5 + 1)).astype(np.int32)
    lab = ids[np.arange(D)[:, None, None] // 3, np.arange(H)[None, :, None] // 4, np.arange(W)[None, None, :] // 5]
    noise = rng.random(shape) < 0.1
    lab[noise] = rng.integers(-1, k, int(noise.sum()))
    return np.ascontiguousarray(lab)


@pytest.mark.parametrize("shape", SHAPES)
def test_sparse_volumes(asv, orc, shape):
    from oracle import evaluate as ev
    rng = np.random.default_rng(sum(shape))
    with asv.Image(lloyd_iters=1) as img:
        for k, g in ((1, 1), (3, 2), (500, 9)):
            lab, truth = _labels(rng, shape, k), np.maximum(_labels(rng, shape, g), 0)
            assert img.evaluate(lab, truth) == ev.evaluate(lab, truth)
            for supsz in (1, 9, 60):
                got, num = img.enforce_connectivity_labels(lab, supsz)
                want, m = orc.enforce_connectivity(lab, supsz)
                assert num == m and np.array_equal(got, want)
