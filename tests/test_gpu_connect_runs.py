"""Connectivity at the edges of its kernels' groups: rows narrower and wider than
a warp, runs that cross warps, volumes that end inside a warp, label -1, none or
all of the segments large enough.  Equal to the CPU restatement."""
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


@pytest.mark.parametrize("shape", SHAPES)
def test_connectivity_edges(asv, orc, shape):
    rng = np.random.default_rng(sum(shape) + 1)
    with asv.Image(lloyd_iters=1) as img:
        for k in (1, 2, 5, 40):
            lab = _blocky(rng, shape, k)
            lab[rng.random(shape) < 0.1] = -1
            for supsz in (1, 8, 60):
                got, num = img.enforce_connectivity_labels(lab, supsz)
                want, m = orc.enforce_connectivity(lab, supsz)
                assert num == m and np.array_equal(got, want)
