"""Connectivity of labels whose segments merge in long chains, one into the one
before: longer than a walk of one round, and than all nodes that walk at once.
Equal to the CPU restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 70000), (1, 70000, 1), (70000, 1, 1), (1, 1, 800000), (3, 300, 200), (900000, 1, 1)])
def test_chains(asv, orc, shape):
    rng = np.random.default_rng(shape[0])
    n = int(np.prod(shape))
    with asv.Image(lloyd_iters=1) as img:
        for lab in (np.arange(n), rng.integers(0, 3, n)):
            lab = lab.astype(np.int32).reshape(shape)
            for supsz in (12, 400):
                got, num = img.enforce_connectivity_labels(lab, supsz)
                want, m = orc.enforce_connectivity(lab, supsz)
                assert num == m and np.array_equal(got, want)
