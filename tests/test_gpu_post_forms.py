"""Post-processing on caller-owned buffers at the edges of its kernels' groups:
buffers not aligned to 16 bytes, volumes that end inside a warp, a thread's eight
voxels or a chunk of 2048, a first voxel of label -1, dead seeds of either rule.
Equal to the CPU restatement."""
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


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_noalloc_edges(asv, orc, shape, offset):
    torch = pytest.importorskip("torch")
    lib, rng, n = asv.load(), np.random.default_rng(sum(shape)), int(np.prod(shape))
    D, H, W = shape
    for kp, dead, minus, first in ((12, 0, 0.0, None), (12, 0, 0.1, None), (12, 0, 0.3, -1), (12, 2, 0.1, None),
                                   (12, 3, 0.0, -1), (20, 6, 0.1, None), (20, 7, 0.2, -1), (3000, 5, 0.0, None)):
        raw = _blocky(rng, shape, kp - dead) + (dead // 2)
        raw[rng.random(shape) < minus] = -1
        if first is not None:
            raw.ravel()[: min(3, n)] = first
        counts = np.zeros((kp + 1, 7), np.int64)
        counts[:, 3] = np.bincount(np.where(raw < 0, kp, raw).ravel(), minlength=kp + 1)
        want, _ = orc.postprocess(raw, counts, kp)
        src = torch.zeros(n + 8, dtype=torch.int32, device="cuda")
        dst = torch.full((n + 8,), -9, dtype=torch.int32, device="cuda")
        src[offset:offset + n] = torch.from_numpy(raw.ravel()).cuda()
        st = lib.asv_check_dead_seeds_noalloc(src.data_ptr() + 4 * offset, dst.data_ptr() + 4 * offset, W, H, D, kp,
                                              torch.cuda.current_stream().cuda_stream)
        assert st == 0
        got = dst.cpu().numpy()
        assert np.array_equal(got[offset:offset + n].reshape(shape), want)
        assert (np.delete(got, np.arange(offset, offset + n)) == -9).all()


def test_noalloc_under_capture(asv, orc):
    torch = pytest.importorskip("torch")
    lib, shape, kp = asv.load(), (4, 64, 40), 20
    D, H, W = shape
    rng = np.random.default_rng(8)
    raws = []
    for dead in (0, 2, 5):
        raw = _blocky(rng, shape, kp - dead)
        raw[rng.random(shape) < 0.1] = -1
        raws.append(raw)
    src = torch.from_numpy(raws[0]).cuda()
    dst = torch.empty_like(src)

    def call():
        return lib.asv_check_dead_seeds_noalloc(src.data_ptr(), dst.data_ptr(), W, H, D, kp,
                                                torch.cuda.current_stream().cuda_stream)

    assert call() == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st = call()
    assert st == 0
    for raw in raws:
        src.copy_(torch.from_numpy(raw))
        graph.replay()
        torch.cuda.synchronize()
        counts = np.zeros((kp + 1, 7), np.int64)
        counts[:, 3] = np.bincount(np.where(raw < 0, kp, raw).ravel(), minlength=kp + 1)
        want, _ = orc.postprocess(raw, counts, kp)
        assert np.array_equal(dst.cpu().numpy(), want)


@pytest.mark.parametrize("kp,dead", [(4095, (0, 4094)), (4096, (3, 4095)), (4098, (4095, 4096)), (9000, (1, 4096, 8191, 8192, 8999)),
                                     (4100, (4096, 4097, 4098, 4099))])
def test_noalloc_scan_rounds(asv, orc, kp, dead):
    """Ranks and chunk carries over several rounds of 4096, sources rounds apart."""
    torch = pytest.importorskip("torch")
    lib, W, H, D = asv.load(), 2048, 1, 4099
    n = W * H * D
    alive = np.setdiff1d(np.arange(kp), dead).astype(np.int32)
    raw = alive[(np.arange(n) // 3) % len(alive)].reshape(D, H, W)
    raw[5:4097] = -1                                # chunks without a source across a round's end
    raw[4097, 0, 9:] = -1
    counts = np.zeros((kp + 1, 7), np.int64)
    counts[:, 3] = np.bincount(np.where(raw < 0, kp, raw).ravel(), minlength=kp + 1)
    want, _ = orc.postprocess(raw, counts, kp)
    src = torch.from_numpy(raw).cuda()
    dst = torch.empty_like(src)
    assert lib.asv_check_dead_seeds_noalloc(src.data_ptr(), dst.data_ptr(), W, H, D, kp,
                                            torch.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(dst.cpu().numpy(), want)
