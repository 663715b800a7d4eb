"""The first two passes of a flood, which start from the drawn seeds instead of
gathering: seeds at corners, edges and faces (whose labels reach many voxels
through the clamped offsets), side by side, and several in one voxel.  Whole
floods, bit-exact against the CPU restatement's passes over the drawn volume;
also where the seed table was replaced after a draw."""
import numpy as np
import pytest

from conftest import mismatch, small_clip

pytestmark = pytest.mark.gpu


def _image(asv, W, H, D, K, full):
    rgb, fwd, bwd = small_clip(asv, W, H, D, seed=W * D)
    img = asv.Image(lloyd_iters=2, full_ladder=full, density_adjust=0)
    img.init_gpu(rgb, K)
    img.upload_flow(fwd, bwd)
    img.initialization()
    img.seed_matrix()
    img.RGB2LAB()
    return img


def _expected(orc, img, seeds, shape):
    i = img.info()
    vol = np.full(shape, -1, np.int32)
    for k, s in enumerate(seeds):
        vol[int(s[2]), int(s[1]), int(s[0])] = k
    lab = img.lab()
    for p in range(i.passes):
        vol = orc.jfa_pass(vol, lab, seeds, i.steps[p], np.float32(i.ratio) * np.float32(2.0 if p >= i.passes - 2 else 1.0))
    return vol


def _places(rng, kind, kp, W, H, D):
    n = np.array([W, H, D])
    if kind == "corners":
        at = rng.integers(0, 2, (kp, 3)) * (n - 1)
        at[::2] = rng.integers(0, n, (len(at[::2]), 3))
    elif kind == "faces":
        at = rng.integers(0, n, (kp, 3))
        ax = rng.integers(0, 3, kp)
        at[np.arange(kp), ax] = np.where(rng.random(kp) < 0.5, 0, n[ax] - 1)
    else:                                           # clusters: neighbours, several in one voxel
        at = np.clip(rng.integers(0, n, (max(kp // 8, 1), 3)).repeat(8, 0)[:kp], 0, n - 1)
        at = np.vstack([at, rng.integers(0, n, (kp - len(at), 3))]) if len(at) < kp else at
        at = np.clip(at + rng.integers(-1, 2, at.shape), 0, n - 1)
    return at


@pytest.mark.parametrize("full", [0, 1])
@pytest.mark.parametrize("kind", ["corners", "faces", "clusters"])
@pytest.mark.parametrize("W,H,D,K", [(50, 41, 18, 40), (64, 33, 9, 12), (30, 30, 30, 30)])
def test_flood_from_seeds(asv, orc, kind, W, H, D, K, full):
    with _image(asv, W, H, D, K, full) as img:
        img.Ld_first_init()
        seeds = img.seeds()
        rng = np.random.default_rng(W + K)
        drawn = {(int(s[0]), int(s[1]), int(s[2])) for s in seeds}
        at = _places(rng, kind, len(seeds), W, H, D)
        # (the seeds drawn first still stand where they were: keep off them)
        at[[tuple(a) in drawn for a in at]] = 0
        if (0, 0, 0) in drawn:
            pytest.skip("a grid seed at the origin")
        seeds[:, :3] = at + 0.5
        img.set_seeds(seeds)
        img.flood(1)
        img.check_dead_seeds()
        assert mismatch(img.raw_labels(), _expected(orc, img, seeds, (D, H, W))) == 0


def test_flood_of_a_plain_draw(asv, orc):
    W, H, D = 60, 44, 20
    with _image(asv, W, H, D, 50, 0) as img:
        for _ in range(2):                          # the second flood reads what the first one left behind
            img.Ld_first_init()
            seeds = img.seeds()
            img.flood(1)
            img.check_dead_seeds()
            assert mismatch(img.raw_labels(), _expected(orc, img, seeds, (D, H, W))) == 0


def test_flood_again_without_a_draw(asv, orc):
    """A flood that follows a flood gathers every pass from the last labels."""
    W, H, D = 48, 40, 16
    with _image(asv, W, H, D, 40, 0) as img:
        img.Ld_first_init()
        seeds = img.seeds()
        img.flood(1)
        img.check_dead_seeds()
        i = img.info()
        raw = img.raw_labels()
        if i.passes % 2 == 0:                       # the labels are in the volume that the first pass reads
            img2_in = raw
        else:
            img2_in = img.labels()
        want = img2_in
        for p in range(i.passes):
            want = orc.jfa_pass(want, img.lab(), seeds, i.steps[p],
                                np.float32(i.ratio) * np.float32(2.0 if p >= i.passes - 2 else 1.0))
        img.flood(2)
        img.check_dead_seeds()
        assert mismatch(img.raw_labels(), want) == 0
