"""Timed cases of the supervoxel engine, over the work its users have it do.

Every case goes through the C ABI (include/asv.h) or its Python mirror with
host buffers that a program keeps pinned, as the engine's own programs do:
a clip segmented from its frames and flow, the same from raw video frames
with the flow computed on the device, the flow alone, windows of a long
video, clips of uneven size in one batch, and what follows a segmentation
(connectivity enforcement, evaluation, the post-processing on a caller's
device buffers).
"""
import ctypes
import math

import numpy as np
import torch

import anisotropic_supervoxel_gb300 as asv

NAMES = ("clip", "video_clip", "flow", "stream", "batch", "connect", "evaluate", "post")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _clip(W, H, D, K, iters, variant=0, full_ladder=0, middlebury=0):
    return dict(kind="clip", W=W, H=H, D=D, K=K, iters=iters, variant=variant, full_ladder=full_ladder,
                middlebury=middlebury)


def listed():
    return [
        # a thumbnail-sized clip: launches and latency count
        dict(name="clip_64x48x12", **_clip(64, 48, 12, 60, 4)),
        # the small plain clip, with the full ladder of powers of two
        dict(name="clip_240x160x30_full", **_clip(240, 160, 30, 200, 10, full_ladder=1)),
        # the usual benchmark clip of the supervoxel literature's size
        dict(name="clip_320x240x85", **_clip(320, 240, 85, 1000, 15)),
        # odd sizes, many small supervoxels, the streaming variant's weights, the reference's default of 20 iterations
        dict(name="clip_427x239x61_dense", **_clip(427, 239, 61, 3000, 20, variant=1)),
        # raw BGR frames: preprocessing, optical flow, segmentation
        dict(name="video_clip_320x240x85", kind="video_clip", W=320, H=240, D=85, K=1000, iters=15),
        # the optical flow alone, forward and backward, of a VGA clip
        dict(name="flow_640x480x16", kind="flow", W=640, H=480, D=16),
        # one window of a long 720p video, flow given
        dict(name="stream_1280x720", kind="stream", W=1280, H=720, seeds_num_100=10000, iters=20, block=30,
             device_flow=False),
        # one window of a smaller video with odd width, flow computed on the device
        dict(name="stream_641x360_flow", kind="stream", W=641, H=360, seeds_num_100=2500, iters=20, block=30,
             device_flow=True),
        # six clips of uneven size segmented together
        dict(name="batch_6_uneven", kind="batch", n=6, W=640, H=480, D=60, K=1000, iters=10),
        # 3D connectivity enforcement of a clip's labels
        dict(name="connect_320x240x85", kind="connect", W=320, H=240, D=85, K=1000),
        # quality measures of a clip's labels against a ground truth
        dict(name="evaluate_320x240x85", kind="evaluate", W=320, H=240, D=85, cell=18),
        # dead-seed relabel and -1 fill on the caller's device buffers
        dict(name="post_320x240x85", kind="post", W=320, H=240, D=85, cell=18, dead=5, minus=0.01),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, least, most):
    """W, H, D of least..most voxels, any parity."""
    D = int(_log(rng, 8, 110))
    area = _log(rng, max(least / D, 40 * 32), max(min(most / D, 1280 * 720), 50 * 40))
    aspect = rng.uniform(1.0, 1.9)
    W = int(math.sqrt(area * aspect))
    return W, max(int(area / W), 24), D


def draw(rng):
    kind = rng.choice(NAMES + ("clip", "clip", "clip", "stream"))     # segmentation is what is called most
    if kind in ("clip", "video_clip", "connect"):
        W, H, D = _dims(rng, 3e4, 9e6)
        s = rng.uniform(8.0, 26.0)                                   # spacing of the seeds
        K = min(max(int(W * H * D / s ** 3), 8), 8000)
        if kind == "connect":
            return dict(kind=kind, W=W, H=H, D=D, K=K)
        iters = rng.randint(4, 20)
        if kind == "video_clip":
            return dict(kind=kind, W=max(W, 48), H=max(H, 36), D=D, K=K, iters=iters)
        return _clip(W, H, D, K, iters, variant=rng.randint(0, 1), full_ladder=int(rng.random() < 0.2))
    if kind == "flow":
        W, H, D = _dims(rng, 3e4, 6e6)
        return dict(kind=kind, W=max(W, 48), H=max(H, 36), D=min(D, 64))
    if kind == "stream":
        W = int(_log(rng, 160, 1280))
        H = int(W * rng.uniform(0.5, 0.75))
        H = min(H, 720)
        s = rng.uniform(14.0, 26.0)
        return dict(kind=kind, W=W, H=H, seeds_num_100=max(int(100 * W * H / s ** 3), 100), iters=rng.randint(5, 20),
                    block=30, device_flow=rng.random() < 0.3)
    if kind == "batch":
        W = int(_log(rng, 120, 640))
        return dict(kind=kind, n=rng.randint(2, 8), W=W, H=int(W * 0.75), D=rng.randint(12, 60), K=rng.randint(100, 1000),
                    iters=rng.randint(4, 10))
    if kind == "evaluate":
        W, H, D = _dims(rng, 1e5, 9e6)
        return dict(kind=kind, W=W, H=H, D=D, cell=min(rng.randint(8, 26), min(W, H) // 6))
    W, H, D = _dims(rng, 2e4, 9e6)
    dead = rng.choice((0, 2, 5))
    return dict(kind=kind, W=W, H=H, D=D, cell=rng.randint(8, 26), dead=dead, minus=rng.choice((0.0, 0.01)))


def _batch_dims(c):
    """n uneven clips from the given largest one down (the same for every seed)."""
    out = []
    for i in range(c["n"]):
        f = 1.0 - 0.55 * i / max(c["n"] - 1, 1)
        W, H = max(int(c["W"] * f), 48), max(int(c["H"] * f), 36)
        out.append((W, H, max(int(c["D"] * (0.4 + 0.6 * ((i * 5) % c["n"]) / c["n"])), 8),
                    max(int(c["K"] * f * f), 24)))
    return out


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _pin(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _video(W, H, n, seed, frame0=0):
    """A seeded synthetic video: textured moving ellipses with noise, and its flow."""
    return asv.synth_clip(W, H, n, n_ellipses=max(6, min(60, W * H // 3000)), noise_sigma=5.0, vmax=3.0, jitter=0.5,
                          seed=seed, frame0=frame0)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _cells(W, H, D, cell, seed, device):
    """Labels of warped cells of about cell^3 voxels, numbered densely in raster order: int32 [D, H, W] on `device`."""
    g = torch.Generator().manual_seed(seed)
    ph = (torch.rand(6, generator=g, dtype=torch.float64) * 6.283).tolist()
    z = torch.arange(D, device=device, dtype=torch.float32)[:, None, None]
    y = torch.arange(H, device=device, dtype=torch.float32)[None, :, None]
    x = torch.arange(W, device=device, dtype=torch.float32)[None, None, :]
    a, f = 0.35 * cell, 6.283 / (3.1 * cell)
    nx, ny, nz = (max(n // cell, 1) for n in (W, H, D))
    ix = ((x + a * torch.sin(f * y + ph[0]) + a * torch.sin(f * z + ph[1])) / cell).floor().clamp(0, nx - 1)
    iy = ((y + a * torch.sin(f * x + ph[2]) + a * torch.sin(f * z + ph[3])) / cell).floor().clamp(0, ny - 1)
    iz = ((z + a * torch.sin(f * x + ph[4]) + a * torch.sin(f * y + ph[5])) / cell).floor().clamp(0, nz - 1)
    return ((iz * ny + iy) * nx + ix).to(torch.int32), nx * ny * nz


def _labels_and_truth(case, seed, device):
    lab, n = _cells(case["W"], case["H"], case["D"], case["cell"], seed, device)
    return lab % 32000, _cells(case["W"], case["H"], case["D"], 3 * case["cell"], seed + 1, device)[0] % 4000


class _State:
    pass


def prepare(case, seed):
    s, k = _State(), case["kind"]
    s.kind, s.case, s.lib = k, dict(case), asv.load()
    if k == "batch":
        dims = _batch_dims(case)
        s.img = asv.Batch(dims, lloyd_iters=case["iters"])
        s.clips = [tuple(_pin(a) for a in _video(W, H, D, 1000 * seed + i)) for i, (W, H, D, _) in enumerate(dims)]
        s.out = [_pinned((D, H, W), torch.int32) for W, H, D, _ in dims]
        return s
    W, H = case["W"], case["H"]
    if k == "stream":
        frames = [_video(W, H, case["block"], seed), _video(W, H, 2 * case["block"] // 3, seed, frame0=case["block"])]
        s.frames = [tuple(_pin(a) for a in f) for f in frames]
        s.out = _pinned((case["block"] + case["block"] // 3, H, W), torch.int32)
        s.img = _open(case)
        return s
    D = case["D"]
    if k in ("clip", "video_clip", "flow", "connect"):
        rgb, fwd, bwd = _video(W, H, D, seed)
        if k in ("video_clip", "flow"):
            # frames as a video decoder gives them: BGR, top row first
            s.rgb = _pin(np.ascontiguousarray(rgb[:, ::-1, :, ::-1]))
        else:
            s.rgb, s.fwd, s.bwd = _pin(rgb), _pin(fwd), _pin(bwd)
        opts = {o: case[o] for o in ("variant", "full_ladder", "middlebury") if o in case}
        s.img = asv.Image(lloyd_iters=case.get("iters", 6), **opts)
        s.out = _pinned((D, H, W), torch.int32)
        if k == "flow":
            s.out = _pinned((D, H, W, 2), torch.float32), _pinned((D, H, W, 2), torch.float32)
        if k == "connect":                       # the labels are on the device when the call comes
            s.img.segment(s.rgb, s.fwd, s.bwd, case["K"])
        return s
    if k == "evaluate":
        lab, truth = _labels_and_truth(case, seed, "cuda")
        s.lab, s.truth = _pin(lab.cpu().numpy()), _pin(truth.cpu().numpy())
        s.img = asv.Image(lloyd_iters=1)
        return s
    lab, n = _cells(W, H, D, case["cell"], seed, "cuda")
    n = min(n, 32767)
    lab = lab % n
    g = torch.Generator().manual_seed(seed)
    gone = torch.randperm(n, generator=g)[: min(case["dead"], n - 1)].to("cuda").to(torch.int32)
    lab[torch.isin(lab, gone)] = -1
    if case["minus"]:
        gd = torch.Generator(device="cuda").manual_seed(seed)
        lab[torch.rand(lab.shape, device="cuda", generator=gd) < case["minus"]] = -1
    s.raw, s.out, s.Kp = lab.contiguous(), torch.empty_like(lab), n
    s.stream = torch.cuda.current_stream().cuda_stream
    return s


def _open(case):
    """The stream of a 400-window video."""
    return asv.Stream(case["W"], case["H"], case["block"] + 400 * (2 * case["block"] // 3),
                      seeds_num_100=case["seeds_num_100"], block_size=case["block"], lloyd_iters=case["iters"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    c, img = s.case, s.__dict__.get("img")
    if s.kind == "clip":
        img._ck(s.lib.asv_segment_clip(img.h, _ptr(s.rgb), _ptr(s.fwd), _ptr(s.bwd), c["W"], c["H"], c["D"], c["K"],
                                       _ptr(s.out)))
        return s.out
    if s.kind == "video_clip":
        img.init_gpu_bgr(s.rgb, c["K"])
        img.compute_flow()
        img.initialization()
        img.seed_matrix()
        img.RGB2LAB()
        img.run_lloyd()
        img._ck(s.lib.asv_get_labels(img.h, _ptr(s.out)))
        return s.out
    if s.kind == "flow":
        img.init_gpu_bgr(s.rgb, 8)
        img.compute_flow()
        img._ck(s.lib.asv_get_flow(img.h, _ptr(s.out[0]), _ptr(s.out[1])))
        return s.out
    if s.kind == "stream":
        at = img.info()
        if at.next_block == at.blocks:           # the video is over: the next one
            img.close()
            s.img = img = _open(c)
            at = img.info()
        rgb, fwd, bwd = s.frames[0 if at.next_block == 0 else 1]
        if c["device_flow"]:
            fwd = bwd = None
        if at.frames_needed != len(rgb):         # a video's last window can be longer
            reps = [i % len(rgb) for i in range(at.frames_needed)]
            rgb, fwd, bwd = (None if a is None else a[reps] for a in (rgb, fwd, bwd))
        return img.push(rgb, fwd, bwd, out=s.out)[1]
    if s.kind == "batch":
        for i, clip in enumerate(s.clips):
            img.upload(i, *clip)
        img.prepare()
        img.run_lloyd()
        for i, o in enumerate(s.out):
            img._ck(s.lib.asv_batch_get_labels(img.h, i, _ptr(o)))
        return s.out
    if s.kind == "connect":
        n = ctypes.c_int()
        img._ck(s.lib.asv_enforce_connectivity(img.h, 0, _ptr(s.out), ctypes.byref(n)))
        return s.out, n.value
    if s.kind == "evaluate":
        return img.evaluate(s.lab, s.truth)
    st = s.lib.asv_check_dead_seeds_noalloc(s.raw.data_ptr(), s.out.data_ptr(), c["W"], c["H"], c["D"], s.Kp, s.stream)
    if st != 0:
        raise RuntimeError(f"asv_check_dead_seeds_noalloc: {st}")
    return s.out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _passes(s, full, maxdim):
    """Passes of the flood's ladder for base step s."""
    n, st = 1, math.floor(0.5 * s)
    if full:
        n += int(math.log2(maxdim)) + 1
    else:
        while st > 0:
            n += 1
            st = 0 if int(st) == 1 else math.floor(0.5 * st + 0.5)
    return n + 2


def _lloyd_work(W, H, D, K, iters, full=0):
    """Bytes and operations of the Lloyd loop: a pass of the flood reads and
    writes each voxel's label and reads its three colour bytes, with at least
    two distances of 22 operations at a boundary; the sums read label and
    colour once more."""
    n = W * H * D
    P = _passes(int((n / max(K, 1)) ** (1 / 3) + 1e-9), full, max(W, H, D))
    return n * iters * (11 * P + 7), n * iters * P * 44


def _flow_work(W, H, D):
    """Ten iterations a level: the two expansions (20 bytes each) and the flow
    in and out; per pixel about 60 operations of the products and 13 + 13
    additions for each of five sums."""
    px = sum(math.ceil(W / 2 ** k) * math.ceil(H / 2 ** k) for k in range(5)) * 2 * (D - 1)
    return 10 * px * 56, 10 * px * (60 + 5 * 26)


def work(case):
    k = case["kind"]
    if k == "batch":
        b = f = 0
        for W, H, D, K in _batch_dims(case):
            wb, wf = _lloyd_work(W, H, D, K, case["iters"])
            b, f = b + wb + 23 * W * H * D, f + wf
        return {"bytes": b, "flops": f}
    W, H = case["W"], case["H"]
    if k == "stream":
        D, new = case["block"], 2 * case["block"] // 3
        b, f = _lloyd_work(W, H, D, case["seeds_num_100"] * new // 100 * D // new, case["iters"])
        b += W * H * new * (3 + 4 + (0 if case["device_flow"] else 16))
        if case["device_flow"]:
            fb, ff = _flow_work(W, H, new + 1)
            b, f = b + fb, f + ff
        return {"bytes": b, "flops": f}
    n = W * H * case["D"]
    if k == "clip":
        b, f = _lloyd_work(W, H, case["D"], case["K"], case["iters"], case["full_ladder"])
        return {"bytes": b + 23 * n, "flops": f}
    if k == "video_clip":
        b, f = _lloyd_work(W, H, case["D"], case["K"], case["iters"])
        fb, ff = _flow_work(W, H, case["D"])
        return {"bytes": b + fb + 7 * n, "flops": f + ff}
    if k == "flow":
        fb, ff = _flow_work(W, H, case["D"])
        return {"bytes": fb + 19 * n, "flops": ff}
    # labels in, labels out (or both label volumes in)
    return {"bytes": 8 * n, "flops": 0}


# ---------------------------------------------------------------------------
# the computed outputs in 64 bits (the others are labels and counts)
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "flow":
        return _exact_flow(case, seed)
    if case["kind"] == "evaluate":
        return _exact_measures(case, seed)
    return None


def _exact_measures(case, seed):
    lab, gt = (t.cpu().numpy().astype(np.int64) for t in _labels_and_truth(case, seed, "cuda"))
    D = lab.shape[0]
    ns, ng = int(lab.max()) + 1, int(gt.max()) + 1
    n = np.bincount((lab * ng + gt).ravel(), minlength=ns * ng).reshape(ns, ng)
    ssz, gsz = n.sum(1), n.sum(0)
    there = gsz > 0
    under = ((n > 0) * ssz[:, None]).sum(0)
    best = n.argmax(1)
    cover = np.bincount(best, weights=n[np.arange(ns), best], minlength=ng)

    def bound(a):
        b = np.zeros(a.shape, bool)
        for ax in range(3):
            d = np.diff(a, axis=ax) != 0
            lo, hi = [slice(None)] * 3, [slice(None)] * 3
            lo[ax], hi[ax] = slice(0, -1), slice(1, None)
            b[tuple(lo)] |= d
            b[tuple(hi)] |= d
        return b

    near = np.pad(bound(lab), 1)
    for ax in range(3):
        near = near | np.roll(near, 1, ax) | np.roll(near, -1, ax)
    near = near[1:-1, 1:-1, 1:-1]
    tb = bound(gt)
    first, last = np.full(ns, D), np.full(ns, -1)
    for z in range(D):
        ids = np.unique(lab[z])
        first[ids] = np.minimum(first[ids], z)
        last[ids] = z
    live = ssz > 0
    truth, hit = int(tb.sum()), int((tb & near).sum())
    return {"undersegmentation": float(((under - gsz)[there] / gsz[there]).mean()),
            "segmentation_accuracy": float((cover[there] / gsz[there]).mean()),
            "boundary_recall": hit / truth if truth else 1.0,
            "mean_duration": float((last - first + 1)[live].mean()), "supervoxels": int(live.sum()),
            "truth_segments": int(there.sum()), "truth_boundary": truth, "recalled": hit}


def _exact_flow(case, seed):
    """The two-frame polynomial-expansion flow (Farneback 2003) in 64 bits:
    5 levels, 5x5 window of sigma 1.1, 13x13 averages, 10 iterations."""
    if case["W"] * case["H"] * case["D"] > 8e6:
        return None
    dev, f8 = "cuda", torch.float64
    rgb = torch.from_numpy(_video(case["W"], case["H"], case["D"], seed)[0]).to(dev).flip(1).long()
    rgb = rgb[..., [2, 1, 0]].permute(0, 3, 1, 2)                       # the BGR frames, then blur, swap and flip back
    fr = torch.nn.functional.pad(rgb.to(f8), (1, 1, 1, 1), mode="reflect").long()
    H, W = case["H"], case["W"]
    acc = sum((2 - abs(j)) * (2 - abs(i)) * fr[:, :, 1 + j:1 + j + H, 1 + i:1 + i + W] for j in (-1, 0, 1) for i in (-1, 0, 1))
    b, g, r = ((acc + 8) >> 4).flip(2).unbind(1)
    img = ((r * 4899 + g * 9617 + b * 1868 + 8192) >> 14).to(f8)

    def at(n, o, step=1, m=None):
        return (torch.arange(m or n, device=dev) * step + o).clamp(0, n - 1)

    imgs = [img]
    while len(imgs) < 5:
        a = imgs[-1]
        h, w = (a.shape[1] + 1) // 2, (a.shape[2] + 1) // 2
        if h < 16 or w < 16:
            break
        k5 = (1, 4, 6, 4, 1)
        a = sum(k5[o + 2] * a[:, :, at(a.shape[2], o, 2, w)] for o in range(-2, 3))
        imgs.append(sum(k5[o + 2] * a[:, at(a.shape[1], o, 2, h)] for o in range(-2, 3)) / 256.0)
    u = np.arange(-2, 3)
    gs = np.exp(-(u * u) / (2 * 1.1 ** 2))
    vv, uu = np.meshgrid(u, u, indexing="ij")
    B = np.stack([np.ones(25), uu.ravel(), vv.ravel(), uu.ravel() ** 2, vv.ravel() ** 2, (uu * vv).ravel()])
    wgt = np.outer(gs, gs).ravel()
    fit = np.linalg.inv((B * wgt) @ B.T) @ (B * wgt)                    # 6 x 25
    D = case["D"]
    src = torch.tensor(list(range(D - 1)) + list(range(1, D)), device=dev)
    dst = torch.tensor(list(range(1, D)) + list(range(D - 1)), device=dev)
    flow = None
    for a in reversed(imgs):
        h, w = a.shape[1:]
        poly = [torch.zeros_like(a) for _ in range(5)]
        for t in range(25):
            tap = a[:, at(h, int(vv.ravel()[t]))][:, :, at(w, int(uu.ravel()[t]))]
            for q in range(5):
                poly[q] += float(fit[q + 1, t]) * (0.5 if q == 4 else 1.0) * tap
        poly = torch.stack(poly, 1)                                     # [D, 5, h, w]: b1 b2 a11 a22 a12
        yy = torch.arange(h, device=dev, dtype=f8)[:, None]
        xx = torch.arange(w, device=dev, dtype=f8)[None, :]
        if flow is None:
            flow = torch.zeros(len(src), 2, h, w, device=dev, dtype=f8)
        else:
            hc, wc = flow.shape[2:]
            sx, sy = wc / w, hc / h
            cx, cy = ((xx + 0.5) * sx - 0.5).clamp(0, wc - 1), ((yy + 0.5) * sy - 0.5).clamp(0, hc - 1)
            x0, y0 = cx.long()[0], cy.long()[:, 0]
            x1, y1 = (x0 + 1).clamp(max=wc - 1), (y0 + 1).clamp(max=hc - 1)
            fx, fy = cx - x0, cy - y0[:, None]
            top = flow[:, :, y0]
            bot = flow[:, :, y1]
            flow = (1 - fy) * ((1 - fx) * top[..., x0] + fx * top[..., x1]) + fy * ((1 - fx) * bot[..., x0] + fx * bot[..., x1])
            flow[:, 0] /= sx
            flow[:, 1] /= sy
        for p0 in range(0, len(src), 8):                                # a few pairs at a time
            fl, ps, pd = flow[p0:p0 + 8], poly[src[p0:p0 + 8]], poly[dst[p0:p0 + 8]].flatten(2)
            for _ in range(10):
                dx, dy = fl[:, 0], fl[:, 1]
                qx, qy = xx + dx, yy + dy
                ok = (qx >= 0) & (qy >= 0) & (qx <= w - 1) & (qy <= h - 1)
                x0, y0 = qx.long().clamp(0, w - 2), qy.long().clamp(0, h - 2)
                fx, fy = qx - x0, qy - y0
                samp = 0.0
                for oy, wy in ((0, 1 - fy), (1, fy)):
                    for ox, wx in ((0, 1 - fx), (1, fx)):
                        idx = ((y0 + oy) * w + x0 + ox).flatten(1)[:, None].expand(-1, 5, -1)
                        samp = samp + (wy * wx)[:, None] * pd.gather(2, idx).view_as(ps)
                a11, a22, a12 = (0.5 * (ps[:, q] + samp[:, q]) for q in (2, 3, 4))
                d1 = -0.5 * (samp[:, 0] - ps[:, 0]) + a11 * dx + a12 * dy
                d2 = -0.5 * (samp[:, 1] - ps[:, 1]) + a12 * dx + a22 * dy
                m = torch.stack([a11 * a11 + a12 * a12, a11 * a12 + a12 * a22, a12 * a12 + a22 * a22,
                                 a11 * d1 + a12 * d2, a12 * d1 + a22 * d2], 1) * ok[:, None]
                m = torch.nn.functional.avg_pool2d(m, (1, 13), 1, (0, 6), divisor_override=1)
                m = torch.nn.functional.avg_pool2d(m, (13, 1), 1, (6, 0), divisor_override=1)
                g11, g12, g22, h1, h2 = m.unbind(1)
                det = g11 * g22 - g12 * g12 + 1e-3
                fl = torch.stack([(g22 * h1 - g12 * h2) / det, (g11 * h2 - g12 * h1) / det], 1)
            flow[p0:p0 + 8] = fl
    fwd = torch.zeros(D, H, W, 2, device=dev, dtype=f8)
    bwd = torch.zeros_like(fwd)
    fwd[:-1] = flow[:D - 1].permute(0, 2, 3, 1)
    bwd[1:] = flow[D - 1:].permute(0, 2, 3, 1)
    return fwd, bwd
