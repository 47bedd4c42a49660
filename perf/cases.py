"""The performance cases: what programs have this library do, at the sizes they
do it.

listed() are the fixed cases, draw() makes more of the same ranges, prepare()
makes what a program holds before the call (images on the GPU, configured
handles, output buffers), run() is one pass through the public Python
interface, work() the bytes and operations that the pass cannot do without,
and exact() the floating-point outputs in 64 bits by plain torch.

Inputs are seeded stereo pairs of the library's generator (fractal texture
with rectangles, slanted planes, or smooth surfaces, and sensor noise).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "module.clutec.cuda_b200"))

import ctstereo as ct  # noqa: E402

BATCH_SIZES = [(320, 240), (640, 480), (1280, 720), (1920, 1080)]
BATCH_DISPS = [32, 64, 128, 256]
NCC, BM1, SAD1, AW1 = ct.CT_COMPAT_NCC, ct.CT_COMPAT_BM1, ct.CT_COMPAT_SAD1, ct.CT_COMPAT_AW1


def listed():
    return [
        # a thumbnail or region of interest: the call's latency and its launches
        {"name": "census_roi", "path": "census", "width": 160, "height": 96, "disps": 64, "disp_min": 0,
         "u16": False, "maps": "checked", "kind": 1},
        # one frame of a depth camera taken to 3D: checked map, its mip-maps and
        # points; odd size, odd disparity count and minimum
        {"name": "frame_to_3d", "path": "frame3d", "width": 801, "height": 603, "disps": 97, "disp_min": 3, "kind": 2},
        # the ordinary frame: Full HD, both directions and the left-right check
        {"name": "census_1080", "path": "census", "width": 1920, "height": 1080, "disps": 128, "disp_min": 0,
         "u16": False, "maps": "checked", "kind": 2},
        # a camera's frames from host memory to host maps
        {"name": "stream_1080", "path": "stream", "width": 1920, "height": 1080, "disps": 128, "frames": 8, "kind": 2},
        # an offline job: pairs of mixed sizes and ranges in one call
        {"name": "batch_mixed", "path": "batch", "pairs": 32, "graph": False, "shapes": 4, "kind": 1},
        # a small SAD matcher
        {"name": "sad_640", "path": "sad", "width": 640, "height": 480, "disps": 64, "radius": 4, "kind": 1},
        # normalised cross-correlation with its scores at Full HD
        {"name": "ncc_1080", "path": "ncc", "width": 1920, "height": 1080, "disps": 128, "radius": 5, "kind": 2},
        # coarse to fine: census at a quarter of the size guides the correlation
        {"name": "ncc_guided_1080", "path": "ncc_guided", "width": 1920, "height": 1080, "disps": 128, "radius": 5,
         "kind": 2},
        # the largest: adaptive windows and sub-pixel disparities
        {"name": "aw_1440", "path": "aw", "width": 2560, "height": 1440, "disps": 256, "kind": 3},
        # the learned check: cost curves and the confidence net's inference
        {"name": "learned_1080", "path": "learned", "width": 1920, "height": 1080, "u16": False, "kind": 1},
        # one gradient of the confidence net's training
        {"name": "net_gradient", "path": "gradient", "samples": 8192},
        # the reference drivers' 4 x uint16 pixels with gates and thresholds
        {"name": "compat_ncc_1080", "path": "compat", "width": 1920, "height": 1080, "disps": 128, "method": NCC,
         "patch": 11, "grad": 2.0, "score": 0.6, "delta": 3.0, "kind": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["census", "census", "census", "frame3d", "stream", "batch", "sad", "ncc", "ncc_guided", "aw",
                       "learned", "gradient", "compat"])
    w = _log(rng, 96, 1920)
    h = max(48, min(1200, int(w * rng.uniform(0.5, 0.8))))
    d = min(_log(rng, 16, 256), max(16, w // 2))
    kind = rng.choice([1, 2, 3])
    size = {"width": w, "height": h, "disps": d}
    if path == "census":
        u16 = rng.random() < 0.5
        return {"path": path, "width": w, "height": h, "disps": d if u16 else min(d, 240),
                "disp_min": rng.choice([0, 0, 1, 6, 11]), "u16": u16, "maps": rng.choice(["checked", "all", "left"]),
                "kind": kind}
    if path == "frame3d":
        return {"path": path, **size, "disp_min": rng.choice([0, 1, 6]), "kind": kind}
    if path == "stream":
        return {"path": path, "width": w, "height": h, "disps": min(d, 240), "frames": rng.randint(1, 12), "kind": kind}
    if path == "batch":
        return {"path": path, "pairs": _log(rng, 1, 32), "graph": rng.random() < 0.5, "shapes": rng.randint(5, 1000),
                "kind": rng.choice([1, 2])}
    if path == "sad":
        return {"path": path, "width": w, "height": h, "disps": min(d, 240), "radius": rng.randint(1, 4), "kind": kind}
    if path == "ncc":
        return {"path": path, **size, "radius": rng.choice([2, 4, 5, 5]), "kind": kind}
    if path == "ncc_guided":
        s = 4
        return {"path": path, "width": max(160, w // s * s), "height": max(96, h // s * s), "disps": max(32, d // s * s),
                "radius": rng.choice([2, 4, 5, 5]), "kind": kind}
    if path == "aw":
        return {"path": path, **size, "kind": kind}
    if path == "learned":
        return {"path": path, "width": max(w, 200), "height": h, "u16": rng.random() < 0.5, "kind": rng.choice([1, 2])}
    if path == "gradient":
        return {"path": path, "samples": _log(rng, 100, 16384)}
    method = rng.choice([NCC, NCC, BM1, SAD1, AW1])
    patch = {NCC: [5, 9, 11], BM1: [5, 9, 11, 15], SAD1: [5, 9, 16], AW1: [3, 5]}[method]
    return {"path": path, "width": min(w, 1280), "height": min(h, 800), "disps": min(d, 128), "method": method,
            "patch": rng.choice(patch), "grad": rng.choice([0.0, 2.0]), "score": rng.choice([0.0, 0.6]),
            "delta": rng.choice([0.0, 3.0]), "kind": kind}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _pair(case, seed, dmax):
    """Host images of a seeded pair (numpy uint8)."""
    left, right, _, _ = ct.synth_pair(case["kind"], seed & 0x7FFFFFFF, case["width"], case["height"], max(1, dmax))
    return left, right


def _up(a):
    t = ct.alloc_image(a.shape[0], a.shape[1], torch.uint8)
    t.copy_(torch.from_numpy(a))
    return t


def _down4(img):
    h, w = img.shape
    return np.round(img.reshape(h // 4, 4, w // 4, 4).mean(axis=(1, 3))).astype(np.uint8)


def _batch_shapes(case):
    r = np.random.default_rng(case["shapes"])
    return [(*BATCH_SIZES[int(r.integers(4))], BATCH_DISPS[int(r.integers(4))]) for _ in range(case["pairs"])]


def _weights():
    p = os.path.join(os.getcwd(), "module.clutec.cuda_b200", "confnet_census128.f32")
    return np.fromfile(p, dtype="<f4")


def _cams(case):
    w, h = case["width"], case["height"]
    return (0.73 * w, 0.73 * w, w / 2, h / 2), 0.12  # (fx, fy, cx, cy), baseline


def _samples(case, seed):
    """Re-centred cost curves and labels of a training batch: a minimum at the
    centre, rising costs beside it, 255 where the match leaves the image."""
    g = np.random.default_rng(seed)
    n = case["samples"]
    slope = g.uniform(1.0, 12.0, (n, 1))
    base = g.uniform(5.0, 70.0, (n, 1))
    x = base + slope * np.abs(np.arange(128)[None, :] - 64.0) + g.normal(0.0, 6.0, (n, 128))
    x = np.clip(x, 0, 196).astype(np.uint8)
    x[np.arange(128)[None, :] >= g.integers(68, 260, (n, 1))] = 255
    y = (slope[:, 0] / (1.0 + base[:, 0] / 20.0) + g.normal(0.0, 0.6, n) > 2.0).astype(np.uint8)
    return x, y


def prepare(case, seed):
    path = case["path"]
    s = {"case": case}
    if path == "gradient":
        x, y = _samples(case, seed)
        s["x"], s["y"] = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
        s["net"] = net = ct.ConfNet()
        net.configure(0, case["samples"])
        net.set_params(_weights())
        s["grad"] = torch.empty(ct.CT_CONFNET_PARAMS, dtype=torch.float32, device="cuda")
        s["loss"] = torch.empty(1, dtype=torch.float32, device="cuda")
        return s
    if path == "batch":
        shapes = _batch_shapes(case)
        s["pairs"] = []
        for i, (w, h, d) in enumerate(shapes):
            left, right = _pair({"kind": case["kind"], "width": w, "height": h}, seed * 1009 + i, d - 1)
            s["pairs"].append((_up(left), _up(right), ct.alloc_image(h, w, torch.int16)))
        s["m"] = m = ct.BatchStereo()
        m.configure(0, shapes, tol=1)
        if case["graph"]:
            m.graph_create(s["pairs"])
        return s
    w, h, d = case["width"], case["height"], case.get("disps", 128)
    if path == "stream":
        s["m"] = m = ct.CensusStream()
        m.configure(0, w, h, d, tol=1)
        s["frames"] = []
        for i in range(case["frames"]):
            if i < 2:  # a camera's two alternating scenes, each frame in a buffer of its own
                scene = _pair(case, seed * 1009 + i, d - 1)
                s.setdefault("scenes", []).append(scene)
            left, right = s["scenes"][i % len(s["scenes"])]
            s["frames"].append((torch.from_numpy(left).clone().pin_memory(), torch.from_numpy(right).clone().pin_memory(),
                                torch.empty((h, w), dtype=torch.uint8).pin_memory()))
        return s
    left, right = _pair(case, seed, case.get("disp_min", 0) + d - 1)
    s["left"], s["right"] = _up(left), _up(right)
    u8, i16, f32 = torch.uint8, torch.int16, torch.float32
    if path == "census":
        s["m"] = m = ct.BlockMatcherCensus()
        m.configure(0, w, h, d, disp_min=case["disp_min"])
        n = 3 if case["maps"] == "all" else 1
        s["out"] = [ct.alloc_image(h, w, i16 if case["u16"] else u8) for _ in range(n)]
    elif path == "frame3d":
        s["m"] = m = ct.BlockMatcherCensus()
        m.configure(0, w, h, d, disp_min=case["disp_min"])
        s["out"] = [ct.alloc_image(h, w, i16) for _ in range(3)]
        pw, _ = ct.disp_mipmap_format(w, h)
        s["mip"] = ct.alloc_image(h, pw, f32)
        s["mip"].zero_()
        (fx, fy, cx, cy), b = _cams(case)
        s["to3d"] = ct.MapDisparityTo3D()
        s["to3d"].configure(0, w, h, ct.pinhole(fx, fy, cx, cy), ct.pinhole(fx, fy, cx, cy, center=(b, 0.0, 0.0)))
        s["points"] = ct.alloc_map3d(h, w)
    elif path == "sad":
        s["m"] = m = ct.BlockMatcherSAD1()
        m.configure(0, w, h, d, radius=case["radius"])
        s["out"] = ct.alloc_image(h, w, u8)
    elif path in ("ncc", "ncc_guided"):
        s["m"] = m = ct.BlockMatcherNCC()
        m.configure(0, w, h, d, radius=case["radius"])
        s["out"], s["score"] = ct.alloc_image(h, w, i16), ct.alloc_image(h, w, f32)
        if path == "ncc_guided":
            s["left4"], s["right4"] = _up(_down4(left)), _up(_down4(right))
            s["coarse_m"] = c = ct.BlockMatcherCensus()
            c.configure(0, w // 4, h // 4, d // 4)
            s["coarse"] = ct.alloc_image(h // 4, w // 4, u8)
    elif path == "aw":
        s["m"] = m = ct.BlockMatcherAW()
        m.configure(0, w, h, d)
        s["out"] = ct.alloc_image(h, w, f32)
    elif path == "learned":
        s["m"] = m = ct.BlockMatcherCensus()
        m.configure(0, w, h, d)
        s["curves"] = ct.CurveVolume(w, h, d)
        dt = i16 if case["u16"] else u8
        s["out"], s["checked"] = ct.alloc_image(h, w, dt), ct.alloc_image(h, w, dt)
        s["net"] = ct.ConfNet()
        s["net"].configure(0, 16)
        s["net"].set_params(_weights())
    else:
        s["m"] = m = ct.BlockMatcherCompat()
        m.configure(0, w, h, case["method"], d, case["patch"], grad_thresh=case["grad"], score_thresh=case["score"],
                    min_delta_thresh=case["delta"])
        s["out"] = ct.alloc_u16x4(h, w)
    return s


def run(s):
    case = s["case"]
    path = case["path"]
    if path == "census":
        if case["maps"] == "checked":
            s["m"].process_lr(s["left"], s["right"], disp_checked=s["out"][0], tol=1)
        elif case["maps"] == "all":
            s["m"].process_lr(s["left"], s["right"], *s["out"], tol=1)
        else:
            s["m"].process(s["out"][0], s["left"], s["right"])
        return list(s["out"])
    if path == "frame3d":
        s["m"].process_lr(s["left"], s["right"], *s["out"], tol=1)
        ct.disp_mipmaps(s["mip"], s["out"][2])
        s["to3d"].process(s["points"], s["out"][2])
        return {"maps": list(s["out"]), "mip": s["mip"], "points": s["points"]}
    if path == "stream":
        for left, right, out in s["frames"]:
            k = s["m"].submit(left, right, out)
        s["m"].wait(k)
        return [f[2] for f in s["frames"]]
    if path == "batch":
        if case["graph"]:
            s["m"].graph_launch()
        else:
            s["m"].process(s["pairs"])
        return [p[2] for p in s["pairs"]]
    if path == "sad":
        s["m"].process(s["out"], s["left"], s["right"])
        return s["out"]
    if path == "ncc":
        s["m"].process(s["out"], s["left"], s["right"], score=s["score"])
        return {"disp": s["out"], "score": s["score"]}
    if path == "ncc_guided":
        s["coarse_m"].process_lr(s["left4"], s["right4"], disp_checked=s["coarse"], tol=1)
        s["m"].process(s["out"], s["left"], s["right"], score=s["score"], disp_init=s["coarse"])
        return {"coarse": s["coarse"], "disp": s["out"], "score": s["score"]}
    if path == "aw":
        s["m"].process(s["out"], s["left"], s["right"])
        return s["out"]
    if path == "learned":
        s["m"].process_curves(s["out"], s["curves"], s["left"], s["right"])
        s["net"].infer(None, s["curves"], s["out"], checked=s["checked"], threshold=0.5)
        return {"disp": s["out"], "checked": s["checked"]}
    if path == "gradient":
        s["net"].loss_grad(s["x"], s["y"], s["grad"], s["loss"])
        return {"grad": s["grad"], "loss": s["loss"]}
    s["m"].process(s["out"], s["left"], s["right"])
    return s["out"]


# ---------------------------------------------------------------------------
# work: inputs read once, outputs written once; operations per pixel and
# disparity of the cost, its running window sums and the selection
# ---------------------------------------------------------------------------

CENSUS_OPS = 9  # two 64-bit halves' xor and popcount (4), box sums (4), selection (1)


def work(case):
    path = case["path"]
    if path == "gradient":
        n = case["samples"]
        macs = 7 * 5 * 32 + 2 * 5 * 32 * 32 + 2 * 32 * 32 + 32 * 64 + 64
        return {"bytes": n * 36 + 8 * 12673, "flops": 3 * 2 * macs * n}
    if path == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(4 * w * h for w, h, _ in shapes), "flops": sum((CENSUS_OPS + 1) * w * h * d + 126 * w * h
                                                                            for w, h, d in shapes)}
    px, d = case["width"] * case["height"], case.get("disps", 128)
    if path == "census":
        maps = 3 if case["maps"] == "all" else 1
        return {"bytes": px * (2 + maps * (2 if case["u16"] else 1)),
                "flops": px * (126 + (CENSUS_OPS + (case["maps"] != "left")) * d)}
    if path == "frame3d":
        return {"bytes": px * (2 + 6 + 16 + 16 / 3), "flops": px * (126 + (CENSUS_OPS + 1) * d + 60)}
    if path == "stream":
        return {"bytes": 3 * px * case["frames"], "flops": px * (126 + (CENSUS_OPS + 1) * d) * case["frames"]}
    if path == "sad":
        return {"bytes": 3 * px, "flops": 8 * px * d}
    if path == "ncc":
        return {"bytes": 8 * px, "flops": 15 * px * d}
    if path == "ncc_guided":
        return {"bytes": 8 * px + 3 * px // 16, "flops": px // 16 * (126 + (CENSUS_OPS + 1) * d // 4) + 15 * px * 16}
    if path == "aw":
        return {"bytes": 6 * px, "flops": 13 * px * d}
    if path == "learned":
        out = 2 * (2 if case["u16"] else 1)
        macs = 7 * 5 * 32 + 2 * 5 * 32 * 32 + 2 * 32 * 32 + 32 * 64 + 64
        return {"bytes": px * (2 + out), "flops": px * (126 + CENSUS_OPS * d + 2 * macs)}
    return {"bytes": 10 * px, "flops": 30 * px * d}


# ---------------------------------------------------------------------------
# exact: floating-point outputs in 64 bits by plain torch
# ---------------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _census(img):
    """9 x 7 census descriptors (int64), 0 near the border."""
    h, w = img.shape
    c = img.to(torch.int16)
    out = torch.zeros((h, w), dtype=torch.int64, device=img.device)
    if h < 7 or w < 9:
        return out
    mid = c[3:h - 3, 4:w - 4]
    bits = torch.zeros(mid.shape, dtype=torch.int64, device=img.device)
    for dy in range(7):
        for dx in range(9):
            bits = bits * 2 + (c[dy:dy + h - 6, dx:dx + w - 8] > mid).to(torch.int64)
    out[3:h - 3, 4:w - 4] = bits
    return out


def _shift(a, d, fill):
    """b[:, x] = a[:, x - d], `fill` outside."""
    b = torch.full_like(a, fill)
    w = a.shape[1]
    if d < w and d > -w:
        b[:, max(0, d):w + min(0, d)] = a[:, max(0, -d):w - max(0, d)]
    return b


def _box(a, r):
    """Centred (2r + 1)^2 box sums; 0 within r of the border."""
    h, w = a.shape
    out = torch.zeros_like(a)
    if h <= 2 * r or w <= 2 * r:
        return out
    v = a[0:h - 2 * r].clone()
    for k in range(1, 2 * r + 1):
        v += a[k:h - 2 * r + k]
    s = v[:, 0:w - 2 * r].clone()
    for k in range(1, 2 * r + 1):
        s += v[:, k:w - 2 * r + k]
    out[r:h - r, r:w - r] = s
    return out


def _inside(h, w, r, dev):
    m = torch.zeros((h, w), dtype=torch.bool, device=dev)
    m[r:h - r, r:w - r] = True
    return m


def _census_checked(left, right, disps, disp_min, tol=1):
    """Left-right checked census disparities (int64, -1: none, -2: rejected)."""
    dev = _dev()
    cl, cr = _census(torch.from_numpy(left).to(dev)), _census(torch.from_numpy(right).to(dev))
    h, w = cl.shape
    table = torch.tensor([bin(i).count("1") for i in range(1 << 16)], dtype=torch.int32, device=dev)
    big = 1 << 20
    inside = _inside(h, w, 2, dev)
    best = [torch.full((h, w), big, dtype=torch.int32, device=dev) for _ in range(2)]
    disp = [torch.full((h, w), -1, dtype=torch.int64, device=dev) for _ in range(2)]
    for d in range(disp_min, disp_min + disps):
        if d >= w:
            break
        x = cl ^ _shift(cr, d, 0)
        cost = sum(table[(x >> k) & 0xFFFF] for k in (0, 16, 32, 48))
        cost = _box(cost, 2)
        ok = inside & _shift(inside, d, False)
        cost = torch.where(ok, cost, big)
        for k, c in ((0, cost), (1, _shift(cost, -d, big))):  # the right pixel x - d has the same windows
            better = c < best[k]
            best[k] = torch.where(better, c, best[k])
            disp[k] = torch.where(better, d, disp[k])
    lr, rl = disp
    xo = torch.arange(w, device=dev)[None, :] - lr
    other = torch.gather(rl, 1, xo.clamp(0, w - 1))
    keep = (lr >= 0) & (xo >= 0) & (other >= 0) & ((other - lr).abs() <= tol)
    return torch.where(lr < 0, -1, torch.where(keep, lr, -2))


def _mipmaps(codes):
    """Packed mip-map image of a disparity code map (float64)."""
    h, w = codes.shape
    half = lambda n: (n - 1) // 2 if n >= 1 else 0  # noqa: E731
    x1 = -(-w // 4) * 4
    out = torch.zeros((h, x1 + half(w)), dtype=torch.float64, device=codes.device)

    def mean121(a, b, c):
        n = (a != 0).double() + 2 * (b != 0).double() + (c != 0).double()
        return torch.where(n > 0, (a + 2 * b + c) / n.clamp(min=1), 0.0)

    level = torch.where((codes >= 1) & (codes <= 0xFFEF), codes, 0).double()
    out[:, :w] = level
    dims, lw, lh = [], w, h
    while half(lw) > 0 and half(lh) > 0:
        lw, lh = half(lw), half(lh)
        dims.append((lw, lh))
    y = 0
    for lw, lh in dims[:-1]:
        t = mean121(level[:, 0:2 * lw:2], level[:, 1:2 * lw + 1:2], level[:, 2:2 * lw + 2:2])
        level = 0.5 * mean121(t[0:2 * lh:2], t[1:2 * lh + 1:2], t[2:2 * lh + 2:2])
        out[y:y + lh, x1:x1 + lw] = level
        y += lh
    return out


def _points(codes, case):
    """Rectified triangulation of a code map (float64): (x, y, z, valid)."""
    (fx, fy, cx, cy), b = _cams(case)
    h, w = codes.shape
    valid = (codes >= 1) & (codes <= 0xFFEF)
    d = torch.where(valid, codes - 1, 1).double()
    yy, xx = torch.meshgrid(torch.arange(h, device=codes.device).double(), torch.arange(w, device=codes.device).double(),
                            indexing="ij")
    hit = d != 0
    z = torch.where(hit, fx * b / torch.where(hit, d, 1.0), 0.0)
    return torch.stack([(xx - cx) / fx * z, (yy - cy) / fy * z, z, (hit & valid).double()], -1)


def _ncc_score(left, right, disps, r, lo=None, hi=None):
    """Largest NCC score over the searched disparities (float64)."""
    dev = _dev()
    a, b = torch.from_numpy(left).to(dev).double(), torch.from_numpy(right).to(dev).double()
    h, w = a.shape
    n = float((2 * r + 1) ** 2)
    sa, sb = _box(a, r), _box(b, r)
    va, vb = n * _box(a * a, r) - sa * sa, n * _box(b * b, r) - sb * sb
    inside = _inside(h, w, r, dev)
    best = torch.full((h, w), -2.0, dtype=torch.float64, device=dev)
    for d in range(min(disps, w)):
        num = n * _box(a * _shift(b, d, 0.0), r) - sa * _shift(sb, d, 0.0)
        vv = va * _shift(vb, d, 0.0)
        s = torch.where(vv < n ** 4, 0.0, num / vv.clamp(min=1.0).sqrt())
        ok = inside & _shift(inside, d, False)
        if lo is not None:
            ok = ok & (lo <= d) & (hi >= d)
        best = torch.where(ok, torch.maximum(best, s), best)
    return torch.where(best > -2.0, best, 0.0)  # no disparity: 0


def _guide(coarse, h, w, s=4, block=16, margin=4):
    """Search ranges per pixel from a coarse disparity map (-1: none)."""
    ys, xs = torch.arange(h, device=coarse.device) // s, torch.arange(w, device=coarse.device) // s
    up = coarse[ys][:, xs]
    up = torch.where(up >= 0, up * s, -1)
    gh, gw = -(-h // block), -(-w // block)
    pad = torch.full((gh * block, gw * block), -1, dtype=up.dtype, device=up.device)
    pad[:h, :w] = up
    t = pad.reshape(gh, block, gw, block).permute(0, 2, 1, 3).reshape(gh, gw, -1)
    hi = t.amax(-1)
    lo = torch.where(t < 0, 1 << 20, t).amin(-1)
    lo, hi = torch.where(hi < 0, 1 << 20, (lo - margin).clamp(min=0)), torch.where(hi < 0, -1, hi + margin)
    grow = lambda v: v.repeat_interleave(block, 0).repeat_interleave(block, 1)[:h, :w]  # noqa: E731
    return grow(lo), grow(hi)


def _aw_subpixel(left, right, disps):
    """Adaptive-window disparities with the parabolic sub-pixel step (float64)."""
    dev = _dev()
    a, b = torch.from_numpy(left).to(dev).int(), torch.from_numpy(right).to(dev).int()
    h, w = a.shape
    r, sh = 3, 3
    ext = r + sh
    none = 1 << 28
    inside = _inside(h, w, ext, dev)
    best = torch.full((h, w), none, dtype=torch.int32, device=dev)
    disp = torch.full((h, w), -1, dtype=torch.int32, device=dev)
    before, after, prev = best.clone(), best.clone(), best.clone()
    for d in range(min(disps, w)):
        s = _box((a - _shift(b, d, 0)).abs(), r)
        c = s.clone()
        c[:, sh:] = torch.minimum(c[:, sh:], s[:, :-sh])
        c[:, :-sh] = torch.minimum(c[:, :-sh], s[:, sh:])
        c[sh:] = torch.minimum(c[sh:], s[:-sh])
        c[:-sh] = torch.minimum(c[:-sh], s[sh:])
        c = torch.where(inside & _shift(inside, d, False), c, none)
        after = torch.where(disp == d - 1, c, after) if d else after
        better = c < best
        before = torch.where(better, prev, before)
        after = torch.where(better, none, after)
        best = torch.where(better, c, best)
        disp = torch.where(better, d, disp)
        prev = c
    den = (before.long() - 2 * best.long() + after.long()).double()
    fit = (disp > 0) & (disp < disps - 1) & (before < none) & (after < none) & (den > 0)
    off = torch.where(fit, (before - after).double() / (2.0 * torch.where(fit, den, 1.0)), 0.0)
    return torch.where(disp < 0, -1.0, disp.double() + off)


def _net_gradient(x, y, flat):
    """Loss and gradient of the confidence net in float64, no roundings."""
    dev = _dev()
    p = torch.from_numpy(flat).to(dev).double().requires_grad_()
    take, at = {}, 0
    for name, shape in (("w1", (32, 1, 5)), ("b1", (32,)), ("w2", (32, 32, 5)), ("b2", (32,)), ("w3", (32, 32, 5)),
                        ("b3", (32,)), ("w4", (64, 32)), ("b4", (64,)), ("w5", (1, 64)), ("b5", (1,))):
        k = math.prod(shape)
        take[name] = p[at:at + k].view(shape)
        at += k
    F = torch.nn.functional
    v = torch.from_numpy(x).to(dev).double()[:, None, 52:87]
    v = F.relu(F.conv1d(v, take["w1"], take["b1"], stride=5))
    v = F.relu(F.conv1d(v, take["w2"], take["b2"], stride=3, padding=1))
    v = F.relu(F.conv1d(v, take["w3"], take["b3"], padding=2)[:, :, 0])
    v = F.relu(F.linear(v, take["w4"], take["b4"]))
    z = F.linear(v, take["w5"], take["b5"])[:, 0]
    loss = F.binary_cross_entropy_with_logits(z, torch.from_numpy(y).to(dev).double())
    loss.backward()
    return {"grad": p.grad, "loss": loss.detach().reshape(1)}


def exact(case, seed):
    path = case["path"]
    if path == "gradient":
        return _net_gradient(*_samples(case, seed), _weights())
    if path not in ("frame3d", "ncc", "ncc_guided", "aw"):
        return None  # integer maps only
    d = case["disps"]
    left, right = _pair(case, seed, case.get("disp_min", 0) + d - 1)
    if path == "frame3d":
        m = _census_checked(left, right, d, case["disp_min"])
        codes = torch.where(m >= 0, m + 1, torch.where(m == -1, 0xFFFF, 0xFFFA))
        return {"maps": [None, None, None], "mip": _mipmaps(codes), "points": _points(codes, case)}
    if path == "ncc":
        return {"disp": None, "score": _ncc_score(left, right, d, case["radius"])}
    if path == "ncc_guided":
        coarse = _census_checked(_down4(left), _down4(right), d // 4, 0)
        lo, hi = _guide(coarse, *left.shape)
        return {"coarse": None, "disp": None, "score": _ncc_score(left, right, d, case["radius"], lo, hi)}
    return _aw_subpixel(left, right, d)
