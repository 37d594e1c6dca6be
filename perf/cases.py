"""Workloads of the stereo engine for timing and comparison, one per way the package is used.

Each case is one call through the public Python API as an application makes it:

* ``plain``          StereoCuda: one single-level match, on device tensors or on host arrays
* ``pyramid``        FasterStereoCuda: one coarse-to-fine match, device tensors or host arrays
* ``batch``          StereoBatch: many pairs of uneven size, one launch, inputs resident
* ``batch_pyramid``  StereoBatchPyramid: many whole pyramids, one launch, inputs resident
* ``float``          float_sgm: the differentiable layer, forward alone or forward + backward

The scenes have the sizes, disparity ranges and textures of the benchmark configurations
(Cone 450x375, KITTI 1242x375, Building 4800x3409, the uneven batch) and are drawn on the GPU
from the seed. A matcher and its buffers are made once per program, so they belong to prepare().
"""
import math
import random

import numpy as np
import torch

import fasterstereocuda_b200 as fsc
from fasterstereocuda_b200.float_sgm import float_sgm

DEVICE = "cuda"
INVALID = -999999.0


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one frame at a time from a camera, images already on the GPU (the Cone size)
        {"name": "plain_cone", "kind": "plain", "width": 450, "height": 375, "min_disp": 0, "disp": 64, "census": 1,
         "p1": 10, "p2": 150, "lr": True, "median": True, "host": False, "scene": "planar"},
        # the reference's own call: host images in, host disparity out (the KITTI size)
        {"name": "plain_kitti_host", "kind": "plain", "width": 1242, "height": 375, "min_disp": 0, "disp": 64,
         "census": 1, "p1": 10, "p2": 150, "lr": True, "median": True, "host": True, "scene": "road"},
        # 5x5 census, the reference's penalties, a range that starts above zero, odd sizes, 128 disparities
        {"name": "plain_128_odd", "kind": "plain", "width": 957, "height": 541, "min_disp": 3, "disp": 128, "census": 0,
         "p1": 8, "p2": 32, "lr": True, "median": True, "host": False, "scene": "planar"},
        # the widest search range, for close objects at video resolution
        {"name": "plain_256", "kind": "plain", "width": 1280, "height": 720, "min_disp": 0, "disp": 256, "census": 1,
         "p1": 10, "p2": 150, "lr": True, "median": True, "host": False, "scene": "planar"},
        # the console's Cone options: one layer, no consistency check, small-region removal, host images
        {"name": "console_cone_host", "kind": "pyramid", "width": 450, "height": 375, "min_disp": 0, "max_disp": 64,
         "layers": 1, "lr": False, "peaks": True, "override": False, "host": True, "scene": "planar"},
        # the headline: three layers at the KITTI size, host images in and disparity out
        {"name": "pyramid_kitti_host", "kind": "pyramid", "width": 1242, "height": 375, "min_disp": 0, "max_disp": 64,
         "layers": 3, "lr": True, "peaks": True, "override": True, "host": True, "scene": "road"},
        # an aerial image (the Building size), four layers, inputs on the GPU
        {"name": "pyramid_building", "kind": "pyramid", "width": 4800, "height": 3409, "min_disp": 0, "max_disp": 256,
         "layers": 4, "lr": True, "peaks": True, "override": True, "host": False, "scene": "fractal"},
        # a server's queue: pairs of many cameras with different sizes and ranges in one launch
        {"name": "batch_uneven", "kind": "batch", "pairs": 32, "width_lo": 320, "width_hi": 1920, "height_lo": 240,
         "height_hi": 1080, "disp_lo": 64, "disp_hi": 128, "sizes": 3, "scene": "planar"},
        # offline processing of recorded drives: 64 whole pyramids in one launch
        {"name": "batch_pyramid_kitti", "kind": "batch_pyramid", "pairs": 64, "width": 1242, "height": 375,
         "min_disp": 0, "max_disp": 64, "layers": 3, "lr": True, "peaks": True, "override": True, "scene": "road"},
        # a training step's SGM layer at full resolution: disparity and the three gradients
        {"name": "float_train", "kind": "float", "batch": 4, "width": 1242, "height": 375, "disp": 64, "grad": True},
        # the same layer on a training crop
        {"name": "float_train_crop", "kind": "float", "batch": 1, "width": 64, "height": 48, "disp": 32, "grad": True},
        # inference with the trained penalties: forward alone, odd sizes, one image
        {"name": "float_infer_odd", "kind": "float", "batch": 1, "width": 641, "height": 479, "disp": 32,
         "grad": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _drawn(rng):
    kind = rng.choice(["plain", "plain", "pyramid", "batch", "batch_pyramid", "float", "float"])
    if kind == "plain":
        d = rng.choice([32, 64, 64, 128, 256])
        census = rng.choice([0, 1])
        p1, p2 = rng.choice([(10, 150), (8, 32), (rng.randint(3, 20), rng.randint(30, 300))])
        return {"kind": kind, "width": _log_int(rng, 450, 1920), "height": _log_int(rng, 240, 1080),
                "min_disp": rng.choice([0, 0, rng.randint(1, 8)]), "disp": d, "census": census, "p1": p1, "p2": p2,
                "lr": rng.random() < 0.8, "median": rng.random() < 0.8, "host": rng.random() < 0.5,
                "scene": rng.choice(["planar", "road"])}
    if kind == "pyramid":
        layers = rng.choice([1, 2, 3, 4])
        return {"kind": kind, "width": _log_int(rng, 450, 4800), "height": _log_int(rng, 375, 3409), "min_disp": 0,
                "max_disp": 64 if layers == 1 else 32 << (layers - 1), "layers": layers, "lr": rng.random() < 0.8,
                "peaks": rng.random() < 0.8, "override": rng.random() < 0.6, "host": rng.random() < 0.5,
                "scene": rng.choice(["planar", "road", "fractal"])}
    if kind == "batch":
        return {"kind": kind, "pairs": _log_int(rng, 2, 32), "width_lo": 320, "width_hi": rng.choice([641, 1242, 1920]),
                "height_lo": 240, "height_hi": rng.choice([375, 1080]), "disp_lo": rng.choice([32, 64]),
                "disp_hi": rng.choice([64, 128]), "sizes": rng.randint(4, 10 ** 6), "scene": "planar"}
    if kind == "batch_pyramid":
        layers = rng.choice([2, 3])
        return {"kind": kind, "pairs": _log_int(rng, 2, 64), "width": _log_int(rng, 450, 1242),
                "height": _log_int(rng, 240, 375), "min_disp": 0, "max_disp": 32 << (layers - 1), "layers": layers,
                "lr": True, "peaks": rng.random() < 0.8, "override": rng.random() < 0.6, "scene": "road"}
    return {"kind": kind, "batch": _log_int(rng, 1, 8), "width": _log_int(rng, 64, 1242),
            "height": _log_int(rng, 48, 375), "disp": rng.choice([32, 64]), "grad": rng.random() < 0.7}


def draw(rng):
    most = {}
    for c in listed():
        most[c["kind"]] = max(most.get(c["kind"], 0), work(c)["flops"])
    most["plain"] = most["pyramid"]  # a large plain image costs what the aerial pyramid does
    while True:
        c = _drawn(rng)
        if work(c)["flops"] <= most[c["kind"]]:
            return c


def _batch_specs(case):
    """(width, height, min_disp, disp) of every pair: sizes a multiple of 32 or odd, two ranges."""
    r = random.Random(case["sizes"])
    out = []
    for i in range(case["pairs"]):
        w, h = r.randint(case["width_lo"], case["width_hi"]), r.randint(case["height_lo"], case["height_hi"])
        if i % 4:
            w, h = max(w // 32 * 32, 320), max(h // 32 * 32, 240)
        out.append((w, h, 0, r.choice([case["disp_lo"], case["disp_hi"]])))
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _match_ops(w, h, d, views):
    # per voxel and view: 2 for the cost (xor, count), 4 paths x 7 (two candidate sums, three minima,
    # cost, normalisation), 4 for the sum and the winner; per pixel 62 census compares of both images
    # at two operations each
    return views * 34.0 * w * h * d + 248.0 * w * h


def work(case):
    kind = case["kind"]
    if kind == "plain":
        px = case["width"] * case["height"]
        return {"bytes": 2.0 * px + 4.0 * px,
                "flops": _match_ops(case["width"], case["height"], case["disp"], 2 if case["lr"] else 1)}
    if kind in ("pyramid", "batch_pyramid"):
        n = case.get("pairs", 1)
        px = case["width"] * case["height"]
        ops = 0.0
        for k in range(case["layers"]):
            d = 32 if case["layers"] > 1 else case["max_disp"]
            ops += _match_ops(case["width"] >> k, case["height"] >> k, d, 2 if case["lr"] else 1)
        return {"bytes": 6.0 * px * n, "flops": ops * n}
    if kind == "batch":
        specs = _batch_specs(case)
        return {"bytes": sum(6.0 * w * h for w, h, _, _ in specs),
                "flops": sum(_match_ops(w, h, d, 2) for w, h, _, d in specs)}
    px = float(case["batch"] * case["width"] * case["height"])
    vox = px * case["disp"]
    if case["grad"]:  # the cost in, its gradient out; penalties, disparity and upstream gradient are maps
        return {"bytes": 4.0 * (2 * vox + 6 * px), "flops": vox * (4 * 7 + 10 + 4 * 8 + 8)}
    return {"bytes": 4.0 * (vox + 3 * px), "flops": vox * (4 * 7 + 10)}


# ---------------------------------------------------------------------------------------------
# seeded scenes
# ---------------------------------------------------------------------------------------------
def _blur(img, sigma):
    r = int(3 * sigma + 0.5)
    k = torch.exp(-0.5 * (torch.arange(-r, r + 1, device=img.device, dtype=torch.float32) / sigma) ** 2)
    k = k / k.sum()
    x = torch.nn.functional.pad(img[None, None], (r, r, r, r), mode="replicate")
    x = (x.unfold(3, 2 * r + 1, 1) * k).sum(-1)
    return (x.unfold(2, 2 * r + 1, 1) * k).sum(-1)[0, 0]


def _noise(g, h, w):
    return torch.rand(h, w, generator=g, device=DEVICE)


def _stretch(t):
    return (t - t.min()) / (t.max() - t.min()).clamp_min(1e-6) * 255.0


def _texture(scene, g, r, h, w):
    if scene == "fractal":  # five octaves of smooth noise
        t = torch.zeros(h, w, device=DEVICE)
        for o in range(5):
            n = _noise(g, max(h >> o, 2) + 1, max(w >> o, 2) + 1)[None, None]
            t += torch.nn.functional.interpolate(n, size=(h, w), mode="bilinear", align_corners=True)[0, 0] * 2.0 ** (o - 4)
        return _stretch(t)
    t = _stretch(_blur(_noise(g, h, w), 1.5))
    if scene == "road":  # a fifth of the image nearly flat
        flat = 0
        while flat < 0.2 * h * w:
            pw, ph = r.randint(max(w // 40, 1), max(w // 8, 2)), r.randint(max(h // 40, 1), max(h // 8, 2))
            x, y = r.randrange(max(w - pw, 1)), r.randrange(max(h - ph, 1))
            t[y:y + ph, x:x + pw] = t[y:y + ph, x:x + pw] * 0.06 + 115.0
            flat += pw * ph
    else:  # six patches with a brightness gradient
        for _ in range(6):
            pw, ph = r.randint(w // 10 + 1, w // 3 + 1), r.randint(h // 10 + 1, h // 3 + 1)
            x, y = r.randrange(max(w - pw, 1)), r.randrange(max(h - ph, 1))
            part = t[y:y + ph, x:x + pw]
            ramp = (r.uniform(40, 215) + r.uniform(-2, 2) * torch.arange(part.shape[1], device=DEVICE)[None, :]
                    + r.uniform(-2, 2) * torch.arange(part.shape[0], device=DEVICE)[:, None])
            t[y:y + ph, x:x + pw] = 0.5 * part + 0.5 * ramp
    return t


def _true_disparity(scene, r, h, w, lo, hi):
    yy = torch.arange(h, device=DEVICE, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=DEVICE, dtype=torch.float32)[None, :]
    span = hi - lo
    if scene == "road":  # ground plane rising to the bottom rows, twelve boxes
        d = (lo + 0.86 * span * yy / max(h - 1, 1)).expand(h, w).clone()
        for _ in range(12):
            bw, bh = r.randint(w // 30 + 1, w // 8 + 1), r.randint(h // 12 + 1, h // 3 + 1)
            x, y = r.randrange(max(w - bw, 1)), r.randrange(max(h - bh, 1))
            d[y:y + bh, x:x + bw] = d[y:y + bh, x:x + bw].clamp_min(lo + span * r.uniform(0.08, 0.8))
        return d
    best = torch.full((h, w), float("inf"), device=DEVICE)
    d = torch.zeros(h, w, device=DEVICE)
    for _ in range(40 if scene == "fractal" else 8):  # planes on the cells of random centres
        cx, cy = r.uniform(0, w), r.uniform(0, h)
        dist = (xx - cx) ** 2 + (yy - cy) ** 2
        plane = (r.uniform(lo, hi) + r.uniform(-0.3, 0.3) * span / w * (xx - cx)
                 + r.uniform(-0.3, 0.3) * span / h * (yy - cy))
        d = torch.where(dist < best, plane, d)
        best = torch.minimum(best, dist)
    return d.clamp(lo, hi)


def _pair(scene, seed, w, h, lo, hi):
    """Left and right uint8 images; the left view samples the right one at x - d, the right gets noise."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    r = random.Random(seed)
    lo, hi = lo + 2.0, lo + max(0.94 * (hi - lo), 3.0)
    pad = int(hi) + 2
    wide = _texture(scene, g, r, h, w + pad)
    d = _true_disparity(scene, r, h, w, lo, hi)
    x = torch.arange(w, device=DEVICE, dtype=torch.float32)[None, :] + pad - d
    x0 = x.floor().clamp(0, w + pad - 2)
    f, i = x - x0, x0.long()
    left = (1 - f) * wide.gather(1, i) + f * wide.gather(1, i + 1)
    right = wide[:, pad:] + torch.randn(h, w, generator=g, device=DEVICE) * (3.0 if scene == "road" else 2.0)
    return left.round().clamp(0, 255).to(torch.uint8).contiguous(), right.round().clamp(0, 255).to(torch.uint8).contiguous()


def _hamming_volume(left, right, d_range):
    """9x7 census Hamming distances [H, W, D] as float32 (partners left of the image: the first column)."""
    def bits(img):
        p = torch.nn.functional.pad(img.float()[None, None], (4, 4, 3, 3), mode="replicate")[0, 0]
        h, w = img.shape
        return torch.stack([p[dy:dy + h, dx:dx + w] < img for dy in range(7) for dx in range(9) if (dy, dx) != (3, 4)])
    a, b = bits(left), bits(right)
    h, w = left.shape
    out = torch.empty(h, w, d_range, device=DEVICE)
    x = torch.arange(w, device=DEVICE)
    for d in range(d_range):
        out[:, :, d] = (a ^ b[:, :, (x - d).clamp_min(0)]).sum(0)
    return out


def _float_inputs(case, seed):
    b, w, h, d = case["batch"], case["width"], case["height"], case["disp"]
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    cost = torch.empty(b, h, w, d, device=DEVICE)
    for k in range(b):
        left, right = _pair("planar", seed * 64 + k, w, h, 0, d)
        cost[k] = _hamming_volume(left, right, d)
    cost += 0.5 * torch.rand(b, h, w, d, generator=g, device=DEVICE)
    # penalty maps a few fitting steps away from their initial 10 and 150
    p1 = 10.0 * (1 + 0.1 * (torch.rand(b, h, w, generator=g, device=DEVICE) - 0.5))
    p2 = 150.0 * (1 + 0.1 * (torch.rand(b, h, w, generator=g, device=DEVICE) - 0.5))
    up = torch.randn(b, h, w, generator=g, device=DEVICE) / (b * h * w)
    return cost, p1, p2, up


# ---------------------------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------------------------
class _Buffer:
    """Device memory of a batch as a tensor: shape, type and address. Tensors made from it hold the batch."""

    def __init__(self, owner, address, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": typestr, "version": 3}


def _wrap(owner, address, shape, typestr):
    return torch.as_tensor(_Buffer(owner, address, shape, typestr), device=DEVICE)


def _plain_option(case):
    return fsc.CuSGMOption(p1=case["p1"], p2_init=case["p2"], cs_type=case["census"], num_paths=4,
                           do_median_filter=case["median"], do_lr_check=case["lr"], lr_threshold=1.0,
                           unique_threshold=0.95, using_constant_p2=True, do_remove_peaks=False)


def _ok(matcher, done):
    if not done:
        raise RuntimeError(matcher.last_error())


def _pyramid_args(case):
    opt = fsc.StereoOption1(width=case["width"], height=case["height"], min_disp=case["min_disp"],
                            max_disp=case["max_disp"], num_layers=case["layers"], do_lr_check=case["lr"],
                            do_rm_peaks=case["peaks"], do_smooth=False)
    return opt, fsc.LevelOverride(1, 10, 150) if case["override"] else None


def _host(t):
    """A page-locked host copy, as the API's own allocator gives applications."""
    a = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    a.copy_(t)
    return a.numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "float":
        cost, p1, p2, up = _float_inputs(case, seed)
        if case["grad"]:
            for t in (cost, p1, p2):
                t.requires_grad_(True)
        return {"kind": kind, "grad": case["grad"], "inputs": (cost, p1, p2), "up": up}
    if kind in ("plain", "pyramid"):
        w, h = case["width"], case["height"]
        hi = case["min_disp"] + case["disp"] if kind == "plain" else case["max_disp"]
        left, right = _pair(case["scene"], seed, w, h, case["min_disp"], hi)
        if kind == "plain":
            m = fsc.StereoCuda()
            _ok(m, m.Init(w, h, case["min_disp"], case["disp"], _plain_option(case)))
        else:
            m = fsc.FasterStereoCuda()
            _ok(m, m.Init(*_pyramid_args(case)))
        if case["host"]:
            left, right, out = _host(left), _host(right), _host(torch.zeros(h, w))
        else:
            out = torch.zeros(h, w, device=DEVICE)
        return {"kind": kind, "host": case["host"], "matcher": m, "images": (left, right), "out": out}
    if kind == "batch":
        pairs = _batch_specs(case)
        m = fsc.StereoBatch()
        _ok(m, m.Init(pairs, fsc.CuSGMOption(p1=10, p2_init=150, cs_type=1, num_paths=4, do_median_filter=True,
                                             do_lr_check=True, lr_threshold=1.0, unique_threshold=0.95,
                                             using_constant_p2=True, do_remove_peaks=False)))
        ranges = [(lo, lo + d) for _, _, lo, d in pairs]
    else:
        opt, override = _pyramid_args(case)
        pairs = [(case["width"], case["height"], case["min_disp"], case["max_disp"])] * case["pairs"]
        m = fsc.StereoBatchPyramid()
        _ok(m, m.Init(pairs, opt, override))
        ranges = [(case["min_disp"], case["max_disp"])] * case["pairs"]
    outs = []
    for i, (p, (lo, hi)) in enumerate(zip(pairs, ranges)):
        w, h = p[0], p[1]
        a, b, c = m.buffers(i)
        left, right = _pair(case["scene"], seed * 1000 + i, w, h, lo, hi)
        _wrap(m, a, (h, w), "|u1").copy_(left)
        _wrap(m, b, (h, w), "|u1").copy_(right)
        outs.append(_wrap(m, c, (h, w), "<f4"))
    return {"kind": kind, "matcher": m, "out": outs}


def run(state):
    kind = state["kind"]
    if kind == "float":
        if not state["grad"]:
            with torch.no_grad():
                return {"disp": float_sgm(*state["inputs"])}
        disp = float_sgm(*state["inputs"])
        gc, g1, g2 = torch.autograd.grad(disp, state["inputs"], state["up"])
        return {"disp": disp.detach(), "grad_cost": gc, "grad_p1": g1, "grad_p2": g2}
    m = state["matcher"]
    if kind in ("plain", "pyramid"):
        left, right = state["images"]
        _ok(m, m.Match(left, right, state["out"]) if state["host"] else m.match_device(left, right, state["out"]))
    else:
        _ok(m, m.run())
    return state["out"]


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
_PATHS = ((1, False), (2, False), (1, True), (2, True))  # down, right, up, left


def _exact_float(case, seed):
    """Hard-min recurrence, soft-argmin and their adjoint in float64, one path at a time."""
    cost, p1, p2, up = (t.double() for t in _float_inputs(case, seed))
    n_d = cost.shape[-1]
    inf = float("inf")

    def padded(t, left, right):  # neighbours in d, infinite outside
        return torch.nn.functional.pad(t, (left, right), value=inf)

    def choices(q, m, a, b):
        jump = m + b
        cand = torch.stack([q, padded(q, 1, 0)[..., :-1] + a, padded(q, 0, 1)[..., 1:] + a, jump.expand_as(q)])
        return cand.min(0)  # the first of equal candidates

    def scan(dim, rev):
        n = cost.shape[dim]
        vol = torch.empty_like(cost)
        order = list(range(n - 1, -1, -1) if rev else range(n))
        prev = None
        for k in order:
            c = cost.select(dim, k)
            if prev is not None:
                m = prev.min(-1, keepdim=True).values
                t = choices(prev, m, p1.select(dim, k)[..., None], p2.select(dim, k)[..., None]).values
                c = c + t - m
            vol.select(dim, k).copy_(c)
            prev = c
        return vol, order

    total = sum(scan(*path)[0] for path in _PATHS)
    weight = torch.softmax(-total, -1)
    levels = torch.arange(n_d, device=DEVICE, dtype=torch.float64)
    disp = (weight * levels).sum(-1)
    if not case["grad"]:
        return {"disp": disp}
    g_sum = -up[..., None] * weight * (levels - disp[..., None])
    gc, g1, g2 = torch.zeros_like(cost), torch.zeros_like(p1), torch.zeros_like(p2)
    for dim, rev in _PATHS:
        vol, order = scan(dim, rev)
        g = torch.zeros_like(vol.select(dim, 0))
        for k, before in zip(reversed(order), list(reversed(order))[1:] + [None]):
            g = g + g_sum.select(dim, k)
            gc.select(dim, k).add_(g)
            if before is None:
                break
            q = vol.select(dim, before)
            m, at = q.min(-1, keepdim=True)
            pick = choices(q, m, p1.select(dim, k)[..., None], p2.select(dim, k)[..., None]).indices
            part = [torch.where(pick == i, g, 0.0) for i in range(4)]
            jumped = part[3].sum(-1, keepdim=True)
            g1.select(dim, k).add_((part[1] + part[2]).sum(-1))
            g2.select(dim, k).add_(jumped[..., 0])
            back = (part[0] + torch.nn.functional.pad(part[1], (0, 1))[..., 1:]
                    + torch.nn.functional.pad(part[2], (1, 0))[..., :-1])
            g = back.scatter_add(-1, at, jumped - g.sum(-1, keepdim=True))
    return {"disp": disp, "grad_cost": gc, "grad_p1": g1, "grad_p2": g2}


def _popcount(v):
    """Set bits of non-negative int64 values."""
    v = v - ((v >> 1) & 0x5555555555555555)
    v = (v & 0x3333333333333333) + ((v >> 2) & 0x3333333333333333)
    v = (v + (v >> 4)) & 0x0F0F0F0F0F0F0F0F
    return ((v & 0x00FF00FF00FF00FF) + ((v >> 8) & 0x00FF00FF00FF00FF)) % 65535


def _census(img, wide, border):
    rx, ry = (4, 3) if wide else (2, 2)
    h, w = img.shape
    v = torch.full((h, w), border, dtype=torch.int64, device=img.device)
    if h <= 2 * ry or w <= 2 * rx:
        return v
    mid = img[ry:h - ry, rx:w - rx]
    acc = torch.zeros(mid.shape, dtype=torch.int64, device=img.device)
    for dy in range(2 * ry + 1):
        for dx in range(2 * rx + 1):
            acc = (acc << 1) | (img[dy:dy + mid.shape[0], dx:dx + mid.shape[1]] < mid)
    v[ry:h - ry, rx:w - rx] = acc
    return v


def _exact_view(case, cost):
    """Four paths, their sum, the winner with the uniqueness test and the parabola: disparities of a view."""
    h, w, n_d = cost.shape
    x0 = max(0, case["min_disp"])
    p1, p2 = case["p1"], case["p2"]
    total = torch.zeros(h, w - x0, n_d, dtype=torch.int64, device=cost.device)
    sub = cost[:, x0:]
    for dim, rev in ((0, False), (1, False), (0, True), (1, True)):
        n = sub.shape[dim]
        prev = None
        for k in (range(n - 1, -1, -1) if rev else range(n)):
            c = sub.select(dim, k).to(torch.int64)
            if prev is not None:
                m = prev.min(-1, keepdim=True).values
                side = torch.nn.functional.pad(prev + p1, (1, 1), value=127)
                t = torch.minimum(torch.minimum(prev, side[..., :-2]), torch.minimum(side[..., 2:], m + p2))
                c = c + t - m
            total.select(dim, k).add_(c & 0xFF)
            prev = c
    levels = torch.arange(n_d, device=cost.device)
    m = total.min(-1, keepdim=True).values
    tied = total == m
    if n_d == 64:  # two halves: one holds d < 32, the other d >= 32 where d - 32 is not tied; rows alternate
        low, high = tied[..., :32], tied[..., 32:] & ~tied[..., :32]
        first_low = torch.where(low.any(-1), low.int().argmax(-1), -1)
        first_high = torch.where(high.any(-1), high.int().argmax(-1) + 32, -1)
        even = (torch.arange(h, device=cost.device) % 2 == 0)[:, None]
        best = torch.where(even, torch.where(first_high >= 0, first_high, first_low),
                           torch.where(first_low >= 0, first_low, first_high))
    else:
        best = tied.int().argmax(-1)
    at = best[..., None]
    c2 = m[..., 0].double()
    c1 = total.gather(-1, (at - 1).clamp_min(0))[..., 0].double()
    c3 = torch.where(best + 1 < n_d, total.gather(-1, (at + 1).clamp_max(n_d - 1))[..., 0], best).double()
    den = (c1 + c3 - 2 * c2).clamp_min(1.0)
    d = best + case["min_disp"] + (c1 - c3 + den) / (2 * den)
    # 1 - 0.95 as the single-precision option value gives it
    loss = float(np.float32(1.0) - np.float32(0.95))
    good = (best > 0) & (torch.minimum(c1, c3) - c2 > (c2.float() * loss).double())
    if n_d == 256:
        good &= best < n_d - 1
    out = torch.full((h, w), INVALID, dtype=torch.float64, device=cost.device)
    out[:, x0:] = torch.where(good, d, INVALID)
    rows = h if n_d == 256 else h // 2 * 2
    out[rows:] = INVALID
    out[:5] = INVALID
    out[max(h - 4, 0):] = INVALID
    out[:, :5] = INVALID
    out[:, max(w - 4, 0):] = INVALID
    return out


def _exact_plain(case, seed):
    w, h, n_d, lo = case["width"], case["height"], case["disp"], case["min_disp"]
    left, right = _pair(case["scene"], seed, w, h, lo, lo + n_d)
    cl = _census(left, case["census"], 0)
    cr = _census(right, case["census"], 0xFFFFFFFF)
    x = torch.arange(w, device=DEVICE)[:, None]
    step = lo + torch.arange(n_d, device=DEVICE)[None, :]

    def volume(a, b, pos):
        pos = torch.where((pos >= 0) & (pos < w), pos, 0)
        out = torch.empty(h, w, n_d, dtype=torch.uint8, device=DEVICE)
        for y in range(0, h, 64):
            out[y:y + 64] = _popcount(a[y:y + 64, :, None] ^ b[y:y + 64][:, pos])
        return out

    cost = volume(cl, cr, x - step)
    disp = _exact_view(case, cost)
    if case["lr"]:
        other = volume(cr, cl, x + step)
        if not case["census"]:  # the 5x5 right view keeps the left cost on the last pixel of each block of D
            x0 = max(0, lo)
            cols = torch.arange(x0, w, device=DEVICE)
            last = ((cols - x0) % n_d == n_d - 1) | (cols == w - 1)
            other[:, cols[last]] = cost[:, cols[last]]
        right_disp = _exact_view(case, other)
        at = torch.arange(w, device=DEVICE)[None, :] - disp
        at = torch.where(at > 0, torch.floor(at + 0.5), -torch.floor(-at + 0.5))
        inside = (disp != INVALID) & (at >= 0) & (at < w)
        r = right_disp.gather(1, at.clamp(0, w - 1).long())
        disp = torch.where(inside & ((disp - r).abs() <= 1.0), (disp + r) / 2, INVALID)
    if case["median"] and w >= 3 and h >= 3:
        last_row = min(h - 2, 2 * ((w - 1) // 2))
        windows = torch.stack([disp[1 + dy:1 + dy + last_row, 1 + dx:w - 1 + dx] for dy in (-1, 0, 1) for dx in (-1, 0, 1)])
        mid = windows.sort(0).values[4]
        disp = disp.clone()
        disp[1:1 + last_row, 1:w - 1] = mid
    return disp


def exact(case, seed):
    """float64 results; None where integer decisions of one pyramid level feed the next."""
    if case["kind"] == "float":
        return _exact_float(case, seed)
    if case["kind"] == "plain":
        return _exact_plain(case, seed)
    return None
