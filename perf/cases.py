"""Workloads of the permutohedral-lattice library, as user programs call it.

Every case names an operation, its sizes and its filter parameters.  Images are synthetic:
gradients, constant rectangles and Gaussian noise of 0.05, clamped to [0, 1], made on the GPU
from the seed alone.  Operations that filter in place run on a copy, so the inputs survive a
pass.
"""
import math

import numpy as np
import torch

import imagestack_b200 as pg
from imagestack_b200 import synth


def listed():
    return [
        # the smallest request a service sees: launches and latency, no throughput
        {"name": "bilateral_64", "op": "bilateral", "w": 64, "h": 64, "t": 1, "c": 3, "fw": 8.0, "ft": 0.0,
         "cs": 0.1, "payload": "fp32"},
        # -gausstransform on a host image, positions (x, y, r, g, b) and values (r, g, b, 1), as
        # the command-line plugin hands them over
        {"name": "gauss_host_512", "op": "gauss_host", "w": 512, "h": 512, "fw": 8.0, "cs": 0.1},
        # one RGB frame per call at the usual sigmas
        {"name": "bilateral_4k", "op": "bilateral", "w": 3840, "h": 2160, "t": 1, "c": 3, "fw": 16.0, "ft": 0.0,
         "cs": 0.1, "payload": "fp32"},
        # a throughput job: four 4K frames in one set of launches, settings picked by the autotuner
        {"name": "batch_4k_x4", "op": "frames", "w": 3840, "h": 2160, "count": 4, "fw": 16.0, "cs": 0.1,
         "payload": "fp32"},
        # grey joint bilateral against a luminance guide, by the lattice and by the bilateral grid
        {"name": "joint_gray_4k", "op": "joint", "w": 3840, "h": 2160, "c": 1, "guide": 1, "fw": 16.0, "cs": 0.1,
         "method": "permutohedral_gpu"},
        {"name": "joint_gray_4k_grid", "op": "joint", "w": 3840, "h": 2160, "c": 1, "guide": 1, "fw": 16.0,
         "cs": 0.1, "method": "grid_gpu"},
        # a high-dimensional Gauss transform of a point cloud: capacity of the hash table
        {"name": "gauss_d16_2m", "op": "cloud", "n": 2000000, "d": 16, "vc": 4},
        # uneven images, each with its own sigmas, FP16 vertex rows, one replayed CUDA graph
        {"name": "mixed_batch_fp16", "op": "mixed", "count": 256, "lo": 128, "hi": 1024, "shapes": 0,
         "payload": "fp16", "graph": True},
        # a video clip with time as a position (d = 6), odd sizes
        {"name": "video_d6", "op": "bilateral", "w": 959, "h": 541, "t": 8, "c": 3, "fw": 8.0, "ft": 2.0,
         "cs": 0.15, "payload": "fp32"},
        # denoising against patch features (d = 8: keys of two words)
        {"name": "nlmeans_d8", "op": "joint", "w": 1280, "h": 720, "c": 3, "guide": 6, "fw": 4.0, "cs": 0.3,
         "method": "permutohedral_gpu"},
        # joint upsampling: splat a half-size image, slice at the full-size guide's positions
        {"name": "upsample_1080p", "op": "upsample", "w": 1920, "h": 1080, "fw": 16.0, "cs": 0.1},
        # a burst of requests to the server, bilateral and joint bilateral, host images
        {"name": "served_burst", "op": "served", "count": 48, "lo": 64, "hi": 1024, "shapes": 5, "payload": "fp16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["bilateral", "bilateral", "gauss_host", "frames", "joint", "joint", "grid", "cloud", "mixed",
                     "video", "nlmeans", "upsample", "served"])
    fw = round(rng.uniform(4.0, 32.0), 2)
    cs = round(rng.uniform(0.05, 0.3), 3)
    if op == "bilateral":
        return {"op": "bilateral", "w": _log(rng, 64, 3840), "h": _log(rng, 64, 2160), "t": 1,
                "c": rng.choice([1, 3, 3]), "fw": fw, "ft": 0.0, "cs": cs,
                "payload": rng.choice(["fp32", "fp32", "fp16", "bf16"])}
    if op == "gauss_host":
        return {"op": "gauss_host", "w": _log(rng, 64, 1024), "h": _log(rng, 64, 1024), "fw": fw, "cs": cs}
    if op == "frames":
        return {"op": "frames", "w": _log(rng, 640, 3840), "h": _log(rng, 360, 2160), "count": rng.randint(2, 4),
                "fw": fw, "cs": cs, "payload": rng.choice(["fp32", "fp16"])}
    if op in ("joint", "grid"):
        return {"op": "joint", "w": _log(rng, 64, 3840), "h": _log(rng, 64, 2160),
                "c": rng.choice([1, 1, 3]), "guide": 1, "fw": fw, "cs": cs,
                "method": "grid_gpu" if op == "grid" else "permutohedral_gpu"}
    if op == "cloud":
        return {"op": "cloud", "n": _log(rng, 20000, 2000000), "d": rng.randint(6, 16), "vc": 4}
    if op == "mixed":
        return {"op": "mixed", "count": _log(rng, 16, 256), "lo": 64, "hi": 1024, "shapes": rng.randint(1, 1 << 20),
                "payload": rng.choice(["fp16", "fp16", "fp32"]), "graph": rng.random() < 0.5}
    if op == "video":
        return {"op": "bilateral", "w": _log(rng, 64, 960), "h": _log(rng, 64, 540), "t": rng.randint(2, 8),
                "c": rng.choice([1, 3, 3]), "fw": round(rng.uniform(4.0, 16.0), 2),
                "ft": round(rng.uniform(1.0, 4.0), 2), "cs": cs, "payload": "fp32"}
    if op == "nlmeans":
        return {"op": "joint", "w": _log(rng, 128, 1280), "h": _log(rng, 128, 720), "c": 3, "guide": rng.choice([4, 6]),
                "fw": round(rng.uniform(3.0, 8.0), 2), "cs": round(rng.uniform(0.2, 0.5), 3),
                "method": "permutohedral_gpu"}
    if op == "upsample":
        return {"op": "upsample", "w": _log(rng, 256, 1920), "h": _log(rng, 256, 1080), "fw": fw, "cs": cs}
    return {"op": "served", "count": rng.randint(8, 48), "lo": 64, "hi": rng.choice([256, 512, 1024]),
            "shapes": rng.randint(1, 1 << 20), "payload": rng.choice(["fp16", "fp32"])}


# ---- inputs ------------------------------------------------------------------------------

DEV = "cuda" if torch.cuda.is_available() else "cpu"


class _Source:
    """Random numbers of one state: `host` for shapes, `dev` for pixels."""

    def __init__(self, seed):
        self.host = np.random.RandomState(seed & 0x7FFFFFFF)
        self.dev = torch.Generator(device=DEV)
        self.dev.manual_seed(seed)

    def image(self, c, h, w, rects):
        """(c, h, w): gradients, constant rectangles and noise, clamped to [0, 1]."""
        abc = self.host.uniform(0.0, 0.5, (c, 3))
        xs = torch.arange(w, device=DEV, dtype=torch.float32) / w
        ys = torch.arange(h, device=DEV, dtype=torch.float32) / h
        out = torch.empty((c, h, w), device=DEV)
        for k in range(c):
            out[k] = float(abc[k, 0]) * xs[None, :] + float(abc[k, 1]) * ys[:, None] + float(abc[k, 2])
        for u in self.host.uniform(size=(rects, 4 + c)):
            x0, y0 = int(u[0] * w), int(u[1] * h)
            rw, rh = int(1 + u[2] * max(w / 4 - 1, 0)), int(1 + u[3] * max(h / 4 - 1, 0))
            for k in range(c):
                out[k, y0:y0 + rh, x0:x0 + rw] = float(u[4 + k])
        out += 0.05 * torch.randn((c, h, w), device=DEV, generator=self.dev)
        return out.clamp_(0.0, 1.0)


def _rects(w, h):
    return 64 if w * h > 1 << 21 else 16


def _luminance(rgb):
    return (0.299 * rgb[0] + 0.587 * rgb[1] + 0.114 * rgb[2])[None].contiguous()


def _features(src, rgb, n):
    """Patch features: n random mixes of a pixel and its four neighbours."""
    mix = src.host.uniform(-1.0, 1.0, (n, 3, 5))
    out = torch.zeros((n,) + tuple(rgb.shape[1:]), device=DEV)
    for j, s in enumerate([(0, 0), (0, 1), (1, 0), (0, -1), (-1, 0)]):
        moved = torch.roll(rgb, s, dims=(1, 2))
        for k in range(n):
            for c in range(3):
                out[k] += float(mix[k, c, j]) * moved[c]
    return out


def _coords(w, h, step=1.0, first=0.0):
    xs = (torch.arange(w, device=DEV, dtype=torch.float32) * step + first).expand(h, w)
    ys = (torch.arange(h, device=DEV, dtype=torch.float32) * step + first)[:, None].expand(h, w)
    return torch.stack([xs, ys])


def _specs(case):
    return synth.batch_specs(case["count"], case["lo"], case["hi"], seed=case["shapes"])


_SERVERS = {}


def _server(payload):
    """One server per payload for the whole program, as a service keeps it."""
    if payload not in _SERVERS:
        _SERVERS[payload] = pg.Server(payload=payload)
    return _SERVERS[payload]


def _inputs(case, seed):
    src = _Source(seed)
    op = case["op"]
    if op == "bilateral":
        if case["t"] == 1:
            return {"image": src.image(case["c"], case["h"], case["w"], _rects(case["w"], case["h"]))}
        scene = src.image(case["c"], case["h"], case["w"], 24)
        frames = [torch.roll(scene, 2 * t, dims=2) + 0.05 * torch.randn(scene.shape, device=DEV, generator=src.dev)
                  for t in range(case["t"])]
        return {"image": torch.stack(frames, 1).contiguous()}
    if op == "gauss_host":
        rgb = src.image(3, case["h"], case["w"], 16)
        return {"pos": torch.cat([_coords(case["w"], case["h"]), rgb]).cpu().numpy(),
                "val": torch.cat([rgb, torch.ones_like(rgb[:1])]).cpu().numpy()}
    if op == "frames":
        return {"image": torch.stack([src.image(3, case["h"], case["w"], _rects(case["w"], case["h"]))
                                      for _ in range(case["count"])])}
    if op == "joint":
        rgb = src.image(3, case["h"], case["w"], _rects(case["w"], case["h"]))
        guide = _luminance(rgb) if case["guide"] == 1 else _features(src, rgb, case["guide"])
        noisy = rgb if case["c"] == 3 else _luminance(rgb)
        return {"image": noisy, "guide": guide}
    if op == "cloud":
        n, d = case["n"], case["d"]
        centres = torch.rand((d, 32), device=DEV, generator=src.dev) * 10.0
        pick = torch.randint(0, 32, (n,), device=DEV, generator=src.dev)
        pos = centres[:, pick] + 0.5 * torch.randn((d, n), device=DEV, generator=src.dev)
        val = torch.rand((case["vc"] + 1, n), device=DEV, generator=src.dev) * 2.0 - 1.0
        val[-1] = 1.0
        return {"pos": pos.reshape(d, 1, n), "val": val.reshape(-1, 1, n)}
    if op == "mixed":
        specs = _specs(case)
        flat = torch.cat([src.image(3, h, w, 16).reshape(-1) for w, h, _, _, _ in specs])
        return {"image": flat}
    if op == "upsample":
        w, h = case["w"], case["h"]
        full = src.image(3, h, w, 32)
        half = torch.nn.functional.avg_pool2d(full[None], 2)[0]
        lw, lh = half.shape[2], half.shape[1]
        return {"slice": torch.cat([_coords(w, h), full]),
                "pos": torch.cat([_coords(lw, lh, 2.0, 0.5), half]),
                "val": torch.cat([half.flip(0), torch.ones_like(half[:1])])}
    images = []
    for k, (w, h, _, _, _) in enumerate(_specs(case)):
        images.append((src.image(3, h, w, 12) if k % 2 == 0 else _luminance(src.image(3, h, w, 12))).cpu().numpy())
    return {"images": images}


def _parts(case, flat):
    """The images of a mixed batch as views into one buffer."""
    out, at = [], 0
    for w, h, _, _, _ in _specs(case):
        out.append(flat[at:at + 3 * w * h].view(3, h, w))
        at += 3 * w * h
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    op = case["op"]
    if op in ("bilateral", "frames", "joint", "mixed"):
        s["work"] = s["image"].clone()
    if op == "mixed":
        specs = _specs(case)
        s["parts"] = _parts(case, s["work"])
        s["fw"], s["cs"] = [x[2] for x in specs], [x[3] for x in specs]
    if op == "frames":
        s["parts"] = list(s["work"])
        # a throughput job lets the tuner finish its trials for the shape before it starts
        for _ in range(40):
            s["work"].copy_(s["image"])
            _frames(s)
            if pg.last_stats()["tuned"] != 1:
                break
    if op == "served":
        specs = _specs(case)
        s["fw"], s["cs"] = [x[2] for x in specs], [x[3] for x in specs]
        s["out"] = [np.empty_like(a) for a in s["images"]]
        s["server"] = _server(case["payload"])
    return s


# ---- one pass ----------------------------------------------------------------------------

def _frames(s):
    case = s["case"]
    n = case["count"]
    pg.bilateral_batch(s["parts"], [case["fw"]] * n, [case["cs"]] * n, payload=case["payload"], autotune=True)


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "bilateral":
        s["work"].copy_(s["image"])
        return pg.Bilateral.apply(s["work"], case["fw"], case["fw"], case["ft"], case["cs"], payload=case["payload"])
    if op == "gauss_host":
        sig = [case["fw"], case["fw"], case["cs"], case["cs"], case["cs"]]
        return pg.GaussTransform.apply(None, s["pos"], s["val"], sig)
    if op == "frames":
        s["work"].copy_(s["image"])
        _frames(s)
        return s["work"]
    if op == "joint":
        s["work"].copy_(s["image"])
        return pg.JointBilateral.apply(s["work"], s["guide"], case["fw"], case["fw"], 0.0, case["cs"],
                                       method=case["method"])
    if op == "cloud":
        return pg.GaussTransform.apply(None, s["pos"], s["val"], [1.0] * case["d"])
    if op == "mixed":
        s["work"].copy_(s["image"])
        pg.bilateral_batch(s["parts"], s["fw"], s["cs"], payload=case["payload"], graph=case["graph"])
        return s["work"]
    if op == "upsample":
        sig = [case["fw"], case["fw"], case["cs"], case["cs"], case["cs"]]
        return pg.GaussTransform.apply(s["slice"], s["pos"], s["val"], sig)
    server = s["server"]
    tickets = []
    for k, (im, out) in enumerate(zip(s["images"], s["out"])):
        if im.shape[0] == 3:
            tickets.append(server.submit(pg.REQ_BILATERAL, im, out, filter_width=s["fw"][k], color_sigma=s["cs"][k]))
        else:
            tickets.append(server.submit(pg.REQ_JOINT_BILATERAL, im, out, ref=im, filter_width=s["fw"][k],
                                         color_sigma=s["cs"][k]))
    for t in tickets:
        server.wait(t)
    return s["out"]


def work(case):
    """Inputs read and outputs written once; the multiply-adds of the splat and the slice."""
    op = case["op"]
    if op in ("bilateral", "frames"):
        n = case["w"] * case["h"] * case.get("t", 1) * case.get("count", 1)
        c = case.get("c", 3)
        d = c + 2 + (1 if case.get("t", 1) > 1 else 0)
        io, vd = 2 * c * n, c + 1
    elif op == "gauss_host":
        n, d, vd = case["w"] * case["h"], 5, 4
        io = 13 * n
    elif op == "joint":
        n, d, vd = case["w"] * case["h"], case["guide"] + 2, case["c"] + 1
        io = (2 * case["c"] + case["guide"]) * n
    elif op == "cloud":
        n, d, vd = case["n"], case["d"], case["vc"] + 1
        io = (d + 2 * vd) * n
    elif op == "upsample":
        full, n = case["w"] * case["h"], (case["w"] // 2) * (case["h"] // 2)
        d, vd = 5, 4
        return {"bytes": 4 * (9 * n + 9 * full), "flops": 2 * (d + 1) * vd * (n + full)}
    else:
        n = sum(x[0] * x[1] for x in _specs(case))
        d, vd = 5, 4
        io = 6 * n
        if op == "served":
            io = sum((6 if k % 2 == 0 else 3) * x[0] * x[1] for k, x in enumerate(_specs(case)))
    return {"bytes": 4 * io, "flops": 4 * (d + 1) * vd * n}


# ---- the same results in 64 bits -----------------------------------------------------------
# The method fixes each point's lattice vertices and weights by single-precision arithmetic in
# a stated order; from there on every sum is in 64 bits.

def _simplex(pos):
    """Per point (columns of pos, (d, n) float32 already divided by the sigmas): the hash of
    each of its d+1 vertex keys, their weights, and the key hash's per-coordinate factors."""
    d, n = pos.shape
    f32 = np.float32
    sf = [f32(f32(1) / f32(math.sqrt(f32((i + 1) * (i + 2)))) * f32(f32(d + 1) * f32(math.sqrt(f32(2.0 / 3)))))
          for i in range(d)]
    sc = [float(x) for x in sf]
    e = [None] * (d + 1)
    e[d] = (pos[d - 1] * float(-d)) * sc[d - 1]
    for i in range(d - 1, 0, -1):
        e[i] = (e[i + 1] - (pos[i - 1] * float(i)) * sc[i - 1]) + (pos[i] * float(i + 2)) * sc[i]
    e[0] = e[1] + (pos[0] * 2.0) * sc[0]
    scale = float(f32(1) / f32(d + 1))
    g, total = [], torch.zeros(n, dtype=torch.int64, device=pos.device)
    for i in range(d + 1):
        v = e[i] * scale
        up, down = torch.ceil(v) * (d + 1), torch.floor(v) * (d + 1)
        g.append(torch.where(up - e[i] < e[i] - down, up, down).to(torch.int64))
        total += g[i]
    total = torch.div(total, d + 1, rounding_mode="trunc")
    diff = [e[i] - g[i].to(torch.float32) for i in range(d + 1)]
    rank = [torch.zeros_like(total) for _ in range(d + 1)]
    for i in range(d):
        for j in range(i + 1, d + 1):
            less = diff[i] < diff[j]
            rank[i] += less
            rank[j] += ~less
    del diff
    for i in range(d + 1):
        rank[i] += total
        high, low = rank[i] > d, rank[i] < 0
        g[i] += (low.to(torch.int64) - high.to(torch.int64)) * (d + 1)
        rank[i] += (low.to(torch.int64) - high.to(torch.int64)) * (d + 1)
    delta = torch.empty((d + 1, n), dtype=torch.float32, device=pos.device)
    for i in range(d + 1):
        delta.scatter_(0, rank[i][None], ((e[i] - g[i].to(torch.float32)) * scale)[None])
    bary = [delta[d] + (1.0 + -delta[0])] + [delta[d - k] - delta[d + 1 - k] for k in range(1, d + 1)]
    del e, delta
    factors = [int(x) | 1 for x in np.random.RandomState(12).randint(-(1 << 62), 1 << 62, d)]
    h = sum(g[i] * factors[i] for i in range(d))
    step, mask = _wrap(sum(factors)), (1 << 64) - 1
    hashes = []
    for r in range(d + 1):
        hr = h + _wrap((r * step) & mask)
        for i in range(d):
            hr = hr - torch.where(rank[i] > d - r, _wrap((d + 1) * factors[i]), 0)
        hashes.append(hr)
    return hashes, bary, factors


def _wrap(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >= 1 << 63 else x


def _find(keys, h):
    at = torch.searchsorted(keys, h).clamp_(max=keys.numel() - 1)
    return at, keys[at] == h


def _lattice(pos, val, slice_pos=None):
    """val (vd, n) splatted at pos (d, n), blurred, sliced at slice_pos or at pos: (vd, m) float64."""
    d, n = pos.shape
    hashes, bary, factors = _simplex(pos)
    keys = torch.unique(torch.cat(hashes))
    rows = torch.zeros((keys.numel(), val.shape[0]), dtype=torch.float64, device=pos.device)
    v64 = val.double().t().contiguous()
    where = []
    for r in range(d + 1):
        at = torch.searchsorted(keys, hashes[r])
        rows.index_add_(0, at, v64 * bary[r].double()[:, None])
        hashes[r] = None
        if slice_pos is None:
            where.append(at.to(torch.int32))
    del v64
    for j in range(d + 1):
        up = _wrap(sum(factors) - ((d + 1) * factors[j] if j < d else 0))
        out = rows * 0.5
        for step in (up, _wrap(-up)):
            at, hit = _find(keys, keys + step)
            out += rows[at].mul_((0.25 * hit)[:, None])
        rows = out
    if slice_pos is None:
        out = torch.zeros((n, val.shape[0]), dtype=torch.float64, device=pos.device)
        for r in range(d + 1):
            out += rows[where[r].to(torch.int64)] * bary[r].double()[:, None]
        return out.t()
    hashes, bary, _ = _simplex(slice_pos)
    out = torch.zeros((slice_pos.shape[1], val.shape[0]), dtype=torch.float64, device=pos.device)
    for r in range(d + 1):
        at, hit = _find(keys, hashes[r])
        out += rows[at] * (bary[r].double() * hit)[:, None]
    return out.t()


def _inv(sigma):
    return float(np.float32(1) / np.float32(sigma))


def _guided_points(image, guide, fw, ft, cs):
    """Positions and values of a joint bilateral of image (c, t, h, w) against guide."""
    c, t, h, w = image.shape
    pos = [guide[k].reshape(-1) * _inv(cs) for k in range(guide.shape[0])]
    grid = torch.meshgrid(torch.arange(t, device=image.device), torch.arange(h, device=image.device),
                          torch.arange(w, device=image.device), indexing="ij")
    pos += [grid[2].reshape(-1).float() * _inv(fw), grid[1].reshape(-1).float() * _inv(fw)]
    if t > 1:
        pos.append(grid[0].reshape(-1).float() * _inv(ft))
    val = torch.cat([image.reshape(c, -1), torch.ones((1, t * h * w), device=image.device)])
    return torch.stack(pos), val


def _normalised(out, shape):
    return (out[:-1] / out[-1]).reshape(shape)


def _joint64(image, guide, fw, ft, cs, method="permutohedral_gpu"):
    shape = image.shape
    if image.dim() == 3:
        image, guide = image[:, None], guide[:, None]
    pos, val = _guided_points(image, guide, fw, ft, cs)
    return _normalised(_grid(pos, val) if method == "grid_gpu" else _lattice(pos, val), shape)


def _grid(pos, val):
    """The bilateral grid: multilinear splat, two [1 2 1]/4 passes per dimension, multilinear slice."""
    d, n = pos.shape
    scaled = pos * float(np.float32(math.sqrt(np.float32(1.0 / 3 + 1.0))))
    low = scaled.min(1).values
    span = scaled.max(1).values - low
    sizes = [int(math.ceil(float(span[j]))) + 1 for j in range(d)]
    f = scaled - low[:, None]
    cell = torch.floor(f)
    frac = (f - cell).double()
    cell = cell.to(torch.int64)
    corners = []
    for corner in range(1 << d):
        w = torch.ones(n, dtype=torch.float64, device=pos.device)
        at = torch.zeros(n, dtype=torch.int64, device=pos.device)
        for j in reversed(range(d)):
            up = (corner >> j) & 1
            w = w * (frac[j] if up else 1.0 - frac[j])
            at = at * sizes[j] + (cell[j] + up).clamp(max=sizes[j] - 1)   # past the end: weight 0
        corners.append((at, w))
    rows = torch.zeros((math.prod(sizes), val.shape[0]), dtype=torch.float64, device=pos.device)
    v64 = val.double().t().contiguous()
    for at, w in corners:
        rows.index_add_(0, at, v64 * w[:, None])
    rows = rows.reshape(tuple(reversed(sizes)) + (val.shape[0],))
    for j in range(d):
        axis, last = d - 1 - j, sizes[j] - 1
        for _ in range(2):
            out = rows * 0.5
            if last > 0:
                out.narrow(axis, 1, last).add_(rows.narrow(axis, 0, last), alpha=0.25)
                out.narrow(axis, 0, last).add_(rows.narrow(axis, 1, last), alpha=0.25)
            rows = out
    rows = rows.reshape(-1, val.shape[0])
    out = torch.zeros((n, val.shape[0]), dtype=torch.float64, device=pos.device)
    for at, w in corners:
        out += rows[at] * w[:, None]
    return out.t()


def exact(case, seed):
    s = _inputs(case, seed)
    op = case["op"]
    if op == "bilateral":
        return _joint64(s["image"], s["image"], case["fw"], case["ft"], case["cs"])
    if op == "joint":
        return _joint64(s["image"], s["guide"], case["fw"], 0.0, case["cs"], case["method"])
    if op == "frames":
        return torch.stack([_joint64(f, f, case["fw"], 0.0, case["cs"]) for f in s["image"]])
    if op == "mixed":
        parts = [_joint64(f, f, x[2], 0.0, x[3]) for f, x in zip(_parts(case, s["image"]), _specs(case))]
        return torch.cat([p.reshape(-1) for p in parts])
    if op == "served":
        out = []
        for im, x in zip(s["images"], _specs(case)):
            f = torch.from_numpy(im).to(DEV)
            out.append(_joint64(f, f, x[2], 0.0, x[3]).cpu().numpy())
        return out
    if op == "cloud":
        d, n = case["d"], case["n"]
        return _lattice(s["pos"].reshape(d, n), s["val"].reshape(-1, n)).reshape(-1, 1, n)
    pos, val = torch.as_tensor(s["pos"], device=DEV), torch.as_tensor(s["val"], device=DEV)
    scale = torch.tensor([_inv(case["fw"])] * 2 + [_inv(case["cs"])] * 3, device=DEV)[:, None]
    flat = pos.reshape(5, -1) * scale
    if op == "gauss_host":
        return _lattice(flat, val.reshape(4, -1)).reshape(val.shape).cpu().numpy()
    out = _lattice(flat, val.reshape(4, -1), s["slice"].reshape(5, -1) * scale)
    return out.reshape((4,) + tuple(s["slice"].shape[1:]))
