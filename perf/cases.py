"""Performance cases of the stereo engine: what its users have it do, through its public entry points.

listed() holds the named cases, draw() gives more of the same ranges, prepare() makes a case's inputs on the
device (host arrays where the entry point takes host buffers), run() is one pass, work() the bytes and
operations that pass cannot do without, exact() its outputs in 64 bits where they are computed numbers with
a plain definition.

Sizes: 96x64 is the smoke test's, 450x375 D64 the single-pair driver's, 720x496 D128 the quarter-scale batch's,
1440x992 the half-scale pairs' (D256 Census, D144 MC-CNN).
"""
import ctypes as C
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(os.getcwd() if os.path.isdir("hbp-isp_b200") else ROOT, "hbp-isp_b200"))

import hbp_b200 as E  # noqa: E402

DEV = "cuda:0"

# kinds of case and the range of each (pixels, aspect ratio H/W, disparities as a share of W, pairs)
PAIR, BATCH, MCCNN, AD, CENSUS, SUPERPIXELS, POST, SERVE = (
    "pair", "batch", "mccnn", "ad_levels", "census", "superpixels", "post", "serve")


def _case(kind, W, H, D=0, name=None, **kw):
    c = {"kind": kind, "W": W, "H": H, "D": D, "pairs": 1, "fp16": 0, "post": 1, "gpu_order": 0, "right": 0,
         "linkage": 2, "num_nb": 4, "sigma": 0.0, "target": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one thumbnail pair from host buffers, bound by launches and host reads
        _case(PAIR, 96, 64, 32, "pair_96x64_d32"),
        # the single-pair driver's image through the Middlebury driver's flow: both views, left-right check,
        # weighted median, planes returned
        _case(PAIR, 450, 375, 64, "pair_450x375_d64_lr", post=2),
        # one quarter-scale pair at a time, FP32: the latency of a caller that waits for each result
        _case(PAIR, 720, 496, 128, "pair_720x496_d128"),
        # the throughput workload: a resident batch of 16 quarter-scale pairs, FP16 messages
        _case(BATCH, 720, 496, 128, "batch16_720x496_d128_fp16", pairs=16, fp16=1),
        # half-scale pairs with 256 disparities, FP32 messages: the largest volumes
        _case(BATCH, 1440, 992, 256, "batch4_1440x992_d256", pairs=4),
        # the reference's published flow: a network's float volume, HBP with alpha 1.3 and tau 0.5
        _case(MCCNN, 1440, 992, 144, "mccnn_1440x992_d144"),
        # AD cost and every pyramid level's map, at a size that no tile divides
        _case(AD, 451, 373, 64, "ad_levels_451x373_d64"),
        # the matching cost by itself, both views: a caller that brings its own optimiser
        _case(CENSUS, 720, 496, 128, "census_720x496_d128", right=1),
        # superpixels by themselves: SegHAC down to 1000 clusters and the label image
        _case(SUPERPIXELS, 720, 496, 0, "superpixels_720x496_1000", target=1000),
        # the post-processing by itself at half scale: left-right check, fill, weighted median
        _case(POST, 1440, 992, 256, "post_1440x992"),
        # the same with the reference's GPU order of the weighted median
        _case(POST, 450, 375, 64, "post_gpu_order_450x375", gpu_order=1),
        # a request server in closed loop with three image sizes at once, FP16 messages
        _case(SERVE, 720, 496, 128, "serve_9_mixed_fp16", pairs=9, fp16=1),
    ]


def _size(rng, lo, hi):
    """W, H with lo..hi pixels spread over their logarithm, any remainder."""
    n = lo * (hi / lo) ** rng.random()
    r = rng.uniform(0.6, 0.95)
    W = max(40, int((n / r) ** 0.5))
    return W, max(32, int(W * r))


def draw(rng):
    kind = rng.choice([PAIR, PAIR, BATCH, BATCH, MCCNN, AD, CENSUS, SUPERPIXELS, POST, SERVE])
    fp16 = rng.randrange(2)
    if kind == PAIR:
        W, H = _size(rng, 4000, 720 * 496)
        return _case(PAIR, W, H, rng.randint(16, max(17, W // 5)), fp16=fp16, post=rng.choice([0, 1, 2]),
                     linkage=rng.choice([2, 2, 0, 3]), num_nb=rng.choice([4, 4, 8]), sigma=rng.choice([0.0, 0.0, 0.7]))
    if kind == BATCH:
        W, H = _size(rng, 20000, 1440 * 992)
        most = max(1, min(12, 3 * 1440 * 992 // (W * H)))
        return _case(BATCH, W, H, rng.randint(16, min(256, W // 5)), pairs=rng.randint(1, most), fp16=fp16)
    if kind == MCCNN:
        W, H = _size(rng, 20000, 1200 * 900)
        return _case(MCCNN, W, H, rng.randint(16, min(144, W // 5)), fp16=fp16)
    if kind == AD:
        W, H = _size(rng, 8000, 720 * 496)
        return _case(AD, W, H, rng.randint(16, max(17, W // 5)), fp16=fp16)
    if kind == CENSUS:
        W, H = _size(rng, 4000, 1440 * 992)
        return _case(CENSUS, W, H, rng.randint(16, max(17, W // 5)), right=rng.randrange(2))
    if kind == SUPERPIXELS:
        W, H = _size(rng, 4000, 1440 * 992)
        return _case(SUPERPIXELS, W, H, target=rng.choice([50, 300, 1000]), linkage=rng.choice([2, 0, 1, 3]),
                     num_nb=rng.choice([4, 8]), sigma=rng.choice([0.0, 0.7, 1.0]))
    if kind == POST:
        W, H = _size(rng, 4000, 1440 * 992)
        order = rng.randrange(2) if W * H < 200000 else 0
        return _case(POST, W, H, max(16, W // 6), gpu_order=order)
    W, H = _size(rng, 20000, 720 * 496)
    return _case(SERVE, W, H, max(16, W // 6), pairs=rng.randint(3, 12), fp16=fp16)


# ---------------------------------------------------------------------------------------------- inputs
def _scene(W, H, D, seed):
    """A piecewise-planar pair as the tests' scenes are (Voronoi segments with slanted disparity planes, noise and
    a sinusoid as texture, the right view a z-buffered warp), made on the device.
    left, right: H x W x 3 bytes; plane: H x W x 3 of the left view; disparities of both views (0: no match)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(DEV).manual_seed(seed)
    n = 16 if W * H <= 450 * 375 else 24 if W * H <= 1080 * 744 else 40
    lo, hi = min(4.0, D / 4), float(D - min(4, D // 4))
    sx, sy = rng.uniform(0, W, n), rng.uniform(0, H, n)
    a, b = rng.uniform(-0.05, 0.05, n), rng.uniform(-0.05, 0.05, n)
    c = rng.uniform(lo, hi, n) - a * sx - b * sy
    base = rng.uniform(0, 255, (n, 3))
    theta, period, phase = rng.uniform(0, np.pi, n), rng.uniform(4, 32, n), rng.uniform(0, 2 * np.pi, n)
    t = lambda v: torch.from_numpy(np.asarray(v)).to(DEV)  # noqa: E731
    ys, xs = torch.meshgrid(torch.arange(H, device=DEV, dtype=torch.float64),
                            torch.arange(W, device=DEV, dtype=torch.float64), indexing="ij")
    best = torch.full((H, W), float("inf"), device=DEV, dtype=torch.float64)
    lab = torch.zeros((H, W), device=DEV, dtype=torch.int64)
    for i in range(n):
        d2 = (xs - sx[i]) ** 2 + (ys - sy[i]) ** 2
        closer = d2 < best
        best = torch.where(closer, d2, best)
        lab[closer] = i
    plane = torch.stack([t(a)[lab], t(b)[lab], t(c)[lab]], -1)
    gt = (plane[..., 0] * xs + plane[..., 1] * ys + plane[..., 2]).clamp(lo, hi)
    arg = 2 * np.pi * (xs * t(np.cos(theta))[lab] + ys * t(np.sin(theta))[lab]) / t(period)[lab] + t(phase)[lab]
    noise = torch.randn((H, W, 3), device=DEV, dtype=torch.float64, generator=gen) * 8
    left = (t(base)[lab] + noise + 20 * torch.sin(arg)[..., None]).round().clamp(0, 255).to(torch.uint8)
    # the larger disparity wins a right pixel, the lower source index among equals
    xr = (xs - gt).round().long()
    ok = (xr >= 0) & (xr < W)
    src = torch.arange(H * W, device=DEV).view(H, W)
    key = (ys.long() * W + xr)[ok]
    val = ((gt * 4096).long() << 32 | ((1 << 31) - src))[ok]
    z = torch.full((H * W,), -1, device=DEV, dtype=torch.int64).scatter_reduce(0, key, val, "amax")
    hit = z >= 0
    source = (1 << 31) - (z & 0xFFFFFFFF)
    right = torch.randint(0, 256, (H * W, 3), device=DEV, dtype=torch.uint8, generator=gen)
    right[hit] = left.view(-1, 3)[source[hit]]
    dispR = torch.zeros(H * W, device=DEV, dtype=torch.float64)
    dispR[hit] = gt.view(-1)[source[hit]]
    return left.contiguous(), right.view(H, W, 3).contiguous(), plane, gt, dispR.view(H, W)


def _network_volume(left, right, D, seed):
    """A float volume [D][H][W] in [0, 1] as a matching network gives it: the 5x5 mean of |grey - grey(x - d)| and noise."""
    gen = torch.Generator(DEV).manual_seed(seed)
    w = torch.tensor([0.114, 0.587, 0.299], device=DEV)
    gl, gr = (left.float() * w).sum(-1), (right.float() * w).sum(-1)
    H, W = gl.shape
    xs = torch.arange(W, device=DEV)
    out = torch.empty((D, H, W), device=DEV)
    for d in range(D):
        diff = (gl - gr[:, (xs - d).clamp(min=0)]).abs()
        out[d] = torch.nn.functional.avg_pool2d(diff[None, None], 5, 1, 2)[0, 0] / 48
    out += torch.randn(out.shape, device=DEV, generator=gen) * 0.02
    return out.clamp_(0, 1)


_handles = {}


def _context():
    """The one engine context that a program keeps; its slabs grow to the largest size it has seen. The BP streams
    of a batch follow the engine's fixed rule, so that a class's first batches explore nothing."""
    if "ctx" not in _handles:
        ctx = E.Context(0)
        E.lib().hbp_set_autotune(ctx.h, 0)
        _handles["ctx"] = ctx
    return _handles["ctx"]


def _server(fp16):
    if ("server", fp16) not in _handles:
        _handles["server", fp16] = E.Server(0, 24 << 30, 4, E.default_params(post=1, msg_fp16=fp16))
    return _handles["server", fp16]


def _mixed(case):
    """The sizes of a served mix: the case's own, a quarter and a ninth of its pixels, in turn."""
    W, H, D = case["W"], case["H"], case["D"]
    return [(max(64, W // k), max(48, H // k), max(16, D // k)) for k in (1 + i % 3 for i in range(case["pairs"]))]


def prepare(case, seed):
    W, H, D, kind = case["W"], case["H"], case["D"], case["kind"]
    s = {"case": case}
    if kind == SERVE:
        s["server"] = _server(case["fp16"])
        s["requests"] = []
        for i, (w, h, d) in enumerate(_mixed(case)):
            left, right = _scene(w, h, d, seed * 64 + i)[:2]
            s["requests"].append((left.cpu().numpy(), right.cpu().numpy(), d))
        return s
    s["ctx"] = _context()
    if kind in (PAIR, BATCH):
        s["prm"] = E.default_params(post=case["post"], msg_fp16=case["fp16"], linkage=case["linkage"],
                                    num_nb=case["num_nb"], sigma=case["sigma"])
    if kind == BATCH:
        pairs = [_scene(W, H, D, seed * 64 + i)[:2] for i in range(case["pairs"])]
        s["disp"] = torch.zeros((len(pairs), H, W), device=DEV)
        ptrs = lambda ts: (C.c_void_p * len(pairs))(*[t.data_ptr() for t in ts])  # noqa: E731
        s["pairs"] = pairs
        s["args"] = (ptrs([p[0] for p in pairs]), ptrs([p[1] for p in pairs]), ptrs(list(s["disp"])))
        return s
    left, right, plane, gt, dispR = _scene(W, H, max(D, 16), seed * 64)
    if kind == PAIR:
        s["left"], s["right"] = left.cpu().numpy(), right.cpu().numpy()
        return s
    s["left"], s["right"] = left, right
    f32 = lambda *shape: torch.zeros(shape, device=DEV)  # noqa: E731
    if kind == CENSUS:
        s["census"] = [torch.zeros((H, W), device=DEV, dtype=torch.int32) for _ in range(2)]
        s["vol"] = [torch.zeros(E.volume_bytes(W, H, D), device=DEV, dtype=torch.uint8) for _ in range(1 + case["right"])]
        s["wta"] = [f32(H, W) for _ in range(1 + case["right"])]
    elif kind == SUPERPIXELS:
        s["labels"] = torch.zeros((H, W), device=DEV, dtype=torch.int32)
    elif kind == MCCNN:
        s["src"] = _network_volume(left, right, D, seed * 64 + 1)
        s["vol"], s["wta"] = f32(E.volume_f32_bytes(W, H, D) // 4), f32(H, W)
        s["disp"], s["plane"] = f32(H, W), f32(H, W, 3)
        s["prm"] = E.default_params(alpha=1.3, msg_fp16=case["fp16"])
    elif kind == AD:
        s["grey"] = [f32(H, W), f32(H, W)]
        s["vol"], s["wta"] = f32(E.volume_f32_bytes(W, H, D) // 4), f32(H, W)
        s["levels"] = f32(24, H, W)  # room for the deepest pyramid; the levels past its last stay zero
        s["prm"] = E.default_params(msg_fp16=case["fp16"])
    else:  # POST: planes as HBP leaves them, an eighth of the 12 x 12 blocks on a wrong plane
        gen = torch.Generator(DEV).manual_seed(seed * 64 + 2)
        bh, bw = -(-H // 12), -(-W // 12)
        wrong = (torch.rand((bh, bw), device=DEV, generator=gen) < 0.125).float()
        shift = torch.randn((bh, bw), device=DEV, generator=gen) * 6 * wrong
        up = lambda v: v.repeat_interleave(12, 0)[:H].repeat_interleave(12, 1)[:, :W]  # noqa: E731
        pl = plane.float()
        pl[..., 2] += up(shift)
        ys, xs = torch.meshgrid(torch.arange(H, device=DEV).float(), torch.arange(W, device=DEV).float(), indexing="ij")
        s["plane0"] = pl.contiguous()
        s["dispL"] = (pl[..., 0] * xs + pl[..., 1] * ys + pl[..., 2]).clamp(0, D - 1).contiguous()
        s["dispR"] = dispR.float().contiguous()
        s["plane"], s["disp"] = torch.empty_like(s["plane0"]), f32(H, W)
        s["fail"] = torch.zeros((H, W), device=DEV, dtype=torch.uint8)
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    W, H, D, kind = case["W"], case["H"], case["D"], case["kind"]
    if kind == SERVE:
        ids = [s["server"].submit(*r) for r in s["requests"]]
        return [s["server"].wait(i)[0] for i in ids]
    ctx = s["ctx"]
    if kind == PAIR:
        return ctx.run_pair(s["left"], s["right"], D, s["prm"], want_plane=case["post"] == 2)
    if kind == BATCH:
        left, right, disp = s["args"]
        E._check(E.lib().hbp_run_batch_d(ctx.h, case["pairs"], left, right, W, H, D, C.byref(s["prm"]), disp, None))
        return s["disp"]
    if kind == CENSUS:
        volR, wtaR = (s["vol"][1], s["wta"][1]) if case["right"] else (None, None)
        ctx.cost_census_d(s["left"], s["right"], W, H, D, *s["census"], s["vol"][0], s["wta"][0], volR, wtaR)
        return {"census": s["census"], "vol": s["vol"], "wta": s["wta"]}
    if kind == SUPERPIXELS:
        ctx.segment_target_d(s["left"], W, H, case["linkage"], case["num_nb"], case["sigma"], case["target"])
        return ctx.segment_labels_d(s["labels"]), s["labels"]
    if kind == MCCNN:
        ctx.cost_f32_d(s["src"], W, H, D, 0.5, s["vol"], s["wta"])
        ctx.segment_d(s["left"], W, H)
        ctx.infer_f32_d(s["vol"], s["wta"], D, 0.5, s["prm"], s["disp"], s["plane"])
        return {"vol": s["vol"], "wta": s["wta"], "disp": s["disp"], "plane": s["plane"]}
    if kind == AD:
        ctx.cost_ad_d(s["left"], s["right"], W, H, D, *s["grey"], s["vol"], s["wta"])
        ctx.segment_d(s["left"], W, H)
        ctx.infer_levels_d(None, s["vol"], s["wta"], D, 30.0, s["prm"], 24, s["levels"])
        return {"grey": s["grey"], "vol": s["vol"], "wta": s["wta"], "levels": s["levels"]}
    s["plane"].copy_(s["plane0"])  # the post-processing works in place
    ctx.lr_check_d(s["dispL"], s["dispR"], s["plane"], s["fail"], s["disp"], W, H)
    median = ctx.weighted_median_gpu_d if case["gpu_order"] else ctx.weighted_median_d
    median(s["left"], s["fail"], s["plane"], s["disp"], W, H)
    return {"fail": s["fail"], "plane": s["plane"], "disp": s["disp"]}


# ---------------------------------------------------------------------------------------------- what a pass needs
def _bp_flops(n):
    """Data cost of BP: 12 operations per pixel, candidate plane and step; about 5.2 steps in each of the 10 + 10 l
    iterations of level l, levels 2 .. L - 2 of a pyramid that shrinks about 3.5 times a level."""
    L = max(4, round(np.log(n) / np.log(3.5)))
    return 12.0 * 4 * n * sum(5.2 * (10 + 10 * l) for l in range(2, L - 1))


def work(case):
    W, H, D, kind = case["W"], case["H"], case["D"], case["kind"]
    n = W * H
    views = 2 if case["post"] == 2 else 1
    match = 4.0 * n * D  # xor, count, compare, select per pixel and disparity
    if kind in (PAIR, BATCH, SERVE):
        sizes = _mixed(case) if kind == SERVE else [(W, H, D)] * case["pairs"]
        px = sum(w * h for w, h, _ in sizes)
        planes = 12 if kind == PAIR and case["post"] == 2 else 0
        return {"bytes": px * (6.0 + 4 + planes),
                "flops": sum(views * (4.0 * w * h * d + _bp_flops(w * h)) for w, h, d in sizes)}
    if kind == CENSUS:
        return {"bytes": n * (6.0 + 8) + (1 + case["right"]) * (4.0 * n + E.volume_bytes(W, H, D)),
                "flops": (1 + case["right"]) * match}
    if kind == SUPERPIXELS:
        return {"bytes": n * (3.0 + 4), "flops": 200.0 * n}
    if kind == MCCNN:
        return {"bytes": 4.0 * n * D + E.volume_f32_bytes(W, H, D) + n * (3.0 + 4 + 4 + 12), "flops": match + _bp_flops(n)}
    if kind == AD:
        return {"bytes": n * (6.0 + 8 + 4 + 4 * 6) + E.volume_f32_bytes(W, H, D), "flops": match + _bp_flops(n)}
    # a fifth of the pixels or so fail; each sorts or selects over a 41 x 41 window
    return {"bytes": n * (8.0 + 12 + 3 + 1 + 12 + 4), "flops": 0.2 * n * 1681 * 10}


# ---------------------------------------------------------------------------------------------- 64-bit results
def _tiled(dhw, fill=0.0):
    """[D][H][W] in the engine's tile order (8 x 4 pixels, disparity-major inside a tile)."""
    D, H, W = dhw.shape
    TX, TY = -(-W // 8), -(-H // 4)
    out = torch.full((D, TY * 4, TX * 8), fill, device=dhw.device, dtype=dhw.dtype)
    out[:, :H, :W] = dhw
    return out.view(D, TY, 4, TX, 8).permute(1, 3, 0, 2, 4).reshape(-1)


def _exact_census(case, s):
    W, H, D = case["W"], case["H"], case["D"]
    k = torch.tensor([114, 587, 299], device=DEV)
    codes = []
    for img in (s["left"], s["right"]):
        g = torch.nn.functional.pad((img.long() * k).sum(-1) // 1000, (4, 4, 3, 3))
        at = lambda r, m: g[r:r + H, m:m + W]  # noqa: E731
        code = torch.zeros((H, W), device=DEV, dtype=torch.int64)
        for bit in range(31):
            r, m = divmod(bit, 9)
            code |= (at(r, m) >= at(6 - r, 8 - m)).long() << bit
        codes.append(code)
    xs = torch.arange(W, device=DEV)

    def popcount(v):
        n = torch.zeros_like(v)
        for bit in range(31):
            n += v >> bit & 1
        return n

    vol = torch.stack([popcount(codes[0] ^ codes[1][:, (xs - d).clamp(min=0)]).clamp(max=25) for d in range(D)])
    vols = [vol]
    if case["right"]:
        vols.append(torch.stack([vol[d][:, (xs + d).clamp(max=W - 1)] for d in range(D)]))
    first = lambda v: (v * D + torch.arange(D, device=DEV)[:, None, None]).amin(0) % D  # noqa: E731
    return {"census": [c.to(torch.int32) for c in codes], "vol": [_tiled(v).to(torch.uint8) for v in vols],
            "wta": [first(v).double() for v in vols]}


def _first_min(vol):
    best, arg = vol[0].clone(), torch.zeros(vol.shape[1:], device=vol.device, dtype=torch.float64)
    for d in range(1, vol.shape[0]):
        less = vol[d] < best
        best = torch.where(less, vol[d], best)
        arg[less] = d
    return arg


def _exact_mccnn(case, s):
    D, xs = case["D"], torch.arange(case["W"], device=DEV)
    vol = torch.stack([s["src"][d][:, xs.clamp(min=d)] for d in range(D)]).clamp_(max=0.5)
    return {"vol": _tiled(vol), "wta": _first_min(vol), "disp": None, "plane": None}


def _exact_ad(case, s):
    W, H, D = case["W"], case["H"], case["D"]
    w = torch.tensor([114.0, 587.0, 299.0], device=DEV, dtype=torch.float64)
    gl, gr = ((img.double() * w).sum(-1) / 1000 for img in (s["left"], s["right"]))
    vol = torch.zeros((D, H, W), device=DEV, dtype=torch.float64)
    for d in range(D):
        vol[d, :, D - 1:] = (gl[:, D - 1:] - gr[:, D - 1 - d:W - d]).abs().clamp(max=30)
    # the winners among equal costs depend on the grey values' rounding
    return {"grey": [gl, gr], "vol": _tiled(vol), "wta": None, "levels": None}


def _exact_post(case, s):
    W, H = case["W"], case["H"]
    plane, dl, dr = s["plane0"].double(), s["dispL"].double(), s["dispR"].double()
    ys, xs = torch.meshgrid(torch.arange(H, device=DEV), torch.arange(W, device=DEV), indexing="ij")
    xr = (xs - dl + 0.5).trunc().long()
    seen = (xr >= 0) & (xr < W)
    fail = seen & ((dr.gather(1, xr.clamp(0, W - 1)) - dl).abs() > 1.5)
    near = torch.nn.functional.max_pool2d(fail[None, None].float(), 3, 1, 1)[0, 0] > 0
    # the nearest pixel on each side outside the dilated mask; the plane with the smaller disparity here
    xl = torch.where(near, -1, xs).cummax(1).values
    xh = torch.where(near, W, xs).flip(1).cummin(1).values.flip(1)
    pick = lambda x: plane[ys, x.clamp(0, W - 1)]  # noqa: E731
    z = lambda p, x, y: p[..., 0] * x + p[..., 1] * y + p[..., 2]  # noqa: E731
    pl, pr = pick(xl), pick(xh)
    use_l = (xl >= 0) & ((xh >= W) | (z(pl, xs, ys) < z(pr, xs, ys)))
    filled = torch.where(use_l[..., None], pl, pr)
    plane = torch.where((fail & ((xl >= 0) | (xh < W)))[..., None], filled, plane)
    # weighted median of the 41 x 41 window's planes at each failed pixel
    out, bgr = plane.clone(), s["left"].long()
    o = torch.arange(-20, 21, device=DEV)
    oy, ox = (v.reshape(-1) for v in torch.meshgrid(o, o, indexing="ij"))
    where = fail.nonzero()
    for f in where.split(8192):
        y, x = f[:, :1], f[:, 1:]
        qy, qx = y + oy, x + ox
        inside = (qy >= 0) & (qy < H) & (qx >= 0) & (qx < W)
        qy, qx = qy.clamp(0, H - 1), qx.clamp(0, W - 1)
        v = torch.where(inside, z(plane[qy, qx], x, y), float("inf"))
        w = torch.exp((bgr[qy, qx] - bgr[y, x]).abs().sum(-1).double() / -10) * inside
        v, at = v.sort(dim=1, stable=True)
        w = w.gather(1, at).cumsum(1)
        m = (w > w[:, -1:] / 2).int().argmax(1, keepdim=True)
        m = at.gather(1, m)
        out[f[:, 0], f[:, 1]] = plane[qy.gather(1, m)[:, 0], qx.gather(1, m)[:, 0]]
    return {"fail": (fail * 255).to(torch.uint8), "plane": out, "disp": z(out, xs, ys)}


def exact(case, seed):
    """Costs and post-processing have a plain definition. A BP result is the end of thousands of discrete choices
    (which plane a node keeps), which take minutes to follow in plain 64-bit code, and the superpixels are whole
    numbers: no value for these."""
    f = {CENSUS: _exact_census, MCCNN: _exact_mccnn, AD: _exact_ad, POST: _exact_post}.get(case["kind"])
    return f(case, prepare(case, seed)) if f else None
