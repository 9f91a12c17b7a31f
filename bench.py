#!/usr/bin/env python
"""Benchmark of the B200 HBP-ISP stereo engine.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

A step is one pass of the stereo path (census cost volume, segmentation
pyramid, hierarchical BP, driver median) over a batch of 16 synthetic
rectified pairs of 720x496 with D = 128: the quarter-scale batch workload.
The scenes are seeded piecewise-planar synthetic pairs standing in for the
Middlebury images the reference benchmarks on (data: "synthetic").

One JSON line on rank 0 (BP messages stored as FP16 unless --fp16 0):
  value       pairs/s with the pairs already in device memory (hbp_run_batch_d)
  e2e         pairs/s served through the request server's C API (hbp_submit /
              hbp_wait) from pinned host buffers, 16 requests in flight: upload,
              whole path and download of each disparity inside the timed region
  latency_ms  p50/p99 of the served requests (submit to result in host memory)
  plain_fp32  the plain FP32 single-pair path (hbp_run_pair, one pair at a
              time) on the same pairs: pairs/s and p50/p99
  roofline    the data-cost kernel (the dominant kernel): algorithmic bytes of
              its launches / their CUDA-event time over the timed region,
              against the measured HBM copy peak; traffic from the committed
              ncu capture, scaled to a 16-view launch
  cpu_baseline the CPU oracle (a port of the reference path, all host cores) on
              one pair of the same workload
  gpu_launches kernels this library launched inside the timed region
With N > 1 (torchrun), every rank runs its own 16 pairs (replicas, weak
scaling); the time is the max over ranks.

--impl reference runs the reference's own build (oracle/_ref/libhbpref.so,
compiled from the reference sources) through its classes, one pair per step,
on rank 0.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "hbp-isp_b200"))

METRIC = "pairs/s and p50/p99 latency at 720×496×D128, FP16-msg served vs plain FP32 path"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--pairs", type=int, default=16)
    ap.add_argument("--W", type=int, default=720)
    ap.add_argument("--H", type=int, default=496)
    ap.add_argument("--D", type=int, default=128)
    ap.add_argument("--fp16", type=int, default=1, help="store BP messages as FP16 (1) or FP32 (0)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--config", default="batch", choices=["batch", "uneven", "precision", "serve", "mccnn"],
                    help="batch: the contract line (16 pairs 720x496 D128); uneven: 32 pairs of mixed "
                         "sizes and disparity ranges in flight together; precision: 8 pairs 1440x992 D256, "
                         "FP16 vs FP32 messages; serve: Poisson arrivals of a size mix; mccnn: the "
                         "reference's published benchmark flow (MC-CNN volume, one view, runtime against "
                         "min_level) at a Middlebury half-resolution size")
    ap.add_argument("--rate", type=float, default=200.0, help="serve: arrivals per second")
    ap.add_argument("--duration", type=float, default=5.0, help="serve: seconds of arrivals")
    ap.add_argument("--rates", default="", help="serve: comma-separated arrival rates, one phase each "
                                                 "(a sweep; overrides --rate)")
    ap.add_argument("--p99-bound-ms", type=float, default=5000.0,
                    help="serve sweep: the p99 latency a sustainable rate must stay within")
    ap.add_argument("--profile-run", action="store_true",
                    help="skip the untimed extra batches (accuracy, isolated roofline): for profiler captures")
    ap.add_argument("--bp-streams", type=int, default=0,
                    help="BP streams of a batch (0: the engine's default; 1 for profiler captures)")
    ap.add_argument("--prep-lanes", type=int, default=8, help="served: the server's preparation lanes")
    ap.add_argument("--window", type=int, default=0,
                    help="served requests in flight (default: twice the pairs per step, so that the "
                         "next pairs are prepared while the BP of the others runs)")
    ap.add_argument("--breakdown", action="store_true",
                    help="after the timed region, one extra step with every BP kernel of every 8th "
                         "BP step event-timed; per-kernel/per-level estimate printed to stderr")
    return ap.parse_args()


class ClockSampler:
    """nvidia-smi samples during the timed region (SM clock, reasons)."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in self.lines:
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6650.0, "fallback"


def make_pairs(n, W, H, D, seed0):
    from scenes import make_scene
    return [make_scene(W, H, D, seed0 + i) for i in range(n)]


def cpu_baseline(scenes, W, H, D):
    """The CPU oracle (a port of the reference path) in its FP64 mode on the
    first two pairs, all host cores; the FP32 mode (the engine's arithmetic)
    on the first pair beside it."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as O
    cores = os.cpu_count() or 1
    t64 = []
    for s in scenes[:2]:
        t0 = time.perf_counter()
        O.driver_median(O.pipeline(s.left, s.right, D, fp64=True)["disp"])
        t64.append(time.perf_counter() - t0)
    t0 = time.perf_counter()
    O.driver_median(O.pipeline(scenes[0].left, scenes[0].right, D)["disp"])
    t32 = time.perf_counter() - t0
    seeds = ", ".join(str(s.seed) for s in scenes[:2])
    return {"value": len(t64) / sum(t64), "unit": "pairs/s", "cores": cores, "kind": "port",
            "mode": "fp64", "fp32_value": 1.0 / t32,
            "sample": f"{len(t64)} pairs {W}x{H} D{D} (seeds {seeds}) through the CPU oracle's FP64 mode, "
                      f"OpenMP on {cores} threads, {sum(t64):.1f} s; fp32_value: its FP32 mode on the "
                      f"first pair, {t32:.1f} s"}


def message_error(scene, D):
    """Lock-step message error of FP32 and FP16 message storage against FP64
    on one pair: the oracle's float run (bit-exact with the engine) with an
    FP64 shadow that takes the same candidate planes and kept slots. Each
    message is compared minus its own minimum (a per-message constant changes
    no decision); raw errors of the stored values beside."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle as O
    out = {"pair_seed": scene.seed}
    for name, fp16 in (("fp32", False), ("fp16", True)):
        _, st = O.pipeline_lockstep(scene.left, scene.right, D, fp16_msg=fp16)
        out[name] = {k: st[k] for k in ("msg_err_max", "msg_err_mean", "msg_ref_mean", "msg_ref_max",
                                        "msg_raw_err_max", "msg_raw_err_mean", "values")}
    return out


# DRAM bytes (read + write) per unit of one launch, from the committed ncu
# captures of 8-view 720x496 D128 launches (profiles/k_*_8x720x496_d128.md):
# k_cost per list position (the mean of its level-2 and level-5 captures,
# 185.8 and 140.7 MB), k_edges per directed edge (level 2, 62.7 MB for
# 4856 blocks of 128).
KCOST_DRAM_BYTES_PER_PIXEL = (185.8e6 + 140.7e6) / 2 / (8 * 357120)
KEDGES_DRAM_BYTES_PER_EDGE = 62.7e6 / (4856 * 128)


KERNEL_NAMES = {"k_edges": "k_edges (message passing, smoothing and normalisation, one thread per "
                           "directed edge; four lanes on small launches)",
                "k_cost": "k_cost (data cost of 4 candidate planes per pixel)"}


def read_kernel_profiles(E, ctx):
    """Summed device ms, launches, algorithmic bytes and units of the event-
    timed k_cost and k_edges launches (every 16th BP tick of the first BP
    stream) since profiling was enabled."""
    import ctypes as C
    out = {}
    for kid, name in ((0, "k_cost"), (1, "k_edges")):
        ms, n, b, u = C.c_double(), C.c_long(), C.c_double(), C.c_double()
        E._check(E.lib().hbp_profile_read_kernel(ctx.h, kid, C.byref(ms), C.byref(n), C.byref(b), C.byref(u)))
        out[name] = (ms.value, n.value, b.value, u.value)
    return out


def autotune_settled(E, ctx, key):
    """Whether the BP-stream autotuner has chosen for the workload class key
    (W, H, D, msg_fp16, post, views)."""
    import ctypes as C
    n = E.lib().hbp_autotune_table(ctx.h, None, 0)
    if n <= 0:
        return False
    buf = (C.c_double * (9 * n))()
    E.lib().hbp_autotune_table(ctx.h, buf, n)
    return any(tuple(int(x) for x in buf[9 * i:9 * i + 6]) == tuple(key) and buf[9 * i + 8] > 0 for i in range(n))


def autotune_rows(E, ctx, explore):
    """The BP-stream autotuner's measurements for this context (hbp_autotune_table)."""
    import ctypes as C
    n = E.lib().hbp_autotune_table(ctx.h, None, 0)
    if n <= 0:
        return None
    buf = (C.c_double * (9 * n))()
    E.lib().hbp_autotune_table(ctx.h, buf, n)
    rows = [list(buf[9 * i:9 * i + 9]) for i in range(n)]
    classes = {}
    for r in rows:
        key = (int(r[0]), int(r[1]), int(r[2]), int(r[3]), int(r[4]), int(r[5]))
        classes.setdefault(key, []).append({"streams": int(r[6]), "bp_ms_per_view": round(r[7], 3),
                                            "chosen": bool(r[8])})
    return {"exploration_batches": explore,
            "classes": [{"W": k[0], "H": k[1], "D": k[2], "msg_fp16": k[3], "post": k[4], "views": k[5],
                         "tried": v} for k, v in classes.items()]}


def roofline_entry(name, prof, peak, peak_kind, hw, where):
    """achieved = the timed launches' algorithmic bytes / their device time;
    traffic = the committed ncu capture's DRAM bytes per unit, times the units
    of an average timed launch."""
    ms, n, b, u = prof
    if ms <= 0 or n <= 0:
        return None
    achieved = b / (ms / 1e3) / 1e9
    per_unit = KCOST_DRAM_BYTES_PER_PIXEL if name == "k_cost" else KEDGES_DRAM_BYTES_PER_EDGE
    e = {"kernel": KERNEL_NAMES[name] + (", timed region: the first of the concurrent BP streams" if where == "live"
                                         else ", BP on one stream (the kernel alone on the device)"),
         "bound": "hbm", "achieved": achieved, "peak": peak, "peak_kind": peak_kind, "unit": "GB/s",
         "frac": achieved / peak, "traffic": per_unit * u / n,
         "traffic_source": f"ncu dram__bytes_read+write per {'list position' if name == 'k_cost' else 'edge'} "
                           f"of an 8-view 720x496 D128 capture (profiles/), times the units of an average "
                           f"timed launch",
         "algorithmic_bytes_per_launch": b / n, "launches_timed": n, "avg_launch_us": 1e3 * ms / n}
    if name == "k_cost":
        e["views_per_launch"] = u / n / hw
    else:
        e["edges_per_launch"] = u / n
        e["note"] = ("instruction-issue bound (ncu: issue slots busy, DRAM a few %), so its HBM fraction "
                     "is low by construction; the issue figures are in profiles/")
    return e


def max_over_ranks(x: float, dist, device) -> float:
    """The slowest rank's duration (every rank gets it); x itself without a
    process group."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(pairs_per_rank: int, steps: int, world: int, seconds: float) -> float:
    """pairs/s of the whole job: every rank's pairs over the slowest rank's time."""
    return pairs_per_rank * steps * world / seconds


KINDS = ["node_select", "", "", "spatial_cand", "data_cost", "edge_msgs",
         "prior_cost", "init_nodes", "map", "cost_edges"]


def breakdown(E, ctx, step):
    """One untimed step with the BP on one stream and its kernels event-timed
    (mode 3): estimated device ms per step by kernel kind and by (kind,
    pyramid level)."""
    import ctypes as C
    n = 10 * 32
    ms, timed, allc = (C.c_double * n)(), (C.c_long * n)(), (C.c_long * n)()
    E._check(E.lib().hbp_set_bp_streams(ctx.h, 1))  # kernels alone: times add up
    E._check(E.lib().hbp_profile_enable(ctx.h, 3))
    step()
    E._check(E.lib().hbp_profile_breakdown(ctx.h, ms, timed, allc))
    E._check(E.lib().hbp_profile_enable(ctx.h, 0))
    E._check(E.lib().hbp_set_bp_streams(ctx.h, 0))
    by_kind, by_level = {}, {}
    for k, name in enumerate(KINDS):
        for lv in range(32):
            i = k * 32 + lv
            if allc[i] == 0 or timed[i] == 0:
                continue
            est = ms[i] / timed[i] * allc[i]
            by_kind[name] = by_kind.get(name, 0.0) + est
            by_level.setdefault(str(lv), {})[name] = {"est_ms": round(est, 3), "launches": allc[i],
                                                      "avg_us": round(1e3 * ms[i] / timed[i], 2)}
    return {"breakdown_est_ms_per_step": {k: round(v, 3) for k, v in by_kind.items()},
            "total_est_ms": round(sum(by_kind.values()), 3), "by_level": by_level}


def run_reference(args, rank):
    """Reference arm: the reference's own build on the pairs of this workload."""
    if rank != 0:
        return
    import ctypes as C
    lib_path = os.path.join(ROOT, "oracle", "_ref", "libhbpref.so")
    if not os.path.exists(lib_path):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libhbpref.so not built "
                          "(make -C oracle/ref needs the reference sources)"}))
        return
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    sys.path.insert(0, os.path.join(ROOT, "tests", "golden"))
    import pyoracle as O
    from make_golden import RefLib
    ref = RefLib(lib_path)
    if args.config == "mccnn":
        run_reference_mccnn(ref)
        return
    W, H, D = args.W, args.H, args.D
    scenes = make_pairs(args.warmup + args.steps, W, H, D, 1000)
    times = []
    for i, s in enumerate(scenes):
        t0 = time.perf_counter()
        disp, _, _ = ref.hbp_pair(s.left, s.right, D)
        O.driver_median(disp)
        dt = time.perf_counter() - t0
        if i >= args.warmup:
            times.append(dt)
    tot = sum(times)
    lat = sorted(t * 1e3 for t in times)
    # the reference's step times have a long tail (its host syncs and
    # allocations per pair): the value is the median step's rate, the mean's
    # beside it
    p50 = lat[len(lat) // 2] if len(lat) % 2 else 0.5 * (lat[len(lat) // 2 - 1] + lat[len(lat) // 2])
    val = 1e3 / p50
    out = {
        "metric": METRIC, "value": val, "unit": "pairs/s", "n_gpus": 1, "steps": args.steps,
        "value_kind": "1 / median step time", "mean_value": len(times) / tot,
        "warmup": args.warmup, "ms_per_step": 1e3 * tot / len(times), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
        "config": {"workload": f"1 synthetic pair {W}x{H} D{D} per step (sample of the 16-pair batch), "
                               "reference build (its CUDA kernels, SegHAC/StereoCost/HBP_ISP classes) "
                               "+ driver median", "W": W, "H": H, "D": D},
        "latency_ms": {"p50": lat[len(lat) // 2], "p99": lat[min(len(lat) - 1, int(0.99 * len(lat)))]},
        "cpu_baseline": {"value": val, "unit": "pairs/s", "cores": 1, "kind": "reference",
                         "sample": f"one pair per step through the reference's own build, driven by one "
                                   f"host thread, {len(times)} steps, median step; the reference runs this "
                                   f"path as CUDA kernels on the GPU"},
        "e2e": {"value": val, "unit": "pairs/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(out))


def run_reference_mccnn(ref):
    """The reference build on the published MC-CNN flow, the same synthetic view and volume
    as run_mccnn: its StereoCost reads the volume from a raw file, then HBP_ISP::run_ms per
    min_level, timed over the scope its benchmark times (HBP_ISP construction + run_ms,
    main_bench_middv3.cu:97-104); median of 2 runs."""
    import ctypes as C
    import torch
    ref.lib.ref_last_hbp_ms.restype = C.c_double
    s, src_d, W, H, D = mccnn_workload(torch)
    src = src_d.cpu().numpy()
    del src_d
    out = {}
    _, _, _, _, levels = ref.hbp_f32(s.left, s.right, src, min_level=2)  # warm-up; pyramid depth
    for m in sorted(PUBLISHED_ADIRONDACK_S, reverse=True):
        if m > levels - 1:
            continue
        ts = []
        for _ in range(2):
            _, _, disp, _, levels = ref.hbp_f32(s.left, s.right, src, min_level=m)
            ts.append(ref.lib.ref_last_hbp_ms())
        bad2 = 100.0 * float(np.mean(np.abs(disp - s.gt)[s.nonocc] > 2.0))
        out[str(m)] = {"hbp_ms": sorted(ts)[0], "bad2_pct": bad2,
                       "published_titan_xp_ms": PUBLISHED_ADIRONDACK_S[m] * 1e3}
    print(json.dumps({"impl": "reference", "config": "mccnn", "levels": levels, "by_min_level": out,
                      "workload": f"1 synthetic view {W}x{H} D{D}, synthetic MC-CNN-like volume, "
                                  "reference build on this GPU, FP32"}))


# runtime.png of the reference (README.md:17-18): Adirondack at trainingH, seconds per view
# on a Titan Xp for min_level 9, 8, ..., 1 (read from the plot, about +-0.03 s)
PUBLISHED_ADIRONDACK_S = {9: 0.42, 8: 0.80, 7: 1.18, 6: 1.61, 5: 2.00, 4: 2.42, 3: 3.05, 2: 4.12, 1: 5.36}


def mccnn_workload(torch):
    """The synthetic stand-in for a Middlebury half-resolution view with its MC-CNN volume:
    a 1440x992 scene (D 144, Adirondack's trainingH size) and a float volume [D][H][W] on
    the device, the 5x5 mean of the grey difference / 48 plus noise, clipped to [0, 1]."""
    from scenes import make_scene
    W, H, D = 1440, 992, 144
    s = make_scene(W, H, D, 8000)
    w = torch.tensor([0.114, 0.587, 0.299], device="cuda")
    gl = torch.from_numpy(s.left).cuda().float() @ w
    gr = torch.from_numpy(s.right).cuda().float() @ w
    xs = torch.arange(W, device="cuda")
    src = torch.empty((D, H, W), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(8001)
    for d in range(D):
        diff = (gl - gr[:, (xs - d).clamp(min=0)]).abs()[None, None]
        src[d] = torch.nn.functional.avg_pool2d(diff, 5, 1, 2, count_include_pad=False)[0, 0] / 48.0
    src += 0.02 * torch.randn(src.shape, device="cuda", generator=gen)
    src.clamp_(0.0, 1.0)
    torch.cuda.synchronize()
    return s, src, W, H, D


def run_mccnn(args, E, torch, local, bad):
    """The flow the reference publishes runtimes for (main_bench_middv3.cu:73-108 with
    cost "MC-CNN", bench_MiddV3_train.sh: alpha 1.3, tau_smooth 0.6): SegHAC on the left
    image, the MC-CNN volume, HBP_ISP::run_ms(min_level), for min_level 9 down to 1, on
    mccnn_workload(). Per min_level: "hbp_ms", the HBP alone (the scope the reference's
    benchmark times, main_bench_middv3.cu:97-104), and "ms", segmentation + volume ingest +
    HBP; medians of 3 runs, device-resident inputs."""
    s, src, W, H, D = mccnn_workload(torch)
    ctx = E.Context(local, W * H, D)
    vol = torch.empty(E.volume_f32_bytes(W, H, D) // 4, device="cuda")
    wta = torch.empty(H * W, device="cuda")
    disp = torch.empty(H * W, device="cuda")
    dl = torch.from_numpy(s.left).cuda()
    out = {}
    try:
        L = ctx.segment_d(dl, W, H)
        for m in sorted(PUBLISHED_ADIRONDACK_S, reverse=True):
            if m > L - 1:
                continue
            row = {}
            for name, f16 in (("fp32", 0), ("fp16", 1)):
                prm = E.default_params(alpha=1.3, min_level=m, msg_fp16=f16, post=0)
                ts, th = [], []
                for rep in range(4):
                    torch.cuda.synchronize()
                    t0 = time.perf_counter()
                    ctx.segment_d(dl, W, H)
                    ctx.cost_f32_d(src, W, H, D, 0.5, vol, wta)
                    torch.cuda.synchronize()
                    t1 = time.perf_counter()
                    ctx.infer_f32_d(vol, wta, D, 0.5, prm, disp)
                    torch.cuda.synchronize()
                    t2 = time.perf_counter()
                    if rep:
                        ts.append((t2 - t0) * 1e3)
                        th.append((t2 - t1) * 1e3)
                d = disp.cpu().numpy().reshape(H, W)
                row[name] = {"ms": sorted(ts)[1], "hbp_ms": sorted(th)[1], "bad2_pct": bad(d, s, 2.0)}
            row["published_titan_xp_ms"] = PUBLISHED_ADIRONDACK_S[m] * 1e3
            row["speedup_fp32_vs_published"] = row["published_titan_xp_ms"] / row["fp32"]["hbp_ms"]
            out[str(m)] = row
    finally:
        ctx.close()
    return {"config": "mccnn", "workload": f"1 synthetic view {W}x{H} D{D} with a synthetic MC-CNN-like "
                                           "float volume; segmentation + ingest + HBP per min_level",
            "levels": L, "by_min_level": out,
            "published": "runtime.png (README.md:17-18), Adirondack trainingH, Titan Xp; not the same "
                         "image: a size-matched comparison, not a like-for-like one"}


def run_config(args, E, torch):
    """The other workloads (one JSON line each, not the contract line)."""
    from scenes import make_scene
    local = int(os.environ.get("LOCAL_RANK", "0"))
    bad = lambda d, s, t: 100.0 * float(np.mean(np.abs(d - s.gt)[s.nonocc] > t))
    if args.config == "uneven":
        rng = np.random.default_rng(7)
        sizes = [(450, 375), (720, 496), (1080, 744), (1440, 992)]
        work = []
        for i in range(32):
            W, H = sizes[rng.integers(4)]
            D = int(rng.choice([64, 128, 192, 256]))
            work.append((make_scene(W, H, D, 5000 + i), D))
        prm = E.default_params(msg_fp16=args.fp16, post=1)
        srv = E.Server(local, budget_bytes=120 << 30, prep_lanes=8, params=prm)
        try:
            for s, D in work[:4]:  # warm-up
                srv.wait(srv.submit(s.left, s.right, D))
            t0 = time.perf_counter()
            ids = [srv.submit(s.left, s.right, D) for s, D in work]
            lat = sorted(srv.wait(i)[1] for i in ids)
            el = time.perf_counter() - t0
        finally:
            srv.close()
        px = sum(s.left.shape[0] * s.left.shape[1] for s, _ in work)
        return {"config": "uneven", "pairs": 32, "value": 32 / el, "unit": "pairs/s",
                "mpixels_per_s": px / el / 1e6, "seconds": el,
                "latency_ms": {"p50": lat[len(lat) // 2], "p99": lat[-1]},
                "workload": "32 synthetic pairs, sizes from {450x375, 720x496, 1080x744, 1440x992}, D from "
                            "{64,128,192,256}, submitted together to the request server (seed 7)",
                "msg": "fp16" if args.fp16 else "fp32"}
    if args.config == "precision":
        W, H, D, n = 1440, 992, 256, 8
        scenes = [make_scene(W, H, D, 6000 + i, n_seg=40) for i in range(n)]
        ctx = E.Context(local, W * H, D)
        import ctypes as C
        dL = [torch.from_numpy(s.left).cuda() for s in scenes]
        dR = [torch.from_numpy(s.right).cuda() for s in scenes]
        out = [torch.empty((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
        arr = lambda ts: (C.c_void_p * n)(*[t.data_ptr() for t in ts])
        res = {}
        for name, f16 in (("fp32", 0), ("fp16", 1)):
            prm = E.default_params(msg_fp16=f16, post=1)
            for _ in range(7):  # warm-up, and the BP-stream autotuner's candidates (2, 3, 4) twice
                E._check(E.lib().hbp_run_batch_d(ctx.h, n, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            E._check(E.lib().hbp_run_batch_d(ctx.h, n, arr(dL), arr(dR), W, H, D, C.byref(prm), arr(out), None))
            torch.cuda.synchronize()
            el = time.perf_counter() - t0
            d = [t.cpu().numpy() for t in out]
            res[name] = {"pairs_per_s": n / el, "disp": d,
                         "bad1_pct": float(np.mean([bad(x, s, 1.0) for x, s in zip(d, scenes)])),
                         "bad2_pct": float(np.mean([bad(x, s, 2.0) for x, s in zip(d, scenes)]))}
        same = [float(np.mean(a == b)) for a, b in zip(res["fp16"]["disp"], res["fp32"]["disp"])]
        for r in res.values():
            r.pop("disp")
        out = {"config": "precision", "workload": f"{n} synthetic pairs {W}x{H} D{D}, 40 segments, "
                                                  "hbp_run_batch_d", "fp32": res["fp32"], "fp16": res["fp16"],
               "fp16_vs_fp32_identical_mean": float(np.mean(same)),
               "fp16_vs_fp32_identical_min": float(np.min(same)),
               "autotune": autotune_rows(E, ctx, 7)}
        if not args.no_cpu_baseline:
            out["message_error_vs_fp64"] = message_error(scenes[0], D)
        ctx.close()
        return out
    if args.config == "mccnn":
        return run_mccnn(args, E, torch, local, bad)
    # serve: Poisson arrivals of the size mix, FP16 messages, 120 GB budget;
    # --rates runs one arrival phase per rate on the same server
    mix = [((450, 375, 64), 0.4), ((720, 496, 128), 0.3), ((1440, 992, 256), 0.2), ((2880, 1984, 384), 0.1)]
    kinds = [m for m, _ in mix]
    pool = {k: make_scene(k[0], k[1], k[2], 7000 + i) for i, k in enumerate(kinds)}
    rates = [float(r) for r in args.rates.split(",")] if args.rates else [args.rate]
    prm = E.default_params(msg_fp16=1, post=1)
    srv = E.Server(local, budget_bytes=120 << 30, prep_lanes=8, params=prm)
    phases = []
    try:
        for k in kinds:  # warm-up, one of each size
            s = pool[k]
            srv.wait(srv.submit(s.left, s.right, k[2]))
        for ri, rate in enumerate(rates):
            rng = np.random.default_rng(11 + ri)
            n_req = max(1, int(rate * args.duration))
            gaps = rng.exponential(1.0 / rate, n_req)
            pick = rng.choice(len(kinds), n_req, p=[p for _, p in mix])
            t0 = time.perf_counter()
            t_next = t0
            ids = []
            for g, j in zip(gaps, pick):
                t_next += g
                dt = t_next - time.perf_counter()
                if dt > 0:
                    time.sleep(dt)
                s = pool[kinds[j]]
                ids.append((srv.submit(s.left, s.right, kinds[j][2]), j))
            t_arr = time.perf_counter() - t0
            lat = [srv.wait(i)[1] for i, _ in ids]
            el = time.perf_counter() - t0
            ls = sorted(lat)
            per = {}
            for (i, j), l in zip(ids, lat):
                per.setdefault(f"{kinds[j][0]}x{kinds[j][1]}xD{kinds[j][2]}", []).append(l)
            px = sum(kinds[j][0] * kinds[j][1] for _, j in ids)
            phases.append({"offered_rate": rate, "arrival_seconds": t_arr, "requests": n_req,
                           "completed_per_s": n_req / el, "mpixels_per_s": px / el / 1e6,
                           "seconds_to_drain": el,
                           "latency_ms": {"p50": ls[len(ls) // 2], "p99": ls[min(len(ls) - 1, int(0.99 * len(ls)))]},
                           "latency_p50_by_size_ms": {k: sorted(v)[len(v) // 2] for k, v in per.items()}})
    finally:
        srv.close()
    out = {"config": "serve", "phases": phases,
           "workload": "Poisson arrivals; 40% 450x375 D64, 30% 720x496 D128, 20% 1440x992 D256, "
                       "10% 2880x1984 D384; FP16 messages; 120 GB admission budget (seeds 11+)"}
    if len(rates) > 1:
        bound = args.p99_bound_ms
        ok = [p["offered_rate"] for p in phases if p["latency_ms"]["p99"] <= bound]
        out["p99_bound_ms"] = bound
        out["highest_rate_within_bound"] = max(ok) if ok else None
    return out


def main():
    args = parse()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return
    import torch
    import hbp_b200 as E

    torch.cuda.set_device(local)
    if args.config != "batch":
        if rank == 0:
            print(json.dumps(run_config(args, E, torch)))
        return
    dist = None
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))
    W, H, D, NP = args.W, args.H, args.D, args.pairs
    scenes = make_pairs(NP, W, H, D, 1000 + rank * NP)
    ctx = E.Context(local, W * H, D)
    stream = torch.cuda.ExternalStream(ctx.stream)
    prm = E.default_params(msg_fp16=args.fp16, post=1)

    dL = [torch.from_numpy(s.left).cuda() for s in scenes]
    dR = [torch.from_numpy(s.right).cuda() for s in scenes]
    disp = [torch.empty((H, W), dtype=torch.float32, device="cuda") for _ in scenes]
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")  # > 126 MB L2
    import ctypes as C
    arrL = (C.c_void_p * NP)(*[t.data_ptr() for t in dL])
    arrR = (C.c_void_p * NP)(*[t.data_ptr() for t in dR])
    arrD = (C.c_void_p * NP)(*[t.data_ptr() for t in disp])

    E._check(E.lib().hbp_set_bp_streams(ctx.h, args.bp_streams))

    def step():
        E._check(E.lib().hbp_run_batch_d(ctx.h, NP, arrL, arrR, W, H, D, C.byref(prm), arrD, None))

    # the BP stream autotuner explores its candidates on the first batches of
    # this workload (untimed, before the warm-up); later batches use its choice
    explore = 0
    if args.bp_streams == 0:
        while explore < 16 and not autotune_settled(E, ctx, (W, H, D, args.fp16, 1, NP)):
            step()
            explore += 1
    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()

    # ------------------------------------------------------------ timed region
    clocks = ClockSampler(local)
    clocks.start()
    E._check(E.lib().hbp_profile_enable(ctx.h, 2))
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    l0 = E.lib().hbp_launch_count()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    for k in range(args.steps):
        with torch.cuda.stream(stream):
            flush.random_(0, 255)  # evict L2 between steps (not timed)
            ev[k][0].record(stream)
        step()
        with torch.cuda.stream(stream):
            ev[k][1].record(stream)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    launches = E.lib().hbp_launch_count() - l0
    clk = clocks.stop()
    ph = (C.c_double * 4)()
    E._check(E.lib().hbp_last_phase_ms(ctx.h, ph))
    phases = {"prepare": ph[0], "bp": ph[1], "post": ph[2], "total": ph[3]}
    ms = sum(a.elapsed_time(b) for a, b in ev)
    live = read_kernel_profiles(E, ctx)
    E._check(E.lib().hbp_profile_enable(ctx.h, 0))

    # the same kernel alone on the device: one more batch (untimed) with the
    # BP on a single stream, every 16th data-cost launch event-timed
    iso = None
    if rank == 0 and not args.profile_run:
        E._check(E.lib().hbp_set_bp_streams(ctx.h, 1))
        E._check(E.lib().hbp_profile_enable(ctx.h, 2))
        with torch.cuda.stream(stream):
            flush.random_(0, 255)
        step()
        iso = read_kernel_profiles(E, ctx)
        E._check(E.lib().hbp_profile_enable(ctx.h, 0))
        E._check(E.lib().hbp_set_bp_streams(ctx.h, args.bp_streams))
    t_max = max_over_ranks(ms, dist, "cuda")
    value = whole_job_rate(NP, args.steps, world, t_max / 1e3)

    # accuracy of the FP16 messages at this workload: the same batch with FP32
    # messages, pixel agreement and bad-2.0 against the generator's ground truth
    accuracy = None
    if args.fp16 and rank == 0 and not args.profile_run:
        prm32 = E.default_params(msg_fp16=0, post=1)
        d16 = [t.cpu().numpy() for t in disp]
        E._check(E.lib().hbp_run_batch_d(ctx.h, NP, arrL, arrR, W, H, D, C.byref(prm32), arrD, None))
        torch.cuda.synchronize()
        d32 = [t.cpu().numpy() for t in disp]
        bad2 = lambda d, s: 100.0 * float(np.mean(np.abs(d - s.gt)[s.nonocc] > 2.0))
        same = [float(np.mean(a == b)) for a, b in zip(d16, d32)]
        accuracy = {"fp16_vs_fp32_identical_mean": float(np.mean(same)),
                    "fp16_vs_fp32_identical_min": float(np.min(same)),
                    "bad2_fp32_pct": float(np.mean([bad2(d, s) for d, s in zip(d32, scenes)])),
                    "bad2_fp16_pct": float(np.mean([bad2(d, s) for d, s in zip(d16, scenes)])),
                    "pairs": NP}
        # the CPU oracle's lock-step run takes a minute or two: at N = 1 only,
        # like the CPU baseline, so no rank waits that long at a barrier
        if not args.no_cpu_baseline and world == 1:
            accuracy["message_error_vs_fp64"] = message_error(scenes[0], D)

    if args.breakdown and rank == 0:
        print(json.dumps(breakdown(E, ctx, step)), file=sys.stderr)

    # ------------------------------------------------------------ end to end
    # Served: the same pairs through the request server's C API from pinned
    # host buffers (upload, whole path, download of the disparity inside the
    # timed region), a closed loop keeping NP requests in flight.
    e2e = None
    lat = []
    plain = None
    if not args.no_e2e:
        pinL = [torch.from_numpy(s.left).pin_memory().numpy() for s in scenes]
        pinR = [torch.from_numpy(s.right).pin_memory().numpy() for s in scenes]
        srv = E.Server(local, budget_bytes=120 << 30, prep_lanes=args.prep_lanes, params=prm)
        try:
            ids = [srv.submit(pinL[i], pinR[i], D) for i in range(NP)]  # warm-up
            for i in ids:
                srv.wait(i)
            if dist:
                dist.barrier()
            # a closed loop that refills as soon as any request completes; enough
            # requests (40 batches' worth) that the ramp-up and the final drain
            # (in-flight count rising from and falling to 0) are a small part
            # of the timed region
            n_req = max(NP * args.steps, 40 * NP)
            window = args.window or 2 * NP
            t0 = time.perf_counter()
            inflight = []
            k = 0
            while k < n_req or inflight:
                while k < n_req and len(inflight) < window:
                    inflight.append(srv.submit(pinL[k % NP], pinR[k % NP], D))
                    k += 1
                done = [i for i in inflight if srv.poll(i)]
                if not done:
                    done = [inflight[0]]  # block on the oldest
                for i in done:
                    lat.append(srv.wait(i)[1])
                    inflight.remove(i)
            el = time.perf_counter() - t0
        finally:
            srv.close()
        el = max_over_ranks(el, dist, "cuda")
        e2e = {"value": whole_job_rate(n_req, 1, world, el), "unit": "pairs/s",
               "h2d_bytes_per_step": NP * 2 * 3 * W * H, "d2h_bytes_per_step": NP * 4 * W * H,
               "requests": n_req,
               "path": f"hbp_submit/hbp_poll/hbp_wait, {n_req} requests, {window} in flight (refilled on "
                       "each completion), messages " + ("fp16" if args.fp16 else "fp32")}
        # the plain FP32 single-pair path (hbp_run_pair, one pair at a time)
        prm32 = E.default_params(msg_fp16=0, post=1)
        out = np.zeros((H, W), np.float32)
        ctx.run_pair(pinL[0], pinR[0], D, prm32)
        plat = []
        t0 = time.perf_counter()
        for k in range(NP):
            a = time.perf_counter()
            E._check(E.lib().hbp_run_pair(ctx.h, pinL[k].ctypes.data_as(C.c_void_p),
                                          pinR[k].ctypes.data_as(C.c_void_p), W, H, D, C.byref(prm32),
                                          out.ctypes.data_as(C.c_void_p), None))
            plat.append((time.perf_counter() - a) * 1e3)
        pel = time.perf_counter() - t0
        plat.sort()
        plain = {"value": NP / pel, "unit": "pairs/s", "p50_ms": plat[len(plat) // 2],
                 "p99_ms": plat[min(len(plat) - 1, int(0.99 * len(plat)))],
                 "path": "hbp_run_pair, FP32 messages, one pair at a time, pinned host buffers"}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(scenes, W, H, D)

    if rank == 0:
        peak, peak_kind = peaks()
        live_roof = {k: roofline_entry(k, v, peak, peak_kind, W * H, "live") for k, v in live.items()}
        iso_roof = {k: roofline_entry(k, v, peak, peak_kind, W * H, "isolated") for k, v in iso.items()} \
            if iso else None
        # the dominant kernel: the larger share of the timed launches' device time
        dom = max(live_roof, key=lambda k: live[k][0])
        lat.sort()
        line = {
            "metric": METRIC,
            "value": value,
            "unit": "pairs/s",
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": t_max / args.steps,
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f16-msg" if args.fp16 else "f32",
            "data": "synthetic",
            "config": {"workload": f"{NP} synthetic pairs {W}x{H} D{D} per step: census cost volume, "
                                   "segmentation pyramid, HBP (min_level 2), driver median",
                       "pairs_per_step": NP, "W": W, "H": H, "D": D,
                       "msg": "fp16" if args.fp16 else "fp32", "parallelism": f"replicas x{world}",
                       "l2": "256 MiB buffer written between timed steps"},
            "latency_ms": {"p50": lat[len(lat) // 2] if lat else None,
                           "p99": lat[min(len(lat) - 1, int(0.99 * len(lat)))] if lat else None,
                           "of": "served requests, submit to result in host memory"},
            "plain_fp32": plain,
            "accuracy": accuracy,
            "roofline": live_roof[dom],
            "roofline_kernels": {"live": live_roof, "isolated": iso_roof,
                                 "device_ms_timed": {k: v[0] for k, v in live.items()}},
            "cpu_baseline": cpu,
            "clocks": clk,
            "e2e": e2e,
            "gpu_launches": launches,
            "phase_ms_last_step": phases,
            "autotune": autotune_rows(E, ctx, explore),
        }
        print(json.dumps(line))
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    ctx.close()


if __name__ == "__main__":
    main()
