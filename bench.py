"""Render benchmark: Mrays/s of the hybrid kd-tree Gaussian ray tracer.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--config NAME] [--impl ours|reference]

A step renders one batch of views of a resident scene.  Configurations:

  scale     (default) 1M-Gaussian cluster+shell scene, one 1920x1080 view;
            the line also carries two short legs on the same GPU: the
            64-view batch of the same scene (`legs.batching`) and the
            serving loop at one request rate (`legs.serving`)
  small     100k Gaussians uniform in the unit cube, one 256x256 view
  batching  the 1M scene, 64 views on spheres of radius 2-4 (16 each at
            256x256, 640x480, 1280x720, 1920x1080) in one persistent launch
  precision 3M Gaussians (256 clusters), 8 views at 1080p, BF16 SH and FP16
            shape arrays with FP32 arithmetic
  serving   4 resident scenes (0.5M/1M/2M/3M), Poisson request streams at
            --rates req/s; p50/p99 latency of the serving loop against the
            plain per-request path
  serving_1080p  the same for the scale scene alone, requests of 1-16
            1920x1080 views
  build     kd-tree build time of the scale scene: device builder against
            the host builder, trees compared word for word
  hybrid    secondary-ray renderer on the scale scene (demo spheres and a
            mirror quad), against the plain render of the same view
Every render line carries `accuracy`: max and RMS RGB error of the batched
frame and of the plain kernel against the FP64 oracle on a ray sample, and
the plain kernel against the oracle-matching FP32 oracle (expected 0).

The batched configuration is the autotuner's (kdgr_autotune), re-ranked:
its three fastest variants are timed again under the timed region's
conditions (L2 flushed before each step) and the fastest is used
(`autotune_reranked` lists both times).
`value` is the batched (persistent, CUDA-graph) form with the scene resident
in HBM, timed with CUDA events per step with an L2 flush (a 512 MB write)
between steps.  `e2e` is the same metric through the C ABI
(kdgr_render_batch) timed on the host clock: from the call (cameras in host
memory) to the frame being readable in pinned host memory, with no other
work on the GPU (the L2 flush runs and completes before the clock starts).
`roofline` is the issue-rate bound the kernel has (it is not bandwidth
bound: its working set stays in L2): warp instructions per launch (from the
ncu capture of the same launch, profiles/instructions.txt) over the
measured kernel time, against 4 warp instructions per SM per cycle at the
SM clock sampled during the timed region.  `roofline.memory` keeps the
algorithmic bytes (L1/L2 demand) and the DRAM bytes of that capture.

`--impl reference` times the reference algorithm's CPU implementation (the
oracle transcription of cudaRenderer.cu, all host threads) on a strided ray
sample of the same workload.  Its process loads only the oracle: the scene
and its kd-tree are prepared by an untimed child process (seeded generation
and the host kd-tree builder, whose trees are byte-identical to the
reference builder's) and read back from files (the tree through the
oracle's .kdt reader).  Multi-GPU: scene replicas, no collective in the data
path (views are independent), weak scaling.
"""
from __future__ import annotations

import argparse
import collections
import importlib
import json
import os
import shutil
import statistics
import subprocess
import sys
import tempfile
import time
from types import SimpleNamespace

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)

METRIC = "Mrays/s at 1080p/1M Gaussians"
UNIT = "Mrays/s"
PEAKS = os.path.join(REPO, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6800.0
PKG = "3dgrt_kdtree_gb300"


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def _scenes():
    """The seeded scene generator (numpy only)."""
    return importlib.import_module(PKG + ".scenes")


# ------------------------------------------------------------------ workload
def make_workload(sc, name: str):
    if name == "small":
        rec = sc.uniform_cube(100_000, seed=0)
        cams = [(sc.front_camera(256, 256), 256, 256)]
        desc = {"workload": "uniform cube, 100k Gaussians, 1 view 256x256", "gaussians": 100_000}
    elif name == "scale":
        rec = sc.cluster_shell(1_000_000, seed=1)
        cams = [(sc.front_camera(1920, 1080), 1920, 1080)]
        desc = {"workload": "cluster+shell, 1M Gaussians, 1 view 1920x1080", "gaussians": 1_000_000}
    elif name == "mid":
        rec = sc.cluster_shell(300_000, seed=1, n_clusters=64)
        cams = [(sc.front_camera(1280, 720), 1280, 720)]
        desc = {"workload": "cluster+shell, 300k Gaussians, 1 view 1280x720", "gaussians": 300_000}
    elif name == "batching":
        rec = sc.cluster_shell(1_000_000, seed=1)
        cams = batching_cameras(sc)
        desc = {"workload": "cluster+shell, 1M Gaussians, 64 mixed-resolution views", "gaussians": 1_000_000}
    elif name == "precision":
        rec = sc.cluster_shell(3_000_000, seed=2, n_clusters=256)
        cams = sc.sphere_cameras(8, seed=12, resolutions=[(1920, 1080)], r_lo=2.5, r_hi=3.5)
        desc = {"workload": "cluster+shell, 3M Gaussians, 8 views 1920x1080, BF16/FP16 storage",
                "gaussians": 3_000_000}
    else:
        raise SystemExit(f"unknown config {name}")
    desc["rays_per_step"] = int(sum(w * h for _, w, h in cams))
    desc["views"] = len(cams)
    return rec, cams, desc


def batching_cameras(sc):
    """64 views on spheres of radius 2-4, 16 each at the four resolutions."""
    return sc.sphere_cameras(64, seed=11)


def common_config(desc: dict, world: int) -> dict:
    """The `config` object both arms print (same workload, same keys)."""
    return {**desc, "l2": "flushed between timed steps (512 MB write)", "parallelism": f"replicas x{world}"}


# ------------------------------------------------------------------ clocks
class ClockSampler:
    """nvidia-smi samples (every 20 ms), each stamped with the host clock as
    it arrives; `stop(t0, t1)` keeps the samples taken inside the timed
    window [t0, t1] (host time.time()).  Started before the warm-up, so the
    sampler is running when the timed region begins."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        import threading
        self.rows = []
        self.first = threading.Event()
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(index), f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "20"], stdout=subprocess.PIPE,
                                      stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.p = None
            return

        def reader():
            for line in self.p.stdout:
                if line.strip():
                    self.rows.append((time.time(), line.split(",")))
                    self.first.set()

        self.th = threading.Thread(target=reader, daemon=True)
        self.th.start()
        self.first.wait(10.0)

    def stop(self, t0: float = None, t1: float = None) -> dict:
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.05)  # the sample after the window's end
        self.p.terminate()
        self.p.wait()
        self.th.join(2.0)
        ok = [(ts, r) for ts, r in self.rows if len(r) >= 8 and r[0].strip().replace(".", "").isdigit()]
        window = "timed region"
        rows = [r for ts, r in ok if t0 is None or t0 <= ts <= t1]
        if not rows and ok and t0 is not None:  # a region shorter than the interval: the nearest samples
            ok.sort(key=lambda x: min(abs(x[0] - t0), abs(x[0] - t1)))
            rows, window = [r for _, r in ok[:2]], "nearest samples to a timed region shorter than the interval"
        sm = [float(r[0]) for r in rows]
        mx = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if "Active" in r[4 + i]
                          and "Not" not in r[4 + i]})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(sm), "interval_ms": 20, "window": window}


# ------------------------------------------------------------------ roofline
def peaks() -> dict:
    try:
        return json.load(open(PEAKS))
    except (OSError, ValueError):
        return {}


def algorithmic_bytes(tr, b_test: int, b_blend: int, b_out: int) -> float:
    """Sum over rays of 8(N_inner+N_leaf) + 4 N_cand + b_test N_cand +
    b_blend N_blend + b_out (counters of the oracle-matching kernel)."""
    n = tr.shape[0]
    return float(8 * (tr["n_inner"].sum(dtype=np.int64) + tr["n_leaf"].sum(dtype=np.int64))
                 + (4 + b_test) * tr["n_cand"].sum(dtype=np.int64) + b_blend * tr["n_blend"].sum(dtype=np.int64)
                 + b_out * n)


def load_capture(key: str):
    """profiles/instructions.txt: `config:form kernel warp_instructions
    dram_bytes duration_ns` per line (# comments), from one ncu capture of
    one launch of the batched kernel."""
    try:
        for line in open(os.path.join(REPO, "profiles", "instructions.txt")):
            f = line.split("#", 1)[0].split()
            if len(f) == 5 and f[0] == key:
                return {"kernel": f[1], "warp_instructions": int(f[2]), "dram_bytes": int(f[3]),
                        "duration_ns": int(f[4])}
    except (OSError, ValueError):
        pass
    return None


def capture_key(config: str, cfg, default) -> str:
    """Key of the capture that counts for a launch with `cfg`: the captures are
    of the default configuration (precision apart); any other runs another
    kernel and has none."""
    key = f"{config}:{'packed' if cfg.precision else 'fp32'}"
    a, b = cfg.as_dict(), default.as_dict()
    return key if all(a[k] == b[k] for k in a if k != "precision") else key + ":other configuration"


def roofline(key: str, ms_step: float, clk: dict, sms: int, alg_bytes: float, rays: int) -> dict:
    """Issue-rate bound of the batched kernel, plus its memory figures."""
    pk = peaks()
    hbm = float(pk.get("hbm_gbs", FALLBACK_HBM_GBS))
    mhz = clk.get("sm_mhz") or float(pk.get("sm_max_mhz", 2070.0))
    mhz_src = "median SM clock sampled in the timed region" if clk.get("sm_mhz") else \
        "SM clock not sampled in the timed region: maximum SM clock of MEASURED_PEAKS.json"
    cap = load_capture(key)
    peak = sms * 4 * mhz * 1e6 / 1e9  # G warp instructions / s
    out = {"bound": "issue", "unit": "G warp-inst/s", "peak": round(peak, 2),
           "peak_source": f"{sms} SMs x 4 schedulers x 1 warp instruction per cycle x {mhz:.0f} MHz ({mhz_src})"}
    if cap:
        ach = cap["warp_instructions"] / (ms_step * 1e-3) / 1e9
        prof_frac = cap["warp_instructions"] / (sms * 4 * 2070e6 * cap["duration_ns"] * 1e-9)
        out.update({"achieved": round(ach, 2), "frac": round(ach / peak, 4),
                    "warp_instructions_per_launch": cap["warp_instructions"],
                    "warp_instructions_per_ray": round(cap["warp_instructions"] / rays, 1),
                    "instructions_from": f"ncu smsp__inst_executed.sum of one launch of {cap['kernel']} "
                                         f"(profiles/instructions.txt); frac of that capture at its own "
                                         f"duration: {prof_frac:.4f}",
                    "traffic": cap["dram_bytes"]})
    else:
        out.update({"achieved": None, "frac": None, "traffic": None,
                    "instructions_from": f"no capture for {key} in profiles/instructions.txt"})
    dram = cap["dram_bytes"] if cap else None
    out["memory"] = {
        "algorithmic_bytes_per_step": alg_bytes, "bytes_per_ray": round(alg_bytes / rays, 1),
        "algorithmic_gbs": round(alg_bytes / (ms_step * 1e-3) / 1e9, 1),
        "note": "algorithmic bytes are L1/L2 demand: the frame's working set stays in the 129 MB L2",
        "dram_bytes_per_launch": dram,
        "dram_gbs": round(dram / (ms_step * 1e-3) / 1e9, 2) if dram else None,
        "dram_frac_of_hbm": round(dram / (ms_step * 1e-3) / 1e9 / hbm, 5) if dram else None,
        "hbm_peak_gbs": hbm, "hbm_peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)" if "hbm_gbs" in pk
        else "fallback 6.8 TB/s"}
    return out


# ------------------------------------------------------------------ our arm
def timed_loop(step_fn, k, flush, stream, dev):
    import torch
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(k)]
    for i in range(k):
        flush.zero_()
        evs[i][0].record(stream)
        step_fn()
        evs[i][1].record(stream)
    torch.cuda.synchronize(dev)
    return [a.elapsed_time(b) for a, b in evs]


def wall_loop(step_fn, k, flush, dev):
    """Host-clock time of each step, the L2 flush completed before the clock starts."""
    import torch
    out = []
    for _ in range(k):
        flush.zero_()
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
        step_fn()
        out.append(1e3 * (time.perf_counter() - t0))
    return out


def rerank(F, scene, views, n_views, rgb, cfg, report, flush, stream, dev, top: int = 3):
    """The autotuner ranks its variants back to back, with the scene's working
    set warm in L2 (as in a frame loop); the timed region flushes L2 before
    every step.  Re-time the autotuner's `top` fastest configurations under
    the timed region's conditions (flush, then the graph replay) and return
    the fastest, with every time."""
    rows = []
    for line in report.splitlines():
        try:
            d = json.loads(line)
        except ValueError:
            continue
        if isinstance(d, dict) and "ms" in d:
            rows.append(d)
    rows.sort(key=lambda d: d["ms"])
    best, best_ms, tried, seen = cfg, None, [], set()
    for d in rows:
        key = tuple(sorted((k, v) for k, v in d.items() if k != "ms"))
        if key in seen:
            continue
        seen.add(key)
        c = F.BatchConfig.default()
        for k, v in d.items():
            if k != "ms":
                setattr(c, k, v)
        b = F.Batch(scene, views, n_views, rgb, None, None, c)
        for _ in range(2):
            b.run()
        ms = statistics.median(timed_loop(b.run, 5, flush, stream, dev))
        b.close()
        tried.append({**{k: v for k, v in d.items() if k != "ms"}, "warm_ms": d["ms"], "flushed_ms": round(ms, 4)})
        if best_ms is None or ms < best_ms:
            best, best_ms = c, ms
        if len(seen) >= top:
            break
    return best, tried


def run_ours(args, rank: int, world: int):
    import torch
    pkg = importlib.import_module(PKG)
    F = pkg.renderer
    dev = torch.device("cuda", int(os.environ.get("LOCAL_RANK", 0)))
    torch.cuda.set_device(dev)
    F.init(dev.index)
    rec, cams, desc = make_workload(pkg.scenes, args.config)
    t0 = time.time()
    tree = pkg.kdtree.build(rec, device="cuda")  # the device builder: same tree as the host builder
    build_s = time.time() - t0
    precision = 1 if args.config == "precision" else 0
    forms = F.FORM_EXACT | (F.FORM_PACKED if precision else F.FORM_FAST)
    scene = F.Scene(tree, rec, forms=forms)
    info = scene.info()
    log(f"[bench] {desc['workload']}: tree {tree.n_nodes} nodes, {tree.offsets.size} ids, depth {tree.depth}, "
        f"built on the device in {build_s:.2f}s; scene {info['device_bytes'] / 1e9:.2f} GB on device")
    views, total_px, offs = F.make_views(cams)
    rays = desc["rays_per_step"]
    rgb = torch.zeros(total_px * 3, device=dev)
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)
    # autotuned persistent-kernel configuration
    reranked = None
    if args.profile:
        cfg = F.BatchConfig.default()
        cfg.precision = precision
    else:
        cfg, report = scene.autotune(views, len(cams), rgb, precision=precision)
        log("[bench] autotuner variants:\n" + report.strip())
        cfg, reranked = rerank(F, scene, views, len(cams), rgb, cfg, report, flush, stream, dev)
        log(f"[bench] autotuner's three fastest re-timed with the L2 flush: {reranked}")
        log(f"[bench] picked {cfg.as_dict()}")
    batch = F.Batch(scene, views, len(cams), rgb, None, None, cfg)
    if args.profile:
        for _ in range(args.warmup + args.steps):
            for (cam, w, h), off in zip(cams, offs):
                scene.render(cam, w, h, rgb[3 * off:3 * (off + w * h)])
        for _ in range(args.warmup + args.steps):
            batch.run()
        torch.cuda.synchronize(dev)
        assert scene.status() == 0
        print(json.dumps({"profile_run": args.config, "launches": args.warmup + args.steps}), flush=True)
        raise SystemExit(0)

    clocks = ClockSampler(dev.index)
    for _ in range(args.warmup):
        batch.run()
    torch.cuda.synchronize(dev)
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize(dev)
    wall0 = time.time()
    ms = timed_loop(batch.run, args.steps, flush, stream, dev)
    wall = time.time() - wall0
    clk = clocks.stop(wall0, wall0 + wall)
    if world > 1:
        torch.distributed.barrier()
    assert scene.status() == 0, "kernel raised an error status"
    R = importlib.import_module(PKG + ".replicas")
    ms_step = R.max_over_ranks(sum(ms) / len(ms), dev)
    value = R.job_throughput(rays, world, ms_step) / 1e6

    # e2e: the public C ABI call with host-side cameras, timed on the host
    # clock until the frame is readable in pinned host memory.  The kernel
    # writes the frame straight into the pinned buffer (page-locked host
    # memory is device-addressable; on GB300 the stores cross NVLink-C2C
    # while the frame renders); the variant with a device buffer and a
    # separate copy is reported beside it.
    host = torch.empty(total_px * 3, dtype=torch.float32, pin_memory=True)
    host_copy = torch.empty(total_px * 3, dtype=torch.float32, pin_memory=True)

    def e2e_step():
        scene.render_batch(views, len(cams), host, cfg=cfg)
        stream.synchronize()

    def e2e_copy_step():
        scene.render_batch(views, len(cams), rgb, cfg=cfg)
        host_copy.copy_(rgb, non_blocking=True)
        stream.synchronize()

    for _ in range(args.warmup):
        e2e_step()
        e2e_copy_step()
    ms_e2e = wall_loop(e2e_step, args.steps, flush, dev)
    ms_e2e_copy = wall_loop(e2e_copy_step, args.steps, flush, dev)
    e2e_step_ms = R.max_over_ranks(statistics.median(ms_e2e), dev)
    e2e_copy_ms = R.max_over_ranks(statistics.median(ms_e2e_copy), dev)
    assert np.array_equal(host.numpy(), host_copy.numpy()), "host-written frame differs from the copied one"
    view_bytes = 96 * len(cams)  # ViewDesc table (96 B per view) copied host->device by kdgr_render_batch
    e2e = {"value": R.job_throughput(rays, world, e2e_step_ms) / 1e6, "unit": UNIT,
           "h2d_bytes_per_step": view_bytes, "d2h_bytes_per_step": int(host.numel() * 4),
           "ms_per_step": e2e_step_ms, "ms_per_step_mean": statistics.mean(ms_e2e),
           "clock": "host perf_counter, median over steps: call -> frame readable in pinned host memory",
           "path": "kdgr_render_batch (C ABI) writing the RGB frame into pinned host memory + stream sync",
           "device_buffer_plus_copy": {
               "value": round(R.job_throughput(rays, world, e2e_copy_ms) / 1e6, 3), "ms_per_step": round(e2e_copy_ms, 4),
               "path": "kdgr_render_batch into device memory + D2H copy into pinned host memory + stream sync"}}

    # plain drop-in (oracle-matching) kernel on the same views, one launch per view
    def plain_step():
        for (cam, w, h), off in zip(cams, offs):
            scene.render(cam, w, h, rgb[3 * off:3 * (off + w * h)])

    batched_host = host.numpy().copy()  # the last batched frame (e2e loop)
    for _ in range(max(1, args.warmup // 2)):
        plain_step()
    pm = timed_loop(plain_step, max(2, args.steps // 2), flush, stream, dev)
    plain_ms = sum(pm) / len(pm)
    torch.cuda.synchronize(dev)
    plain_host = rgb.cpu().numpy().copy()

    # counters of the oracle-matching kernel -> algorithmic bytes per step
    tr_cat = trace_counters(pkg, scene, cams, dev)
    b_test, b_blend = (32, 96 + 2) if precision else (48, 192 + 4)
    alg_bytes = algorithmic_bytes(tr_cat, b_test, b_blend, 12)
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    counters = {k: float(tr_cat[k].mean()) for k in ("n_inner", "n_leaf", "n_cand", "n_hit", "n_blend",
                                                     "n_restart")}
    out = {
        "metric": METRIC if args.config == "scale" else f"Mrays/s ({args.config})",
        "value": round(value, 3), "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(ms_step, 4), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "bf16/fp16 storage, fp32 arithmetic" if precision else "f32", "data": "synthetic",
        "config": common_config(desc, world),
        "form": "batched persistent kernel, CUDA graph", "autotuned": cfg.as_dict(),
        "autotune_reranked": reranked,
        "e2e": {k: (round(v, 4) if isinstance(v, float) else v) for k, v in e2e.items()},
        "roofline": roofline(capture_key(args.config, cfg, F.BatchConfig.default()), ms_step, clk, sms, alg_bytes,
                             rays),
        "gpu_launches": args.steps,
        "clocks": clk,
        "forms": {"plain_ms_per_step": plain_ms,
                  "plain_mrays_s": round(rays / (plain_ms * 1e-3) / 1e6, 3) if plain_ms else None,
                  "batched_over_plain": round(plain_ms / ms_step, 3) if plain_ms else None},
        "counters_per_ray": counters,
        "tree": {"nodes": tree.n_nodes, "ids": int(tree.offsets.size), "depth": tree.depth, "builder": "device",
                 "build_s": round(build_s, 2)},
        "wall_s_timed": round(wall, 3),
    }
    check = rank == 0 and not args.no_cpu_baseline
    if check:
        out["cpu_baseline"] = cpu_baseline(tree, rec, cams, args.cpu_seconds)
        out["accuracy"] = accuracy(tree, rec, cams, offs, batched_host, plain_host)
    if args.config == "scale" and not args.no_legs and rank == 0:
        out["legs"] = {"batching": leg_batching(pkg, scene, tree, rec, dev, flush, stream, args, check)}
    batch.close()
    scene.close()
    if args.config == "scale" and not args.no_legs and rank == 0:
        del flush
        torch.cuda.empty_cache()
        srv = run_serving_rates(pkg, [args.leg_rate], args.leg_seconds)
        out["legs"]["serving"] = {"rate_req_s": args.leg_rate, "seconds": args.leg_seconds, **srv["results"],
                                  "setup": srv["setup"]}
    return out


def trace_counters(pkg, scene, cams, dev):
    import torch
    tr_all = []
    dt = np.dtype(pkg.capi.TRACE_DTYPE)
    for cam, w, h in cams:
        tr = torch.zeros(w * h * dt.itemsize, dtype=torch.uint8, device=dev)
        tmp = torch.zeros(w * h * 3, device=dev)
        scene.render_trace(cam, w, h, tmp, None, None, tr)
        torch.cuda.synchronize(dev)
        tr_all.append(np.frombuffer(tr.cpu().numpy().tobytes(), dtype=dt))
    return np.concatenate(tr_all)


def leg_batching(pkg, scene, tree, rec, dev, flush, stream, args, check: bool):
    """The 64-view batch of the same 1M scene (one persistent launch, CUDA
    graph, autotuned) against the plain kernel, one launch per view."""
    import torch
    F = pkg.renderer
    cams = batching_cameras(pkg.scenes)
    views, total, offs = F.make_views(cams)
    rays = int(sum(w * h for _, w, h in cams))
    rgb = torch.zeros(total * 3, device=dev)
    cfg, report = scene.autotune(views, len(cams), rgb, precision=0)
    cfg, _ = rerank(F, scene, views, len(cams), rgb, cfg, report, flush, stream, dev)
    batch = F.Batch(scene, views, len(cams), rgb, None, None, cfg)
    for _ in range(2):
        batch.run()
    k = max(3, args.steps // 5)
    ms = statistics.mean(timed_loop(batch.run, k, flush, stream, dev))
    torch.cuda.synchronize(dev)
    batched_host = rgb.cpu().numpy().copy()
    batch.close()

    def plain_step():
        for (cam, w, h), off in zip(cams, offs):
            scene.render(cam, w, h, rgb[3 * off:3 * (off + w * h)])

    plain_step()
    pms = statistics.mean(timed_loop(plain_step, 2, flush, stream, dev))
    torch.cuda.synchronize(dev)
    assert scene.status() == 0
    out = {"workload": "cluster+shell, 1M Gaussians, 64 views (16 each at 256x256, 640x480, 1280x720, "
                       "1920x1080) in one persistent launch", "rays_per_step": rays, "steps": k,
           "ms_per_step": round(ms, 3), "mrays_s": round(rays / (ms * 1e-3) / 1e6, 2),
           "plain_ms_per_step": round(pms, 3), "plain_mrays_s": round(rays / (pms * 1e-3) / 1e6, 2),
           "batched_over_plain": round(pms / ms, 3), "autotuned": cfg.as_dict()}
    if check:
        plain_host = rgb.cpu().numpy().copy()
        out["accuracy"] = accuracy(tree, rec, cams, offs, batched_host, plain_host, n_target=20000)
    return out


# ------------------------------------------------------------------ serving
def poisson_requests(rate: float, seconds: float, n_scenes: int, seed: int, resolutions=None):
    """[(arrival_s, scene, [(Camera, W, H)])]: Poisson arrivals, 1-16 views per
    request, each view's resolution uniform over `resolutions` (default: the
    four of the mixed set), scene uniform."""
    sc = _scenes()
    res = resolutions or sc.RESOLUTIONS
    rng = np.random.default_rng(seed)
    t, out = 0.0, []
    while True:
        t += rng.exponential(1.0 / rate)
        if t > seconds:
            return out
        nv = int(rng.integers(1, 17))
        cams = []
        for _ in range(nv):
            w, h = res[int(rng.integers(0, len(res)))]
            d = rng.normal(0.0, 1.0, 3)
            d /= np.linalg.norm(d)
            cams.append((sc.look_at(d * rng.uniform(2.0, 4.0), aspect=w / h), w, h))
        out.append((t, int(rng.integers(0, n_scenes)), cams))


class PinnedRing:
    """Output buffers of the served client: ranges of one page-locked slab,
    handed out in submission order and given back when their request has
    been waited for.  The server's kernel writes page-locked buffers
    directly.  When the slab is full the client waits for its oldest
    request first (time reported as client_wait_s: non-zero only when the
    offered load exceeds what the GPU serves)."""

    def __init__(self, torch, n_floats: int):
        self.slab = torch.empty(n_floats, dtype=torch.float32, pin_memory=True)
        self.n = n_floats
        self.live = collections.deque()  # (start, end, ticket, submit delay s)
        self.head = 0
        self.waited = 0.0
        self.lat_ms = []  # per request: scheduled arrival -> done

    def _retire_oldest(self, srv):
        _, _, t, delay = self.live.popleft()
        t0 = time.perf_counter()
        rc, st = srv.wait(t, timeout_ms=600_000)
        self.waited += time.perf_counter() - t0
        assert rc == 0, rc
        self.lat_ms.append(1e3 * delay + st["latency_ms"])
        if not self.live:
            self.head = 0

    def take(self, srv, n: int):
        """A slab range of n floats; returns (start, view)."""
        assert n <= self.n
        while True:
            tail = self.live[0][0] if self.live else 0
            if not self.live or self.head > tail:
                if self.head + n <= self.n:
                    start = self.head
                    break
                if self.live and n < tail:
                    start = 0
                    break
            elif self.head + n < tail:
                start = self.head
                break
            self._retire_oldest(srv)
        self.head = start + n
        return start, self.slab[start:start + n]

    def add(self, start: int, n: int, ticket: int, delay: float):
        """delay: seconds from the request's scheduled arrival to its submit."""
        self.live.append((start, start + n, ticket, delay))

    def drain(self, srv):
        while self.live:
            self._retire_oldest(srv)


SERVING_SETS = {
    # the serving config: four scenes, views of the four resolutions
    "mix": {"sizes": [500_000, 1_000_000, 2_000_000, 3_000_000], "resolutions": None},
    # the headline config served: the 1M scene, 1920x1080 views
    "1m_1080p": {"sizes": [1_000_000], "resolutions": [(1920, 1080)]},
}


def run_serving_rates(pkg, rates, seconds, scene_set: str = "mix"):
    """Resident cluster+shell scenes (the "mix" set: 0.5M/1M/2M/3M, seeds
    1-4; "1m_1080p": the 1M scene of seed 1 with 1920x1080 views only) under
    a 60 GB budget; Poisson request streams at each rate, served by the
    continuous-batching server, and by the plain per-request path (one
    request at a time, one plain-kernel launch per view) for comparison.
    Both clients receive frames in page-locked host memory written by the
    kernels themselves."""
    import threading
    import torch
    F = pkg.renderer
    F.init(0)
    sizes, resolutions = SERVING_SETS[scene_set]["sizes"], SERVING_SETS[scene_set]["resolutions"]
    srv = F.Server(hbm_budget_bytes=60 << 30, arena_bytes=8 << 30, lanes=3, max_views_per_launch=256)
    plain_scenes, slots = [], []
    t0 = time.time()
    for i, n in enumerate(sizes):
        rec = pkg.scenes.cluster_shell(n, seed=i + 1)
        tree = pkg.kdtree.build(rec, device="cuda")
        slots.append(srv.add_scene(tree, rec))
        plain_scenes.append(F.Scene(tree, rec, forms=F.FORM_EXACT))
    setup = {"seconds": round(time.time() - t0, 1), "resident_gb": round(srv.stats()["resident_bytes"] / 1e9, 2),
             "budget_gb": 60.0 * (1 << 30) / 1e9}
    log(f"[bench] serving: {len(sizes)} scenes built and resident in {setup['seconds']}s, {setup['resident_gb']} GB")
    pct = lambda v, p: v[min(len(v) - 1, int(p * (len(v) - 1) + 0.5))]
    max_req = 16 * 1920 * 1080 * 3  # floats of the largest request
    ring = PinnedRing(torch, 1 << 30)  # 4 GiB of served output in flight
    plain_out = torch.empty(max_req, dtype=torch.float32, pin_memory=True)
    # untimed warm-up, one small request per scene through both paths
    # (first launches load their kernels and run one-time queries)
    for i, slot in enumerate(slots):
        cams = [(pkg.scenes.front_camera(256, 256), 256, 256)]
        views, total, _ = F.make_views(cams)
        off, buf = ring.take(srv, total * 3)
        ring.add(off, total * 3, srv.submit(slot, views, 1, buf), 0.0)
        plain_scenes[i].render(cams[0][0], 256, 256, plain_out[:total * 3])
    ring.drain(srv)
    torch.cuda.synchronize()
    results = {}
    for rate in rates:
        reqs = poisson_requests(rate, seconds, len(sizes), seed=int(rate), resolutions=resolutions)
        rays = sum(w * h for _, _, cams in reqs for _, w, h in cams)
        # served
        srv.reset_stats()
        ring.waited = 0.0
        ring.lat_ms = []
        start = time.time()
        for arr, scene, cams in reqs:
            now = time.time() - start
            if arr > now:
                time.sleep(arr - now)
            views, total, _ = F.make_views(cams)
            off, buf = ring.take(srv, total * 3)
            ticket = srv.submit(slots[scene], views, len(cams), buf)
            ring.add(off, total * 3, ticket, max(0.0, time.time() - start - arr))
        ring.drain(srv)
        st = srv.stats()
        served_lat = sorted(ring.lat_ms)
        # plain path: FIFO, one request at a time, plain kernel per view
        dev = torch.device("cuda:0")
        q, lat, lock = [], [], threading.Lock()
        done_evt = threading.Event()

        def worker():
            stream = torch.cuda.current_stream(dev)
            while True:
                with lock:
                    item = q.pop(0) if q else None
                if item is None:
                    if done_evt.is_set():
                        return
                    time.sleep(0.0005)
                    continue
                arr_abs, scene, cams = item
                off = 0
                for cam, w, h in cams:
                    plain_scenes[scene].render(cam, w, h, plain_out[off:off + w * h * 3])
                    off += w * h * 3
                stream.synchronize()
                lat.append(1e3 * (time.time() - arr_abs))

        th = threading.Thread(target=worker)
        th.start()
        start = time.time()
        for arr, scene, cams in reqs:
            now = time.time() - start
            if arr > now:
                time.sleep(arr - now)
            with lock:
                q.append((start + arr, scene, cams))
        done_evt.set()
        th.join()
        plain_wall = time.time() - start
        lat.sort()
        results[str(int(rate))] = {
            "requests": len(reqs), "rays": int(rays),
            # latency from the request's scheduled arrival, as for plain;
            # server_* from its submit (later than arrival only while the
            # client waits for output space: client_wait_s)
            "served": {"p50_ms": round(pct(served_lat, 0.5), 2), "p99_ms": round(pct(served_lat, 0.99), 2),
                       "server_p50_ms": round(st["p50_ms"], 2), "server_p99_ms": round(st["p99_ms"], 2),
                       "mean_ms": round(st["mean_ms"], 2), "mrays_per_s": round(st["mrays_per_s"], 1),
                       "launches": st["launches"], "max_views_per_launch": st["max_views_per_launch"],
                       "client_wait_s": round(ring.waited, 3)},
            "plain": {"p50_ms": round(pct(lat, 0.5), 2), "p99_ms": round(pct(lat, 0.99), 2),
                      "mrays_per_s": round(rays / plain_wall / 1e6, 1)},
        }
        r = results[str(int(rate))]
        r["p99_plain_over_served"] = round(r["plain"]["p99_ms"] / max(r["served"]["p99_ms"], 1e-9), 2)
        log(f"[bench] rate {rate}: {r}")
    srv.close()
    for s in plain_scenes:
        s.close()
    return {"results": results, "setup": setup}


def run_serving(args):
    pkg = importlib.import_module(PKG)
    hd = args.config == "serving_1080p"
    rates = [float(r) for r in (args.rates or ("20,40,80,160" if hd else "50,100,200,400")).split(",")]
    res = run_serving_rates(pkg, rates, args.serve_seconds, "1m_1080p" if hd else "mix")
    results = res["results"]
    key = str(int(rates[0]))
    workload = ("the 1M cluster+shell scene (seed 1) resident, Poisson requests of 1-16 views at 1920x1080"
                if hd else "4 resident cluster+shell scenes (0.5M/1M/2M/3M), Poisson requests of 1-16 "
                           "views at 256x256/640x480/1280x720/1920x1080, 60 GB budget")
    return {
        "metric": f"served p99 latency at {key} req/s", "value": results[key]["served"]["p99_ms"], "unit": "ms",
        "n_gpus": 1, "steps": len(rates), "warmup": 0, "higher_is_better": False, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": workload, "form": "continuous-batching server, 3 lanes",
                   "seconds_per_rate": args.serve_seconds},
        "serving": results, "setup": res["setup"],
    }


# ------------------------------------------------------------------ CPU arm
def _oracle():
    sys.path.insert(0, os.path.join(REPO, "oracle"))
    return importlib.import_module("oracle")


def oracle_scene(tree, rec):
    O = _oracle()
    return O.OracleScene(tree.nodes, tree.offsets, tree.aabb, O.invert_scales(rec))


def cpu_sample(S, cams, seconds: float, threads: int = 0, precision: str = "f32"):
    """Render a strided ray sample of every view with the oracle (CPU), sized
    to about `seconds` of work.  Returns (Mrays/s, rays, stride, threads, s)."""
    O = _oracle()
    nthr = threads or os.cpu_count() or 1

    def run(stride):
        n = 0
        t = time.time()
        for cam, w, h in cams:
            pix = np.arange(0, w * h, stride, dtype=np.uint32)
            O.render(S, cam, w, h, pixels=pix, threads=nthr, precision=precision)
            n += pix.size
        return n, time.time() - t

    total = sum(w * h for _, w, h in cams)
    stride = max(1, total // 20000)
    n, dt = run(stride)
    rate = n / max(dt, 1e-6)
    stride = max(1, int(total / max(rate * seconds, 1)))
    n, dt = run(stride)
    return n / dt / 1e6, n, stride, nthr, dt


def accuracy(tree, rec, cams, offs, batched, plain, n_target: int = 40000):
    """Max and RMS RGB error of the batched frame against the FP64 oracle,
    and of the plain kernel against the FP64 and the oracle-matching FP32
    oracle, on a strided ray sample of every view."""
    O = _oracle()
    S = oracle_scene(tree, rec)
    total = sum(w * h for _, w, h in cams)
    stride = max(1, total // n_target)
    eb, ep, ep32 = [], [], []
    for (cam, w, h), off in zip(cams, offs):
        pix = np.arange(0, w * h, stride, dtype=np.uint32)
        x, y = pix % w, pix // w
        idx = off + (h - 1 - y).astype(np.int64) * w + x
        r64 = O.render(S, cam, w, h, pixels=pix, precision="f64")[0]
        r32 = O.render(S, cam, w, h, pixels=pix, precision="f32")[0]
        eb.append(batched.reshape(-1, 3)[idx].astype(np.float64) - r64)
        ep.append(plain.reshape(-1, 3)[idx].astype(np.float64) - r64)
        ep32.append(plain.reshape(-1, 3)[idx] - r32)
    eb, ep, ep32 = np.concatenate(eb), np.concatenate(ep), np.concatenate(ep32)
    return {"vs": "FP64 oracle (CPU transcription in double)", "sampled_rays": int(eb.shape[0]),
            "batched_max_abs": float(np.abs(eb).max()), "batched_rms": float(np.sqrt((eb ** 2).mean())),
            "plain_max_abs": float(np.abs(ep).max()), "plain_rms": float(np.sqrt((ep ** 2).mean())),
            "plain_vs_fp32_oracle_max_abs": float(np.abs(ep32).max())}


def cpu_baseline(tree, rec, cams, seconds):
    S = oracle_scene(tree, rec)
    mr, n, stride, nthr, dt = cpu_sample(S, cams, seconds)
    mr1, n1, _, _, dt1 = cpu_sample(S, cams, max(1.0, seconds / 4), threads=1)
    mr64, n64, _, _, dt64 = cpu_sample(S, cams, max(1.0, seconds / 4), precision="f64")
    return {"value": round(mr, 4), "unit": UNIT, "cores": nthr, "kind": "port",
            "sample": f"every {stride}th ray of each view ({n} rays, {dt:.1f}s), oracle FP32 transcription "
                      f"of cudaRenderer.cu with OpenMP over rays",
            "single_thread_value": round(mr1, 4), "single_thread_sample": f"{n1} rays, {dt1:.1f}s",
            "fp64_value": round(mr64, 4), "fp64_sample": f"{n64} rays, {dt64:.1f}s, {nthr} threads",
            "cpu_model": cpu_model()}


def cpu_model() -> str:
    try:
        out = subprocess.run(["lscpu"], capture_output=True, text=True, timeout=10).stdout
        for line in out.splitlines():
            if line.startswith("Model name:"):
                return line.split(":", 1)[1].strip()
    except (OSError, subprocess.SubprocessError):
        pass
    try:
        for line in open("/proc/cpuinfo"):
            if line.lower().startswith(("model name", "cpu part")):
                return line.split(":", 1)[1].strip()
    except OSError:
        pass
    import platform
    return platform.machine()


def prepare_reference_inputs(config: str, out_dir: str) -> None:
    """Untimed input preparation of the reference arm, run as its own process:
    the seeded scene and its kd-tree (host builder, trees byte-identical to
    the reference builder's) written as files: scene.npy (activated 64-float
    records), tree.kdt (the reference's binary format) and meta.json
    (cameras, workload description, build time)."""
    pkg = importlib.import_module(PKG)
    rec, cams, desc = make_workload(pkg.scenes, config)
    t0 = time.time()
    tree = pkg.kdtree.build(rec)
    build_s = time.time() - t0
    np.save(os.path.join(out_dir, "scene.npy"), rec)
    pkg.kdtree.write_kdt(tree, os.path.join(out_dir, "tree.kdt"))
    meta = {"desc": desc, "build_s": build_s,
            "cams": [{"cam": {"pos": list(c.pos), "uaxis": list(c.uaxis), "vaxis": list(c.vaxis),
                              "naxis": list(c.naxis), "fovy": c.fovy, "aspect": c.aspect, "near_c": c.near_c},
                      "w": w, "h": h} for c, w, h in cams]}
    json.dump(meta, open(os.path.join(out_dir, "meta.json"), "w"))


def run_reference(args):
    """The reference's render algorithm on the host cores: the oracle
    transcription of cudaRenderer.cu, all host threads, on a strided ray
    sample per step.  This process loads the oracle only."""
    O = _oracle()
    work = tempfile.mkdtemp(prefix="kdgr_ref_")
    try:
        t0 = time.time()
        subprocess.run([sys.executable, os.path.abspath(__file__), "--prepare-reference", work, "--config",
                        args.config], check=True, stdout=subprocess.DEVNULL)
        prep_s = time.time() - t0
        meta = json.load(open(os.path.join(work, "meta.json")))
        rec = np.load(os.path.join(work, "scene.npy"))
        nodes, offsets, aabb = O.read_kdt(os.path.join(work, "tree.kdt"))
    finally:
        shutil.rmtree(work, ignore_errors=True)
    desc = meta["desc"]
    cams = [(SimpleNamespace(**c["cam"]), c["w"], c["h"]) for c in meta["cams"]]
    S = O.OracleScene(nodes, offsets, aabb, O.invert_scales(rec))
    per_step = max(2.0, min(20.0, 60.0 / max(1, args.steps + args.warmup)))
    res = []
    for i in range(args.warmup + args.steps):
        mr, n, stride, nthr, dt = cpu_sample(S, cams, per_step)
        if i >= args.warmup:
            res.append((mr, n, stride, dt))
    value = statistics.mean(r[0] for r in res)
    return {
        "metric": METRIC if args.config == "scale" else f"Mrays/s ({args.config})", "impl": "reference",
        "value": round(value, 4), "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(1e3 * statistics.mean(r[3] for r in res), 2), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": common_config(desc, args.gpus),
        "form": "CPU transcription of the reference render kernel (oracle, OpenMP over rays)",
        "cpu_baseline": {"value": round(value, 4), "unit": UNIT, "cores": nthr, "kind": "port",
                         "sample": f"every {res[-1][2]}th ray per view, {res[-1][1]} rays per step",
                         "cpu_model": cpu_model()},
        "e2e": {"value": round(value, 4), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "inputs": {"prepared_by": "untimed child process: seeded scene generation and the host kd-tree builder "
                                  "(trees byte-identical to the reference builder's, tests/test_kdtree.py); "
                                  "read here from scene.npy and tree.kdt through the oracle's .kdt reader",
                   "prep_s": round(prep_s, 1), "host_build_s": round(meta["build_s"], 2),
                   "reference_builder": "not run here: it builds only from the reference's own sources, which "
                                        "the GPU host does not have"},
    }


def run_build(args):
    """Tree build time on the bench scene: device builder against the host
    builder (all host cores), trees compared word for word."""
    pkg = importlib.import_module("3dgrt_kdtree_gb300")
    pkg.renderer.init(0)
    rec, _, desc = make_workload(pkg.scenes, "scale")
    pkg.kdtree.build(pkg.scenes.uniform_cube(20_000, seed=5), device="cuda")  # context and pools warm
    times = []
    for _ in range(max(1, args.steps)):
        t0 = time.time()
        g = pkg.kdtree.build(rec, device="cuda")
        times.append(time.time() - t0)
    t0 = time.time()
    h = pkg.kdtree.build(rec)
    host_s = time.time() - t0
    same = bool(np.array_equal(g.nodes, h.nodes) and np.array_equal(g.offsets, h.offsets))
    dev_s = statistics.median(times)
    return {"metric": "kd-tree build seconds (1M cluster+shell, reference builder flags)", "value": round(dev_s, 3),
            "unit": "s", "n_gpus": 1, "steps": len(times), "warmup": 1, "higher_is_better": False,
            "config": {"workload": desc["workload"], "max_level": 24, "force_split": 16, "sah_mode": 1},
            "host_builder_s": round(host_s, 2), "host_cores": os.cpu_count(), "speedup": round(host_s / dev_s, 2),
            "identical_trees": same, "nodes": int(g.n_nodes), "ids": int(g.offsets.size), "depth": int(g.depth),
            "triangles": int(g.stats["n_triangles"])}


def run_hybrid(args):
    """Secondary-ray renderer (the reference's SECONDARY_RAY build) on the
    1M scene at 1080p: the reference's two demo spheres (glass, mirror) and
    a mirror quad behind the scene; primary rays per second, the plain
    render of the same view beside it, and a bit-exactness check of a ray
    sample against the oracle."""
    import torch
    pkg = importlib.import_module("3dgrt_kdtree_gb300")
    F = pkg.renderer
    dev = torch.device("cuda", 0)
    F.init(0)
    rec, cams, desc = make_workload(pkg.scenes, "scale")
    tree = pkg.kdtree.build(rec, device="cuda")
    scene = F.Scene(tree, rec, forms=F.FORM_EXACT)
    quad = np.array([[-1.6, -1.6, -1.7, 1.6, -1.6, -1.7, 1.6, 1.6, -1.7],
                     [-1.6, -1.6, -1.7, 1.6, 1.6, -1.7, -1.6, 1.6, -1.7]], np.float32)
    mat = F.mesh_material_default()
    sec = F.Secondary(F.demo_spheres(), quad, mat)
    cam, w, h = cams[0]
    rgb = torch.zeros(w * h * 3, device=dev)
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    stream = torch.cuda.current_stream(dev)

    def timed(fn, k):
        out = []
        for _ in range(k):
            flush.zero_()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            fn()
            b.record(stream)
            torch.cuda.synchronize(dev)
            out.append(a.elapsed_time(b))
        return sum(out) / len(out)

    clocks = ClockSampler(0)
    for _ in range(args.warmup):
        scene.render_hybrid(cam, w, h, sec, rgb)
    t0 = time.time()
    ms = timed(lambda: scene.render_hybrid(cam, w, h, sec, rgb), args.steps)
    clk = clocks.stop(t0, time.time())
    torch.cuda.synchronize(dev)
    hyb = rgb.cpu().numpy().copy()
    for _ in range(args.warmup):
        scene.render(cam, w, h, rgb)
    plain_ms = timed(lambda: scene.render(cam, w, h, rgb), args.steps)
    assert scene.status() == 0
    out = {"metric": "Mrays/s (hybrid secondary rays, primary rays counted)", "value": round(w * h / (ms * 1e-3) / 1e6, 3),
           "unit": UNIT, "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 4),
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
           "config": {"workload": desc["workload"] + ", 2 demo spheres (glass, mirror) + mirror quad, <=5 bounces",
                      "l2": "flushed between timed steps (512 MB write)"},
           "plain_ms_per_step": round(plain_ms, 4), "hybrid_over_plain_time": round(ms / plain_ms, 3),
           "clocks": clk, "gpu_launches": args.steps}
    if not args.no_cpu_baseline:
        O = _oracle()
        S = oracle_scene(tree, rec)
        pix = np.arange(0, w * h, 211, dtype=np.uint32)
        sph = [(tuple(x.center), x.radius, x.material.material, x.material.reflectivity, x.material.ior,
                tuple(x.material.color)) for x in F.demo_spheres()]
        want = O.render_hybrid(S, cam, w, h, spheres=sph, tris=quad,
                               tri_material=(mat.material, mat.reflectivity, mat.ior, tuple(mat.color)), pixels=pix)
        x, y = pix % w, pix // w
        got = hyb.reshape(-1, 3)[(h - 1 - y).astype(np.int64) * w + x]
        out["accuracy"] = {"vs": "oracle FP32 hybrid transcription", "sampled_rays": int(pix.size),
                           "max_abs": float(np.abs(got - want).max())}
    sec.close()
    scene.close()
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--config", default="scale",
                    choices=["scale", "small", "mid", "batching", "precision", "serving", "serving_1080p", "build",
                             "hybrid"])
    ap.add_argument("--rates", default=None,
                    help="serving: Poisson request rates (req/s; default 50,100,200,400, or 20,40,80,160 for "
                         "serving_1080p)")
    ap.add_argument("--serve-seconds", type=float, default=4.0, help="serving: arrivals per rate")
    ap.add_argument("--leg-rate", type=float, default=50.0, help="scale: request rate of the serving leg")
    ap.add_argument("--leg-seconds", type=float, default=3.0, help="scale: arrivals of the serving leg")
    ap.add_argument("--no-legs", action="store_true", help="scale: skip the batching and serving legs")
    ap.add_argument("--profile", action="store_true",
                    help="profiling run: default kernel config, no L2-flush buffer, no e2e/plain/CPU legs")
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cpu-seconds", type=float, default=10.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--prepare-reference", metavar="DIR", help=argparse.SUPPRESS)
    args = ap.parse_args()
    if args.prepare_reference:
        prepare_reference_inputs(args.config, args.prepare_reference)
        return
    if args.warmup < 3:
        log("[bench] warmup raised to 3")
        args.warmup = 3
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    if args.impl == "reference":
        if rank != 0:
            return
        print(json.dumps(run_reference(args)), flush=True)
        return
    if world > 1:
        import torch
        torch.distributed.init_process_group("nccl")
    if args.config == "build":
        out = run_build(args)
    elif args.config == "hybrid":
        out = run_hybrid(args)
    elif args.config in ("serving", "serving_1080p"):
        out = run_serving(args)
    else:
        out = run_ours(args, rank, world)
    if rank == 0:
        print(json.dumps(out), flush=True)
    if world > 1:
        import torch
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
