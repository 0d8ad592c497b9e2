#!/usr/bin/env python
"""Benchmark: interpolated Mpix/s of the per-frame interpolation path at 1080p.

Workload (the configuration the headline metric is quoted on): 1920x1080
main camera plus left/right aux cameras at +-0.3 m (6 source views per
keyframe pair), soft shadows on, seeded procedural scene (64 spheres,
|v| <= 0.5 m/s, 30 Hz keyframes), client at 120 Hz (frames_per_anchor 4,
shadow_frames_per_anchor 4), plain method (mode 0: 3x3 window, 3 search
iterations).

One step = one keyframe interval = 3 interpolated 1080p client frames
(t = 0.25, 0.5, 0.75) between a resident keyframe pair; steps cycle over
``--pairs`` resident pairs.  Inputs are larger than L2: each frame touches
~0.8 GB (6 source views of colour, z, f16 motion, shadow A/B/Info plus the
renderer's keys and flow fields), and 6 keyframes x 3 cameras (~1.6 GB) stay
resident.

value: device-resident throughput (CUDA events on the rendering stream).
e2e:   the same metric through the C ABI with host buffers: each step
       uploads the newly arrived keyframe data from pinned host memory
       (colour, z, motion and shadow images of the new keyframe for the 3
       cameras, plus the earlier keyframe's forward motion and shadows; colour
       and shadow images as RGB, expanded to RGBA on the device: the shadow
       images' alpha is never read and the colour comes from opaque RGB sources)
       and reads the 3 output frames back.

--impl reference times the reference's per-frame algorithm on the host
cores (the C oracle, OpenMP over all threads: the reference has no CPU
implementation and its GPU code cannot be built on the GPU host), one 1080p
frame per step.

Multi-GPU: replicas only (every frame is independent); each rank renders its
own seeded stream, no collective on the data path; time = max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

W, H = 1920, 1080
AUX = (-0.3, 0.3)
TS = (1, 2, 3)            # b of t = b / 4
FPA = SFPA = 4
METRIC = "interp Mpix/s @1080p"
WORKLOAD = "1080p interpolation, 3 cameras (main + aux +-0.3 m), soft shadows, t in {0.25,0.5,0.75}, plain search (mode 0)"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=34)   # 102 timed frames (3 per step)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--pairs", type=int, default=5)
    ap.add_argument("--seed", type=int, default=2024)
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="bounded CPU-baseline sample")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-per-frame", action="store_true", help="skip the single-frame-call comparison")
    ap.add_argument("--no-quality", action="store_true", help="skip PSNR / SSIM against the analytic ground truth")
    ap.add_argument("--no-graph-batch", action="store_true", help="skip the mixed-resolution batch under a CUDA graph")
    ap.add_argument("--no-serving", action="store_true", help="skip the serving loop with simulated clients")
    ap.add_argument("--serve-seconds", type=float, default=60.0, help="real time of the serving loop (the configuration's 60 s)")
    ap.add_argument("--serve-learned", type=int, default=1, help="serve with the learned initialiser when its weights exist")
    ap.add_argument("--serve-slots", type=int, default=4, help="concurrent batches (streams) of the serving loop")
    ap.add_argument("--pressure-seconds", type=float, default=20.0,
                    help="real time of the serving loop under pressure (more clients than the budget admits)")
    ap.add_argument("--no-pressure", action="store_true", help="skip the serving loop under pressure")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned-initialiser comparison")
    ap.add_argument("--no-small-frame", action="store_true", help="skip the 640x360 single-frame timing")
    ap.add_argument("--no-reference-gpu", action="store_true", help="skip timing the reference's own GPU build")
    ap.add_argument("--no-arith-compare", action="store_true",
                    help="skip timing the same steps under IEEE arithmetic (the line itself uses the reference's GPU arithmetic)")
    ap.add_argument("--clock-log", default=None, help="write the raw nvidia-smi clock samples of the timed region to this CSV")
    return ap.parse_args()


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def profile_traffic(kernel: str):
    """dram bytes per launch for `kernel` from the committed ncu summaries
    (line 'traffic_bytes_per_launch <kernel> <bytes>')."""
    d = os.path.join(ROOT, "profiles")
    if not os.path.isdir(d):
        return None
    for fn in sorted(os.listdir(d)):
        if not fn.endswith((".md", ".txt")):
            continue
        for line in open(os.path.join(d, fn)):
            parts = line.strip().strip("`").split()
            if len(parts) == 3 and parts[0] == "traffic_bytes_per_launch" and parts[1] == kernel:
                return float(parts[2])
    return None


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled during the timed region."""

    def __init__(self, index: int, path: str | None = None):
        self.index = index
        self.proc = None
        self.path = path  # raw samples are written here when given (--clock-log)

    def start(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                          "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        time.sleep(0.3)
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except Exception:
            self.proc.kill()
            out = ""
        if self.path:
            with open(self.path, "w") as f:
                f.write(out)
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in out.splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


def dist_env():
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    local = int(os.environ.get("LOCAL_RANK", 0))
    return rank, world, local


def max_over_ranks(value: float, world: int, device=None) -> float:
    """The largest value over all ranks (the slowest replica's time); the only
    collective of the benchmark: replicas share no data."""
    if world <= 1:
        return value
    import torch
    import torch.distributed as dist
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ------------------------------------------------------------------ CPU (oracle port)

def cpu_frames(seq, pairs):
    out = []
    for p in range(pairs):
        fr = seq.frame(p)
        for b in TS:
            out.append((fr, seq.client(p, b)))
    return out


def time_cpu(frames, budget_s: float, max_frames: int):
    """Times the oracle port (all OpenMP threads) frame by frame; returns (Mpix/s, frames, seconds)."""
    import numpy as np

    import oracle
    n, t_total, i = 0, 0.0, 0
    prev = np.zeros((H, W, 4), np.uint8)
    while n < max_frames and (t_total < budget_s or n == 0):
        fr, cl = frames[i % len(frames)]
        call = oracle.prepared_call(fr, cl, prev)
        t0 = time.perf_counter()
        call()
        t_total += time.perf_counter() - t0
        n += 1
        i += 1
    return (n * W * H / 1e6 / t_total if n else 0.0), n, t_total


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    import oracle
    from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence

    oracle.build()
    seq = Sequence(W, H, 2, seed=args.seed, aux_offsets=AUX, shadows=True)
    frames = cpu_frames(seq, 1)
    time_cpu(frames, float("inf"), args.warmup)              # warm-up frames
    mpix_s, n, secs = time_cpu(frames, float("inf"), args.steps)  # exactly K frames
    cores = os.cpu_count()
    line = {
        "impl": "reference", "metric": METRIC, "value": round(mpix_s, 3), "unit": "Mpix/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(secs * 1e3 / n, 3), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "step": "one 1080p interpolated frame (t cycling 0.25/0.5/0.75)"},
        "cpu_baseline": {"value": round(mpix_s, 3), "unit": "Mpix/s", "cores": cores, "kind": "port",
                         "sample": f"{n} frames of the workload, C oracle restating src/renderer.cu, OpenMP over {cores} threads"},
        "e2e": {"value": round(mpix_s, 3), "unit": "Mpix/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


# ------------------------------------------------------------------ GPU (ours)

def main_ours(args):
    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import _build, native
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, DeviceView, Renderer
    from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence

    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    _build.build_all()
    dev = torch.device("cuda", local)
    P = args.pairs
    seq = Sequence(W, H, P + 1, seed=args.seed + rank, aux_offsets=AUX, shadows=True)
    n_cams = 1 + len(AUX)

    # ---- resident keyframes: per keyframe k, camera c: colour, z, motions, shadows
    def up(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    res = {}
    for k in range(P + 1):
        for c in range(n_cams):
            kf = seq.keyframe(k, c)
            res[(k, c)] = dict(color=up(kf.color), z=up(kf.z), mf=up(kf.motion_fwd), mb=up(kf.motion_bwd),
                               sf=[up(a) for a in kf.shadow_fwd], sb=[up(a) for a in kf.shadow_bwd],
                               vp=kf.viewproj.astype(np.float32), ivp=np.linalg.inv(kf.viewproj).astype(np.float32))

    def dview(d, forward):
        sh = d["sf"] if forward else d["sb"]
        return DeviceView(d["color"], d["z"], d["mf"] if forward else d["mb"], sh[0], sh[1], sh[2], d["vp"], d["ivp"])

    frames = []
    for p in range(P):
        fr = DeviceFrame(dview(res[(p, 0)], True), dview(res[(p + 1, 0)], False))
        for c in range(1, n_cams):
            fr.aux_curr.append(dview(res[(p, c)], True))
            fr.aux_next.append(dview(res[(p + 1, c)], False))
            fr.aux_priority.append(3)
        frames.append(fr)
    from imagebasedspatiotemporalinterpolation_gb300.renderer import render_info
    clients = [[render_info(seq.client(p, b)) for b in TS] for p in range(P)]
    out = torch.zeros((H, W, 4), dtype=torch.uint8, device=dev)
    r = Renderer()
    # the reference's own GPU arithmetic (its -use_fast_math build, CMakeLists.txt:36): every
    # key, flow and pixel bit-exact against the reference's sm_103a build; the IEEE mode
    # (bit-exact against the reference compiled for the CPU) is timed beside it
    r.set_arithmetic(native.ARITH_REFERENCE_GPU)
    stream = torch.cuda.current_stream(dev)

    outs = [torch.zeros((H, W, 4), dtype=torch.uint8, device=dev) for _ in TS]

    def step(s):
        p = s % P
        r.render_batch(outs, clients[p], frames[p], chain=True, stream=stream)

    for s in range(args.warmup):
        step(s)
    torch.cuda.synchronize()

    # ---- timed region (device-resident inputs): one batched call per keyframe interval
    sev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    clocks = ClockSampler(local, args.clock_log)
    r.timing()          # discard warm-up
    r.enable_timing(True)
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clocks.start()
    t0.record(stream)
    for s in range(args.steps):
        sev[s][0].record(stream)
        step(s)
        sev[s][1].record(stream)
    t1.record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    r.enable_timing(False)
    ms = t0.elapsed_time(t1)
    tim = r.timing()
    ms = max_over_ranks(ms, world, dev)
    step_ms = sorted(a.elapsed_time(b) for a, b in sev)
    n_frames = args.steps * len(TS)
    value = world * n_frames * W * H / 1e6 / (ms / 1e3)

    # ---- the same steps under IEEE arithmetic (ISTI_ARITH_IEEE: -fmad=false and correctly
    # rounded division and roots, bit-exact against the reference's code run on the CPU)
    arith = None
    if not args.no_arith_compare:
        r.set_arithmetic(native.ARITH_IEEE)
        for s in range(args.warmup):
            step(s)
        torch.cuda.synchronize()
        r.timing()
        r.enable_timing(True)
        f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f0.record(stream)
        for s in range(args.steps):
            step(s)
        f1.record(stream)
        torch.cuda.synchronize()
        r.enable_timing(False)
        ftim = r.timing()
        fcalls = max(1, ftim["frames"] // len(TS))
        fms = f0.elapsed_time(f1)
        arith = {"arithmetic": "IEEE (bit-exact against the CPU oracle)", "value": round(n_frames * W * H / 1e6 / (fms / 1e3), 2), "unit": "Mpix/s",
                 "ms_per_step": round(fms / args.steps, 4),
                 "kernels_ms_per_call": {"key_init": round(ftim["init_ms"] / fcalls, 4), "splat_kernel": round(ftim["splat_ms"] / fcalls, 4),
                                         "reproj_kernel": round(ftim["reproj_ms"] / fcalls, 4)}}
        r.set_arithmetic(native.ARITH_REFERENCE_GPU)

    # ---- the same frames through the single-frame call (isti_render), for comparison
    per_frame = None
    if not args.no_per_frame:
        fev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(n_frames)]
        torch.cuda.synchronize()
        a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a0.record(stream)
        fi = 0
        for s in range(args.steps):
            p = s % P
            for ci in clients[p]:
                fev[fi][0].record(stream)
                r.render(out, ci, frames[p], stream)
                fev[fi][1].record(stream)
                fi += 1
        a1.record(stream)
        torch.cuda.synchronize()
        frame_ms = sorted(a.elapsed_time(b) for a, b in fev)
        per_frame = {"value": round(n_frames * W * H / 1e6 / (a0.elapsed_time(a1) / 1e3), 2), "unit": "Mpix/s",
                     "p50_frame_ms": round(frame_ms[len(frame_ms) // 2], 4),
                     "p99_frame_ms": round(frame_ms[min(len(frame_ms) - 1, int(0.99 * len(frame_ms)))], 4)}

    # ---- e2e: host buffers through the C ABI, uploads + read-back inside the timed region
    e2e = None
    if not args.no_e2e:
        e2e = run_e2e(args, seq, res, clients, r, dev, world)

    # ---- the batched mixed-resolution workload under one CUDA graph (reported beside the line)
    graph_batch = None
    if not args.no_graph_batch:
        graph_batch = run_graph_batch(args, dev, rank)

    # ---- the serving loop: simulated clients in real time (reported beside the line)
    serving = None
    if not args.no_serving:
        serving = run_serving(args, dev, rank)
        if not args.no_pressure:
            serving["pressure"] = run_serving(args, dev, rank, pressure=True)

    # ---- learned initialiser vs plain at 1080p, one 640x360 frame per call, the reference's own GPU build
    learned = None if args.no_learned else run_learned(args, dev, rank)
    small_frame = None if args.no_small_frame else run_small_frame(args, dev, rank)
    reference_gpu = None
    if rank == 0 and not args.no_reference_gpu:
        reference_gpu = run_reference_gpu(args, dev, seq, per_frame["p50_frame_ms"] if per_frame else None)

    # ---- roofline of the dominant kernel.  Algorithmic bytes per interpolated output pixel
    # (the per-unit figure of the path): every source view's inputs once and the output once,
    # 6 views x (4 z + 6 f16 motion + 4 colour + 12 shadow A/B/Info) + 4 = 160 B.  Split by the
    # kernel that reads them: splat z + motion (60 B), reprojection colour + shadows + output
    # (100 B); one launch processes len(TS) frames of W x H output pixels.  The batched call
    # reads each input once for all its frames, so "achieved" is the effective bandwidth of the
    # per-frame data flow; the inputs-once figure is reported beside it.
    px = W * H
    n_views = 2 * n_cams
    calls = max(1, tim["frames"] // len(TS))  # one batched call per step
    out_px = len(TS) * px
    alg = {"splat_kernel": n_views * (4 + 6) * out_px, "reproj_kernel": (n_views * (4 + 12) + 4) * out_px}
    once = {"splat_kernel": n_views * (4 + 6) * px, "reproj_kernel": n_views * (4 + 12) * px + len(TS) * 4 * px}
    per_launch_ms = {"splat_kernel": tim["splat_ms"] / calls, "reproj_kernel": tim["reproj_ms"] / calls}
    dom = max(per_launch_ms, key=per_launch_ms.get)
    peak, peak_kind = peaks()
    achieved = alg[dom] / (per_launch_ms[dom] / 1e3) / 1e9
    traffic = profile_traffic(dom)
    roof = {"kernel": dom, "bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
            "frac": round(achieved / peak, 4), "peak_kind": peak_kind, "traffic": traffic,
            "algorithmic_bytes_per_launch": alg[dom], "bytes_per_output_px": alg[dom] // out_px,
            "inputs_once_bytes_per_launch": once[dom],
            "inputs_once_frac": round(once[dom] / (per_launch_ms[dom] / 1e3) / 1e9 / peak, 4)}

    # ---- quality of the interpolated frames of pair 0 against the analytic ray-cast of
    # the client camera at its own time (outside the timed region), by the GPU metric
    # kernels (PSNR / SSIM of the reference's evaluation script)
    quality = None
    if rank == 0 and not args.no_quality:
        from imagebasedspatiotemporalinterpolation_gb300.metrics import Quality
        qouts = [torch.zeros((H, W, 4), dtype=torch.uint8, device=dev) for _ in TS]
        r.render_batch(qouts, clients[0], frames[0], chain=True, stream=stream)
        q = Quality(W, H, dev)
        vals = []
        for o, b in zip(qouts, TS):
            truth = up(seq.ground_truth(0, b))
            vals.append(q(o, truth))
            vals[-1]["flip"] = q.flip(o, truth)
        qa, qb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        qa.record(stream)
        for _ in range(10):
            q.launch(qouts[0], truth)
        qb.record(stream)
        fa, fb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        fa.record(stream)
        for _ in range(10):
            q.flip(qouts[0], truth)
        fb.record(stream)
        torch.cuda.synchronize()
        mean = lambda key: sum(v[key] for v in vals) / len(vals)
        quality = {"psnr_db": round(mean("psnr"), 3), "ssim": round(mean("ssim"), 5), "flip": round(mean("flip"), 5),
                   "per_t": {str(t): {"psnr_db": round(v["psnr"], 3), "ssim": round(v["ssim"], 5), "flip": round(v["flip"], 5)}
                             for t, v in zip(TS, vals)},
                   "reference": "analytic ray-cast of the client camera at its time (procedural scene)",
                   "psnr_ssim_kernel_ms": round(qa.elapsed_time(qb) / 10, 4),
                   "flip_ms": round(fa.elapsed_time(fb) / 10, 4)}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        import oracle
        oracle.build()
        host_seq = Sequence(W, H, 2, seed=args.seed, aux_offsets=AUX, shadows=True)
        mpix_s, n, secs = time_cpu(cpu_frames(host_seq, 1), args.cpu_seconds, 30)
        cpu = {"value": round(mpix_s, 3), "unit": "Mpix/s", "cores": os.cpu_count(), "kind": "port",
               "sample": f"{n} frames ({secs:.1f} s) of the same workload, C oracle (OpenMP, all threads)"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 2), "unit": "Mpix/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "arithmetic": "reference GPU (fast-math; bit-exact against the reference's sm_103a build)",
                       "width": W, "height": H, "source_views": n_views, "frames_per_step": len(TS),
                       "resident_pairs": P, "mode": 0, "l2": "inputs larger than L2 (~0.8 GB touched per frame)",
                       "parallelism": f"replicas x{world}"},
            "p50_step_ms": round(step_ms[len(step_ms) // 2], 4),
            "p99_step_ms": round(step_ms[min(len(step_ms) - 1, int(0.99 * len(step_ms)))], 4),
            "kernels_ms_per_call": {"key_init": round(tim["init_ms"] / calls, 4),
                                    "splat_kernel": round(per_launch_ms["splat_kernel"], 4),
                                    "reproj_kernel": round(per_launch_ms["reproj_kernel"], 4)},
            "per_frame_api": per_frame,
            "arith_ieee": arith,
            "learned_vs_plain": learned,
            "frame_640x360": small_frame,
            "reference_gpu": reference_gpu,
            "graph_batch_mixed": graph_batch,
            "serving": serving,
            "gpu_launches": tim["kernel_launches"],
            "clocks": clk,
            "e2e": e2e,
            "roofline": roof,
            "cpu_baseline": cpu,
            "quality": quality,
        }
        print(json.dumps(line), flush=True)
    r.close()
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


def run_reference_gpu(args, dev, seq, ours_frame_ms):
    """The reference's own renderer.cu built for sm_103a with its -use_fast_math flags
    (oracle/_ref/libisti_ref_gpu.so, staged from the reference sources), timed on this GPU
    as its frame loop runs it: one Renderer::render per client frame on the legacy default
    stream (its memsets, splat launches, host synchronisation, aux-info copy and
    reprojection launch), CUDA events around each call.  Same keyframes and client frames
    as the main workload.  A baseline reported beside the line, not the measured product."""
    import numpy as np

    import oracle
    if not oracle.reference_gpu_available():
        return {"unavailable": "reference sources not staged (oracle/build_ref.py needs the reference tree)"}
    out = {}
    for name, (sq, ts) in {"frame_1080p_6views_shadows": (seq, TS)}.items():
        frame = sq.frame(0)
        ms = oracle.time_reference_gpu(frame, [sq.client(0, b) for b in ts], warmup=max(3, args.warmup), repeats=10)
        p50 = float(np.median(ms))
        out[name] = {"ms_per_frame_p50": round(p50, 4), "ms_per_frame_p99": round(float(np.percentile(ms, 99)), 4),
                     "mpix_s": round(sq.width * sq.height / 1e6 / (p50 / 1e3), 2), "frames_timed": int(ms.size)}
    out["frame_1080p_6views_shadows"]["ours_per_frame_call_ms_p50"] = ours_frame_ms
    out["build"] = "src/renderer.cu unmodified, nvcc -arch sm_103a -use_fast_math --expt-relaxed-constexpr (CMakeLists.txt:36)"
    return out


def run_small_frame(args, dev, rank):
    """One interpolated frame at t = 0.5 between two 640x360
    keyframes, main camera only, mode 0, no shadows.  Device-resident keyframes, one
    isti_render call per step on 5 resident pairs in turn; the reference GPU build and the
    CPU port (the C oracle, all threads) timed on the same frames."""
    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import native
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer, render_info
    from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence
    import oracle

    w, h, pairs = 640, 360, 5
    seq = Sequence(w, h, pairs + 1, seed=args.seed + 11 + rank)
    frames = [DeviceFrame.from_host(seq.frame(p), dev) for p in range(pairs)]
    host_clients = [seq.client(p, 2) for p in range(pairs)]
    clients = [render_info(c) for c in host_clients]  # marshalled once, like the main line's
    out = torch.zeros((h, w, 4), dtype=torch.uint8, device=dev)
    r = Renderer()
    r.set_arithmetic(native.ARITH_REFERENCE_GPU)  # as the reference GPU build timed beside it
    for s in range(max(3, args.warmup)):
        r.render(out, clients[s % pairs], frames[s % pairs])
    n = max(60, args.steps * 3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(n)]
    torch.cuda.synchronize()
    for s, (a, b) in enumerate(ev):
        a.record()
        r.render(out, clients[s % pairs], frames[s % pairs])
        b.record()
    torch.cuda.synchronize()
    ms = sorted(a.elapsed_time(b) for a, b in ev)
    r.timing()
    r.enable_timing(True)           # a second pass for the per-kernel split (its events cost host time)
    for s in range(n):
        r.render(out, clients[s % pairs], frames[s % pairs])
    torch.cuda.synchronize()
    r.enable_timing(False)
    tim = r.timing()
    # the same calls replayed from one CUDA graph: the device time without the host's per-call work
    stream = torch.cuda.Stream(dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            for s in range(pairs):
                r.render(out, clients[s], frames[s], stream)
        graph.replay()
        g0, g1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        g0.record(stream)
        for _ in range(n // pairs):
            graph.replay()
        g1.record(stream)
    torch.cuda.synchronize()
    graph_ms = g0.elapsed_time(g1) / ((n // pairs) * pairs)
    r.close()
    res = {"workload": "640x360, main camera only, t = 0.5, mode 0, no shadows (one isti_render call per frame)",
           "arithmetic": "reference GPU (fast-math)",
           "mpix_s": round(n * w * h / 1e6 / (sum(ms) / 1e3), 2), "p50_frame_ms": round(ms[len(ms) // 2], 4),
           "p99_frame_ms": round(ms[min(len(ms) - 1, int(0.99 * len(ms)))], 4),
           "kernels_ms_per_frame": {"key_init": round(tim["init_ms"] / n, 4), "splat_kernel": round(tim["splat_ms"] / n, 4),
                                    "reproj_kernel": round(tim["reproj_ms"] / n, 4)},
           "graph_replayed_ms_per_frame": round(graph_ms, 4)}
    if rank == 0 and oracle.reference_gpu_available():
        rg = oracle.time_reference_gpu(seq.frame(0), [host_clients[0]], warmup=5, repeats=30)
        res["reference_gpu_ms_per_frame_p50"] = round(float(np.median(rg)), 4)
    if rank == 0 and not args.no_cpu_baseline:
        oracle.build()
        fr = seq.frame(0)
        call = oracle.prepared_call(fr, host_clients[0], np.zeros((h, w, 4), np.uint8))
        call()
        t0, k = time.perf_counter(), 0
        while time.perf_counter() - t0 < min(args.cpu_seconds, 5.0) or k == 0:
            call()
            k += 1
        secs = time.perf_counter() - t0
        res["cpu_baseline"] = {"value": round(k * w * h / 1e6 / secs, 3), "unit": "Mpix/s", "cores": os.cpu_count(), "kind": "port",
                               "sample": f"{k} frames ({secs:.1f} s), C oracle (OpenMP, all threads)"}
    return res


def run_learned(args, dev, rank):
    """Learned initialiser vs the plain method (held-out scenes of its training distribution):
    1920x1080 held-out seeds of the training distribution (U[16, 256] spheres, |v| <= 1
    m/s, camera rotation <= 5 degrees per keyframe interval), main camera only, t in
    {0.25, 0.5, 0.75}.  Per step one call renders the 3 frames of a keyframe pair: the plain
    path (isti_render_batch: splat + 3x3 window + 3 search iterations) or the learned path
    (isti_render_learned: U-Net on tcgen05 + 1 search iteration + per-tile plain fallback),
    on the same device-resident keyframes.  Quality: PSNR of each frame against the analytic
    ray-cast of the client camera at its time, previous output = the previous ground truth
    frame (temporal hole filling), for both paths."""
    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import train_flownet
    from imagebasedspatiotemporalinterpolation_gb300.metrics import Quality
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer
    from imagebasedspatiotemporalinterpolation_gb300.scene import Sequence

    if not os.path.exists(train_flownet.DEFAULT_WEIGHTS):
        return {"unavailable": "no trained weights (run train_flownet)"}
    net = train_flownet.load()
    w, h, n_seeds = 1920, 1080, 2
    seqs, frames, clients, truths, prevs = [], [], [], [], []
    for i in range(n_seeds):
        seed = train_flownet.EVAL_SEED_BASE + 7 + i
        rng = np.random.default_rng(seed)
        sq = Sequence(w, h, 2, seed=seed, n_spheres=int(rng.integers(16, 257)), max_speed=1.0, max_rot_deg=5.0, max_step_m=0.1)
        seqs.append(sq)
        frames.append(DeviceFrame.from_host(sq.frame(0), dev))
        clients.append([sq.client(0, b) for b in TS])
        gt = [torch.from_numpy(sq.ground_truth(0, b)).to(dev) for b in [0] + list(TS)]
        gt[0] = torch.from_numpy(sq.frame(0).fwd.color).to(dev)
        truths.append(gt[1:])
        prevs.append(gt[:-1])
    r = Renderer()
    outs = [torch.zeros((h, w, 4), dtype=torch.uint8, device=dev) for _ in TS]
    paths = {"plain": lambda i: r.render_batch(outs, clients[i], frames[i], chain=False),
             "learned": lambda i: r.render_learned(outs, clients[i], frames[i], net, 1)}
    res = {}
    for name, fn in paths.items():
        for s in range(max(3, args.warmup)):
            fn(s % n_seeds)
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        torch.cuda.synchronize()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        for s, (a, b) in enumerate(ev):
            a.record()
            fn(s % n_seeds)
            b.record()
        t1.record()
        torch.cuda.synchronize()
        ms = sorted(a.elapsed_time(b) for a, b in ev)
        total = t0.elapsed_time(t1)
        res[name] = {"mpix_s": round(args.steps * len(TS) * w * h / 1e6 / (total / 1e3), 2), "p50_call_ms": round(ms[len(ms) // 2], 4),
                     "p99_call_ms": round(ms[min(len(ms) - 1, int(0.99 * len(ms)))], 4)}
    # quality (outside the timed regions)
    q = Quality(w, h, dev)
    psnr = {k: [] for k in paths}
    vs_plain, fallback = [], []
    for i in range(n_seeds):
        got = {}
        for name in paths:
            o = [p.clone() for p in prevs[i]]
            if name == "plain":
                r.render_batch(o, clients[i], frames[i], chain=False)
            else:
                r.render_learned(o, clients[i], frames[i], net, 1)
                fb, tiles = r.learned_stats()
                fallback.append(fb / max(1, tiles))
            got[name] = o
            psnr[name] += [q(a, t)["psnr"] for a, t in zip(o, truths[i])]
        vs_plain += [q(a, b)["psnr"] for a, b in zip(got["learned"], got["plain"])]
    r.close()
    net.close()
    mean = lambda v: float(sum(v) / len(v))
    res["ratio_learned_over_plain"] = round(res["learned"]["mpix_s"] / res["plain"]["mpix_s"], 3)
    res["psnr_vs_truth_db"] = {k: round(mean(v), 3) for k, v in psnr.items()}
    res["dpsnr_db"] = round(mean(psnr["plain"]) - mean(psnr["learned"]), 3)
    res["psnr_learned_vs_plain_db"] = round(mean([v for v in vs_plain if v != float("inf")] or [float("inf")]), 2)
    res["fallback_tile_frac"] = round(mean(fallback), 4)
    res["workload"] = ("1920x1080 held-out seeds, main camera only, 3 frames (t = 0.25/0.5/0.75) per call, "
                       "learned: 1 search iteration (plain: 3) + per-tile plain fallback")
    return res


GB_RES = ((1280, 720), (1920, 1080), (2064, 2208))
GB_PAIRS = 16
GB_EYES = (-0.032, 0.032)  # half the interpupillary distance, metres
SV_CLIENTS = 16
PRESSURE_CLIENTS = 256        # open sessions under pressure: more than the 120 GB budget admits
PRESSURE_SESSION_S = 8.0      # mean session length under pressure (a closing client is replaced)
PRESSURE_MAX_WAITING = 8      # back-pressure: waiting requests per eye before refusing


def run_serving(args, dev, rank, pressure=False):
    """The serving workload of the benchmark list: 16 simulated clients, each sending stereo
    frame requests as a Poisson process at a rate drawn from U[90, 120] Hz and receiving a
    new keyframe pair every 1/30 s, at 1280x720 / 1920x1080 / 2064x2208 per eye in turn,
    main camera only, no shadows; keyframes resident on the device, admission against a
    120 GB budget, 4 slots, batches of up to 8 frames.  Runs in real time for
    --serve-seconds, then drains; latency is from a request's scheduled arrival to the loop
    seeing its batch done.  Keyframe pairs are uploaded from pinned host memory as they
    arrive (each client cycles through two pre-rendered pairs of its resolution).

    pressure=True: 256 open sessions of the same kind for --pressure-seconds, each ending
    after an exponential session (mean 8 s) and replaced by a new client: more clients than
    the budget admits (the rest wait, deferred, in arrival order) and more frames than the
    device renders (an eye with 8 requests waiting refuses the next)."""
    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import scene
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame
    from imagebasedspatiotemporalinterpolation_gb300.serving import CudaBackend, PinnedPair, Server, SimClient, eye_info, simulate

    rng = np.random.default_rng(args.seed + 7 + rank)
    seqs = {}
    for j, (w, h) in enumerate(GB_RES):
        seq = scene.Sequence(w, h, 3, seed=args.seed + 301 * (j + 1) + rank)
        seqs[(w, h)] = (seq, [PinnedPair(seq.frame(p)) for p in range(2)])
    max_w, max_h = max(GB_RES, key=lambda r: r[0] * r[1])
    from imagebasedspatiotemporalinterpolation_gb300 import train_flownet
    weights = train_flownet.DEFAULT_WEIGHTS if (args.serve_learned and os.path.exists(train_flownet.DEFAULT_WEIGHTS)) else None
    backend = CudaBackend(dev, learned_weights=weights)
    server = Server(backend, hbm_budget=120 << 30, n_slots=args.serve_slots, max_batch=8,
                    slot_pixels=max_w * max_h, slot_views=2, max_waiting=PRESSURE_MAX_WAITING if pressure else None)
    # every slot's renderer (and network) sized once for the largest batch (no allocation while serving)
    big_seq = seqs[(max_w, max_h)][0]
    big = DeviceFrame.from_host(big_seq.frame(0), dev)
    outs = [torch.zeros((max_h, max_w, 4), dtype=torch.uint8, device=dev) for _ in range(8)]
    infos = [eye_info(big_seq, 0, b / 8, GB_EYES[0]) for b in range(8)]
    for slot in server.slots:
        stream, renderer = slot[0], slot[1]
        renderer.render_batch(outs, infos, big, chain=True, stream=stream)
        if len(slot) > 2:
            renderer.render_learned(outs, infos, big, slot[2], 1, chain=True, stream=stream)
    torch.cuda.synchronize()
    del outs, big
    sims = []
    n_clients = PRESSURE_CLIENTS if pressure else SV_CLIENTS
    seconds = args.pressure_seconds if pressure else args.serve_seconds
    for c in range(n_clients):
        w, h = GB_RES[c % len(GB_RES)]
        seq, pairs = seqs[(w, h)]
        server.open_client(c, w, h, len(GB_EYES), pairs[0])
        sims.append(SimClient(c, seq, pairs, rate_hz=float(rng.uniform(90.0, 120.0)), phase_s=float(rng.uniform(0.0, 1.0 / 30))))
    torch.cuda.synchronize()
    st = simulate(server, sims, seconds=seconds, eyes=GB_EYES, seed=args.seed + rank,
                  session_mean_s=PRESSURE_SESSION_S if pressure else None,
                  rate_hz=(lambda g: g.uniform(90.0, 120.0)) if pressure else None)
    torch.cuda.synchronize()
    out = {"mpix_per_s": round(st["mpix_per_s"], 1), "p50_ms": round(st["p50_ms"], 3), "p99_ms": round(st["p99_ms"], 3),
           "requests": st["requests"], "offered_requests": st["offered_requests"], "refused_requests": st["refused_requests"],
           "batches": st["batches"], "frames_per_batch": round(st["frames_per_batch"], 2), "keyframe_uploads": st["uploads"],
           "clients": st["clients"], "admitted": st["admitted"], "seconds": seconds,
           "reserved_gb": round(st["peak_reserved_bytes"] / 2**30, 2), "budget_gb": 120, "slots": args.serve_slots,
           "method": "learned initialiser (1 iteration) + per-tile plain fallback" if weights else "plain",
           "learned_batches": backend.learned_batches, "plain_batches": backend.plain_batches,
           "workload": f"{n_clients} clients, stereo requests Poisson U[90,120] Hz, keyframe pairs 30 Hz, 1280x720 / 1920x1080 / "
                       "2064x2208 per eye, main camera only, continuous batching"}
    if pressure:
        out.update({"refused_not_admitted": st["refused_not_admitted"], "refused_queue_full": st["refused_queue_full"],
                    "max_waiting_per_eye": PRESSURE_MAX_WAITING, "sessions_closed": st["sessions_closed"],
                    "clients_opened": st["clients_opened"], "deferred_clients": st["deferred_clients"],
                    "peak_waiting_clients": st["peak_waiting_clients"],
                    "admission_wait_p50_ms": round(st["admission_wait_p50_ms"], 1),
                    "admission_wait_p99_ms": round(st["admission_wait_p99_ms"], 1),
                    "session_mean_s": PRESSURE_SESSION_S})
    del server, backend
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return out


def run_graph_batch(args, dev, rank):
    """The batched workload of the benchmark list: 16 keyframe pairs x 3 t values x 2 eyes,
    the pairs at 1280x720, 1920x1080 and 2064x2208 in turn (6, 5, 5 pairs: 241.7 Mpix per
    batch), main-camera buffers only (no aux cameras, no shadows), plain method.  Each
    pair's 6 frames are one isti_render_batch call; the 16 calls are captured once into a
    CUDA graph, replayed `warmup` times untimed and `steps` times timed (keyframes
    resident; inputs and intermediates of a replay far larger than L2).  Afterwards one
    pair per resolution is checked against per-frame isti_render calls."""
    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import scene
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, Renderer, render_info

    def eye_client(seq, k, b, offset):
        t = b / seq.fpa
        pose = seq.poses[k].lerp(seq.poses[k + 1], t)
        eye = pose.eye + scene.right_vector(pose.yaw, pose.pitch) * offset
        vp = seq.proj_main @ scene.view_matrix(eye, pose.yaw, pose.pitch)
        return scene.Client(seq.width, seq.height, float(np.float32(t)), vp.astype(np.float32),
                            np.linalg.inv(vp).astype(np.float32), seq.fpa, seq.sfpa, False, 0)

    jobs, first_of_res = [], []
    for j, (w, h) in enumerate(GB_RES):
        n_pairs = len(range(j, GB_PAIRS, len(GB_RES)))
        seq = scene.Sequence(w, h, n_pairs + 1, seed=args.seed + 101 * (j + 1) + rank)
        first_of_res.append(len(jobs))
        for k in range(n_pairs):
            infos = [render_info(eye_client(seq, k, b, e)) for b in TS for e in GB_EYES]
            jobs.append((w, h, DeviceFrame.from_host(seq.frame(k), dev), infos))
    mpix = sum(w * h * len(infos) for w, h, _, infos in jobs) / 1e6
    r = Renderer()
    r.set_autotune(True)   # the uncaptured first pass tunes each resolution's reprojection launch
    stream = torch.cuda.Stream(dev)
    outs = [[torch.zeros((h, w, 4), dtype=torch.uint8, device=dev) for _ in infos] for w, h, _, infos in jobs]
    with torch.cuda.stream(stream):
        for (w, h, frame, infos), o in zip(jobs, outs):   # sizes the arena and tunes before the capture
            r.render_batch(o, infos, frame, chain=False, stream=stream)
    stream.synchronize()
    tuned = [{"size": f"{t['width']}x{t['height']}", "regs": t["regs"], "row_pairs": t["row_pairs"],
              "key_tiles": "plain loads" if t["plain_tiles"] else "TMA",
              "reproj_ms": round(t["best_ms"], 4), "rule_reproj_ms": round(t["rule_ms"], 4)} for t in r.tuning()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        with torch.cuda.graph(graph, stream=stream):
            for (w, h, frame, infos), o in zip(jobs, outs):
                r.render_batch(o, infos, frame, chain=False, stream=stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(max(args.warmup, 3)):
            graph.replay()
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        stream.synchronize()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        for e0, e1 in ev:
            e0.record(stream)
            graph.replay()
            e1.record(stream)
        t1.record(stream)
    stream.synchronize()
    ms = t0.elapsed_time(t1) / args.steps
    batch_ms = sorted(a.elapsed_time(b) for a, b in ev)
    # outside the timed region: the replayed frames equal per-frame calls (one pair per resolution)
    single = Renderer()
    for idx in first_of_res:
        w, h, frame, infos = jobs[idx]
        o = outs[idx]
        for k, info in enumerate(infos):
            ref = torch.zeros((h, w, 4), dtype=torch.uint8, device=dev)
            single.render(ref, info, frame, stream)
            stream.synchronize()
            if not torch.equal(ref, o[k]):
                raise RuntimeError(f"graph batch: {w}x{h} frame {k} differs from the per-frame call")
    single.close()
    r.close()

    # the same batch as ONE persistent launch (isti_render_pairs with unit sizes set, which asks for
    # it: a cooperative kernel over a device work queue of init / splat / reprojection units; without
    # them pairs of this size are rendered as batches), captured once and replayed; its
    # frames must equal the 48-launch graph's bit for bit
    persistent = None
    try:
        rp = Renderer()
        rp.set_pair_units(32, 256)
        pouts = [[torch.zeros_like(o) for o in os_] for os_ in outs]
        pjobs = [(po, infos, frame) for po, (w, h, frame, infos) in zip(pouts, jobs)]
        with torch.cuda.stream(stream):
            rp.render_pairs(pjobs, stream=stream)       # sizes the arena outside the capture
        stream.synchronize()
        pgraph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            with torch.cuda.graph(pgraph, stream=stream):
                rp.render_pairs(pjobs, stream=stream)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(max(args.warmup, 3)):
                pgraph.replay()
            pev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
            stream.synchronize()
            p0, p1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            p0.record(stream)
            for e0, e1 in pev:
                e0.record(stream)
                pgraph.replay()
                e1.record(stream)
            p1.record(stream)
        stream.synchronize()
        pms = p0.elapsed_time(p1) / args.steps
        pb = sorted(a.elapsed_time(b) for a, b in pev)
        same = all(torch.equal(a, b) for po, o in zip(pouts, outs) for a, b in zip(po, o))
        if not same:
            raise RuntimeError("persistent launch: frames differ from the per-pair launches")
        if rp.device_status() != 0:
            raise RuntimeError("persistent launch: a bounded wait gave up")
        # work-unit sizes (isti_renderer_set_pair_units), uncaptured calls; the output must not change
        sizes = []
        for rows, kib in ((16, 64), (8, 64), (32, 256), (64, 1024)):
            rp.set_pair_units(rows, kib)
            with torch.cuda.stream(stream):
                for _ in range(2):
                    rp.render_pairs(pjobs, stream=stream)
                u0, u1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                u0.record(stream)
                for _ in range(5):
                    rp.render_pairs(pjobs, stream=stream)
                u1.record(stream)
            stream.synchronize()
            ok = all(torch.equal(a, b) for po, o in zip(pouts, outs) for a, b in zip(po, o)) and rp.device_status() == 0
            sizes.append({"splat_rows": rows, "init_unit_kib": kib, "ms_per_batch": round(u0.elapsed_time(u1) / 5, 4), "equal": ok})
        rp.close()
        persistent = {"value": round(mpix / (pms / 1e3), 2), "unit": "Mpix/s", "ms_per_batch": round(pms, 4),
                      "p50_batch_ms": round(pb[len(pb) // 2], 4), "p99_batch_ms": round(pb[min(len(pb) - 1, int(0.99 * len(pb)))], 4),
                      "launches_per_batch": 1, "equal_to_per_pair_launches": True, "unit_sizes_uncaptured": sizes}
    except Exception as ex:  # reported, not fatal: the per-pair graph is the reference line
        persistent = {"error": str(ex)[:300]}
    return {"value": round(mpix / (ms / 1e3), 2), "unit": "Mpix/s", "mpix_per_batch": round(mpix, 2),
            "persistent_single_launch": persistent,
            "frames_per_batch": sum(len(infos) for _, _, _, infos in jobs), "ms_per_batch": round(ms, 4),
            "p50_batch_ms": round(batch_ms[len(batch_ms) // 2], 4),
            "p99_batch_ms": round(batch_ms[min(len(batch_ms) - 1, int(0.99 * len(batch_ms)))], 4),
            "launches_per_batch": 3 * len(jobs), "autotuned": tuned,
            "workload": "16 pairs x 3 t x 2 eyes at 1280x720 / 1920x1080 / 2064x2208, main camera only, "
                        "no shadows, mode 0, one CUDA graph per batch, reprojection launches chosen by the autotuner"}


def run_e2e(args, seq, res, clients, r, dev, world):
    """Streams keyframes from pinned host memory through the C ABI.  Per step the
    newly arrived keyframe's data goes up (3 cameras: colour, z, backward motion
    and shadows; plus the earlier keyframe's forward motion and shadows), the 3
    frames are rendered, the 3 frames come back.  Each keyframe's images sit in
    one pinned host slab and one device slab, ordered so that what a step needs
    of it is one contiguous range: 2 large copies per step.  Colour travels as
    packed RGB, shadows as sparse entries (isti_unpack_shadows: the pixels whose
    shadow-info field is non-zero, the only ones the renderer reads); both are
    expanded on the device.  Every keyframe of the cycle has its own device slab,
    so when the steps wrap around to the first pair its earlier keyframe is still
    resident, as in an endless stream.  Three streams overlap the upload of step
    s + 1 and the read-back of step s - 1 with the rendering of step s; the timed
    region spans all of them."""
    import ctypes as C

    import numpy as np
    import torch

    from imagebasedspatiotemporalinterpolation_gb300 import native
    from imagebasedspatiotemporalinterpolation_gb300.renderer import DeviceFrame, DeviceView, pack_shadow_entries

    P = args.pairs
    n_cams = 1 + len(AUX)
    # Slab layout of one keyframe: [arrival part | forward part], each grouped by kind over
    # the cameras.  arrival = colour (packed RGB), z, backward motion, backward shadow entries;
    # forward = forward motion, forward shadow entries.  The colour images come from RGB
    # sources (alpha 255, what an RGB PNG decodes to; asserted below).  Shadow entries have a
    # size of their own per keyframe and camera, so each keyframe has its own layout.
    zb, mot, rgb = H * W * 4, H * W * 6, H * W * 3   # each a multiple of 256 bytes
    pad = lambda n: (n + 255) // 256 * 256
    host, layouts, packs = [], [], []
    for k in range(P + 1):
        kfs = [seq.keyframe(k, c) for c in range(n_cams)]
        for kf in kfs:
            if not (kf.color[..., 3] == 255).all():
                raise RuntimeError("e2e uploads colour as RGB: the source colour must be opaque")
        # the shadow images in (A, B, Info) order: the renderer's shadow_a, shadow_b, shadow_info
        pk = {("sb", c): pack_shadow_entries(kfs[c].shadow_bwd[2], kfs[c].shadow_bwd[0], kfs[c].shadow_bwd[1]) for c in range(n_cams)}
        pk.update({("sf", c): pack_shadow_entries(kfs[c].shadow_fwd[2], kfs[c].shadow_fwd[0], kfs[c].shadow_fwd[1]) for c in range(n_cams)})
        layout, off = {}, 0
        for kind in ("color", "z", "mb", "sb", "mf", "sf"):
            for c in range(n_cams):
                n = {"color": rgb, "z": zb, "mb": mot, "mf": mot}[kind] if kind not in ("sb", "sf") else pk[(kind, c)].nbytes
                layout[(kind, c)] = (off, n)
                off += pad(n)
        layout["A"] = layout[("mf", 0)][0]   # arrival part = [0, A), forward part = [A, total)
        layout["total"] = off
        slab = torch.zeros(off, dtype=torch.uint8).pin_memory()
        put = lambda key, arr: slab[layout[key][0]:layout[key][0] + layout[key][1]].copy_(
            torch.from_numpy(np.ascontiguousarray(arr).reshape(-1).view(np.uint8)))
        for c, kf in enumerate(kfs):
            put(("color", c), kf.color[..., :3])
            put(("z", c), np.asarray(kf.z, np.float32))
            put(("mb", c), np.asarray(kf.motion_bwd, np.float16))
            put(("mf", c), np.asarray(kf.motion_fwd, np.float16))
            for kind in ("sb", "sf"):
                if layout[(kind, c)][1]:
                    put((kind, c), pk[(kind, c)])
        host.append(slab)
        layouts.append(layout)
        packs.append({key: len(v) for key, v in pk.items()})
    ring = [torch.empty(layouts[k]["total"], dtype=torch.uint8, device=dev) for k in range(P + 1)]
    # RGBA images the renderer reads, per slot: arrival [colour per camera, then A, B, Info
    # per camera] and forward [A, B, Info per camera]
    rgba_arr = [torch.empty((4 * n_cams, H, W, 4), dtype=torch.uint8, device=dev) for _ in range(P + 1)]
    rgba_fwd = [torch.empty((3 * n_cams, H, W, 4), dtype=torch.uint8, device=dev) for _ in range(P + 1)]

    def dev_field(slot, kind, c, dtype, shape):
        lo, n = layouts[slot][(kind, c)]
        return ring[slot][lo:lo + n].view(dtype).view(*shape)

    ring_fields = []
    for slot in range(P + 1):
        per_cam = []
        for c in range(n_cams):
            per_cam.append(dict(color=rgba_arr[slot][c], z=dev_field(slot, "z", c, torch.float32, (H, W)),
                                mb=dev_field(slot, "mb", c, torch.float16, (H, W, 3)), mf=dev_field(slot, "mf", c, torch.float16, (H, W, 3)),
                                sb=[rgba_arr[slot][n_cams + 3 * c + i] for i in range(3)],
                                sf=[rgba_fwd[slot][3 * c + i] for i in range(3)]))
        ring_fields.append(per_cam)
    lib = native.load()
    outs_dev = [[torch.zeros((H, W, 4), dtype=torch.uint8, device=dev) for _ in TS] for _ in range(2)]
    outs_host = [[torch.empty((H, W, 4), dtype=torch.uint8).pin_memory() for _ in TS] for _ in range(2)]
    up, comp, down = torch.cuda.Stream(dev), torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    xp = torch.cuda.Stream(dev, priority=-1)   # expansion of the uploaded colour and shadow data
    ups = [up, xp]
    ev = lambda: torch.cuda.Event()
    up_done, comp_done, down_done = {}, {}, {}
    counters = {"h2d": 0, "d2h": 0, "launches": 0}
    resident = {}  # ring slot -> keyframe index whose arrival part it holds

    last_use = {}  # (ring slot, "arr" | "fwd") -> last step that read that part
    last_frame = []  # [pair, DeviceFrame] of the latest step

    # entries last unpacked into each slot's shadow images: the next unpack clears only their
    # pixels (the images are zero elsewhere) instead of the whole images
    prev_entries = {(slot, kind, c): torch.empty(max(16, packs[slot][(kind, c)] * 16), dtype=torch.uint8, device=dev)
                    for slot in range(P + 1) for kind in ("sb", "sf") for c in range(n_cams)}
    prev_n = {}

    def expand(slot, part, k):
        """Device-side expansion of one uploaded part of keyframe k in its slot (stream xp)."""
        st = C.c_void_p(xp.cuda_stream)
        launches = 0
        if part == "arr":
            lo = layouts[slot][("color", 0)][0]
            native.check(lib.isti_rgb8_to_rgba8(rgba_arr[slot].data_ptr(), ring[slot][lo:].data_ptr(), n_cams * H * W, st))
            launches += 1
        kind = "sb" if part == "arr" else "sf"
        for c in range(n_cams):
            a_, b_, info = ring_fields[slot][c][kind]
            lo, _ = layouts[slot][(kind, c)]
            n = packs[k][(kind, c)]
            key = (slot, kind, c)
            if n * 16 > prev_entries[key].numel():
                raise RuntimeError("e2e: a slot received more shadow entries than its buffer holds")
            nc = prev_n.get(key)
            native.check(lib.isti_unpack_shadows(info.data_ptr(), a_.data_ptr(), b_.data_ptr(), H * W,
                                                 C.c_void_p(ring[slot][lo:].data_ptr() if n else None), n,
                                                 C.c_void_p(prev_entries[key].data_ptr() if nc is not None else None), nc or 0, st))
            launches += (3 if nc is None else (1 if nc else 0)) + (1 if n else 0)   # clears, scatter
            if n:
                with torch.cuda.stream(xp):
                    prev_entries[key][:n * 16].copy_(ring[slot][lo:lo + n * 16], non_blocking=True)
                launches += 1
            prev_n[key] = n
        return launches

    def step(s, count):
        p = s % P
        k0, k1 = p, p + 1
        s0, s1 = k0, k1
        copies = []  # (slot, part, keyframe): the arrival part of k1, the forward part of k0
        if resident.get(s0) != k0:   # first step only: keyframe 0 is never a newly arrived one
            copies.append((s0, "arr", k0))
        copies += [(s0, "fwd", k0), (s1, "arr", k1)]
        for slot, part, _ in copies:   # wait until no earlier step still reads the range
            if (slot, part) in last_use:
                up.wait_event(comp_done[last_use[(slot, part)]])
        for slot, part, k in copies:
            A, total = layouts[k]["A"], layouts[k]["total"]
            lo, hi = (0, A) if part == "arr" else (A, total)
            with torch.cuda.stream(up):
                ring[slot][lo:hi].copy_(host[k][lo:hi], non_blocking=True)
            # the expansion runs on its own high-priority stream, so the link keeps copying
            copied = ev()
            copied.record(up)
            xp.wait_event(copied)
            n_launch = expand(slot, part, k)
            if count:
                counters["h2d"] += hi - lo
                counters["launches"] += n_launch
        resident[s0], resident[s1] = k0, k1
        up_done[s] = [ev()]
        up_done[s][0].record(xp)
        for key in ((s0, "arr"), (s0, "fwd"), (s1, "arr")):
            last_use[key] = s
        views = []
        for c in range(n_cams):
            d0, d1 = res[(k0, c)], res[(k1, c)]
            f0, f1 = ring_fields[s0][c], ring_fields[s1][c]
            views.append((DeviceView(f0["color"], f0["z"], f0["mf"], *f0["sf"], d0["vp"], d0["ivp"]),
                          DeviceView(f1["color"], f1["z"], f1["mb"], *f1["sb"], d1["vp"], d1["ivp"])))
        fr = DeviceFrame(views[0][0], views[0][1], [v[0] for v in views[1:]], [v[1] for v in views[1:]], [3] * (n_cams - 1))
        last_frame[:] = [p, fr]
        od = outs_dev[s % 2]
        for e_ in up_done[s]:
            comp.wait_event(e_)
        if s - 2 in down_done:
            comp.wait_event(down_done[s - 2])      # output set s % 2 has been read back
        r.render_batch(od, clients[p], fr, chain=True, stream=comp)
        comp_done[s] = ev()
        comp_done[s].record(comp)
        down.wait_event(comp_done[s])
        with torch.cuda.stream(down):
            for i, o in enumerate(od):
                outs_host[s % 2][i].copy_(o, non_blocking=True)
                if count:
                    counters["d2h"] += o.numel()
            down_done[s] = ev()
            down_done[s].record(down)

    for s in range(args.warmup):
        step(s, False)
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record(up)
    for s in range(args.warmup, args.warmup + args.steps):
        step(s, True)
    for st in ups + [comp]:
        down.wait_stream(st)
    t1.record(down)
    torch.cuda.synchronize()
    ms = max_over_ranks(t0.elapsed_time(t1), world, dev)
    value = world * args.steps * len(TS) * W * H / 1e6 / (ms / 1e3)

    # outside the timed region: the streamed views of the last step render what the
    # resident keyframes of the same pair render (slab layout and RGB expansion checked)
    p, fr = last_frame
    d_views = [(DeviceView(res[(p, c)]["color"], res[(p, c)]["z"], res[(p, c)]["mf"], *res[(p, c)]["sf"], res[(p, c)]["vp"],
                           res[(p, c)]["ivp"]),
                DeviceView(res[(p + 1, c)]["color"], res[(p + 1, c)]["z"], res[(p + 1, c)]["mb"], *res[(p + 1, c)]["sb"],
                           res[(p + 1, c)]["vp"], res[(p + 1, c)]["ivp"])) for c in range(n_cams)]
    resident_fr = DeviceFrame(d_views[0][0], d_views[0][1], [v[0] for v in d_views[1:]], [v[1] for v in d_views[1:]],
                              [3] * (n_cams - 1))
    got = [torch.zeros((H, W, 4), dtype=torch.uint8, device=dev) for _ in TS]
    want = [torch.zeros_like(g) for g in got]
    r.render_batch(got, clients[p], fr, chain=True, stream=comp)
    r.render_batch(want, clients[p], resident_fr, chain=True, stream=comp)
    comp.synchronize()
    if not all(torch.equal(a, b) for a, b in zip(got, want)):
        raise RuntimeError("e2e: frames rendered from the streamed keyframes differ from the resident ones")
    return {"value": round(value, 2), "unit": "Mpix/s", "h2d_bytes_per_step": counters["h2d"] // args.steps,
            "d2h_bytes_per_step": counters["d2h"] // args.steps, "ms_per_step": round(ms / args.steps, 4),
            "expand_ops_per_step": counters["launches"] / args.steps,
            "pipeline": "one contiguous slab per keyframe, 2 uploads per step (colour as RGB, shadows as sparse "
                        "entries of the pixels the renderer reads, both expanded on the device) / render / read-back overlapped"}


def main():
    args = parse()
    if args.impl == "reference":
        return run_reference(args)
    return main_ours(args)


if __name__ == "__main__":
    sys.exit(main())
