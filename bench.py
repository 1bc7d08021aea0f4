#!/usr/bin/env python
"""Benchmark of the GB300 MNAD RTM hot path.

Workload (one "step" = one pass over the batch): batched RTM of the
1201 x 401 @ 12.5 m Gaussian-random-field model with three dipping
reflectors, 64 shots every 187.5 m, 20 Hz Ricker, dt = 1 ms, 4 s, BF16
source snapshots, FP64 image stack -- per shot the reference workflow of
SRC/migration/main_Acoustic_RTM.m:221-253 (true-model forward, background
forward with snapshots, scattered data, adjoint with imaging).  Inputs are
seeded synthetic models (no dataset).

value    : grid-point updates per second over all propagations (Gpts/s),
           device-timed with CUDA events, inputs resident in HBM.
e2e      : same metric through the public C ABI (mnad_run_jobs) with host
           buffers, host<->device copies inside the timed region.
plain    : the single-shot drop-in path (mnad_fwd_pde_exact x2 +
           mnad_born_adj per shot, serial), same metric.
serving  : the served shot stream (Poisson arrivals of mixed modeling / RTM
           jobs of four grid sizes and three record lengths) through the
           continuous-batching server: throughput, p50/p99 job latency.
--impl reference : the reference algorithm (literal FP64 sparse-operator
           restatement) on the host cores, shots in a process pool.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG_ROOT = os.path.join(ROOT, "mnad-modeling-rtm_gb300")
for p in (ROOT, PKG_ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)

METRIC = "RTM shots/hr & MNAD Gpts/s, batched vs plain, rel err ≤1e-4; p99 shot latency"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="random-field", choices=["random-field", "faulted-salt"],
                    help="random-field: batched RTM of 64 shots over a 401x1201 Gaussian random field (default); "
                         "faulted-salt: RTM of 16 shots over a 1201x4001 faulted model with FP16 checkpoints")
    ap.add_argument("--shots", type=int, default=None, help="shots per pass (random-field: 64, faulted-salt: 16)")
    ap.add_argument("--nt", type=int, default=None,
                    help="record length in steps (random-field: 4000, faulted-salt: 6000)")
    ap.add_argument("--checkpoint-every", type=int, default=360, help="faulted-salt: checkpoint interval (steps)")
    ap.add_argument("--plain-shots", type=int, default=8)
    ap.add_argument("--f32-steps", type=int, default=2,
                    help="random-field: timed passes of the FP32-snapshot leg (0: skip the leg)")
    ap.add_argument("--no-oracle", action="store_true", help="skip the FP64-oracle error of the checked shot")
    ap.add_argument("--no-extras", action="store_true", help="skip e2e, plain and CPU legs")
    ap.add_argument("--ref-steps", type=int, default=12, help="reference arm: time steps per worker sample")
    ap.add_argument("--kernel", default="auto", choices=["auto", "direct", "tma", "tma_narrow", "tma2", "tune"])
    ap.add_argument("--serve-jobs", type=int, default=512, help="served stream length (0: skip the leg)")
    ap.add_argument("--serve-rate", type=float, default=None, help="arrivals per second (default: from the seed)")
    return ap.parse_args()


# ---------------------------------------------------------------------------
class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms while running."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, val in zip(names, f[5:9]):
                if val.lower() == "active":
                    reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6800.0, "fallback"


FLOPS_PER_POINT = 137        # of the stencil and the update, without the CPML strips


def fp32_peak(sm_max_mhz):
    """TFLOP/s of the FP32 pipes: 128 lanes per SM, two operations per lane and cycle."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152
    return sms * 128 * 2 * (sm_max_mhz or 2070.0) * 1e6 / 1e12


def kernel_roof(kernel, pts, nbytes, seconds, hbm_peak, fp32):
    """What bounds a step kernel and how near it is: HBM for the kernels that move the
    state once per step (algorithmic bytes), the FP32 rate for the on-chip kernel, which
    keeps the state in shared memory."""
    if kernel == "resident":
        a = FLOPS_PER_POINT * pts / seconds / 1e12
        return {"bound": "fp32", "achieved": round(a, 2), "peak": round(fp32, 1), "unit": "TFLOP/s", "frac": round(a / fp32, 4),
                "peak_kind": "128 lanes x SMs x 2 x max SM clock"}
    a = nbytes / seconds / 1e9
    return {"bound": "hbm", "achieved": round(a, 1), "peak": hbm_peak, "unit": "GB/s", "frac": round(a / hbm_peak, 4)}


def profile_traffic():
    """DRAM bytes per point-update of the step kernel from the committed ncu summary."""
    path = os.path.join(ROOT, "profiles", "traffic.json")
    try:
        with open(path) as f:
            return json.load(f)
    except (OSError, ValueError):
        return None


# ---------------------------------------------------------------------------
def dist_setup(n):
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    return rank, world, local


def barrier_sync(world):
    import torch
    torch.cuda.synchronize()
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
        torch.cuda.synchronize()


def allmax(x, world):
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def allsum(x, world):
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.SUM)
    return float(t.item())


# ---------------------------------------------------------------------------
def cpu_baseline(sv, seconds=15.0):
    """C OpenMP FP64 port of the reference algorithm on one shot (bounded)."""
    import numpy as np
    from oracle import coracle
    sh = sv.shots[0]
    w = sv.w
    coracle.fwd(sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr, sv.v, sv.dt, 2, w, sv.d_pml)   # warm the thread pool
    probe = 20
    t = time.perf_counter()
    coracle.fwd(sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr, sv.v, sv.dt, probe, w, sv.d_pml)
    per = (time.perf_counter() - t) / probe
    n = max(probe, min(sv.nt, int(seconds / max(per, 1e-6))))
    t = time.perf_counter()
    coracle.fwd(sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr, sv.v, sv.dt, n, w, sv.d_pml)
    el = time.perf_counter() - t
    pts = float(sv.nz * sv.nx * n)
    return {"value": pts / el / 1e9, "unit": "Gpts/s", "cores": coracle.threads(), "kind": "port",
            "sample": f"one forward propagation of {sv.name} shot 0, {n} of {sv.nt} steps "
                      f"({sv.nz}x{sv.nx} padded), FP64 matrix-free C/OpenMP restatement, {el:.1f} s"}


def oracle_rtm(sv, sh):
    """FP64 C/OpenMP oracle of one RTM shot (true forward, background forward
    with snapshots, adjoint of the scattered data): the reference workflow of
    SRC/migration/main_Acoustic_RTM.m:221-253 for that shot."""
    from oracle import coracle
    from oracle import mnad_oracle as P
    nf = P.snapshot_nf(sv.vs, sv.nt)
    T = sv.T or P.snapshot_plan(sv.vs, sv.nt)[1]
    ncols = max(2 * nf + 1, sv.nt // T)
    a = (sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr)
    t = time.perf_counter()
    data = coracle.fwd(*a, sv.v, sv.dt, sv.nt, sv.w, sv.d_pml)["datau"]
    bg = coracle.fwd(*a, sv.vs, sv.dt, sv.nt, sv.w, sv.d_pml, indx=1, T=T, ncols=ncols)
    im = coracle.adj(sv.dx, sv.dz, sv.nt, sv.dt, sv.vs, sh.xr, sh.zr, data - bg["datau"], sv.d_pml, bg["UU"], T)
    return {"scattered": data - bg["datau"], "illum": bg["illum"], "image": im, "T": T,
            "seconds": time.perf_counter() - t}


def rel_l2(a, b):
    import numpy as np
    a, b = np.ravel(np.asarray(a), order="F"), np.ravel(np.asarray(b), order="F")
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def shot_errors(job, ref, k):
    """rel-L2 of one benchmarked shot's outputs against the FP64 oracle."""
    return {"shot": k, "scattered_gather": rel_l2(job.data, ref["scattered"]),
            "illumination": rel_l2(job.illum, ref["illum"]), "image": rel_l2(job.image, ref["image"]),
            "oracle": "FP64 matrix-free C/OpenMP restatement of the reference",
            "bars": {"scattered_gather": 1e-4, "image": 1e-4, "image_bf16_snapshots": 1e-2}}


def plain_path(ctx, sv, nshots):
    """Single-shot drop-in calls, serial: fwd(true), fwd(background, indx=1),
    scattered data on the host, adjoint (the reference's per-shot calls).
    One untimed shot first (memory pool, module loading), then `nshots`
    timed shots."""
    def shot(k):
        sh = sv.shots[k % len(sv.shots)]
        a = (sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr)
        data = ctx.fwd(*a, sv.v, sv.dt, sv.nt, sv.w, sv.d_pml, ss=k + 1)
        bg = ctx.fwd(*a, sv.vs, sv.dt, sv.nt, sv.w, sv.d_pml, ss=k + 1, indx=1)
        ctx.adj(sv.dx, sv.dz, sv.nt, sv.dt, sv.vs, sh.xr, sh.zr, data - bg, sv.d_pml, ss=k + 1)
        ctx.wavefield_release(k + 1)

    shot(0)
    t = time.perf_counter()
    for k in range(nshots):
        shot(k)
    el = time.perf_counter() - t
    pts = 3.0 * sv.nz * sv.nx * sv.nt * nshots
    return {"value": pts / el / 1e9, "unit": "Gpts/s", "shots_per_hr": nshots / el * 3600.0,
            "shots": nshots, "seconds": el}


def serving_leg(device, njobs, rate=None, seed=0, kernel="auto"):
    """Served shot stream through mnad.Server: a submitter thread replays the
    Poisson schedule in real time, the main thread collects completions.
    Throughput counts the grid-point updates of all jobs over the wall time
    from the first arrival to the last completion."""
    import threading
    import numpy as np
    import mnad
    from mnad import workflow
    sched, pools, rate = workflow.served_stream(seed=seed, njobs=njobs, rate=rate)
    # warm-up server (module load, first allocations of the memory pool)
    with mnad.Server(device, kernel=kernel) as w:
        for sj in sched[:4]:
            w.wait(w.submit(workflow.served_shot_job(workflow.ServedJob(0, sj.kind, (256, 256), 200, sj.fc, 0, 100),
                                                     pools)), timeout_s=600)
    srv = mnad.Server(device, kernel=kernel, chunk_steps=64)
    tickets = [None] * len(sched)
    ready = threading.Semaphore(0)
    err = []

    def submitter():
        t0 = time.perf_counter()
        try:
            for k, sj in enumerate(sched):
                job = workflow.served_shot_job(sj, pools)
                delay = sj.arrival_s - (time.perf_counter() - t0)
                if delay > 0:
                    time.sleep(delay)
                tickets[k] = srv.submit(job)
                ready.release()
        except Exception as e:     # surfaced by the collector
            err.append(e)
            for _ in range(len(sched)):
                ready.release()

    th = threading.Thread(target=submitter)
    t_start = time.perf_counter()
    th.start()
    bad = 0
    kinds = {"model": 0, "rtm": 0}
    for k in range(len(sched)):
        ready.acquire()
        if err:
            break
        job = srv.wait(tickets[k], timeout_s=3600)
        kinds[job.kind] += 1
        if not np.all(np.isfinite(job.data)) or (job.kind == "rtm" and not np.all(np.isfinite(job.image))):
            bad += 1
    th.join()
    wall = time.perf_counter() - t_start
    st = srv.stats()
    srv.close()
    if err:
        raise err[0]
    return {"workload": "served shot stream of mixed modeling / RTM jobs on 256x256 to 1024x2048 grids",
            "jobs": len(sched), "model_jobs": kinds["model"],
            "rtm_jobs": kinds["rtm"], "arrival_rate_per_s": round(rate, 3),
            "grids": [f"{g[0]}x{g[1]}" for g in workflow.SERVED_GRIDS], "seconds": list(workflow.SERVED_SECONDS),
            "value": round(st["point_updates"] / wall / 1e9, 3), "unit": "Gpts/s",
            "jobs_per_s": round(st["completed"] / wall, 3),
            "rtm_jobs_per_hr": round(kinds["rtm"] / wall * 3600.0, 1),
            "p50_ms": round(st["p50_ms"], 1), "p99_ms": round(st["p99_ms"], 1), "max_ms": round(st["max_ms"], 1),
            "wall_s": round(wall, 2), "busy_s": round(st["busy_s"], 2), "failed": st["failed"],
            "non_finite_outputs": bad, "snapshots": "f32", "chunk_steps": 64}


def run_ours(args):
    import numpy as np
    rank, world, local = dist_setup(args.gpus)
    import mnad
    from mnad import shards, workflow
    if args.workload == "faulted-salt":
        sv = workflow.faulted_salt_survey(seed=0, nshots=256, nt=args.nt, first=rank * args.shots, count=args.shots)
        ctx = mnad.Context(local, kernel=args.kernel, checkpoint_every=args.checkpoint_every, checkpoint_codec="f16")
        data_desc = "synthetic (seeded faulted layered model with a salt body)"
        wl = {"workload": "large-grid RTM with checkpoint-and-recompute, 1201x4001 faulted model with a salt body",
              "grid": "1201x4001 (+2x40 CPML) @ 12.5 m", "checkpoints": f"f16 every {args.checkpoint_every} steps",
              "snapshot_buffer": "f32 segment", "propagations_per_shot": "3 + 1 recomputed background forward"}
    else:
        # weak scaling: every rank images args.shots shots of one survey
        sv = workflow.random_field_survey(seed=0, nshots=args.shots * world, nt=args.nt)
        sv.shots = shards.shard(sv.shots, rank, world)
        ctx = mnad.Context(local, snapshot_codec=sv.codec, kernel=args.kernel)
        data_desc = "synthetic (seeded Gaussian random field + dipping reflectors)"
        wl = {"workload": "batched RTM, 401x1201 Gaussian random field with dipping reflectors",
              "grid": "401x1201 (+2x40 CPML) @ 12.5 m",
              "snapshots": sv.codec, "propagations_per_shot": 3}
    jobs = workflow.shot_jobs(sv, "rtm")
    # the shot whose outputs are checked against the FP64 oracle after the
    # timed passes also keeps its scattered data (downloads are not timed)
    kcheck = len(jobs) // 2
    jobs[kcheck].data = np.zeros((sv.nt, jobs[kcheck].xr.size), order="F")
    m0 = ctx.memory()
    plan = ctx.plan(jobs)
    mem_per_shot = (ctx.memory() - m0) / max(len(jobs), 1)
    for _ in range(max(args.warmup, 0)):
        plan.run()
    barrier_sync(world)
    sampler = ClockSampler(local)
    sampler.start()
    run_ms, step_ms = [], []
    phase_ms = [0.0, 0.0]
    launches = 0
    t0 = time.perf_counter()
    for _ in range(args.steps):
        plan.run()
        tm = plan.timing()
        ph = plan.phases()
        phase_ms[0] += ph["forward_ms"]
        phase_ms[1] += ph["adjoint_ms"]
        run_ms.append(tm["run_ms"])
        step_ms.append(tm["step_ms"])
        launches += plan.launches() + 2 + len(jobs)   # step kernels + source seeding + residuals
    barrier_sync(world)
    wall = time.perf_counter() - t0
    clocks = sampler.stop()
    status = ctx.status()
    pts, abytes = plan.work()
    kernels = plan.kernels()     # step kernel of each phase (the tuner's choice under --kernel tune)
    total_s = allmax(sum(run_ms) / 1e3, world)
    pts_all = allsum(pts * args.steps, world)
    value = pts_all / total_s / 1e9
    ms_per_step = total_s * 1e3 / args.steps
    shots_hr = allsum(len(jobs) * args.steps, world) / total_s * 3600.0
    peak, peak_kind = peaks()
    fp32 = fp32_peak(clocks.get("sm_max_mhz"))
    tr = profile_traffic()
    traffic = None
    if tr and "bytes_per_point_update" in tr and args.workload == "random-field":
        traffic = tr["bytes_per_point_update"] * pts / (plan.timing()["step_launches"])
    roof = {"traffic": traffic, "peak_kind": f"{peak_kind} hbm_gbs",
            "kernel": "mnad::step_" + (kernels["forward"] or "tma"),
            "kernels_by_phase": kernels,
            "algorithmic_bytes_per_launch": abytes / plan.timing()["step_launches"],
            **kernel_roof(kernels["forward"], pts * args.steps, abytes * args.steps, sum(step_ms) / 1e3, peak, fp32)}
    if roof["bound"] == "fp32":
        roof["traffic"] = None
    # the same roofline split by phase (forwards with snapshots; adjoints with imaging)
    ph = plan.phases()
    roof["phases"] = {}
    for name, ms in zip(("forward", "adjoint"), phase_ms):
        b = ph[name + "_bytes"]
        # its share of the point updates: by algorithmic bytes, which are near 40 per update in both
        r = kernel_roof(kernels[name], pts * b / abytes * args.steps, b * args.steps, ms / 1e3, peak, fp32) if ms > 0 else {}
        roof["phases"][name] = {"ms_per_step": round(ms / args.steps, 1), "achieved": r.get("achieved"), "frac": r.get("frac"),
                                "unit": r.get("unit")}
    # the one exchange of the path: the FP64 image / illumination stack over ranks
    t = time.perf_counter()
    im, il, _ = plan.stack()
    if world > 1:
        im, il, _ = shards.reduce_stack(im, il)
    stack = {"shots_total": int(allsum(len(jobs), world)), "reduce_ms": round((time.perf_counter() - t) * 1e3, 2),
             "image_norm": float(np.linalg.norm(im))}
    check_oracle = rank == 0 and not args.no_oracle and args.workload == "random-field"
    extras = {"stack": stack}
    ref = None
    if check_oracle:
        plan.download()
        ref = oracle_rtm(sv, sv.shots[kcheck])
        extras["rel_err"] = dict(shot_errors(jobs[kcheck], ref, kcheck), snapshots=sv.codec,
                                 oracle_seconds=round(ref["seconds"], 1))
    plan.close()
    if args.workload == "random-field" and args.f32_steps > 0:
        # the same batch with FP32 snapshots: the leg whose image error meets
        # the 1e-4 bar (BF16 snapshots round every d2u value to 8 bits)
        jobs32 = workflow.shot_jobs(sv, "rtm")
        jobs32[kcheck].data = np.zeros((sv.nt, jobs32[kcheck].xr.size), order="F")
        ctx.set_options(snapshot_codec="f32")
        plan32 = ctx.plan(jobs32)
        plan32.run()
        barrier_sync(world)
        ms32 = []
        for _ in range(args.f32_steps):
            plan32.run()
            ms32.append(plan32.timing()["run_ms"])
        barrier_sync(world)
        t32 = allmax(sum(ms32) / 1e3, world)
        leg = {"value": round(allsum(pts * args.f32_steps, world) / t32 / 1e9, 3), "unit": "Gpts/s",
               "shots_per_hr": round(allsum(len(jobs32) * args.f32_steps, world) / t32 * 3600.0, 1),
               "ms_per_step": round(t32 * 1e3 / args.f32_steps, 2), "steps": args.f32_steps, "snapshots": "f32"}
        if ref is not None:
            plan32.download()
            leg["rel_err"] = shot_errors(jobs32[kcheck], ref, kcheck)
        plan32.close()
        ctx.set_options(snapshot_codec=sv.codec)
        extras["f32_snapshots"] = leg
    if not args.no_extras:
        # e2e through the C ABI with host buffers in pinned memory (upload, run,
        # download inside the timed region)
        pinned = []

        def pin(a):
            import torch
            t = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
            pinned.append(t)
            x = t.numpy().reshape(a.shape, order="F")
            x[...] = a
            return x

        models = {}
        for j in jobs:
            for name in ("v", "vs"):
                a = getattr(j, name)
                if a is not None:
                    if id(a) not in models:
                        models[id(a)] = pin(a)
                    setattr(j, name, models[id(a)])
            j.image = pin(np.zeros_like(j.image))
            j.illum = pin(np.zeros_like(j.illum))
            if j.data is not None:
                j.data = pin(np.zeros_like(j.data))
        h0, d0 = ctx.transfers()
        barrier_sync(world)
        t = time.perf_counter()
        ctx.run_jobs(jobs)
        e2e_s = time.perf_counter() - t
        h1, d1 = ctx.transfers()
        e2e_s = allmax(e2e_s, world)
        extras["e2e"] = {"value": round(allsum(pts, world) / e2e_s / 1e9, 3), "unit": "Gpts/s",
                         "h2d_bytes_per_step": int(h1 - h0), "d2h_bytes_per_step": int(d1 - d0),
                         "shots_per_hr": round(allsum(len(jobs), world) / e2e_s * 3600.0, 1),
                         "api": "mnad_run_jobs", "host_buffers": "pinned"}
        if rank == 0 and args.plain_shots > 0:
            extras["plain"] = plain_path(ctx, sv, args.plain_shots)
            extras["plain"]["value"] = round(extras["plain"]["value"], 3)
            extras["plain"]["snapshots"] = sv.codec
            if "f32_snapshots" in extras:
                # the plain path with the FP32 leg's snapshots (its denominator)
                ctx.set_options(snapshot_codec="f32")
                p32 = plain_path(ctx, sv, args.plain_shots)
                ctx.set_options(snapshot_codec=sv.codec)
                p32["value"] = round(p32["value"], 3)
                p32["snapshots"] = "f32"
                extras["f32_snapshots"]["plain"] = p32
        if rank == 0:
            extras["cpu_baseline"] = cpu_baseline(sv)
    ctx.close()
    if rank == 0 and args.serve_jobs > 0 and not args.no_extras and args.workload == "random-field":
        extras["serving"] = serving_leg(local, args.serve_jobs, args.serve_rate, kernel=args.kernel)
        # the same stream all at once: the server's capacity (latency is then queueing)
        cap = serving_leg(local, args.serve_jobs, 1e6, kernel=args.kernel)
        extras["serving"]["capacity"] = {k: cap[k] for k in ("value", "unit", "jobs_per_s", "rtm_jobs_per_hr",
                                                            "p50_ms", "p99_ms", "wall_s", "failed")}
    if rank == 0:
        line = {"metric": METRIC, "value": round(value, 3), "unit": "Gpts/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 2),
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": data_desc,
                "config": dict(wl, shots=len(jobs), nt=sv.nt, dt=sv.dt, image="f64",
                               parallelism=f"replicas x{world}",
                               l2="state per step >> L2 (inputs larger than L2)",
                               device_bytes_per_shot=int(mem_per_shot)),
                "shots_per_hr": round(shots_hr, 1), "roofline": roof, "clocks": clocks,
                "gpu_launches": launches, "wall_s": round(wall, 2), "device_status": status}
        line.update(extras)
        if "plain" in extras:
            line["batched_vs_plain"] = round(value / extras["plain"]["value"], 2)
            if "plain" in extras.get("f32_snapshots", {}):
                extras["f32_snapshots"]["batched_vs_plain"] = round(
                    extras["f32_snapshots"]["value"] / extras["f32_snapshots"]["plain"]["value"], 2)
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


# ---------------------------------------------------------------------------
_REF = {}


def _ref_init(seed, nshots, nt):
    from mnad import workflow
    from oracle import mnad_oracle as P
    sv = workflow.random_field_survey(seed=seed, nshots=nshots, nt=nt)
    _REF["sv"] = sv
    _REF["A"] = P.a_gen(sv.dx, sv.dz, sv.dt, sv.v)


def _ref_shot(args):
    k, nsteps = args
    from oracle import mnad_oracle as P
    sv = _REF["sv"]
    sh = sv.shots[k % len(sv.shots)]
    t = time.perf_counter()
    P.fwd_pde_exact_mnad(sv.dx, sh.xs, sh.xr, sv.dz, sh.zs, sh.zr, sv.v, sv.dt, nsteps, sv.w, sv.d_pml,
                         A=_REF["A"])
    return time.perf_counter() - t, float(sv.nz * sv.nx * nsteps)


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import multiprocessing as mp
    workers = os.cpu_count() or 1
    ctx = mp.get_context("spawn")
    with ctx.Pool(workers, initializer=_ref_init, initargs=(0, args.shots, args.nt)) as pool:
        tasks = [(k, args.ref_steps) for k in range(workers)]
        for _ in range(max(args.warmup, 0)):
            pool.map(_ref_shot, [(k, 1) for k in range(workers)])
        vals = []
        t0 = time.perf_counter()
        for _ in range(args.steps):
            t = time.perf_counter()
            res = pool.map(_ref_shot, tasks)
            el = time.perf_counter() - t
            vals.append(sum(r[1] for r in res) / el / 1e9)
        wall = time.perf_counter() - t0
    value = statistics.median(vals)
    sample = (f"{workers} worker processes (parfor analogue), each one shot of the 401x1201 random-field survey "
              f"for {args.ref_steps} time steps (401x1201 + 2x40 CPML), literal FP64 sparse-operator "
              f"restatement (SciPy)")
    line = {"metric": METRIC, "value": round(value, 5), "unit": "Gpts/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(wall * 1e3 / args.steps, 1),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded Gaussian random field + dipping reflectors)",
            "config": {"workload": "batched RTM, 401x1201 Gaussian random field with dipping reflectors",
                       "grid": "401x1201 (+2x40 CPML) @ 12.5 m",
                       "shots": args.shots, "nt": args.nt, "parallelism": f"{workers} host processes"},
            "impl": "reference",
            "cpu_baseline": {"value": round(value, 5), "unit": "Gpts/s", "cores": workers, "kind": "port",
                             "sample": sample},
            "e2e": {"value": round(value, 5), "unit": "Gpts/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


if __name__ == "__main__":
    a = parse()
    if a.shots is None:
        a.shots = 16 if a.workload == "faulted-salt" else 64
    if a.nt is None:
        a.nt = 6000 if a.workload == "faulted-salt" else 4000
    if a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)
