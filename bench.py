#!/usr/bin/env python
"""Benchmark: the cuSten plain stencil sweep, FP64, on GB300.

One step = one Compute of each of the twelve cuSten operators on an n x n field (default 16384^2):
X and Y 5-point 4th-order d2/dx2 [-1,16,-30,16,-1]/(12h^2) (periodic and non-periodic), XY 3x3
cross-derivative [1,0,-1;0,0,0;-1,0,1]/(4h^2) (p, np), and the Fun variants applying c^3 - c before
the same stencil (X, Y 5-point; XY 3x3 5-point Laplacian [0,1,0;1,-4,1;0,1,0]/h^2), all with numTiles=1
on device-resident data. Input sin(3x)cos(5y) + U(-1e-3, 1e-3) from seed 1 (synthetic).
Metric: Gpts/s = 12 * n^2 points per step / step time. Every field (2 GiB) is larger than L2.

Extra keys: per-operator Gpts/s; roofline of the stencil kernel against measured HBM bandwidth and
against the measured FP64 FMA rate (the FP64 kernels are FP64-pipe bound on GB300); the FP32
precision variant (same sweep in FP32 with its error against FP64); e2e through the reference-facing
API with host (managed) buffers, numTiles=4 and HOST offload; and the CPU baseline (plain host loop,
same weights and FMA order, all host threads, bounded row sample).

--impl reference: the reference has no CPU stencil implementation, so the reference arm times the
plain host loop port (oracle) on the same workload sample; it prints the same JSON keys.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

# ncu DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) per stencil launch: the mean over the 12
# launches of one timed sweep at 16384^2 (FP64, L2 not flushed between launches), 1.032 x the algorithmic
# 16 B per point. Other sizes scale it by the point count: every launch streams its field once.
TRAFFIC_16384 = 4431034304.0

def operators(n: int):
    """(name, variant, H, L, R, V, T, B, weights, fun_id, dfma_per_point) of the 12-operator sweep."""
    from custen_gb300.inputs import sweep_operators
    return sweep_operators(n)


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


class ClockSampler:
    """nvidia-smi clocks/throttle reasons during the timed region."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.lines: list[str] = []
        self.t = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.dev), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self.t:
            self.t.join(timeout=2)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 8:
                continue
            try:
                sm.append(float(parts[0]))
                smax.append(float(parts[1]))
            except ValueError:
                continue
            for nm, val in zip(names, parts[4:8]):
                if val.lower() == "active":
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": max(smax), "reasons": sorted(reasons),
                "samples": len(sm)}


def reduce_max(value: float, dist=None, device=None) -> float:
    """Max over ranks (the slowest replica sets the job's time)."""
    if dist is None:
        return value
    import torch
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_throughput(points_per_rank: float, world: int, ms_per_step: float) -> float:
    """Whole-job points per second (weak scaling: every rank processes points_per_rank per step)."""
    return world * points_per_rank / (ms_per_step * 1e-3)


def measured_peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            pass
    return {}


# ----------------------------------------------------------------------------------------------
# CPU leg: plain host loop (oracle port), all host threads, bounded row sample
# ----------------------------------------------------------------------------------------------
def cpu_sample(n: int, rows: int, threads: int):
    import concurrent.futures as cf

    import numpy as np

    import oracle
    from custen_gb300.inputs import field
    oracle.build()
    # rows sampled from the real n x n field: build only the rows the sample reads (+ halos)
    full_rows = rows + 4
    rng_field = field(n, full_rows, 1)   # same generator, shape (full_rows, n)
    out = np.zeros_like(rng_field)
    ops = operators(n)

    def one_pass():
        pts = 0
        with cf.ThreadPoolExecutor(max_workers=threads) as ex:
            futs = []
            chunk = max(1, rows // threads)
            for (_, v, H, L, R, V, T, B, w, fun, _) in ops:
                for y0 in range(2, 2 + rows, chunk):
                    y1 = min(2 + rows, y0 + chunk)
                    futs.append(ex.submit(oracle.host_loop, rng_field, out, np.asarray(w), H, L, V, T, fun >= 0,
                                          y0, y1))
                pts += rows * n
            for f in futs:
                f.result()
        return pts

    return one_pass


def cpu_single_thread(n: int, rows: int = 256) -> dict:
    """The same plain host loop on one thread, over a smaller sample of rows."""
    one = cpu_sample(n, rows, 1)
    one()
    t0 = time.perf_counter()
    pts = one()
    dt = time.perf_counter() - t0
    return {"value": round(pts / dt / 1e9, 4), "unit": "Gpts/s", "cores": 1,
            "sample": f"{rows} rows x {n} columns per operator, 12 operators, plain host loop, 1 thread"}


def cpu_ch_sample(steps: int = 40, n: int = 256) -> dict:
    """The serial Cahn-Hilliard solver (oracle port of cuPentSpeedUp/serialCahnADITiming/serialCahnADI.c,
    single-threaded as the reference program is) on config 1's grid: 256^2, lx = 2 pi, bounded steps."""
    import numpy as np

    import oracle
    c0 = np.random.default_rng(0).uniform(-0.1, 0.1, (n, n))
    o = oracle.CHOracle(c0)
    o.step(2)
    t0 = time.perf_counter()
    o.step(steps)
    dt = time.perf_counter() - t0
    return {"value": round(steps / dt, 2), "unit": "steps/s", "gpt_steps_per_s": round(n * n * steps / dt / 1e9, 5),
            "cores": 1, "kind": "port", "sample": f"{n}^2 grid, {steps} steps (serial ADI solver, one thread)"}


def reference_gpu(args) -> dict:
    """The reference's own device code rebuilt for sm_103a on this GPU (cubins compiled unchanged from the
    reference sources; host loops restated in oracle/ref_runner.cpp and oracle/ref_ch_runner.cpp)."""
    try:
        import numpy as np
        import torch
        if not torch.cuda.is_available():
            return {"unavailable": "no GPU visible"}
        import oracle
        if oracle.reference_kernels() is None:
            return {"unavailable": "reference cubins not built (they are compiled from the reference sources)"}
    except Exception as e:  # noqa: BLE001
        return {"unavailable": f"{type(e).__name__}: {e}"[:200]}
    dev = torch.device("cuda", 0)
    n = args.n
    out = {}
    x = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
    g = torch.Generator(device=dev)
    g.manual_seed(1)
    f = (torch.sin(3 * x)[None, :] * torch.cos(5 * x)[:, None] +
         (torch.rand((n, n), device=dev, dtype=torch.float64, generator=g) * 2e-3 - 1e-3)).contiguous()
    o = torch.zeros_like(f)
    per, best_block, total = {}, {}, 0.0
    for (nm, v, H, L, R, V, T, B, w, fun, _) in operators(n):
        wt = torch.tensor(w, dtype=torch.float64, device=dev)
        d = 0 if v < 4 else (1 if v < 8 else 2)
        num_sten = H * V if d == 2 else (H if d == 0 else V)
        func = oracle.reference_fun_ptr(fun) if fun >= 0 else 0
        best = None
        for bx, by in ((32, 8), (32, 16), (32, 32)):   # the reference's BLOCK_X x BLOCK_Y, best of three

            def call():
                oracle.reference_compute(v, n, n, 1, bx, by, o.data_ptr(), f.data_ptr(), wt.data_ptr(),
                                         num_sten=num_sten, H=H, L=L, R=R, V=V, T=T, B=B, num_coe=len(w), func=func)
            call()
            reps = 3
            t0 = time.perf_counter()
            for _ in range(reps):
                call()
            dt = (time.perf_counter() - t0) / reps
            if best is None or dt < best[0]:
                best = (dt, f"{bx}x{by}")
        total += best[0]
        per[nm] = round(n * n / best[0] / 1e9, 3)
        best_block[nm] = best[1]
    out["stencil_sweep"] = {"gpts_s": round(12 * n * n / total / 1e9, 3), "unit": "Gpts/s", "per_op": per,
                            "block_per_op": best_block,
                            "config": f"{n}^2, the 12 operators of the headline sweep, numTiles 1, each operator at "
                                      f"its best BLOCK_X x BLOCK_Y of 32x8, 32x16, 32x32",
                            "method": "reference kernels, one launch per Compute, wall time of each synchronised "
                                      "Compute (XpFun with the shared-memory layout its kernel indexes)"}
    # WENO advection
    rng = np.random.default_rng(1)
    u = torch.tensor(rng.uniform(-1, 1, (n, n)), device=dev)
    vv = torch.tensor(rng.uniform(-1, 1, (n, n)), device=dev)
    h = 2 * math.pi / n
    oracle.reference_weno(n, n, 1, 32, 8, o.data_ptr(), f.data_ptr(), u.data_ptr(), vv.data_ptr(), 1 / h, 1 / h)
    t0 = time.perf_counter()
    for _ in range(3):
        oracle.reference_weno(n, n, 1, 32, 8, o.data_ptr(), f.data_ptr(), u.data_ptr(), vv.data_ptr(), 1 / h, 1 / h)
    dt = (time.perf_counter() - t0) / 3
    out["weno"] = {"gpts_s": round(n * n / dt / 1e9, 3), "config": f"{n}^2, BLOCK 32x8, u, v ~ U(-1, 1)"}
    # cuPentBatch's kernels
    if oracle.ReferenceCahnHilliardGPU.available():
        pm, pb = 256, 1 << 18
        base = pent_inputs(torch, dev, pm, pb)
        work = [a.clone() for a in base[:5]]
        copy_ms = event_ms(torch, lambda: [a.copy_(b) for a, b in zip(work, base[:5])])
        f_ms = event_ms(torch, lambda: ([a.copy_(b) for a, b in zip(work, base[:5])],
                                        oracle.reference_pent(True, [a.data_ptr() for a in work], pm, pb))) - copy_ms
        bb = base[5].clone()
        bcopy_ms = event_ms(torch, lambda: bb.copy_(base[5]))
        s_ms = event_ms(torch, lambda: (bb.copy_(base[5]), oracle.reference_pent(
            False, [a.data_ptr() for a in work] + [bb.data_ptr()], pm, pb))) - bcopy_ms
        rows = pm * pb
        out["pent_batch"] = {"factor_grows_s": round(rows / (f_ms * 1e-3) / 1e9, 2),
                             "solve_grows_s": round(rows / (s_ms * 1e-3) / 1e9, 2),
                             "config": f"{pb} systems x {pm} unknowns, 64-thread blocks (BLOCK_INV)",
                             "method": "pentFactorBatch / pentSolveBatch, event time (each launch synchronised)"}
        del base, work, bb
        torch.cuda.empty_cache()
    del f, o, u, vv
    torch.cuda.empty_cache()
    # Cahn-Hilliard: the reference program, one grid at a time
    if oracle.ReferenceCahnHilliardGPU.available():
        step_s = {}
        for m in (64, 128, 256, 512, 1024, 2048):
            c0 = np.random.default_rng(m).uniform(-0.1, 0.1, (m, m))
            r = oracle.ReferenceCahnHilliardGPU(c0)
            r.step(2)
            k = 20 if m <= 1024 else 8
            t0 = time.perf_counter()
            r.step(k)
            step_s[m] = (time.perf_counter() - t0) / k
            r.close()
        sizes = [int(v) for v in np.random.default_rng(2).choice([64, 128, 256, 512, 1024], size=args.ch_sims)]
        total_b = sum(step_s[m] * args.ch_steps for m in sizes)
        served = served_workload(args)
        ms = sorted(step_s)

        def t_of(m):   # piecewise linear in m^2 between the measured sizes (multiples of 64)
            for lo, hi in zip(ms, ms[1:]):
                if m <= hi:
                    a = (m * m - lo * lo) / (hi * hi - lo * lo)
                    return step_s[lo] + a * (step_s[hi] - step_s[lo])
            return step_s[ms[-1]]
        t, ttc = 0.0, []
        for arr, m, k in zip(*served):
            start = max(t, arr)
            t = start + k * t_of(m)
            ttc.append(t - arr)
        # measured: the first grids of the batched list, one at a time for the full step count
        sub = sizes[:args.plain_grids]
        crng = np.random.default_rng(4)
        t0 = time.perf_counter()
        for m in sub:
            r = oracle.ReferenceCahnHilliardGPU(crng.uniform(-0.1, 0.1, (m, m)))
            r.step(args.ch_steps)
            r.close()
        sub_wall = time.perf_counter() - t0
        sub_model = sum(step_s[m] * args.ch_steps for m in sub)
        out["ch_plain_loop"] = {
            "measured_subset": {"grids": len(sub), "sizes": sub, "steps": args.ch_steps, "wall_s": round(sub_wall, 3),
                                "steps_per_s": round(len(sub) * args.ch_steps / sub_wall, 1),
                                "model_wall_s": round(sub_model, 3),
                                "measured_over_model": round(sub_wall / sub_model, 3),
                                "note": "the reference program run end to end on each grid (set-up, factorisation "
                                        "and every step with its synchronisations), wall clock"},
            "step_ms_by_n": {str(m): round(v * 1e3, 4) for m, v in step_s.items()},
            "batched_config_steps_per_s": round(len(sizes) * args.ch_steps / total_b, 1),
            "served_config": {"makespan_s": round(t, 3), "steps_per_s": round(sum(served[2]) / t, 1),
                              "ttc_p50_s": round(float(np.percentile(ttc, 50)), 3),
                              "ttc_p99_s": round(float(np.percentile(ttc, 99)), 3)},
            "method": "cuPentCahnADITiming device code unchanged, its host loop restated (device synchronisation "
                      "after every kernel); per-size step time x steps summed over the batch; served: FCFS over "
                      "the request stream with step times interpolated in n^2 between measured sizes"}
    else:
        out["ch_plain_loop"] = {"unavailable": "reference CH cubin not built"}
    return out


def run_reference_arm(args, world, rank):
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    rows = args.cpu_rows
    one = cpu_sample(args.n, rows, threads)
    for _ in range(args.warmup):
        one()
    t0 = time.perf_counter()
    pts = 0
    for _ in range(args.steps):
        pts += one()
    dt = time.perf_counter() - t0
    v = pts / dt / 1e9
    line = {
        "impl": "reference", "metric": "stencil Gpts/s", "value": round(v, 4), "unit": "Gpts/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(dt / args.steps * 1e3, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"stencil sweep FP64 {args.n}^2, 12 cuSten operators (sample of {rows} rows each)",
                   "nx": args.n, "ny": args.n},
        "cpu_baseline": {"value": round(v, 4), "unit": "Gpts/s", "cores": threads, "kind": "port",
                         "sample": f"{rows} rows x {args.n} columns per operator, 12 operators, plain host loop",
                         "single_thread": cpu_single_thread(args.n)},
        "e2e": {"value": round(v, 4), "unit": "Gpts/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "cpu_ch": cpu_ch_sample(),
    }
    if not args.skip_ref_gpu:
        line["gpu_sm103a"] = reference_gpu(args)
    print(json.dumps(line), flush=True)


# ----------------------------------------------------------------------------------------------
# GPU arm
# ----------------------------------------------------------------------------------------------
def run_gpu(args, world, rank, local):
    import numpy as np
    import torch

    import custen_gb300 as cs

    cs.build()
    # Kernel configurations: tuned at each handle's first (warm-up) Compute and cached (autotune.cu)
    cs.set_tune_cache(str(ROOT / "_build" / f"tune_cache_rank{rank}.json"))
    cs.set_stage_chunk_bytes(args.stage_chunk_mb << 20)
    cs.set_autotune(args.autotune)
    torch.cuda.set_device(local)
    cs._check(cs.lib().custen_set_device(local))
    dev = torch.device("cuda", local)
    pg = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=dev)
        pg = dist

    n = args.n
    ops = operators(n)
    stream = torch.cuda.current_stream(dev)

    # ---- e2e: reference-facing API with host buffers (numTiles=4, HOST offload) ----
    # The e2e legs run first. On this machine sustained GPU compute slows host<->device DMA for a while
    # afterwards (in bursts, for minutes); an e2e workload by itself does not, so the e2e is measured
    # before this process's compute legs rather than after them. e2e.link carries the host link
    # measured alongside it.
    e2e = e2e_managed = None
    if not args.skip_e2e:
        e2e = run_e2e(args, cs, np, local, ops, "pinned")
        if not args.skip_e2e_managed:
            e2e_managed = run_e2e(args, cs, np, local, ops, "managed", steps=1)

    def make_field(dtype):
        x = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
        g = torch.Generator(device=dev)
        g.manual_seed(1)
        f = torch.sin(3 * x)[None, :] * torch.cos(5 * x)[:, None]
        f = f + (torch.rand((n, n), device=dev, dtype=torch.float64, generator=g) * 2e-3 - 1e-3)
        return f.to(dtype).contiguous()

    def build_handles(dtype_t, cs_dtype, num_tiles=1, managed=False, one_output=False):
        inp = make_field(dtype_t)
        outs, hs, keep = [], [], []
        shared_out = torch.zeros((n, n), device=dev, dtype=dtype_t) if one_output else None
        for (nm, v, H, L, R, V, T, B, w, fun, _) in ops:
            wt = torch.tensor(w, device=dev, dtype=dtype_t)
            o = shared_out if one_output else torch.zeros((n, n), device=dev, dtype=dtype_t)
            func = cs.builtin_function(fun, cs_dtype) if fun >= 0 else None
            h = cs.Stencil(v, n, n, o, inp, wt, H=H, L=L, R=R, V=V, T=T, B=B, num_tiles=num_tiles, block_x=32,
                           block_y=8, dtype=cs_dtype, device=local, ncoef=len(w), func=func)
            h.set_stream(stream)
            outs.append(o)
            hs.append(h)
            keep.append(wt)
        return inp, outs, hs, keep

    def timed_sweep(hs, steps, warmup):
        for _ in range(warmup):
            for h in hs:
                h.compute()
        torch.cuda.synchronize(dev)
        if pg:
            pg.barrier()
        ev = [[(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in hs]
              for _ in range(steps)]
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        launches0 = cs.kernel_launches()
        torch.cuda.synchronize(dev)
        t0.record(stream)
        for s in range(steps):
            for k, h in enumerate(hs):
                ev[s][k][0].record(stream)
                h.compute()
                ev[s][k][1].record(stream)
        t1.record(stream)
        torch.cuda.synchronize(dev)
        launches = cs.kernel_launches() - launches0
        total_ms = t0.elapsed_time(t1)
        # per operator: the median of its timed Computes
        per_op = [sorted(ev[s][k][0].elapsed_time(ev[s][k][1]) for s in range(steps))[steps // 2]
                  for k in range(len(hs))]
        return total_ms, per_op, launches

    def timed_group(hs, steps, warmup):
        """K steps, each one custen_compute_group call over the handles (every operator on its handle's own
        stream between a fork and a join on `stream`), bracketed by events on `stream`."""
        for _ in range(warmup):
            cs.compute_group(hs, cs.DEVICE, stream)
        torch.cuda.synchronize(dev)
        if pg:
            pg.barrier()
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        launches0 = cs.kernel_launches()
        torch.cuda.synchronize(dev)
        t0.record(stream)
        for _ in range(steps):
            cs.compute_group(hs, cs.DEVICE, stream)
        t1.record(stream)
        torch.cuda.synchronize(dev)
        return t0.elapsed_time(t1), cs.kernel_launches() - launches0

    # ---- FP64 sweep (headline) ----
    # Stream order first (each operator's Compute timed with events: the per-operator figures and the
    # kernel roofline), then the headline: the same twelve Computes per step as one custen_compute_group
    # call, so that each launch's tail overlaps the next operator's start. With --one-output the operators
    # share their output field and stay in stream order.
    inp64, outs64, hs64, keep64 = build_handles(torch.float64, cs.F64, one_output=args.one_output)
    sampler = ClockSampler(local)
    sampler.start()
    total_ms, per_op, launches = timed_sweep(hs64, args.steps, args.warmup)
    stream_ms = reduce_max(total_ms, pg, dev) / args.steps
    group_ms = None
    if not args.one_output and not args.stream_order:
        group_total, launches = timed_group(hs64, args.steps, args.warmup)
        group_ms = reduce_max(group_total, pg, dev) / args.steps
    clocks = sampler.stop()
    ms_per_step = group_ms if group_ms is not None else stream_ms
    pts_step = len(ops) * n * n
    value = job_throughput(pts_step, world, ms_per_step) / 1e9
    stream_value = job_throughput(pts_step, world, stream_ms) / 1e9

    peaks = measured_peaks()
    hbm_peak = peaks.get("hbm_gbs") or 6800.0
    hbm_src = "measured" if peaks.get("hbm_gbs") else "fallback"
    kernel_ms = sum(per_op)
    bytes_alg = 16.0 * n * n * len(ops)
    achieved_gbs = bytes_alg / (kernel_ms * 1e-3) / 1e9
    fp64_rate = cs.probe_fma_rate(cs.F64)
    dfma = sum(o[10] for o in ops) * n * n
    achieved_fma = dfma / (kernel_ms * 1e-3)

    per = {}
    for (nm, v, *_rest), ms in zip(ops, per_op):
        dfma_pt = _rest[-1]
        per[nm] = {"gpts_s": round(n * n / (ms * 1e-3) / 1e9, 3), "ms": round(ms, 4),
                   "config": hs64[len(per)].config(),
                   "hbm_gbs": round(16.0 * n * n / (ms * 1e-3) / 1e9, 1),
                   "fp64_frac": round(dfma_pt * n * n / (ms * 1e-3) / fp64_rate, 3)}

    # ---- the six Fun operators again with the indirect call (library function fusion off) ----
    fun_indirect = None
    if not args.skip_indirect:
        fun_hs = [(nm, h) for (nm, *_r), h in zip(ops, hs64) if nm.endswith("Fun")]
        cs.set_fun_fusion(False)
        try:
            _, per_ind, _ = timed_sweep([h for _, h in fun_hs], max(1, args.steps), 1)
        finally:
            cs.set_fun_fusion(True)
        fun_indirect = {"per_op": {nm: {"gpts_s": round(n * n / (ms * 1e-3) / 1e9, 3), "ms": round(ms, 4)}
                                   for (nm, _), ms in zip(fun_hs, per_ind)},
                        "sweep_gpts_s_with_indirect_fun": round(
                            pts_step / ((kernel_ms - sum(per[nm]["ms"] for nm, _ in fun_hs) + sum(per_ind)) * 1e-3)
                            / 1e9, 3),
                        "note": "the Fun operators use the library's c^3 - c device functions; the headline runs "
                                "them fused (one cube per input value, then the coefficients as weights, "
                                "bit-identical); here each output point calls the function through its "
                                "pointer, as a user-defined function does"}

    # ---- FP32 precision variant: same sweep in FP32, error against the FP64 outputs ----
    fp32 = fp32_small = None
    if not args.skip_fp32 and not args.one_output:   # the error needs every FP64 operator's own output
        fp32_small = run_precision(cs, torch, dev, 4096)
        inp32, outs32, hs32, keep32 = build_handles(torch.float32, cs.F32)
        ms32, per32, _ = timed_sweep(hs32, max(1, args.steps), 3)
        fp32 = {"gpts_s": round(pts_step / (ms32 / max(1, args.steps) * 1e-3) / 1e9, 3),
                "hbm_gbs": round(8.0 * pts_step / (sum(per32) * 1e-3) / 1e9, 1), "per_op": {}}
        g32, _ = timed_group(hs32, max(1, args.steps), 3)
        fp32["group"] = {"gpts_s": round(pts_step / (g32 / max(1, args.steps) * 1e-3) / 1e9, 3),
                         "gbs": round(8.0 * pts_step / (g32 / max(1, args.steps) * 1e-3) / 1e9, 1),
                         "note": "the same sweep as one custen_compute_group call per step"}
        for (nm, *_r), ms, o32, o64, h32 in zip(ops, per32, outs32, outs64, hs32):
            d = o32.double() - o64
            fp32["per_op"][nm] = {
                "gpts_s": round(n * n / (ms * 1e-3) / 1e9, 3), "config": h32.config(),
                "gbs": round(8.0 * n * n / (ms * 1e-3) / 1e9, 1),
                "max_abs_err": float(d.abs().max().item()),
                "rel_l2": float((d.norm() / o64.norm()).item()),
            }
        del inp32, outs32, hs32, keep32
        torch.cuda.synchronize(dev)

    # ---- config 2 across sizes: n = 1024 .. 8192, numTiles 1 and 4 (16384 is the headline above) ----
    sizes_out = None
    if not args.skip_sizes:
        sizes_out = run_size_sweep(cs, torch, dev, local)

    # ---- WENO5 advection (the thirteenth operator), FP64 ----
    weno = None
    if not args.skip_weno:
        weno = run_weno(cs, torch, dev, n, fp64_rate)

    # ---- batched pentadiagonal systems (cuPentBatch) ----
    pent = None
    if not args.skip_pent:
        pent = run_pent(cs, torch, dev, hbm_peak, batch=args.pent_batch)

    # ---- e2e again, after the compute legs above: the spread between the two readings is the box's state
    # (sustained GPU compute slows host<->device DMA afterwards), reported beside the first reading ----
    e2e_after = None
    if e2e is not None and not args.skip_e2e_after:
        e2e_after = run_e2e(args, cs, np, local, ops, "pinned")

    # ---- CPU baseline (rank 0 only) ----
    cpu = None
    if rank == 0 and not args.skip_cpu:
        threads = os.cpu_count() or 1
        one = cpu_sample(n, args.cpu_rows, threads)
        one()
        t0c = time.perf_counter()
        pts = one()
        dtc = time.perf_counter() - t0c
        cpu = {"value": round(pts / dtc / 1e9, 4), "unit": "Gpts/s", "cores": threads, "kind": "port",
               "sample": f"{args.cpu_rows} rows x {n} columns per operator, 12 operators, plain host loop, "
                         f"{threads} threads",
               "single_thread": cpu_single_thread(n)}

    for h in hs64:
        h.destroy()
    del inp64, outs64, keep64
    torch.cuda.synchronize(dev)
    torch.cuda.empty_cache()

    ch_batched = ch_served = cpu_ch = None
    if not args.skip_ch:
        ch_batched = run_ch_batched(args, cs)
        ch_served = None if args.skip_served else run_ch_served(args, cs)
        pts_b = ch_batched["points"] * args.ch_steps
        ch_batched["roofline"] = {
            "bound": "fp64", "algorithmic_bytes_per_point_step": 56,
            "achieved_gbs": round(56.0 * ch_batched["fp64"]["gpt_steps_per_s"], 1), "hbm_peak_gbs": hbm_peak,
            "hbm_frac": round(56.0 * ch_batched["fp64"]["gpt_steps_per_s"] / hbm_peak, 4),
            "fp64_ops_per_point_step": 26,
            "fp64_frac": round(26e9 * ch_batched["fp64"]["gpt_steps_per_s"] / fp64_rate, 3),
            "note": "FP64-pipe bound: about 26 FP64 operations per point and step (right-hand side 12.7, x sweep "
                    "4, y sweep 5.7, update 3.7) against 56 compulsory bytes"}
        del pts_b
        if rank == 0 and not args.skip_cpu:
            cpu_ch = cpu_ch_sample()

    if rank == 0:
        line = {
            "metric": "stencil Gpts/s", "value": round(value, 3), "unit": "Gpts/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic: sin(3x)cos(5y)+U(-1e-3,1e-3), seed 1",
            "config": {"workload": f"cuSten stencil sweep FP64 {n}^2: 12 operators (X/Y 5-pt p/np, XY 3x3 "
                                   f"cross p/np, Fun c^3-c X/Y/XY p/np), numTiles=1, device-resident",
                       "schedule": ("one custen_compute_group call per step: the 12 independent handles, on "
                                    "three streams" if group_ms is not None else
                                    "12 Computes per step in stream order"),
                       "nx": n, "ny": n, "numTiles": 1, "l2": f"inputs larger than L2 ({n * n * 8 / 2**30:.3g} GiB per field)" if n * n * 8 > 129e6
                       else f"field of {n * n * 8 / 2**20:.3g} MiB fits in L2 (not the headline size)",
                       "parallelism": f"replicas x{world}"},
            "roofline": {"bound": "hbm", "achieved": round(achieved_gbs, 1), "peak": hbm_peak, "unit": "GB/s",
                         "frac": round(achieved_gbs / hbm_peak, 4),
                         "traffic": args.traffic if args.traffic is not None else round(TRAFFIC_16384 * (n / 16384) ** 2),
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum per launch, mean of the "
                                           "12 operators of one timed sweep at 16384^2" +
                                           ("" if n == 16384 else ", scaled by the point count"),
                         "peak_source": f"{hbm_src} hbm_gbs",
                         "note": "16 B/pt algorithmic; FP64 kernels are bound by the FP64 FMA pipe (binding): at "
                                 "the measured FP64 FMA rate the sweep's operators cap at 1.4-2.5 TB/s",
                         "binding": {"bound": "fp64", "achieved": round(achieved_fma / 1e9, 1),
                                     "peak": round(fp64_rate / 1e9, 1), "unit": "G FMA/s",
                                     "frac": round(achieved_fma / fp64_rate, 4),
                                     "peak_source": "measured live (custen_probe_fma_rate)",
                                     "hbm_frac_at_fp64_peak": round(achieved_gbs / hbm_peak * fp64_rate / achieved_fma,
                                                                    4)}},
            "fp64": {"achieved_fma_s": round(achieved_fma / 1e9, 1), "peak_fma_s": round(fp64_rate / 1e9, 1),
                     "unit": "G FMA/s", "frac": round(achieved_fma / fp64_rate, 4),
                     "peak_source": "measured live (custen_probe_fma_rate)"},
            "per_op": per,
            "stream_order": {"value": round(stream_value, 3), "ms_per_step": round(stream_ms, 3),
                             "note": "the same step as 12 Computes in stream order, each timed with events "
                                     "(per_op; the roofline's kernel times)"},
            "gpu_launches": launches,
            "clocks": clocks,
        }
        if fp32 is not None:
            line["fp32"] = fp32
        if fp32_small is not None:
            line["fp32_4096"] = fp32_small
        if e2e is not None:
            line["e2e"] = e2e
            if e2e_after is not None:
                line["e2e"]["after_compute"] = {
                    k: e2e_after[k] for k in ("value", "unit", "ms_per_step", "h2d_bytes_per_step", "d2h_bytes_per_step")}
                if "link" in e2e_after:
                    line["e2e"]["after_compute"]["link"] = {k: e2e_after["link"][k]
                                                           for k in ("each_way_gbs", "link_each_way_gbs", "frac")}
                line["e2e"]["spread"] = {
                    "first": e2e["value"], "after_compute": e2e_after["value"],
                    "note": "value is the reading taken first, before this process's compute legs; after_compute is "
                            "the same leg after the FP64/FP32 sweeps, size sweep, WENO and pentadiagonal legs "
                            "(about a minute of GPU compute)"}
        if e2e_managed is not None:
            line["e2e_managed"] = e2e_managed
        if cpu is not None:
            line["cpu_baseline"] = cpu
        if fun_indirect is not None:
            line["fun_indirect"] = fun_indirect
        if sizes_out is not None:
            line["sizes"] = sizes_out
        if weno is not None:
            line["weno"] = weno
        if pent is not None:
            line["pent_batch"] = pent
        if cpu_ch is not None:
            line["cpu_baseline_ch"] = cpu_ch
        if ch_batched is not None:
            line["ch_batched"] = ch_batched
            if ch_served is not None:
                line["ch_served"] = ch_served
        print(json.dumps(line), flush=True)
    if pg:
        pg.barrier()
        pg.destroy_process_group()


def link_each_way_gbs(local: int, nbytes: int = 1 << 30, reps: int = 3) -> float:
    """Host-link rate with both directions busy at once: a pinned host->device and a device->host copy of
    nbytes each, on two streams, started together; nbytes / the time both take (best of reps). The
    staged e2e path moves rows both ways at the same time, so this is its ceiling."""
    import torch
    dev = torch.device("cuda", local)
    count = nbytes // 8
    h_in = torch.ones(count, dtype=torch.float64, pin_memory=True)
    h_out = torch.empty(count, dtype=torch.float64, pin_memory=True)
    d_in = torch.empty(count, dtype=torch.float64, device=dev)
    d_out = torch.ones(count, dtype=torch.float64, device=dev)
    s1, s2 = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    best = float("inf")
    for _ in range(reps + 1):
        torch.cuda.synchronize(dev)
        t0 = time.perf_counter()
        with torch.cuda.stream(s1):
            d_in.copy_(h_in, non_blocking=True)
        with torch.cuda.stream(s2):
            h_out.copy_(d_out, non_blocking=True)
        torch.cuda.synchronize(dev)
        best = min(best, time.perf_counter() - t0)
    del h_in, h_out, d_in, d_out
    return nbytes / best / 1e9


def run_e2e(args, cs, np, local, ops, kind="pinned", steps=None):
    """The same sweep through the reference-facing API on host buffers, numTiles=4, HOST offload,
    host<->device traffic inside the timed region.

    kind "pinned": fields in pinned host memory; each Compute streams the rows through device staging
    slots (copy-in, kernel and copy-out of successive chunks overlap). kind "managed": fields in managed
    memory, the reference's own HOST path (cudaMemPrefetchAsync of each tile to the device and back).
    The byte counts are the library's own counters of what Compute moved."""
    import ctypes

    n = args.e2e_n
    steps = steps or args.e2e_steps
    nbytes = n * n * 8
    lib = cs.lib()
    allocs = []

    def host(nb):
        p = ctypes.c_void_p()
        fn = lib.custen_malloc_host if kind == "pinned" else lib.custen_malloc_managed
        cs._check(fn(ctypes.byref(p), nb))
        allocs.append(p.value)
        return p.value

    def arr(ptr, count):
        return np.frombuffer((ctypes.c_char * (8 * count)).from_address(ptr), dtype=np.float64)

    from custen_gb300.inputs import field
    inp = host(nbytes)
    arr(inp, n * n)[:] = field(n, n, 1).ravel()
    outs, hs = [], []
    for (nm, v, H, L, R, V, T, B, w, fun, _) in ops:
        o = host(nbytes)
        arr(o, n * n)[:] = 0.0
        wp = host(8 * len(w))
        arr(wp, len(w))[:] = w
        func = cs.builtin_function(fun, cs.F64) if fun >= 0 else None
        hs.append(cs.Stencil(v, n, n, o, inp, wp, H=H, L=L, R=R, V=V, T=T, B=B, num_tiles=4, block_x=32, block_y=8,
                             ncoef=len(w), func=func, device=local))
        outs.append(o)
    for h in hs:
        h.compute(cs.HOST)
    cs._check(lib.custen_device_synchronize())
    link = link_each_way_gbs(local) if kind == "pinned" else None
    per_buffer = host_buffer_rates(lib, local, [inp] + outs, nbytes) if kind == "pinned" else None
    h2d0, d2h0 = cs.transfer_bytes()
    launches0 = cs.kernel_launches()
    t0 = time.perf_counter()
    for _ in range(steps):
        for h in hs:
            h.compute(cs.HOST)
        cs._check(lib.custen_device_synchronize())
        _ = float(arr(outs[-1], 1)[0])  # host read of the result
    dt = (time.perf_counter() - t0) / steps
    h2d1, d2h1 = cs.transfer_bytes()
    launches = (cs.kernel_launches() - launches0) // steps
    for h in hs:
        h.destroy()
    for p in allocs:
        (lib.custen_free_host if kind == "pinned" else lib.custen_free)(p)
    what = ("pinned host buffers, rows streamed through device staging slots in 32 MiB chunks"
            if kind == "pinned" else "managed buffers, tiles prefetched to the device and back (reference HOST path)")
    out = {"value": round(len(ops) * n * n / dt / 1e9, 3), "unit": "Gpts/s",
           "h2d_bytes_per_step": (h2d1 - h2d0) // steps, "d2h_bytes_per_step": (d2h1 - d2h0) // steps,
           "ms_per_step": round(dt * 1e3, 2), "steps": steps, "kernel_launches_per_step": launches,
           "path": f"{n}^2, 12 operators, numTiles=4, Compute(HOST) per operator; {what}"}
    if link:
        each_way = max(h2d1 - h2d0, d2h1 - d2h0) / steps / dt / 1e9
        out["link"] = {"each_way_gbs": round(each_way, 1), "link_each_way_gbs": round(link, 1),
                       "frac": round(each_way / link, 3), "host_buffers": per_buffer,
                       "note": "the host link measured just before, both directions busy at once (1 GiB each way); "
                               "host_buffers: one-way copy rates of every host buffer of this leg"}
    return out


def host_buffer_rates(lib, local, ptrs, nbytes, probe=1 << 28):
    """One-way copy rate of pinned host buffers of nbytes each (host->device and device->host, the first
    min(probe, nbytes) bytes of each): the slowest and the median. A buffer whose pages sit far from
    the GPU shows here."""
    import ctypes
    import torch
    probe = min(probe, nbytes)   # never past the end of a buffer
    dev = torch.device("cuda", local)
    d = torch.empty(probe // 8, dtype=torch.float64, device=dev)
    rates = {"h2d": [], "d2h": []}
    for p in ptrs:
        for direction in ("h2d", "d2h"):
            src, dst = (p, d.data_ptr()) if direction == "h2d" else (d.data_ptr(), p)
            lib.custen_memcpy(ctypes.c_void_p(dst), ctypes.c_void_p(src), probe)   # warm
            torch.cuda.synchronize(dev)
            t0 = time.perf_counter()
            lib.custen_memcpy(ctypes.c_void_p(dst), ctypes.c_void_p(src), probe)
            torch.cuda.synchronize(dev)
            rates[direction].append(probe / (time.perf_counter() - t0) / 1e9)
    del d
    out = {}
    for direction, r in rates.items():
        if r:
            r.sort()
            out[direction] = {"min_gbs": round(r[0], 1), "median_gbs": round(r[len(r) // 2], 1), "buffers": len(r)}
    return out


# ----------------------------------------------------------------------------------------------
# Stencil sweep across sizes (config 2) and the WENO operator
# ----------------------------------------------------------------------------------------------
def run_size_sweep(cs, torch, dev, local, sizes=(1024, 2048, 4096, 8192), tiles=(1, 4), group=True):
    """The 12-operator FP64 sweep at smaller grids, device-resident, numTiles 1 and 4. For n <= 2048 the
    sweep is captured once in a CUDA graph and the graph is replayed (launch latency would dominate),
    in stream order and again as one custen_compute_group call (the operators free to overlap);
    otherwise sweeps are timed with events. Median of the timed repetitions."""
    out = {}
    for n in sizes:
        ops = operators(n)
        x = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
        inp = (torch.sin(3 * x)[None, :] * torch.cos(5 * x)[:, None]).contiguous()
        for nt in tiles:
            outs, hs, keep = [], [], []
            for (nm, v, H, L, R, V, T, B, w, fun, _) in ops:
                wt = torch.tensor(w, device=dev, dtype=torch.float64)
                o = torch.zeros((n, n), device=dev, dtype=torch.float64)
                func = cs.builtin_function(fun, cs.F64) if fun >= 0 else None
                hs.append(cs.Stencil(v, n, n, o, inp, wt, H=H, L=L, R=R, V=V, T=T, B=B, num_tiles=nt, block_x=32,
                                     block_y=8, dtype=cs.F64, device=local, ncoef=len(w), func=func))
                outs.append(o)
                keep.append(wt)
            side = torch.cuda.Stream(dev)
            with torch.cuda.stream(side):
                for h in hs:
                    h.compute(stream=side)
            torch.cuda.synchronize(dev)
            graph = None
            if n <= 2048:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, capture_error_mode="relaxed"):
                    cap = torch.cuda.current_stream(dev)
                    for h in hs:
                        h.compute(stream=cap)
                graph.replay()
                torch.cuda.synchronize(dev)
            reps, times = 20, []
            s = torch.cuda.current_stream(dev)
            for _ in range(reps):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(s)
                if graph is not None:
                    graph.replay()
                else:
                    for h in hs:
                        h.compute(stream=s)
                e1.record(s)
                torch.cuda.synchronize(dev)
                times.append(e0.elapsed_time(e1))
            ms = sorted(times)[len(times) // 2]
            out[f"{n}_tiles{nt}"] = {"gpts_s": round(len(ops) * n * n / (ms * 1e-3) / 1e9, 3),
                                     "ms_per_sweep": round(ms, 4), "timing": "graph replay" if graph else "events"}
            if group:
                # the twelve operators are independent (one input, twelve outputs): one custen_compute_group
                # call runs them on three of the handles' streams, so that one launch's tail overlaps the next
                g2 = None
                if graph is not None:
                    g2 = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g2, capture_error_mode="relaxed"):
                        cs.compute_group(hs, cs.DEVICE, torch.cuda.current_stream(dev))
                    g2.replay()
                else:
                    cs.compute_group(hs, cs.DEVICE, s)
                torch.cuda.synchronize(dev)
                times = []
                for _ in range(reps):
                    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    e0.record(s)
                    if g2 is not None:
                        g2.replay()
                    else:
                        cs.compute_group(hs, cs.DEVICE, s)
                    e1.record(s)
                    torch.cuda.synchronize(dev)
                    times.append(e0.elapsed_time(e1))
                ms2 = sorted(times)[len(times) // 2]
                out[f"{n}_tiles{nt}"]["group"] = {
                    "gpts_s": round(len(ops) * n * n / (ms2 * 1e-3) / 1e9, 3), "ms_per_sweep": round(ms2, 4),
                    "timing": ("graph replay of " if g2 is not None else "events around ") +
                              "one custen_compute_group call over the 12 handles"}
                del g2
            for h in hs:
                h.destroy()
            del graph, outs, keep
        del inp
        torch.cuda.synchronize(dev)
    return out


def pent_inputs(torch, dev, m, batch):
    """Diagonally dominant interleaved systems (seeded): ds, dl, d, du, dw, b of shape (m, batch)."""
    g = torch.Generator(device=dev)
    g.manual_seed(0)

    def r():
        return torch.rand((m, batch), device=dev, dtype=torch.float64, generator=g) * 2 - 1
    ds, dl, du, dw, b = r(), r(), r(), r(), r()
    d = torch.rand((m, batch), device=dev, dtype=torch.float64, generator=g) * 3 + 5
    ds[:2] = 0
    dl[:1] = 0
    du[m - 1:] = 0
    dw[m - 2:] = 0
    return [ds, dl, d, du, dw, b]


def event_ms(torch, fn, reps=5):
    fn()
    torch.cuda.synchronize()
    times = []
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        fn()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    return sorted(times)[len(times) // 2]


def run_precision(cs, torch, dev, n, steps=20):
    """The precision variant at a second size (n^2, device-resident, numTiles 1): every stencil in FP64 and
    in FP32 on the same input (cast from FP64), the FP32 error against the FP64 output (max abs, rel L2)
    and the achieved GB/s of both (median of `steps` timed Computes)."""
    x = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
    g = torch.Generator(device=dev)
    g.manual_seed(1)
    f64 = (torch.sin(3 * x)[None, :] * torch.cos(5 * x)[:, None]
           + (torch.rand((n, n), device=dev, dtype=torch.float64, generator=g) * 2e-3 - 1e-3)).contiguous()
    f32 = f64.float().contiguous()
    s = torch.cuda.current_stream(dev)
    per = {}
    for (nm, v, H, L, R, V, T, B, w, fun, _) in operators(n):
        res = {}
        for dt_t, cdt, f in ((torch.float64, cs.F64, f64), (torch.float32, cs.F32, f32)):
            wt = torch.tensor(w, device=dev, dtype=dt_t)
            o = torch.zeros((n, n), device=dev, dtype=dt_t)
            func = cs.builtin_function(fun, cdt) if fun >= 0 else None
            h = cs.Stencil(v, n, n, o, f, wt, H=H, L=L, R=R, V=V, T=T, B=B, block_x=32, block_y=8, dtype=cdt,
                           ncoef=len(w), func=func)
            for _ in range(3):
                h.compute(stream=s)
            times = []
            for _ in range(steps):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(s)
                h.compute(stream=s)
                e1.record(s)
                torch.cuda.synchronize(dev)
                times.append(e0.elapsed_time(e1))
            h.destroy()
            res[cdt] = (o, sorted(times)[steps // 2], wt)
        d = res[cs.F32][0].double() - res[cs.F64][0]
        per[nm] = {"fp32_gbs": round(8.0 * n * n / (res[cs.F32][1] * 1e-3) / 1e9, 1),
                   "fp64_gbs": round(16.0 * n * n / (res[cs.F64][1] * 1e-3) / 1e9, 1),
                   "max_abs_err": float(d.abs().max().item()),
                   "rel_l2": float((d.norm() / res[cs.F64][0].norm()).item())}
    del f64, f32
    torch.cuda.empty_cache()
    return {"n": n, "per_op": per,
            "note": "fields of 134 MB (FP64, about the size of L2) and 67 MB (FP32, inside L2): the GB/s here "
                    "are not HBM figures"}


def run_pent(cs, torch, dev, hbm_peak, m=256, batch=1 << 18):
    """cuPentBatch's factorisation and solve over `batch` interleaved systems of m unknowns (the layout's
    wire format), and the inverted-pivot solve; 72 B per row of compulsory traffic in each."""
    base = pent_inputs(torch, dev, m, batch)
    work = [a.clone() for a in base[:5]]
    rows = m * batch
    copy_ms = event_ms(torch, lambda: [a.copy_(b) for a, b in zip(work, base[:5])])
    f_ms = event_ms(torch, lambda: ([a.copy_(b) for a, b in zip(work, base[:5])],
                                    cs.pent_factor_batch(*work, m, batch))) - copy_ms
    bb = base[5].clone()
    bcopy_ms = event_ms(torch, lambda: bb.copy_(base[5]))
    s_ms = event_ms(torch, lambda: (bb.copy_(base[5]), cs.pent_solve_batch(*work, bb, m, batch))) - bcopy_ms
    rd = work[2].clone()
    cs.pent_invert_pivots(rd, m, batch)
    r_ms = event_ms(torch, lambda: (bb.copy_(base[5]), cs.pent_solve_batch(work[0], work[1], rd, work[3], work[4], bb,
                                                                            m, batch, inverted_pivots=True))) - bcopy_ms
    out = {"config": f"{batch} systems x {m} unknowns, interleaved [row * batch + system], FP64"}
    for nm, ms in (("factor", f_ms), ("solve", s_ms), ("solve_inverted_pivots", r_ms)):
        out[nm] = {"grows_s": round(rows / (ms * 1e-3) / 1e9, 2), "ms": round(ms, 4),
                   "hbm_gbs": round(72.0 * rows / (ms * 1e-3) / 1e9, 1),
                   "hbm_frac": round(72.0 * rows / (ms * 1e-3) / 1e9 / hbm_peak, 4)}
    out["note"] = ("factor and exact solve: bit-identical to cuPentBatch, FP64-bound by their correctly rounded "
                   "divisions; inverted pivots: HBM-bound")
    del base, work, bb, rd
    torch.cuda.empty_cache()
    return out


def run_weno(cs, torch, dev, n, fp64_rate):
    """cuStenCompute2DXYWENOADVp at n^2: out = u * WENO5_x + v * WENO5_y, u, v ~ U(-1, 1), 32 B/pt."""
    import numpy as np
    rng = np.random.default_rng(1)
    x = torch.arange(n, device=dev, dtype=torch.float64) * (2 * math.pi / n)
    f = (torch.sin(3 * x)[None, :] * torch.cos(5 * x)[:, None]).contiguous()
    u = torch.tensor(rng.uniform(-1, 1, (n, n)), device=dev)
    v = torch.tensor(rng.uniform(-1, 1, (n, n)), device=dev)
    o = torch.zeros_like(f)
    h = 2 * math.pi / n
    op = cs.WenoAdvection(n, n, o, f, u, v, dx=h, dy=h, block_x=32, block_y=8)
    s = torch.cuda.current_stream(dev)
    op.compute(stream=s)
    torch.cuda.synchronize(dev)
    times = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        op.compute(stream=s)
        e1.record(s)
        torch.cuda.synchronize(dev)
        times.append(e0.elapsed_time(e1))
    op.destroy()
    ms = sorted(times)[len(times) // 2]
    gpts = n * n / (ms * 1e-3) / 1e9
    del f, u, v, o
    torch.cuda.empty_cache()
    return {"gpts_s": round(gpts, 3), "ms": round(ms, 3), "hbm_gbs": round(32.0 * gpts, 1),
            "config": f"{n}^2, periodic, u, v ~ U(-1, 1), dx = dy = 2 pi / n",
            "note": "FP64-pipe bound: about 100 FP64 operations per point (conversions and most of the eight "
                    "correctly rounded divisions on the other pipes) against 32 bytes"}


# ----------------------------------------------------------------------------------------------
# Cahn-Hilliard ADI: batched (config 4) and served (config 5)
# ----------------------------------------------------------------------------------------------
def plain_step_seconds(cs, n: int, steps: int = 10) -> float:
    """One grid at a time, one step per launch sequence with a synchronisation after every step (the
    structure of the reference's plain loop, cuPentCahnADI.cu:528-596), timed per step."""
    import numpy as np
    b = cs.CahnHilliardBatch([n])
    b.set_state(0, np.random.default_rng(n).uniform(-0.1, 0.1, (n, n)))
    b.step(2, graph=False)
    b.synchronize()
    t0 = time.perf_counter()
    for _ in range(steps):
        b.step(1, graph=False)
        b.synchronize()
    dt = (time.perf_counter() - t0) / steps
    b.close()
    return dt


def run_plain_loop(cs, sizes, steps):
    """One grid at a time through this library, one step per launch sequence with a synchronisation after
    every step (the structure of the reference's plain loop, cuPentCahnADI.cu:528-596), measured end to
    end over the given grids in order. Returns the wall time in seconds."""
    import numpy as np
    crng = np.random.default_rng(4)
    t0 = time.perf_counter()
    for n in sizes:
        b = cs.CahnHilliardBatch([n])
        b.set_state(0, crng.uniform(-0.1, 0.1, (n, n)))
        for _ in range(steps):
            b.step(1, graph=False)
            b.synchronize()
        b.close()
    return time.perf_counter() - t0


def run_ch_batched(args, cs):
    """512 periodic grids, N uniform over {64,...,1024} (seed 2), c0 ~ U(-0.1, 0.1), 500 steps; the FP64
    batch and the FP32-stencil batch start from the same fields, and the FP32-stencil result is compared
    with the FP64 one grid by grid."""
    import numpy as np
    rng = np.random.default_rng(2)
    sizes = [int(v) for v in rng.choice([64, 128, 256, 512, 1024], size=args.ch_sims)]
    steps = args.ch_steps
    out = {"config": f"{args.ch_sims} grids, N uniform over {{64..1024}} (seed 2), {steps} steps, lx = 2 pi, "
                     f"gamma 0.01, dt = 0.1 dx", "points": int(sum(n * n for n in sizes))}
    finals = {}
    for label, dt in (("fp64", cs.F64), ("fp32_stencil", cs.F32)):
        b = cs.CahnHilliardBatch(sizes, rhs_dtype=dt)
        crng = np.random.default_rng(3)
        for k, n in enumerate(sizes):
            b.set_state(k, crng.uniform(-0.1, 0.1, (n, n)))
        mean0 = [b.mean(k) for k in range(len(sizes))]
        b.step(2)
        b.synchronize()
        if args.ch_config >= 0:
            b.set_config(args.ch_config)
            cfg_name = b.config()
        else:
            cfg_name = b.autotune(steps=4) if args.autotune else b.config()   # state restored by the tuner
        l0 = b.launches()
        t0 = time.perf_counter()
        b.step(steps)
        b.synchronize()
        wall = time.perf_counter() - t0
        out[label] = {"wall_s": round(wall, 4), "steps_per_s": round(len(sizes) * steps / wall, 1),
                      "gpt_steps_per_s": round(out["points"] * steps / wall / 1e9, 3),
                      "ms_per_step": round(wall / steps * 1e3, 4), "launches": b.launches() - l0,
                      "graphs": "pairs of steps", "kernel_config": cfg_name,
                      "max_mass_drift": max(abs(b.mean(k) - mean0[k]) for k in range(len(sizes)))}
        finals[label] = [b.state(k)[0] for k in range(len(sizes))]
        b.close()
    # conditioning of the problem: FP64 from c0 rounded to FP32 (a perturbation of FP32 rounding size), the
    # same step count; phase separation amplifies any perturbation, so this is the yardstick for the
    # FP32-stencil error above
    b = cs.CahnHilliardBatch(sizes)
    crng = np.random.default_rng(3)
    for k, n in enumerate(sizes):
        b.set_state(k, crng.uniform(-0.1, 0.1, (n, n)).astype(np.float32).astype(np.float64))
    b.set_config(args.ch_config)
    b.step(2 + steps)
    b.synchronize()
    finals["fp64_c0_fp32"] = [b.state(k)[0] for k in range(len(sizes))]
    b.close()
    # the FP32-stencil variant against the FP64 one (the pinned path: parity-tested against the oracle at
    # these sizes), per grid size after 2 + steps steps from the same fields
    err = {}
    for k, n in enumerate(sizes):
        r = finals["fp64"][k]
        a, p = finals["fp32_stencil"][k], finals["fp64_c0_fp32"][k]
        e = err.setdefault(str(n), {"grids": 0, "max_rel_l2": 0.0, "median_rel_l2": [], "max_abs": 0.0,
                                    "fp64_c0_fp32_max_rel_l2": 0.0})
        e["grids"] += 1
        rl = float(np.linalg.norm(a - r) / np.linalg.norm(r))
        e["max_rel_l2"] = max(e["max_rel_l2"], rl)
        e["median_rel_l2"].append(rl)
        e["max_abs"] = max(e["max_abs"], float(np.abs(a - r).max()))
        e["fp64_c0_fp32_max_rel_l2"] = max(e["fp64_c0_fp32_max_rel_l2"], float(np.linalg.norm(p - r) / np.linalg.norm(r)))
    for e in err.values():
        e["median_rel_l2"] = float(np.median(e["median_rel_l2"]))
    del finals
    out["fp32_stencil"]["error_vs_fp64"] = {
        "by_n": dict(sorted(err.items(), key=lambda kv: int(kv[0]))), "steps": steps + 2,
        "note": "relative L2 and max abs of each FP32-stencil grid against the same grid in FP64 (same c0, same "
                "step count), maxima (and median rel L2) per grid size. fp64_c0_fp32_max_rel_l2: FP64 run from c0 "
                "rounded to FP32 against the FP64 run, the problem's own amplification of a perturbation of that "
                "size over these steps. max_mass_drift: |mean(c_end) - mean(c0)|, FP64 compensated sums on the "
                "device"}
    # plain loop on the same GPU: one grid at a time, measured on the first grids of the list, beside the
    # per-size model used for the whole list
    per_size = {n: plain_step_seconds(cs, n) for n in sorted(set(sizes))}
    plain_total = sum(per_size[n] * steps for n in sizes)
    sub = sizes[:args.plain_grids]
    sub_wall = run_plain_loop(cs, sub, steps)
    sub_model = sum(per_size[n] * steps for n in sub)
    out["plain_loop"] = {"steps_per_s": round(len(sizes) * steps / plain_total, 1),
                         "wall_s_estimated": round(plain_total, 3),
                         "step_ms_by_n": {str(n): round(v * 1e3, 4) for n, v in per_size.items()},
                         "method": "this library's kernels, one grid per launch sequence, synchronised per "
                                   "step; per-size step time x steps, summed over grids",
                         "measured_subset": {
                             "grids": len(sub), "sizes": sub, "steps": steps, "wall_s": round(sub_wall, 3),
                             "steps_per_s": round(len(sub) * steps / sub_wall, 1),
                             "model_wall_s": round(sub_model, 3), "measured_over_model": round(sub_wall / sub_model, 3),
                             "note": "the first grids of the list run one at a time for the full step count, each "
                                     "step synchronised, wall clock end to end (grid set-up included)"}}
    out["speedup_vs_plain_loop"] = round(out["fp64"]["steps_per_s"] / out["plain_loop"]["steps_per_s"], 2)
    out["speedup_vs_plain_loop_measured"] = round(
        out["fp64"]["steps_per_s"] / out["plain_loop"]["measured_subset"]["steps_per_s"], 2)
    return out


def served_workload(args, rate=None, count=None, seed=3):
    """(arrival times, grid sizes, step counts) of the served request stream: Poisson arrivals (mean rate,
    seed 3), N log-uniform 128-2048 rounded to a multiple of 32, steps U(100, 5000)."""
    import numpy as np
    rng = np.random.default_rng(seed)
    R = count or args.served_requests
    gaps = rng.exponential(1.0 / (rate or args.served_rate), size=R)
    arrivals = [float(a) for a in np.cumsum(gaps) - gaps[0]]
    sizes = [int(max(128, min(2048, round(math.exp(v) / 32) * 32)))
             for v in rng.uniform(math.log(128), math.log(2048), size=R)]
    steps = [int(v) for v in rng.integers(100, 5001, size=R)]
    return arrivals, sizes, steps


def serve(args, cs, arrivals, sizes, steps):
    """Run one request stream through the server; its figures."""
    import numpy as np
    R = len(sizes)
    srv = cs.CahnHilliardServer(hbm_budget_bytes=150e9, chunk_steps=args.served_chunk, keep_results=False)
    for k in range(R):
        srv.submit(sizes[k], steps[k], arrival=float(arrivals[k]), seed=1000 + k)
    srv.run()
    st = srv.stats()
    res = [srv.result(k, field=False) for k in range(R)]
    srv.close()
    ttc = np.array([r["ttc"] for r in res])
    wait = np.array([r["admit"] - r["arrival"] for r in res])
    drift = max(abs(r["mean_end"] - r["mean0"]) for r in res)
    total_steps = int(sum(steps))
    return {"requests": R, "makespan_s": round(st["makespan"], 3),
            "arrivals_span_s": round(float(arrivals[-1]), 3),
            "arrivals_span_over_makespan": round(float(arrivals[-1]) / st["makespan"], 3),
            "steps_per_s": round(total_steps / st["makespan"], 1),
            "gpt_steps_per_s": round(st["point_steps"] / st["makespan"] / 1e9, 3),
            "ttc_p50_s": round(float(np.percentile(ttc, 50)), 3), "ttc_p99_s": round(float(np.percentile(ttc, 99)), 3),
            "admission_wait_p50_s": round(float(np.percentile(wait, 50)), 4),
            "admission_wait_p99_s": round(float(np.percentile(wait, 99)), 4),
            "max_resident": st["max_active"], "peak_resident_gb": round(st["peak_bytes"] / 1e9, 2),
            "max_mass_drift": drift}


def fcfs_plain(per_size, arrivals, sizes, steps):
    """The plain sequential loop over a request stream: first come first served, one grid at a time."""
    import numpy as np
    t, ttc = 0.0, []
    for a, n, k in zip(arrivals, sizes, steps):
        start = max(t, float(a))
        t = start + k * per_size[n]
        ttc.append(t - float(a))
    return {"makespan_s": round(t, 3), "steps_per_s": round(int(sum(steps)) / t, 1),
            "ttc_p50_s": round(float(np.percentile(ttc, 50)), 3), "ttc_p99_s": round(float(np.percentile(ttc, 99)), 3),
            "method": "FCFS queue over the measured per-size step time of one grid at a time"}


def run_ch_served(args, cs):
    """Poisson arrivals (mean rate, seed 3), N log-uniform 128-2048 rounded to 32, steps U(100, 5000),
    c0 ~ U(-0.1, 0.1), HBM budget 150 GB, a fixed number of requests.

    At the configured 200 requests/s the offered load is far above what one GPU serves, so every request
    arrives within the first fraction of a second and the run drains a full queue. A second stream at 0.9 of
    the throughput measured on the first (same size and step distributions, seed 4) keeps requests arriving
    while others complete, so admission happens continuously over the whole run."""
    arrivals, sizes, steps = served_workload(args)
    out = serve(args, cs, arrivals, sizes, steps)
    out["config"] = (f"{len(sizes)} requests, Poisson {args.served_rate}/s (seed 3), N log-uniform 128-2048 "
                     f"(multiples of 32), steps U(100, 5000), budget 150 GB, chunk {args.served_chunk} steps")
    rate = 0.9 * len(sizes) / out["makespan_s"]
    c_arr, c_sizes, c_steps = served_workload(args, rate=rate, count=args.served_continuous, seed=4)
    cont = serve(args, cs, c_arr, c_sizes, c_steps)
    cont["config"] = (f"{len(c_sizes)} requests, Poisson {rate:.2f}/s (0.9 x the requests/s served above; seed 4), "
                      f"same N and step distributions, budget 150 GB, chunk {args.served_chunk} steps")
    per_size = {n: plain_step_seconds(cs, n, steps=5) for n in sorted(set(sizes) | set(c_sizes))}
    out["plain_loop"] = fcfs_plain(per_size, arrivals, sizes, steps)
    out["speedup_vs_plain_loop"] = round(out["steps_per_s"] / out["plain_loop"]["steps_per_s"], 2)
    cont["plain_loop"] = fcfs_plain(per_size, c_arr, c_sizes, c_steps)
    cont["speedup_vs_plain_loop"] = round(cont["steps_per_s"] / cont["plain_loop"]["steps_per_s"], 2)
    out["continuous"] = cont
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=16384)
    ap.add_argument("--e2e-n", type=int, default=16384)
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--cpu-rows", type=int, default=4096)
    ap.add_argument("--skip-fp32", action="store_true")
    ap.add_argument("--skip-e2e", action="store_true")
    ap.add_argument("--skip-e2e-managed", action="store_true")
    ap.add_argument("--skip-e2e-after", action="store_true", help="skip the second e2e reading after the compute legs")
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--skip-ch", action="store_true")
    ap.add_argument("--skip-served", action="store_true")
    ap.add_argument("--ch-sims", type=int, default=512)
    ap.add_argument("--ch-steps", type=int, default=500)
    ap.add_argument("--served-requests", type=int, default=96)
    ap.add_argument("--served-rate", type=float, default=200.0)
    ap.add_argument("--served-chunk", type=int, default=16)
    ap.add_argument("--served-continuous", type=int, default=48,
                    help="requests of the second served stream (arrivals at 0.9 x the measured throughput)")
    ap.add_argument("--plain-grids", type=int, default=32,
                    help="grids of the batched workload run one at a time for the measured plain loop")
    ap.add_argument("--skip-ref-gpu", action="store_true")
    ap.add_argument("--skip-sizes", action="store_true")
    ap.add_argument("--skip-weno", action="store_true")
    ap.add_argument("--skip-indirect", action="store_true")
    ap.add_argument("--stream-order", action="store_true",
                    help="time the headline as 12 Computes in stream order instead of one grouped call per step")
    ap.add_argument("--one-output", action="store_true",
                    help="the FP64 sweep's operators all write one output field (4 GiB on the device at 16384^2 "
                         "instead of 26; the same work and DRAM traffic per launch)")
    ap.add_argument("--skip-pent", action="store_true")
    ap.add_argument("--pent-batch", type=int, default=1 << 18, help="systems in the pentadiagonal leg (256 unknowns each)")
    ap.add_argument("--ch-config", type=int, default=-1,
                    help="pin the CH batch kernel configuration (0..21) instead of tuning it")
    ap.add_argument("--stage-chunk-mb", type=int, default=0,
                    help="chunk size of the host-memory staging path (0: the library default)")
    ap.add_argument("--autotune", type=int, default=1, choices=[0, 1, 2],
                    help="kernel configuration choice: 0 defaults, 1 tune at the first Compute (default), 2 always")
    ap.add_argument("--traffic", type=float, default=None,
                    help="dram bytes per launch from an ncu capture (default: the 16384^2 capture of the "
                         "sweep, scaled to --n by the point count)")
    args = ap.parse_args()
    world, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference_arm(args, world, rank)
        return
    run_gpu(args, world, rank, local)


if __name__ == "__main__":
    main()
