#!/usr/bin/env python
"""Benchmark of the HAL-CPP hot path on one GB300 (or N replicas).

Headline workload (one "step"): 200 ADI ticks of a 2048x2048 FP32 field at
D*dt/dx^2 = 5.0, decay 0.01, a constant source field, zero-flux edges
(f' = ADI(f) - 0.01 f + s per tick, PDEGrid2D semantics).  The metric is
cell-updates per second over all GPUs.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

* value      -- device time of the resident run (inputs already in HBM),
                L2 flushed between steps (a 512 MB write), CUDA events on the
                handle's stream.
* e2e        -- the same ticks through hal_cuda_adi_run_ticks_host: field and
                source copied in from pinned host memory and the field copied
                back, inside the timed region, every step.
* roofline   -- the dominant kernel's algorithmic bytes per launch over its
                CUDA-event launch time (hal_cuda_adi_profile), against the
                measured HBM copy bandwidth.
* cpu_baseline -- the CPU oracle (a C restatement of the reference's FP64 CPU
                backend, 1 thread as the reference ships) on a bounded sample.
* secondary  -- the explicit 2048^2 tick, the 1M-agent force pass, 512
                batched wells, the adjoint gradient, and the FP64 per-cell
                rate diffusion / advection stencils.

--impl reference times the CPU oracle alone (all host threads) on the same
workload, one bounded sample per step.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "hal-cpp_gb300"))

N = 2048
TICKS = 200
RATE = 5.0
DECAY = 0.01
CELLS = N * N
ADI_COL_BYTES = 8    # x-sweep: read f, write w (FP32)
ADI_ROW_BYTES = 16   # y-sweep: read w, f, src; write f'
EXPLICIT_BYTES = 8   # fused tick: read f, write f'
FLUSH_BYTES = 512 << 20


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as fh:
            p = json.load(fh)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    return rank, local, world


def max_over_ranks(ms, dist=None, device="cuda"):
    """The job's time: the largest of the ranks' timed milliseconds (every
    rank receives it).  Single process: ms itself."""
    if dist is None:
        return ms
    import torch

    t = torch.tensor([ms], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_value(world, units_per_rank_step, ms_step):
    """Whole-job throughput: every replica processes units_per_rank_step units
    per step, and the job's step takes the slowest rank's ms_step."""
    return world * units_per_rank_step / (ms_step * 1e-3)


class Clocks:
    """nvidia-smi sampling during the timed region."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.path = os.path.join("/tmp", f"hal_bench_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                 "-i", str(self.device), "-lms", "100"], stdout=self.fh, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, smax, reasons = [], [], set()
        names = ["active", "hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
                 "sw_power_cap"]
        with open(self.path) as fh:
            for line in fh:
                parts = [p.strip() for p in line.split(",")]
                if len(parts) < 9:
                    continue
                try:
                    sm.append(float(parts[1]))
                    smax.append(float(parts[2]))
                except ValueError:
                    continue
                for name, val in zip(names[1:], parts[5:9]):
                    if val.lower().startswith("active"):
                        reasons.add(name)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax),
                "samples": len(sm), "reasons": sorted(reasons)}


def profile_traffic(kernel):
    """DRAM bytes per launch recorded by an ncu capture under profiles/
    ("traffic_bytes_per_launch <kernel> <value>" lines), or None."""
    pdir = os.path.join(ROOT, "profiles")
    if not os.path.isdir(pdir):
        return None
    for name in sorted(os.listdir(pdir)):
        if not name.endswith((".md", ".txt")):
            continue
        with open(os.path.join(pdir, name)) as fh:
            for line in fh:
                parts = line.replace("`", " ").split()
                if len(parts) >= 3 and parts[0] == "traffic_bytes_per_launch" and parts[1] == kernel:
                    try:
                        return float(parts[2])
                    except ValueError:
                        pass
    return None


def accuracy(got, ref, what):
    """max-abs and relative L2 error of an FP32 device result against the
    FP64 oracle run from the same float32 inputs."""
    d = np.asarray(got, dtype=np.float64) - np.asarray(ref, dtype=np.float64)
    den = float(np.linalg.norm(ref))
    return {"max_abs": float(np.abs(d).max()), "rel_l2": float(np.linalg.norm(d) / (den if den > 0 else 1.0)),
            "vs": what}


def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build(ref=False)
    return pyoracle.Oracle


def cpu_baseline_adi(threads, min_seconds=8.0, max_ticks=40):
    """The oracle's FP64 ADI tick on the full 2048^2 workload, timed on the
    host; returns (cell-updates/s, ticks timed)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle
    from halcuda import workloads

    pyoracle.build(ref=False)
    w = workloads.adi_inputs(N, seed=2)
    f = w["field"].copy()
    src = w["src"]
    # one untimed tick to page everything in
    f = pyoracle.Oracle.run_ticks(1, f, N, N, RATE, decay=DECAY, src_dense=src, ticks=1,
                                  threads=threads)
    ticks = 0
    t0 = time.perf_counter()
    while ticks < max_ticks:
        f = pyoracle.Oracle.run_ticks(1, f, N, N, RATE, decay=DECAY, src_dense=src, ticks=1,
                                      threads=threads)
        ticks += 1
        if time.perf_counter() - t0 >= min_seconds and ticks >= 2:
            break
    dt = time.perf_counter() - t0
    return ticks * CELLS / dt, ticks, dt


def run_reference(args):
    rank, _, world = dist_env()
    if rank != 0:
        return 0
    threads = os.cpu_count() or 1
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle
    from halcuda import workloads

    pyoracle.build(ref=False)
    w = workloads.adi_inputs(N, seed=2)
    f = w["field"].copy()
    ticks_per_sample = 4
    for _ in range(args.warmup):
        f = pyoracle.Oracle.run_ticks(1, f, N, N, RATE, decay=DECAY, src_dense=w["src"],
                                      ticks=ticks_per_sample, threads=threads)
    times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        f = pyoracle.Oracle.run_ticks(1, f, N, N, RATE, decay=DECAY, src_dense=w["src"],
                                      ticks=ticks_per_sample, threads=threads)
        times.append(time.perf_counter() - t0)
    total = sum(times)
    value = ticks_per_sample * CELLS * len(times) / total
    sample = (f"{ticks_per_sample} FP64 ADI ticks of the 2048x2048 workload per step "
              f"(oracle C restatement, {threads} threads)")
    line = {
        "impl": "reference", "metric": "cell-updates/s", "value": value, "unit": "cell-updates/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * total / len(times), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": config_block(world),
        "cpu_baseline": {"value": value, "unit": "cell-updates/s", "cores": threads, "kind": "port",
                         "sample": sample},
        "e2e": {"value": value, "unit": "cell-updates/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def config_block(world):
    return {"workload": f"adi-{N}x{N}-r{RATE:g}-decay{DECAY:g}-source-zeroflux-{TICKS}ticks",
            "grid": [N, N], "ticks_per_step": TICKS, "diffRate": RATE, "decay": DECAY,
            "boundaries": "zero-flux", "precision": "fp32 device, fp64 plan",
            "l2": "flushed between steps (512 MB write)",
            "parallelism": f"replicas x{world}"}


def secondary_explicit(hal, torch, stream, warm=5, iters=50):
    from halcuda import workloads

    w = workloads.explicit_inputs(N, seed=1)
    with hal.Diffusion(N, N) as d:
        d.set_stream(stream.cuda_stream)
        d.set_field(w["field"])
        d.set_point_sources(w["src_idx"], w["src_val"])
        d.run_ticks(warm * 10, 0.2, 0.001)
        d.sync()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ticks = 100
        times = []
        for _ in range(iters // 10 or 1):
            ev0.record(stream)
            d.run_ticks(ticks, 0.2, 0.001)
            ev1.record(stream)
            ev1.synchronize()
            times.append(ev0.elapsed_time(ev1))
        ms_tick = min(times) / ticks
        ms_launch = d.profile(iters, 0.2, 0.001)
        # accuracy: 10 ticks from the float32 start against the FP64 oracle
        f32 = w["field"].astype(np.float32)
        d.set_field(f32)
        d.run_ticks(10, 0.2, 0.001)
        got = d.get_field()
    O = _oracle()
    t0 = time.perf_counter()
    ref = O.run_ticks(0, f32.astype(np.float64), N, N, 0.2, decay=0.001, src_idx=w["src_idx"], src_val=w["src_val"],
                      ticks=10)
    cpu_s = time.perf_counter() - t0
    peak, _ = peaks()
    # several ticks per launch, the field in registers between them: the FP32
    # pipe bounds a tick (11 operations per cell: 4 differences, 3 additions of
    # them, the rate, the decay, the source, the commit), not the passes over
    # memory that one launch per tick made
    sm_hz = 2.07e9
    ops, fp32 = 11 * CELLS / (ms_tick * 1e-3) / 1e9, 152 * 128 * sm_hz / 1e9
    equivalent = EXPLICIT_BYTES * CELLS / (ms_tick * 1e-3) / 1e9
    return {"workload": "explicit-2048x2048-r0.2-decay0.001-64sources-zeroflux",
            "value": CELLS / (ms_tick * 1e-3), "unit": "cell-updates/s",
            "ms_per_tick_graph": ms_tick,
            "roofline": {"kernel": "TickPatch", "bound": "fp32", "achieved": ops, "peak": fp32,
                         "unit": "Gop/s", "frac": ops / fp32,
                         "one_pass_per_tick_gbs": equivalent, "measured_copy_gbs": peak,
                         "launch_ms_basis": "graph replay of 100 ticks, four ticks per launch",
                         "single_tick_launch_ms": ms_launch},
            "accuracy": accuracy(got, ref, "FP64 oracle, 10 ticks from the same float32 field"),
            "cpu_baseline": {"value": 10 * CELLS / cpu_s, "unit": "cell-updates/s", "cores": 1, "kind": "port",
                             "sample": "10 FP64 ticks of the same 2048x2048 workload (oracle, 1 thread)"},
            "note": "100-tick graph replays; 33.5 MB ping-pong set is L2-resident"}


def secondary_agents(hal, stream, iters=20):
    from halcuda import workloads

    import torch

    w = workloads.agent_inputs(1_000_000, N, seed=3)
    n = w["radii"].size
    with hal.Agents(N, N, n) as ag:
        ag.set_stream(stream.cuda_stream)
        ag.upload(w["positions"], w["radii"])
        ag.profile(3, 1.0, 0.1)
        ms = ag.profile(iters, 1.0, 0.1)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        # back-to-back dispatches: the stage kernels chained by programmatic
        # launches, as a caller runs them (the stage times above put an event
        # between stages, which breaks the chain)
        ag.dispatch(1.0, 0.1)
        e0.record(stream)
        for _ in range(iters):
            ag.dispatch(1.0, 0.1)
        e1.record(stream)
        e1.synchronize()
        ms_chained = e0.elapsed_time(e1) / iters
        # resident SphericalAgent2D ticks: forces + vel/cap/move/friction,
        # positions never leave the device
        ag.step(3, 1.0, 0.1, friction=0.5, maxVel=0.5)
        e0.record(stream)
        ag.step(iters, 1.0, 0.1, friction=0.5, maxVel=0.5)
        e1.record(stream)
        e1.synchronize()
        ms_step = e0.elapsed_time(e1) / iters
        # accuracy: FP32 forces of the starting positions against FP64
        ag.upload(w["positions"], w["radii"])
        ag.dispatch(1.0, 0.1)
        got = ag.download()
    O = _oracle()
    pos64 = np.asarray(w["positions"], dtype=np.float32).astype(np.float64)
    rad64 = np.asarray(w["radii"], dtype=np.float32).astype(np.float64)
    t0 = time.perf_counter()
    ref, _, _ = O.accumulate_forces(pos64, rad64, 1.0, 0.1, N, N, False, False)
    cpu_s = time.perf_counter() - t0
    # algorithmic bytes of the whole dispatch: 28 B/agent + 16 B/bin
    bytes_tick = 28 * n + 16 * CELLS
    peak, _ = peaks()
    ach = bytes_tick / (ms_chained * 1e-3) / 1e9
    return {"workload": "agents-1M-in-2048x2048-R1-k0.1-walls",
            "value": n / (ms_chained * 1e-3), "unit": "agents/s",
            "ms_per_dispatch": ms_chained,
            "ms_per_dispatch_basis": "mean of back-to-back dispatches (chained stage launches)",
            "ms_by_stage": {"count": ms[0], "scan": ms[1], "scatter": ms[2], "stabilize": ms[3],
                            "forces": ms[4], "whole": ms[5],
                            "basis": "an event between stages, which breaks the launch chain"},
            "resident_step": {"ms_per_tick": ms_step, "agents_per_s": n / (ms_step * 1e-3),
                              "note": "hal_cuda_agents_step: dispatch + fused vel/CapVelocity/ForceMove/"
                                      "ApplyFriction, friction 0.5, maxVel 0.5, no host copies"},
            "roofline": {"kernel": "whole dispatch", "bound": "hbm", "achieved": ach,
                         "peak": peak, "unit": "GB/s", "frac": ach / peak,
                         "traffic": None},
            "accuracy": accuracy(got, ref, "FP64 CpuAgentForceBackend2D restatement on the same float32 positions"),
            "binning": "bit-exact (tests)",
            "cpu_baseline": {"value": n / cpu_s, "unit": "agents/s", "cores": 1, "kind": "port",
                             "sample": "one FP64 AccumulateForces of the same 1M agents (oracle, 1 thread)"}}


def secondary_coupled(hal, torch, stream, ticks=100, cpu_ticks=2):
    """1M moving agents coupled to a 2048^2 ADI field: each tick is the
    resident agent step (bins, forces, SphericalAgent2D move) followed by the
    ADI tick whose commit removes 0.001 of the field per agent in each cell,
    for 100 ticks: as one hal_cuda_adi_run_coupled call (the ticks replayed
    from one graph), and as alternating step / tick calls on one stream."""
    from halcuda import workloads

    ag_in = workloads.agent_inputs(1_000_000, N, seed=3)
    fd_in = workloads.adi_inputs(N, seed=2)
    n = ag_in["radii"].size
    f32 = fd_in["field"].astype(np.float32)
    s32 = fd_in["src"].astype(np.float32)
    args = (1.0, 0.1, False, False)
    with hal.Agents(N, N, n) as ag, hal.Adi(N, N) as a:
        a.set_stream(stream.cuda_stream)
        ag.set_stream(stream.cuda_stream)
        a.set_field(f32)
        a.set_source(s32)
        a.set_uptake(ag, 0.001)

        def run(k):
            for _ in range(k):
                ag.step(1, *args, friction=0.5, maxVel=-1.0)
                a.run_ticks(1, RATE, DECAY)

        def fused(k):
            a.run_coupled(ag, k, RATE, DECAY, False, False, 1.0, 0.1, 0.5, -1.0)

        def timed(fn):
            # the warm-up runs the timed tick count, so the timed run replays
            # the graphs it captured
            ag.upload(ag_in["positions"], ag_in["radii"])
            a.set_field(f32)
            fn(ticks)
            a.sync()
            ag.upload(ag_in["positions"], ag_in["radii"])
            a.set_field(f32)
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            fn(ticks)
            e1.record(stream)
            e1.synchronize()
            return e0.elapsed_time(e1) / ticks

        ms_calls = timed(run)
        ms_tick = timed(fused)
        ag.set_stream(None)
        a.set_stream(None)
    # the same coupled tick on the CPU: FP64 forces, the FP64 agent update and
    # the FP64 ADI tick with the per-cell counts (oracle, 1 thread)
    O = _oracle()
    p = ag_in["positions"].astype(np.float64)
    rad = ag_in["radii"].astype(np.float64)
    v = np.zeros_like(p)
    f = f32.astype(np.float64)
    s = s32.astype(np.float64)
    t0 = time.perf_counter()
    for _ in range(cpu_ticks):
        dv, off, _ = O.accumulate_forces(p, rad, 1.0, 0.1, N, N, False, False)
        p, v = O.agents_move(p, v, dv, N, N, False, False, 0.5, -1.0)
        f = O.run_ticks(1, f, N, N, RATE, decay=DECAY, src_dense=s, uptake_count=np.diff(off).astype(np.int32),
                        uptake=0.001, ticks=1)
    cpu_s = (time.perf_counter() - t0) / cpu_ticks
    # algorithmic bytes of one coupled tick: ADI 24 B/cell plus the y-sweep's
    # read of the cell offsets (4 B/cell); the agent step's binning and forces
    # (28 B/agent + 16 B/bin) plus its move (read and write position and
    # velocity, 16 B/agent)
    bytes_tick = (24 + 4) * CELLS + (28 + 16) * n + 16 * CELLS
    peak, _ = peaks()
    ach = bytes_tick / (ms_tick * 1e-3) / 1e9
    return {"workload": "coupled-1M-agents-2048x2048-adi-r5-uptake0.001-100ticks",
            "value": n / (ms_tick * 1e-3), "unit": "agents/s",
            "cell_updates_per_s": CELLS / (ms_tick * 1e-3), "ms_per_coupled_tick": ms_tick,
            "ms_per_coupled_tick_basis": "hal_cuda_adi_run_coupled, 100 ticks in one call (one cached graph)",
            "ms_per_coupled_tick_alternating_calls": ms_calls,
            "roofline": {"kernel": "whole coupled tick (agent step + ADI tick)", "bound": "hbm", "achieved": ach,
                         "peak": peak, "unit": "GB/s", "frac": ach / peak, "traffic": None,
                         "bytes_per_tick": bytes_tick},
            "cpu_baseline": {"value": n / cpu_s, "unit": "agents/s", "cores": 1, "kind": "port",
                             "ms_per_coupled_tick": cpu_s * 1e3,
                             "sample": f"{cpu_ticks} FP64 coupled ticks of the same workload (oracle forces, "
                                       "agent update and ADI tick with uptake, 1 thread)"},
            "parity": "bins bit-exact every 10th tick and field rel-L2 <= 1e-5 over 100 ticks "
                      "(tests/test_coupled_gpu.py)"}


def secondary_wells(hal, torch, stream, ticks=20, plain_ticks=3):
    """512 independent wells (109M cells, 5.2M agents): one batched tick of
    every well against per-well launches of the single-grid handles."""
    from halcuda import workloads

    w = workloads.wells_inputs()
    R, k = w["interactionRad"], w["springConstant"]
    wells = w["wells"]
    cells_exp = sum(d["xDim"] * d["yDim"] for d in wells if d["kind"] == "explicit")
    cells_adi = sum(d["xDim"] * d["yDim"] for d in wells if d["kind"] == "adi")
    cells_ag = sum(d["xDim"] * d["yDim"] for d in wells if d["maxAgents"] > 0)
    n_ag = int(w["counts"].sum())
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    with hal.Wells(wells) as b:
        b.set_stream(stream.cuda_stream)
        for i, f in enumerate(w["fields"]):
            b.set_field(i, f)
        b.set_agents(w["counts"], w["positions"], w["radii"])
        b.run_ticks(4, R, k)  # warm-up; captures both parities' graphs
        b.sync()
        l0 = hal.launch_count()
        ev0.record(stream)
        b.run_ticks(ticks, R, k)
        ev1.record(stream)
        ev1.synchronize()
        launches_per_tick = (hal.launch_count() - l0) / ticks
        ms_batched = ev0.elapsed_time(ev1) / ticks
        stages = b.profile(3, R, k)

    # the same wells, one single-grid handle per well, launched one by one
    starts = np.concatenate([[0], np.cumsum(w["counts"])]).astype(np.int64)
    handles = []
    try:
        for i, d in enumerate(wells):
            h = (hal.Adi if d["kind"] == "adi" else hal.Diffusion)(d["xDim"], d["yDim"])
            h.set_stream(stream.cuda_stream)
            h.set_field(w["fields"][i])
            ag = None
            a, e = int(starts[i]), int(starts[i + 1])
            if e > a:
                ag = hal.Agents(d["xDim"], d["yDim"], e - a)
                ag.set_stream(stream.cuda_stream)
                ag.upload(w["positions"][2 * a: 2 * e], w["radii"][a:e])
            handles.append((h, ag, d))

        def plain_tick():
            for h, ag, d in handles:
                h.run_ticks(1, d["diffRate"], d["decay"])
                if ag is not None:
                    ag.dispatch(R, k)

        plain_tick()
        plain_tick()
        torch.cuda.synchronize()
        ev0.record(stream)
        for _ in range(plain_ticks):
            plain_tick()
        ev1.record(stream)
        ev1.synchronize()
        ms_plain = ev0.elapsed_time(ev1) / plain_ticks
    finally:
        for h, ag, _ in handles:
            h.close()
            if ag is not None:
                ag.close()

    # algorithmic bytes of one tick: explicit 8 B/cell, ADI 20 B/cell (x-sweep
    # 8, y-sweep 12 without a source), agents 28 B/agent + 16 B/bin
    bytes_tick = 8 * cells_exp + 20 * cells_adi + 28 * n_ag + 16 * cells_ag
    peak, _ = peaks()
    ach = bytes_tick / (ms_batched * 1e-3) / 1e9
    cells = cells_exp + cells_adi
    cpu_cells, cpu_agents, cpu_s, cpu_threads = cpu_baseline_wells()
    return {"workload": "wells-512-side64..1024-explicit+adi-agents0..20000",
            "value": cells / (ms_batched * 1e-3), "unit": "cell-updates/s",
            "cpu_baseline": {"value": cpu_cells, "unit": "cell-updates/s", "agents_per_s": cpu_agents,
                             "ms_per_tick": cpu_s * 1e3, "cores": cpu_threads, "kind": "port",
                             "sample": "one FP64 tick of all 512 wells (explicit or ADI tick with decay, and the "
                                       "agent force pass) with the wells spread over every host thread, as "
                                       "MultiWellExperiment::StepMultiThread does (oracle)"},
            "agents_per_s": n_ag / (ms_batched * 1e-3),
            "ms_per_tick_batched": ms_batched, "ms_per_tick_per_well_launches": ms_plain,
            "speedup_vs_per_well_launches": ms_plain / ms_batched,
            "kernel_launches_per_tick": launches_per_tick,
            "agent_bins": "per well, bins of 1x1 to 8x8 cells (the largest holding at most one agent on "
                          "average at the well's capacity), ordered by (cell, agent index) within a bin",
            "ms_by_stage": {"explicit": stages[0], "adi_x": stages[1], "adi_y": stages[2],
                            "agents": stages[3], "tick": stages[4]},
            "cells": cells, "agents": n_ag,
            "roofline": {"kernel": "whole batched tick", "bound": "hbm", "achieved": ach, "peak": peak,
                         "unit": "GB/s", "frac": ach / peak, "traffic": None}}


def secondary_stencil64(hal, torch, stream, iters=20):
    """The FP64 per-cell rate diffusion and upwind advection stencils
    (Internal::Diffusion2 / Advection2) on a 2048^2 grid with per-cell rates
    and velocities, called through the C ABI with pinned host arrays (copies
    inside the timed call), beside the kernel launch time and the CPU oracle
    on the same grid."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build(ref=False)
    rng = np.random.default_rng(12)

    def pinned(a):
        t = torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).pin_memory()
        return t, t.numpy()

    keep = []
    arrays = {}
    for name, a in (("f", rng.random(CELLS)), ("d", np.zeros(CELLS)), ("rx", rng.random(CELLS) * 0.24),
                    ("ry", rng.random(CELLS) * 0.24), ("vx", rng.random(CELLS) - 0.5),
                    ("vy", rng.random(CELLS) - 0.5)):
        t, v = pinned(a)
        keep.append(t)
        arrays[name] = v
    f, d, rx, ry, vx, vy = (arrays[k] for k in ("f", "d", "rx", "ry", "vx", "vy"))
    # per cell: algorithmic bytes (field read, deltas read+write, per-cell
    # arrays read) and FP64 operations (the reference's adds, subtracts and
    # multiplies; the FP64 pipe, not HBM, bounds these kernels on GB300)
    forms = {"diffuse_var": (hal.STENCIL_DIFFUSE_VAR, 40, 12, lambda h: h.diffuse_var(f, d, rx, ry, 0, 0)),
             "advect": (hal.STENCIL_ADVECT, 24, 6, lambda h: h.advect(f, d, 0.2, -0.1, 0, 0)),
             "advect_var": (hal.STENCIL_ADVECT_VAR, 40, 8, lambda h: h.advect_var(f, d, vx, vy, 0, 0))}
    cpu_fn = {"diffuse_var": lambda: pyoracle.Oracle.diffuse_var(f, d, rx, ry, N, N, 0, 0),
              "advect": lambda: pyoracle.Oracle.advect(f, d, 0.2, -0.1, N, N, 0, 0),
              "advect_var": lambda: pyoracle.Oracle.advect_var(f, d, vx, vy, N, N, 0, 0)}
    peak, _ = peaks()
    fp64_peak = hal.fp64_issue_rate() / 1e9
    out = {}
    with hal.Diffusion(N, N) as h:
        h.set_stream(stream.cuda_stream)
        for name, (kind, bpc, opc, call) in forms.items():
            d[:] = 0.0
            call(h)
            call(h)
            walls = []
            for _ in range(iters // 4 or 1):
                d[:] = 0.0
                t0 = time.perf_counter()
                call(h)
                walls.append(time.perf_counter() - t0)
            e2e_ms = statistics.median(walls) * 1e3
            ms = h.stencil64_profile(kind, iters, 0.2, -0.1, 0, 0)
            t0 = time.perf_counter()
            cpu_fn[name]()
            cpu_ms = (time.perf_counter() - t0) * 1e3
            gbs = bpc * CELLS / (ms * 1e-3) / 1e9
            gops = opc * CELLS / (ms * 1e-3) / 1e9
            out[name] = {"kernel_ms": ms, "e2e_ms": e2e_ms, "cpu_oracle_ms": cpu_ms,
                         "value": CELLS / (ms * 1e-3), "e2e_value": CELLS / (e2e_ms * 1e-3),
                         "unit": "cell-updates/s", "bytes_per_cell": bpc, "fp64_ops_per_cell": opc,
                         "roofline": {"bound": "fp64", "achieved": gops, "peak": fp64_peak,
                                      "unit": "G FP64 ops/s", "frac": gops / fp64_peak,
                                      "peak_kind": "measured live (hal_cuda_fp64_issue_rate)",
                                      "hbm": {"achieved": gbs, "peak": peak, "unit": "GB/s", "frac": gbs / peak}}}
    return {"workload": "fp64-stencils-2048x2048-zeroflux-per-cell-rates-and-velocities", "forms": out,
            "note": "FP64, bit-identical to the reference; e2e = one C-ABI call on pinned host arrays "
                    "(wall clock, copies in and out); cpu = the oracle, 1 thread"}


def secondary_pdegrid_adi(hal, torch, stream, warm=2, iters=10):
    """The FP64 DiffusionADI tick of the device-resident PDEGrid2D
    (DiffusionADI + MulAll + Update, bit-identical to the reference's
    PDEGrid2D) on a 2048^2 zero-flux grid, beside the CPU oracle's FP64 ADI
    step on the same field.  Each line's Thomas solve is one dependent FP64
    chain, and a warp's FP64 instruction takes 64 cycles on GB300, so the
    chains are bound by L x 7 FP64 instructions x 64 cycles per sweep."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle

    pyoracle.build(ref=False)
    rng = np.random.default_rng(14)
    f0 = rng.random(CELLS)
    with hal.PDEGrid(N, N) as g:
        g.set_stream(stream.cuda_stream)
        g.set_state(f0)

        def tick():
            g.diffusion_adi(5.0)
            g.apply_all(2, -0.01)  # HAL_CUDA_CELL_MUL
            g.update()

        for _ in range(warm):
            tick()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(stream):
            e0.record()
            for _ in range(iters):
                tick()
            e1.record()
        e1.synchronize()
        ms = e0.elapsed_time(e1) / iters
    t0 = time.perf_counter()
    pyoracle.Oracle.diffuse_adi(f0, np.zeros(CELLS), 5.0, N, N, False, False)
    cpu_ms = (time.perf_counter() - t0) * 1e3
    sm_hz = 2.07e9
    # per cell and sweep: 4.25 FP64 operations of the right-hand side and 10 of
    # the segments' elimination, back substitution and correction; a warp's FP64
    # instruction holds its scheduler's pipe for 64 cycles (4 x 152 of them)
    fp64_floor_ms = 2 * CELLS * 14.25 / 32 * 64 / (4 * 152 * sm_hz) * 1e3
    return {"workload": "pdegrid-fp64-adi-2048x2048-r5-zeroflux (DiffusionADI + MulAll + Update)",
            "ms_per_tick": ms, "value": CELLS / (ms * 1e-3), "unit": "cell-updates/s",
            "cpu_oracle_adi_ms": cpu_ms, "cpu_cores": 1,
            "speedup_vs_cpu_adi_step": cpu_ms / ms,
            "fp64_bound": {"bound": "fp64 issue (64 cycles per warp instruction and scheduler)",
                           "fp64_instructions_per_cell_and_sweep": 14.25,
                           "floor_ms_per_tick_at_2070_mhz": fp64_floor_ms, "frac_of_tick": fp64_floor_ms / ms},
            "note": "FP64, bit-identical to the reference's PDEGrid2D; the CPU figure is the oracle's "
                    "DiffusionADI step alone (1 thread)"}


def secondary_interface_calls(timeout=600):
    """Per-call times of Diffuse, DiffuseADI and AccumulateForces through the
    C++ backend classes on host std::vector<double> data (upload, kernels and
    readback in every call), beside the single-threaded CPU oracle on the same
    call: the counterpart of the reference's examples/BackendBenchmark.cpp
    sections 1 and 4 (hal-cpp_gb300/cpp/tests/interface_bench.cpp)."""
    exe = os.path.join(ROOT, "hal-cpp_gb300", "_build", "cpp", "interface_bench")
    if not os.path.exists(exe):
        return {"unavailable": "interface_bench not built (hal-cpp_gb300/cpp/build_cpp.py)"}
    res = subprocess.run([exe], capture_output=True, text=True, timeout=timeout)
    if res.returncode != 0:
        return {"unavailable": f"interface_bench exited {res.returncode}: {res.stderr[-300:]}"}
    rows = [json.loads(line) for line in res.stdout.splitlines() if line.startswith("{")]
    return {"calls": rows, "cpu": "oracle (the reference CPU backends restated), 1 thread",
            "note": "one call per interface invocation; GPU times include the host-device copies"}


def cpu_baseline_wells(threads=None, ticks=1):
    """MultiWellExperiment::StepMultiThread (include/Hal/Tools/
    MultiWellExperiment.h:95-103) on the host: each of the 512 wells' FP64
    tick (explicit or ADI, with decay) and agent force pass, the wells spread
    over all host threads (Hal::MultiThread, include/Hal/Concurrency/
    MultiThread.h:83-91); returns (cell-updates/s, agents/s, s per tick)."""
    import concurrent.futures as cf

    from halcuda import workloads

    O = _oracle()
    threads = threads or os.cpu_count() or 1
    w = workloads.wells_inputs()
    starts = np.concatenate([[0], np.cumsum(w["counts"])]).astype(np.int64)
    fields = [f.astype(np.float64) for f in w["fields"]]
    pos64 = w["positions"].astype(np.float64)
    rad64 = w["radii"].astype(np.float64)

    def step(i):
        d = w["wells"][i]
        fields[i] = O.run_ticks(1 if d["kind"] == "adi" else 0, fields[i], d["xDim"], d["yDim"], d["diffRate"],
                                decay=d["decay"], ticks=1)
        a, e = int(starts[i]), int(starts[i + 1])
        if e > a:
            O.accumulate_forces(pos64[2 * a: 2 * e], rad64[a:e], w["interactionRad"], w["springConstant"],
                                d["xDim"], d["yDim"], False, False)

    order = sorted(range(len(w["wells"])), key=lambda i: -w["wells"][i]["xDim"] * w["wells"][i]["yDim"])
    with cf.ThreadPoolExecutor(max_workers=threads) as ex:
        list(ex.map(step, order))  # warm-up tick
        t0 = time.perf_counter()
        for _ in range(ticks):
            list(ex.map(step, order))
        dt = (time.perf_counter() - t0) / ticks
    cells = sum(d["xDim"] * d["yDim"] for d in w["wells"])
    return cells / dt, int(w["counts"].sum()) / dt, dt, threads


def cpu_baseline_adjoint(steps=20, n=512):
    """The FP64 CPU forward and reverse-mode gradient of the variable-rate ADI
    model (the oracle's restatement) on the workload's 512^2 grid, over a
    bounded number of steps; returns (ms per forward step, ms per gradient
    step, their ratio)."""
    from halcuda import workloads

    O = _oracle()
    w = workloads.adjoint_inputs(n)
    f0 = w["f0"].astype(np.float64)
    D = w["D"].astype(np.float64)
    src = w["src"].astype(np.float64)
    t0 = time.perf_counter()
    f = f0
    for _ in range(steps):
        f, _ = O.dadi_step(f, D, n, n, decay=w["decay"], src=src)
    t_fwd = time.perf_counter() - t0
    t0 = time.perf_counter()
    O.dadi_loss_grad(f0, np.zeros_like(f0), D, w["decay"], src, n, n, steps)
    t_grad = time.perf_counter() - t0
    return 1e3 * t_fwd / steps, 1e3 * t_grad / steps, t_grad / t_fwd


def secondary_adjoint(hal, directions=None):
    """Parameter recovery on 512^2: the gradient of the field misfit after 500
    variable-rate ADI steps (checkpoints every 22) with respect to D(x), decay
    and source; its device time against one forward pass, and central finite
    differences (h = 1e-3) of the device loss on random directions."""
    from halcuda import workloads

    w = workloads.adjoint_inputs()
    n, steps = w["xDim"], w["steps"]
    dirs = w["fd_directions"] if directions is None else directions
    h = w["fd_h"]
    rng = np.random.default_rng(6)
    with hal.Adjoint(n, n) as a:
        a.set_problem(w["f0"], np.zeros_like(w["f0"]), steps, w["checkpoint_every"])
        _, target = a.forward(w["D_true"], w["decay"], w["src"], want_field=True)
        a.set_problem(w["f0"], target, steps, w["checkpoint_every"])
        fwd, grad = [], []
        for _ in range(3):
            a.forward(w["D"], w["decay"], w["src"])
            loss, gD, gK, gS = a.gradient(w["D"], w["decay"], w["src"])
            t = a.times()
            fwd.append(t[0])
            grad.append(t[1])
        ms_fwd, ms_grad = min(fwd), min(grad)
        # the same gradient with every state kept (no recomputation)
        a.set_problem(w["f0"], target, steps, 0)
        keep = []
        for _ in range(3):
            _, gD0, _, _ = a.gradient(w["D"], w["decay"], w["src"])
            keep.append(a.times()[1])
        ms_keep = min(keep)
        keep_equal = bool(np.array_equal(gD0, gD))
        a.set_problem(w["f0"], target, steps, w["checkpoint_every"])
        _, fT = a.forward(w["D"], w["decay"], w["src"], want_field=True)
        # the FP32 forward's error against the FP64 model bounds the rounding
        # noise of the FP64-reduced loss, and so of each central difference
        _, fT64, *_ = _oracle().dadi_loss_grad(w["f0"], target, w["D"], w["decay"], w["src"], n, n, steps,
                                               grad=False)
        eps_f = float(np.linalg.norm(fT.astype(np.float64) - fT64))
        noise = 4.0 * (np.sqrt(2.0 * loss) * eps_f + 0.5 * eps_f * eps_f) / h
        g64 = gD.astype(np.float64)
        errs, ok = [], 0
        for _ in range(dirs):
            v = rng.standard_normal(n * n).astype(np.float32)
            f = lambda t: a.forward(w["D"] + np.float32(t) * v, w["decay"], w["src"])
            f1 = (f(h) - f(-h)) / (2 * h)
            dd = float(g64 @ v.astype(np.float64))
            errs.append(abs(f1 - dd) / max(abs(dd), 1e-30))
            ok += abs(f1 - dd) <= 2e-2 * abs(dd) + noise
    cpu_fwd, cpu_grad, cpu_ratio = cpu_baseline_adjoint()
    return {"workload": "adjoint-512x512-500steps-ckpt22-D0.5..5-decay0.005",
            "value": ms_grad / ms_fwd, "unit": "t(gradient)/t(forward)", "higher_is_better": False,
            "cpu_baseline": {"ms_per_forward_step": cpu_fwd, "ms_per_gradient_step": cpu_grad,
                             "ratio": cpu_ratio, "cores": 1, "kind": "port",
                             "gpu_ms_per_forward_step": ms_fwd / steps, "gpu_ms_per_gradient_step": ms_grad / steps,
                             "sample": "20 FP64 steps of the same 512x512 model: the forward, then the loss and "
                                       "its reverse-mode gradient with every state kept (oracle, 1 thread)"},
            "ms_forward": ms_fwd, "ms_gradient": ms_grad, "loss": loss,
            "keep_all_states": {"ms_gradient": ms_keep, "ratio": ms_keep / ms_fwd,
                                "gradient_bit_identical": keep_equal,
                                "note": "checkpoint interval 0: every state kept (1.5 GB), nothing recomputed"},
            "fd": {"directions": dirs, "h": h, "median_rel_err": float(np.median(errs)),
                   "max_rel_err": float(np.max(errs)),
                   "within_2pct_plus_noise_bound": int(ok), "noise_bound": noise,
                   "forward_err_vs_fp64": eps_f / float(np.linalg.norm(fT64))},
            "note": "loss reduced in FP64 from the FP32 final field; the FD noise bound is 4 (|r| e + e^2/2) / h "
                    "with e the measured |f_T - f_T(FP64)|"}


def profile_case(case, n, iters):
    """Small, fixed launches of one hot kernel for an ncu capture: the case's
    inputs at grid side n, one untimed warm-up launch sequence, then `iters`
    individually launched iterations (no CUDA graph), so that
    `ncu -k <kernel> -c <k>` sees plain launches with few launches before them.

        adi N K        K ADI ticks (x-sweep + y-sweep) of the N^2 workload
        explicit N K   K fused explicit ticks
        agents N K     K dispatches of the agent workload scaled to N^2 cells
        stencil64 N K  K x (FP64 per-cell rate diffusion, advection, per-cell advection)
        wells 0 K      K batched ticks of the 512 wells
        adjoint N K    one gradient of K steps, checkpoints every 10
        coupled N K    K coupled ticks (agent step + ADI tick with uptake)
        pdegrid_adi N K  K FP64 PDEGrid2D ticks (DiffusionADI + MulAll + Update)
    """
    import halcuda as hal
    from halcuda import workloads

    if case == "adi":
        w = workloads.adi_inputs(n, seed=2, blobs=20)
        with hal.Adi(n, n) as a:
            a.set_field(w["field"])
            a.set_source(w["src"])
            a.profile(1, RATE, DECAY)
            ms = a.profile(iters, RATE, DECAY)
        print(f"adi {n}^2: x-sweep {ms[0]*1e3:.1f} us, y-sweep {ms[1]*1e3:.1f} us")
    elif case == "explicit":
        w = workloads.explicit_inputs(n, seed=1)
        with hal.Diffusion(n, n) as d:
            d.set_field(w["field"])
            d.set_point_sources(w["src_idx"], w["src_val"])
            d.profile(1, 0.2, 0.001)
            ms = d.profile(iters, 0.2, 0.001)
        print(f"explicit {n}^2: tick {ms*1e3:.1f} us")
    elif case == "agents":
        agents = max(1, int(1_000_000 * (n / 2048) ** 2))
        w = workloads.agent_inputs(agents, n, seed=3)
        import torch

        with hal.Agents(n, n, agents) as ag:
            ag.upload(w["positions"], w["radii"])
            ag.profile(1, 1.0, 0.1)
            ms = ag.profile(iters, 1.0, 0.1)
            # back-to-back dispatches (chained launches, no events between stages)
            st = torch.cuda.ExternalStream(ag.stream())
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            ag.dispatch(1.0, 0.1)
            e0.record(st)
            for _ in range(iters):
                ag.dispatch(1.0, 0.1)
            e1.record(st)
            e1.synchronize()
            chained = e0.elapsed_time(e1) / iters
            ag.step(2, 1.0, 0.1, friction=0.5, maxVel=0.5)
            e0.record(st)
            ag.step(iters, 1.0, 0.1, friction=0.5, maxVel=0.5)
            e1.record(st)
            e1.synchronize()
            stepped = e0.elapsed_time(e1) / iters
        print(f"agents {agents} in {n}^2: " + ", ".join(f"{v*1e3:.1f}" for v in ms) + " us "
              "(count, scan, scatter, stabilize, forces, whole; events between stages); "
              f"chained dispatch {chained*1e3:.1f} us, resident step {stepped*1e3:.1f} us")
    elif case == "stencil64":
        rng = np.random.default_rng(12)
        cells = n * n
        f, d = rng.random(cells), np.zeros(cells)
        rx, ry = rng.random(cells) * 0.24, rng.random(cells) * 0.24
        vx, vy = rng.random(cells) - 0.5, rng.random(cells) - 0.5
        with hal.Diffusion(n, n) as h:
            for _ in range(iters):
                h.diffuse_var(f, d.copy(), rx, ry, 0, 0)
                h.advect(f, d.copy(), 0.2, -0.1, 0, 0)
                h.advect_var(f, d.copy(), vx, vy, 0, 0)
        print(f"stencil64 {n}^2: {iters} x (diffuse_var, advect, advect_var)")
    elif case == "wells":
        w = workloads.wells_inputs()
        with hal.Wells(w["wells"]) as b:
            for i, f in enumerate(w["fields"]):
                b.set_field(i, f)
            b.set_agents(w["counts"], w["positions"], w["radii"])
            b.run_ticks(1, w["interactionRad"], w["springConstant"])  # autotune + graph capture
            b.sync()
            ms = b.profile(iters, w["interactionRad"], w["springConstant"])
            # the graph-replayed tick, whose three branches run concurrently
            import torch

            st = torch.cuda.ExternalStream(b.stream())
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            b.run_ticks(2, w["interactionRad"], w["springConstant"])
            e0.record(st)
            b.run_ticks(iters, w["interactionRad"], w["springConstant"])
            e1.record(st)
            e1.synchronize()
            replay = e0.elapsed_time(e1) / iters
        print("wells: " + ", ".join(f"{v:.3f}" for v in ms) + " ms (explicit, adi x, adi y, agents, tick; "
              f"stages in order); graph-replayed tick {replay:.3f} ms")
    elif case == "adjoint":
        rng = np.random.default_rng(4)
        f0 = workloads.gaussian_blobs(n, rng, 8).astype(np.float32)
        D = workloads.rate_field(n, rng).astype(np.float32)
        src = (rng.random(n * n) * 0.01).astype(np.float32)
        with hal.Adjoint(n, n) as a:
            a.set_problem(f0, np.roll(f0, 3), iters, 10)
            a.forward(D, 0.005, src)
            a.gradient(D, 0.005, src)
            t = a.times()
        print(f"adjoint {n}^2, {iters} steps: forward {t[0]:.2f} ms, gradient {t[1]:.2f} ms")
    elif case == "coupled":
        agents = max(1, int(1_000_000 * (n / 2048) ** 2))
        ag_in = workloads.agent_inputs(agents, n, seed=3)
        fd_in = workloads.adi_inputs(n, seed=2, blobs=20)
        with hal.Agents(n, n, agents) as ag, hal.Adi(n, n) as a:
            ag.set_stream(a.stream())
            ag.upload(ag_in["positions"], ag_in["radii"])
            a.set_field(fd_in["field"])
            a.set_source(fd_in["src"])
            a.set_uptake(ag, 0.001)
            for _ in range(iters + 1):
                ag.step(1, 1.0, 0.1, friction=0.5, maxVel=-1.0)
                a.run_ticks(1, RATE, DECAY)
            a.sync()
            ag.set_stream(None)
        print(f"coupled {agents} agents in {n}^2: {iters + 1} ticks")
    elif case == "pdegrid_adi":
        rng = np.random.default_rng(14)
        with hal.PDEGrid(n, n) as g:
            g.set_state(rng.random(n * n))
            for _ in range(iters + 1):
                g.diffusion_adi(5.0)
                g.apply_all(2, -0.01)  # HAL_CUDA_CELL_MUL
                g.update()
            g.get_state()
        print(f"pdegrid FP64 ADI {n}^2: {iters + 1} ticks")
    else:
        raise SystemExit(f"unknown profile case {case}")
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=40)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-secondary", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--profile-case", default=None,
                    help="run one small fixed case for an ncu capture instead of the benchmark "
                         "(adi, explicit, agents, stencil64, wells, adjoint, coupled, pdegrid_adi)")
    ap.add_argument("--profile-size", type=int, default=2048, help="grid side of the profile case")
    ap.add_argument("--profile-iters", type=int, default=3, help="launch iterations of the profile case")
    args = ap.parse_args()
    if args.profile_case is not None:
        return profile_case(args.profile_case, args.profile_size, args.profile_iters)
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        return run_reference(args)

    import torch

    import halcuda as hal
    from halcuda import workloads

    rank, local, world = dist_env()
    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    torch.cuda.set_device(local)
    if hal.lib().hal_cuda_set_device(local) != 0:
        raise RuntimeError(hal.last_error())

    w = workloads.adi_inputs(N, seed=2)
    field = torch.from_numpy(w["field"].astype(np.float32)).pin_memory()
    src = torch.from_numpy(w["src"].astype(np.float32)).pin_memory()
    field_np = field.numpy()
    src_np = src.numpy()
    stream = torch.cuda.Stream()
    flush = torch.empty(FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")

    adi = hal.Adi(N, N)
    adi.set_stream(stream.cuda_stream)
    adi.set_field(field_np)
    adi.set_source(src_np)

    def one_step():
        adi.run_ticks(TICKS, RATE, DECAY)

    # warm-up (also captures the graph)
    for _ in range(args.warmup):
        one_step()
    adi.sync()

    ev_s = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ev_e = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    clocks = Clocks(local)
    if dist is not None:
        dist.barrier()
    torch.cuda.synchronize()
    launches0 = hal.launch_count()
    clocks.start()
    for k in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
        ev_s[k].record(stream)
        one_step()
        ev_e[k].record(stream)
    torch.cuda.synchronize()
    clk = clocks.stop()
    launches = hal.launch_count() - launches0
    if dist is not None:
        dist.barrier()
    total_ms = max_over_ranks(sum(s.elapsed_time(e) for s, e in zip(ev_s, ev_e)), dist)
    ms_step = total_ms / args.steps
    value = job_value(world, CELLS * TICKS, ms_step)

    # per-kernel launch times: the mean of 200 back-to-back launches of each
    # sweep replayed from a graph (the steady state of the timed region),
    # and, for reference, single launches between CUDA events
    adi.profile_graph(20, RATE, DECAY)
    ms_col, ms_row = adi.profile_graph(TICKS, RATE, DECAY)
    adi.profile(5, RATE, DECAY)
    ms_col1, ms_row1 = adi.profile(50, RATE, DECAY)
    col_gbs = ADI_COL_BYTES * CELLS / (ms_col * 1e-3) / 1e9
    row_gbs = ADI_ROW_BYTES * CELLS / (ms_row * 1e-3) / 1e9
    if ms_row >= ms_col:
        dom, dom_gbs, dom_bytes = "AdiSweep<kSweepTick>", row_gbs, ADI_ROW_BYTES
    else:
        dom, dom_gbs, dom_bytes = "AdiSweep<kSweepW>", col_gbs, ADI_COL_BYTES
    peak, peak_kind = peaks()
    tick_gbs = (ADI_COL_BYTES + ADI_ROW_BYTES) * CELLS * TICKS / (ms_step * 1e-3) / 1e9

    # end to end through the host-buffer C-ABI call: every step copies the
    # field and the source in from pinned host memory and the field back out;
    # the call updates the host field in place, so each step continues from
    # the last one's result (no host-side copy inside the timed region)
    e2e_host = field.clone().pin_memory()
    e2e_np = e2e_host.numpy()
    for _ in range(2):
        adi.run_ticks_host(e2e_np, src_np, TICKS, RATE, DECAY)
    e2e_ms = []
    for _ in range(max(3, min(args.steps, 10))):
        with torch.cuda.stream(stream):
            flush.zero_()
        torch.cuda.synchronize()
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        adi.run_ticks_host(e2e_np, src_np, TICKS, RATE, DECAY)
        t1.record(stream)
        t1.synchronize()
        e2e_ms.append(t0.elapsed_time(t1))
    e2e_step = max_over_ranks(statistics.median(e2e_ms), dist)
    e2e_value = job_value(world, CELLS * TICKS, e2e_step)

    acc = None
    if rank == 0:
        # 10 ticks from the same float32 field and source against the FP64
        # oracle (the reference CPU backend's arithmetic)
        adi.set_field(field_np)
        adi.run_ticks(10, RATE, DECAY)
        got = adi.get_field()
        ref = _oracle().run_ticks(1, field_np.astype(np.float64), N, N, RATE, decay=DECAY,
                                  src_dense=src_np.astype(np.float64), ticks=10, threads=os.cpu_count() or 1)
        acc = accuracy(got, ref, "FP64 oracle, 10 ticks from the same float32 field and source")

    secondary = None
    if not args.no_secondary and rank == 0:
        secondary = {"explicit": secondary_explicit(hal, torch, stream),
                     "agents": secondary_agents(hal, stream),
                     "coupled": secondary_coupled(hal, torch, stream),
                     "wells": secondary_wells(hal, torch, stream),
                     "adjoint": secondary_adjoint(hal),
                     "stencil64": secondary_stencil64(hal, torch, stream),
                     "pdegrid_adi": secondary_pdegrid_adi(hal, torch, stream),
                     "interface_calls": secondary_interface_calls()}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        v, ticks, dt = cpu_baseline_adi(threads=1)
        cpu = {"value": v, "unit": "cell-updates/s", "cores": 1, "kind": "port",
               "sample": f"{ticks} FP64 ticks of the same 2048x2048 ADI workload "
                         f"({dt:.1f} s, 1 thread, as the reference CPU backend ships)"}

    adi.close()
    if rank == 0:
        line = {
            "metric": "cell-updates/s", "value": value, "unit": "cell-updates/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic: 200 seeded Gaussian blobs, U[0,0.01) source (numpy PCG64)",
            "config": config_block(world),
            "roofline": {"kernel": dom, "bound": "hbm", "achieved": dom_gbs, "peak": peak,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": dom_gbs / peak,
                         "traffic": profile_traffic(dom),
                         "bytes_per_launch": dom_bytes * CELLS,
                         "launch_ms": {"x-sweep AdiSweep<kSweepW>": ms_col,
                                       "y-sweep AdiSweep<kSweepTick>": ms_row},
                         "launch_ms_basis": "mean of 200 back-to-back launches replayed from a CUDA graph",
                         "isolated_launch_ms": {"x-sweep AdiSweep<kSweepW>": ms_col1,
                                                "y-sweep AdiSweep<kSweepTick>": ms_row1},
                         "achieved_by_kernel": {"x-sweep AdiSweep<kSweepW>": col_gbs,
                                                "y-sweep AdiSweep<kSweepTick>": row_gbs},
                         "tick_achieved": tick_gbs,
                         "tick_frac": tick_gbs / peak,
                         "note": "working set (3 x 16.8 MB + scratch) stays in the 126 MB L2 "
                                 "across the ticks of a step"},
            "cpu_baseline": cpu,
            "accuracy": acc,
            "e2e": {"value": e2e_value, "unit": "cell-updates/s",
                    "h2d_bytes_per_step": 2 * CELLS * 4, "d2h_bytes_per_step": CELLS * 4,
                    "ms_per_step": e2e_step,
                    "call": "hal_cuda_adi_run_ticks_host (pinned host field + source in, field out)"},
            "gpu_launches": int(launches),
            "clocks": clk,
            "secondary": secondary,
        }
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
