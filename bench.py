#!/usr/bin/env python
"""Throughput benchmark of the GB300 force-evaluation path (atom-steps/s).

Default workload (one GB300): EAM aluminium, FCC 40^3 cells = 256,000 atoms,
a = 4.05 A, Gaussian displacements 0.05 A (seed 2), Maxwell-Boltzmann
300 K (seed 3), 5000-knot tabulated EAM (tests/golden/tables/eam.aluminum5000,
the reference eam.aluminum resampled), Verlet skin 0.3 A with a
displacement-triggered rebuild, velocity Verlet dt = 2 fs.  One "step" is one
RunKernel iteration: kick-drift, (rebuild when triggered), EAM density and
force, kick, energy ledger.

Timing: W untimed warm-up steps, then K steps each bracketed by CUDA events
on the library's stream, with an L2 flush (a 512 MB write, read back) enqueued before
every step outside the events.  `value` = atoms * K / sum(step times).  `e2e`
repeats the K steps through the public C ABI (omdg_step_io) with pinned host
buffers: every step uploads positions and velocities, steps, and reads
positions, velocities, forces and the energy ledger back.

The default run also times, as sub-objects of its one JSON line, Tersoff Si
diamond 40^3 = 512,000 atoms at 1000 K and the neural surrogate on the same
cell (with its force RMSE against Tersoff), each with its HBM and
instruction-issue roofs (the MLP: its tensor-pipe fraction) and a one-core
CPU baseline (--no-sub leaves them out).

--impl reference times the oracle's CPU restatement of the same path
(oracle/omd_oracle.c, compiled on this host, pinned to the reference's own
outputs) on the same box as the GPU arm, in as many OpenMP threads as the
host has, with both of the reference's rebuild policies: the list rebuilt
every step (its default) and every 10 steps (comm.refresh 10).
"""
from __future__ import annotations

import argparse
import json
import math
import multiprocessing as mp
import os
import statistics
import subprocess
import tempfile
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

TABLE = os.path.join(ROOT, "tests", "golden", "tables", "eam.aluminum5000")
METRIC = "atom-steps/s on 1 GB300, EAM/Tersoff vs NN surrogate at <=30 meV/A force RMSE"
UNIT = "atom-steps/s"

SI_DIR = os.path.join(ROOT, "tests", "golden", "tables")

WORKLOADS = {
    # name: kind, description, lattice cells, lattice constant, Gaussian sigma, temperature, dt, seeds
    "eam_al_256k": dict(kind="eam", desc="EAM Al FCC 40^3 = 256,000 atoms, 5000-knot table, skin 0.3, dt 2 fs",
                        ncell=40, a=4.05, sigma=0.05, temp=300.0, dt=0.002, seeds=(2, 3)),
    "eam_al_1m": dict(kind="eam", desc="EAM Al FCC 64^3 = 1,048,576 atoms, 5000-knot table, skin 0.3, dt 2 fs",
                      ncell=64, a=4.05, sigma=0.05, temp=300.0, dt=0.002, seeds=(2, 3)),
    "eam_al_32k": dict(kind="eam", desc="EAM Al FCC 20^3 = 32,000 atoms, 5000-knot table, skin 0.3, dt 2 fs",
                       ncell=20, a=4.05, sigma=0.05, temp=300.0, dt=0.002, seeds=(2, 3)),
    "tersoff_si_512k": dict(kind="tersoff", desc="Tersoff Si diamond 40^3 = 512,000 atoms, R 2.7 D 0.15, skin 0.3, "
                            "1000 K, dt 1 fs", ncell=40, a=5.431, sigma=0.03, temp=1000.0, dt=0.001, seeds=(4, 5)),
    "sw_si_512k": dict(kind="sw", desc="Stillinger-Weber Si diamond 40^3 = 512,000 atoms, rc 3.771, skin 0.3, "
                       "1000 K, dt 1 fs", ncell=40, a=5.431, sigma=0.03, temp=1000.0, dt=0.001, seeds=(4, 5)),
    "nn_si_512k": dict(kind="nn", desc="neural Tersoff surrogate (32 descriptors, 32-64-64-1 BF16 tensor-core "
                       "network, Tersoff fallback) on Si diamond 40^3 = 512,000 atoms, 1000 K, skin 0.3, dt 1 fs",
                       ncell=40, a=5.431, sigma=0.03, temp=1000.0, dt=0.001, seeds=(4, 5)),
    "impact_256": dict(kind="impact", desc="impact ensemble: 256 Si diamond slabs of 1,000-16,000 atoms (log-uniform, "
                       "1.30M atoms), periodic x/y, free surface, 300 K, one Ar at 10-500 eV each; Tersoff + the reference's "
                       "Ar-Si ZBL table (zero past 3.2 A), skin 0.3 A (per-replica rebuilds), dt 0.5 fs; all replicas "
                       "in one context", ncell=0, a=5.431, sigma=0.03, temp=300.0, dt=0.0005, seeds=(6, 6), skin=0.3),
    "lj_ar_4000": dict(kind="lj", desc="LJ Ar FCC 10^3 = 4000 atoms, FP64, rc 2.5 sigma, skin 0.3, 100 K, dt 1 fs",
                       ncell=10, a=5.26, sigma=0.0, temp=100.0, dt=0.001, seeds=(1, 1)),
}

# Algorithmic bytes per atom for one launch of each kernel (neighbour list of
# N_f int32 entries, FP32 packs/forces, FP64 x and v):
#   eam_density  24 (own position) + 4 N_f (list) + 4 (F' write)
#   eam_force    24 + 4 N_f + 4 (F'_i) + 12 (f) + 4 (energy); with the step's
#                second half-kick in its epilogue (eam_force_kick) + 48 (v)
#   kick_drift   read x v f, write x v + 32 B position pack
#   kick         read v f, write v
ALG_BYTES = {
    "eam_density": lambda nf: 24 + 4 * nf + 4,
    "eam_force": lambda nf: 24 + 4 * nf + 4 + 12 + 4,
    "eam_force_kick": lambda nf: 24 + 4 * nf + 4 + 12 + 4 + 48,  # + v read and written by the fused half-kick
    "tersoff_centre": lambda nf: 24 + 4 * nf + 4,
    "nn_descriptors": lambda nf: 24 + 4 * nf + 128,
    "nn_force": lambda nf: 24 + 4 * nf + 128 + 4 + 16,
    "sw_centre": lambda nf: 24 + 4 * nf + 4,
    "pair64": lambda nf: 24 + 4 * nf + 16,
    "pair32": lambda nf: 24 + 4 * nf + 16,
    "kick_drift": lambda nf: 108 + 32,
    "kick": lambda nf: 24 + 12 + 24,
}
# one step: the force passes of the workload's potential + velocity Verlet (108 B)
STEP_ALG_BYTES = {
    "eam": lambda nf: 2 * (24 + 4 * nf) + 24 + 108,
    "tersoff": lambda nf: 24 + 4 * nf + 16 + 108,
    "sw": lambda nf: 24 + 4 * nf + 16 + 108,
    "lj": lambda nf: 24 + 4 * nf + 16 + 108,
    "nn": lambda nf: 24 + 4 * nf + 16 + 108,
    "impact": lambda nf: 24 + 4 * nf + 16 + 108,
}


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def slowest_rank_ms(total_ms, world, torch, device):
    """The timed region of the slowest rank (each rank's sum of its step
    times; replicas only, so this max is the one collective)."""
    if world <= 1:
        return total_ms
    t = torch.tensor([total_ms], dtype=torch.float64, device=device)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    torch.distributed.barrier()
    return float(t.item())


# ------------------------------------------------------------------ clocks
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        # the samples go to a temporary file (OMDG_CLOCKS_DIR to keep them elsewhere)
        out = os.environ.get("OMDG_CLOCKS_DIR") or tempfile.gettempdir()
        self.path = os.path.join(out, "clocks_bench_%d.csv" % os.getpid())

    def start(self):
        try:
            os.makedirs(os.path.dirname(self.path), exist_ok=True)
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                                          "--format=csv,noheader,nounits", "-lms", "200"], stdout=self.fh,
                                         stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            t = [x.strip() for x in line.split(",")]
            if len(t) < 9:
                continue
            try:
                sm.append(float(t[1]))
                smax.append(float(t[2]))
            except ValueError:
                continue
            for k, nm in enumerate(names):
                if t[5 + k].lower() == "active":
                    reasons.add(nm)
        try:
            os.remove(self.path)
        except OSError:
            pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax), "reasons": sorted(reasons),
                "samples": len(sm)}


# ------------------------------------------------------------------ inputs
def make_workload(name, ncell=None):
    from objectmd_gb300 import inputs

    w = dict(WORKLOADS[name])
    nc = ncell or w["ncell"]
    sp, sv = w["seeds"]
    if w["kind"] == "impact" and not ncell:
        e = inputs.impact_ensemble(seed=w["seeds"][0], temp=w["temp"], sigma=w["sigma"], a=w["a"])
        w["ensemble"] = e
        return w, e["x"], e["v"], e["lo"], e["hi"]
    if w["kind"] == "impact":  # one slab of ncell^3 cells (CPU samples), Si only
        x, lo, hi = inputs.lattice(inputs.DIAMOND_BASIS, (nc, nc, nc), w["a"], 0.125)
        x = inputs.perturb(x, w["sigma"], sp, lo, hi, (True, True, False))
        v = inputs.maxwell_boltzmann(len(x), w["temp"], inputs.md_mass("silicon"), sv)
        hi = np.array([hi[0], hi[1], hi[2] + 10.0])
        lo = np.array([0.0, 0.0, -0.5 * w["a"]])
        return w, x, v, lo, hi
    if w["kind"] == "eam":
        x, v, (lo, hi) = inputs.eam_aluminium(ncell=nc, a=w["a"], sigma=w["sigma"], temp=w["temp"], seed_pos=sp,
                                              seed_vel=sv)
    elif w["kind"] == "lj":
        x, v, (lo, hi) = inputs.lj_argon(ncell=nc, a=w["a"], temp=w["temp"], seed_vel=sv)
    else:
        x, v, (lo, hi) = inputs.diamond_silicon(ncell=nc, a=w["a"], sigma=w["sigma"], temp=w["temp"], seed_pos=sp,
                                                seed_vel=sv)
    return w, x, v, lo, hi


def make_context(w, x, v, lo, hi, device=0, tune=True):
    from objectmd_gb300 import inputs, omdg

    ctx = omdg.Context(device)
    kind = w["kind"]
    if kind == "impact":
        e = w["ensemble"]
        ctx.set_replicas(e["natoms"], e["lo"], e["hi"], (1, 1, 0))
        ctx.set_atoms(x, v, types=e["types"], masses=e["masses"], znum=e["znum"])
        ctx.add_tersoff(os.path.join(SI_DIR, "tersoff.silicon27"))
        # Ar-Si: the reference's own table (TForcePair, test/si-impact/main.cpp:71)
        ctx.add_pair_table(os.path.join(SI_DIR, "pair.ar-si.zbl"), 1, 0)
        ctx.set_neighbor(skin=w.get("skin", 1.0), rebuild_every=0)
        ctx.set_timestep(w["dt"])
        ctx.set_first_step_mode(True)
        if tune:
            ctx.autotune(3)
        return ctx
    ctx.set_box(lo, hi)
    elem, z = {"eam": ("aluminum", 13.0), "lj": ("argon", 18.0)}.get(kind, ("silicon", 14.0))
    ctx.set_atoms(x, v, masses=[inputs.md_mass(elem)], znum=[z])
    if kind == "eam":
        ctx.add_eam(TABLE)
    elif kind == "lj":
        ctx.add_pair_table(os.path.join(SI_DIR, "pair.lj.argon"), fp64=True)
    elif kind == "tersoff":
        ctx.add_tersoff(os.path.join(SI_DIR, "tersoff.silicon27"))
    elif kind == "nn":
        ctx.add_nn(NN_MODEL, os.path.join(SI_DIR, "tersoff.silicon27"))
    else:
        ctx.add_sw(os.path.join(SI_DIR, "sw.silicon"))
    ctx.set_neighbor(skin=w.get("skin", 0.3), rebuild_every=0)
    ctx.set_timestep(w["dt"])
    ctx.set_first_step_mode(True)
    if tune:
        ctx.autotune(3)
    return ctx


def mean_neighbours(ctx):
    off, j, c = ctx.neighbors()
    return float(len(j)) / max(1, len(off) - 1)


# MLP of the surrogate, per atom: z1 = G W1 (32x64), z2 = a1 W2 (64x64) and the
# two products of the force backward pass (64x64, 64x32), 2 flops per MAC
MLP_FLOP_PER_ATOM = 2 * (32 * 64 + 64 * 64 + 64 * 64 + 64 * 32)


def mlp_roof(kernels, n):
    """The surrogate network kernel against the measured sustained BF16 rate."""
    t = kernels["nn_mlp"]["ms_per_launch"]
    tf = MLP_FLOP_PER_ATOM * n / (t * 1e-3) / 1e12
    sus = load_peaks().get("bf16_sustained")
    return {"bound": "tensor", "kernel": "nn_mlp", "flop_per_atom": MLP_FLOP_PER_ATOM, "achieved": round(tf, 2),
            "peak": sus, "unit": "TFLOP/s", "frac": round(tf / sus, 4) if sus else None,
            "peak_source": "measured (MEASURED_PEAKS.json bf16_tflops_sustained)"}


def load_inst(kernel):
    """Warp instructions per atom of one launch (committed ncu figures)."""
    p = os.path.join(ROOT, "profiles", "instructions_per_atom.txt")
    try:
        for line in open(p):
            f = line.split()
            if len(f) == 2 and f[0] == kernel:
                return float(f[1])
    except OSError:
        pass
    return None


def issue_roof(kernel, n, t_ms, torch, device):
    """Instruction-issue roof: every SM sub-partition issues one warp
    instruction a cycle at the maximum SM clock (MEASURED_PEAKS.json)."""
    ipa = load_inst(kernel)
    if ipa is None or not t_ms:
        return None
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    try:
        mhz = float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["sm_max_mhz"])
    except Exception:
        mhz = 2070.0
    peak = 4 * sms * mhz * 1e6 / 1e12
    achieved = ipa * n / (t_ms * 1e-3) / 1e12
    return {"bound": "issue", "kernel": kernel, "warp_instructions_per_atom": ipa, "achieved": round(achieved, 4),
            "peak": round(peak, 4), "unit": "T warp-instructions/s", "frac": round(achieved / peak, 4),
            "source": "ncu smsp__inst_executed per atom (profiles/instructions_per_atom.txt) / CUDA-event time"}


def timed_steps(ctx, n, steps, stream, flush_l2, torch):
    """Device time of `steps` graph-replayed steps, each bracketed by events
    on the context stream with an L2 flush before it; then the per-kernel
    times of the same number of eagerly launched steps."""
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    st0 = ctx.stats()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for k in range(steps):
            flush_l2()
            starts[k].record(stream)
            ctx.step_async(1)
            ends[k].record(stream)
    ctx.sync()
    torch.cuda.synchronize()
    st1 = ctx.stats()
    total_ms = sum(s.elapsed_time(e) for s, e in zip(starts, ends))
    ctx.set_profiling(True)
    with torch.cuda.stream(stream):
        for k in range(steps):
            flush_l2()
            ctx.step_async(1)
    ctx.sync()
    kt = ctx.kernel_times()
    ctx.set_profiling(False)
    kernels = {k: {"ms_per_launch": ms / max(1, c), "launches": c} for k, (ms, c) in kt.items()}
    return total_ms, kernels, st1["rebuilds"] - st0["rebuilds"], st1["launches"] - st0["launches"]


# the solve's bytes a cell: T 8, its three face conductances 24, capacity and its reciprocal 16, S and E 8
# each, map 4, mask 1 read; A 8 written
FDTD_CELL_BYTES = 77


def fdtd_report(device, torch, n=256, steps=100):
    """The finite-difference heat solver (omdg_fdtd) on an n^3 periodic grid
    with a hot block: cells/s over `steps` host-driven steps (wall clock,
    synchronised), and the stencil's HBM roof (FDTD_CELL_BYTES per cell; the
    grid, 1.3 GB of arrays at n = 256, is ten times the L2).  The FP64 pipe
    binds it (79 % busy in ncu)."""
    from objectmd_gb300 import omdg

    dim = n ** 3
    with omdg.FDTD(n, n, n, "a pppppp", "a" * dim, device=device) as g:
        g.set_spacestep(1.0)
        g.set_timestep(0.05)
        g.set_cell("* 300 @ %d,%d,%d,%d,%d,%d=2000" % (n // 3, n // 3, n // 3, n // 2, n // 2, n // 2))
        g.step(3)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        g.step(steps)
        t1 = time.perf_counter()
        a = g.vector()
    sec = (t1 - t0) / steps
    peaks = load_peaks()
    gbs = FDTD_CELL_BYTES * dim / sec / 1e9
    return {"workload": "finite-difference heat solver %d^3 = %d cells, periodic, FP64" % (n, dim),
            "cells_per_s": dim / sec, "ms_per_step": sec * 1e3, "steps": steps,
            "timing": "wall clock over host-driven omdg_fdtd_step calls (one kernel each)",
            "roofline": {"bound": "hbm", "kernel": "fd_solve", "achieved": round(gbs, 1), "peak": peaks["hbm"],
                         "unit": "GB/s", "frac": round(gbs / peaks["hbm"], 4),
                         "alg_bytes_per_cell": FDTD_CELL_BYTES},
            "field_range": [float(a.min()), float(a.max())]}


def sub_workload(name, args, device, torch, flush_l2):
    """Another configured workload, measured as the main one (device-timed
    atom-steps/s, per-kernel times, HBM and issue roofs, one-core CPU
    baseline); for the surrogate also its force RMSE against Tersoff, plain
    Tersoff on the same cell and the MLP's tensor-pipe fraction."""
    w, x, v, lo, hi = make_workload(name)
    n = len(x)
    ctx = make_context(w, x, v, lo, hi, device=device, tune=not args.no_tune)
    stream = torch.cuda.ExternalStream(ctx.stream(), device=device)
    ctx.step(max(3, args.warmup))
    nf = mean_neighbours(ctx)
    total_ms, kernels, rebuilds, launches = timed_steps(ctx, n, args.steps, stream, flush_l2, torch)
    value = n * args.steps / (total_ms * 1e-3)
    peaks = load_peaks()
    out = {"workload": w["desc"], "value": value, "unit": UNIT, "ms_per_step": total_ms / args.steps,
           "atoms": n, "mean_neighbours": round(nf, 2), "neighbour_rebuilds_in_timed_steps": rebuilds,
           "gpu_launches": launches, "kernels": {k: round(v_["ms_per_launch"] * 1e3, 2) for k, v_ in kernels.items()},
           "kernels_unit": "us per launch"}
    cand = [(k, v_) for k, v_ in kernels.items() if k in ALG_BYTES]
    if cand:
        dom_name, dom = max(cand, key=lambda kv: kv[1]["ms_per_launch"] * kv[1]["launches"])
        alg = ALG_BYTES[dom_name](nf) * n
        ach = alg / (dom["ms_per_launch"] * 1e-3) / 1e9
        out["roofline"] = {"bound": "hbm", "kernel": dom_name, "achieved": round(ach, 1), "peak": peaks["hbm"],
                           "unit": "GB/s", "frac": round(ach / peaks["hbm"], 4), "traffic": load_traffic(dom_name, n),
                           "peak_source": peaks["src"], "alg_bytes_per_launch": int(alg)}
        out["issue_roofline"] = issue_roof(dom_name, n, dom["ms_per_launch"], torch, device)
    if "nn_mlp" in kernels:
        out["mlp_roofline"] = mlp_roof(kernels, n)
    if w["kind"] == "nn":
        out["surrogate"] = surrogate_report(ctx, w, x, v, lo, hi, device, args, torch)
    ctx.close()
    if not args.no_cpu:
        out["cpu_baseline"] = cpu_baseline(argparse.Namespace(**dict(vars(args), workload=name)))
    return out


# ------------------------------------------------------------------ GB300 arm
def run_gpu(args):
    import torch

    rank, world, local = dist_env()
    device = local if torch.cuda.device_count() > local else 0
    torch.cuda.set_device(device)
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl", init_method="env://")
    w, x, v, lo, hi = make_workload(args.workload, args.ncell)
    desc = w["desc"] if not args.ncell else "%s (ncell %d)" % (w["desc"], args.ncell)
    if args.skin is not None:
        w["skin"] = args.skin
        desc += " (skin %g A)" % args.skin
    n = len(x)
    ctx = make_context(w, x, v, lo, hi, device=device, tune=not args.no_tune)
    for kv in args.launch:
        k, val = kv.split("=")
        ctx.set_launch(k, int(val))
    if args.eager:
        ctx.set_profiling(True)
    stream = torch.cuda.ExternalStream(ctx.stream(), device=device)
    flush = torch.empty(args.flush_mb * (1 << 20) // 4, dtype=torch.float32, device="cuda")
    flush_sink = torch.empty((), dtype=torch.float32, device="cuda")

    def flush_l2():
        # write a buffer larger than L2, then read it back: the step starts
        # with none of its data in L2, and the write's dirty lines are
        # written back here rather than by the step's first kernel
        flush.zero_()
        torch.sum(flush, 0, out=flush_sink)

    # warm-up (FirstRun, graph capture, tuning effects)
    ctx.step(max(3, args.warmup))
    nf = mean_neighbours(ctx)

    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    st0 = ctx.stats()
    nrep = len(w["ensemble"]["natoms"]) if w["kind"] == "impact" and "ensemble" in w else 0
    rb0 = ctx.replica_builds(nrep) if nrep else None
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    clocks = ClockSampler(device)
    clocks.start()
    t_wall0 = time.perf_counter()
    with torch.cuda.stream(stream):
        for k in range(args.steps):
            flush_l2()
            starts[k].record(stream)
            ctx.step_async(1)
            ends[k].record(stream)
    ctx.sync()
    torch.cuda.synchronize()
    t_wall1 = time.perf_counter()
    clk = clocks.stop()
    st1 = ctx.stats()
    replica_rebuilds = None
    if nrep:
        rb = ctx.replica_builds(nrep) - rb0
        replica_rebuilds = {"replicas": nrep, "replica_builds_in_timed_steps": int(rb.sum()),
                            "mean_replicas_rebuilt_per_step": round(float(rb.sum()) / args.steps, 2),
                            "atoms_rebuilt_per_step": round(float((rb * np.asarray(w["ensemble"]["natoms"])).sum())
                                                            / args.steps, 1)}
    step_ms = [s.elapsed_time(e) for s, e in zip(starts, ends)]
    total_ms = slowest_rank_ms(sum(step_ms), world, torch, "cuda")
    value = world * n * args.steps / (total_ms * 1e-3)
    launches = st1["launches"] - st0["launches"]
    rebuilds = st1["rebuilds"] - st0["rebuilds"]
    led = ctx.ledger()

    # per-kernel CUDA-event times over the same number of steps (eager launch
    # sequence of the same kernels, L2 flushed before every step)
    ctx.set_profiling(True)
    with torch.cuda.stream(stream):
        for k in range(args.steps):
            flush_l2()
            ctx.step_async(1)
    ctx.sync()
    kt = ctx.kernel_times()
    ctx.set_profiling(args.eager)
    kernels = {k: {"ms_per_launch": ms / max(1, c), "launches": c} for k, (ms, c) in kt.items()}
    dom = max(((k, v_) for k, v_ in kernels.items() if k in ALG_BYTES),
              key=lambda kv: kv[1]["ms_per_launch"] * kv[1]["launches"])
    dom_name, dom_t = dom[0], dom[1]["ms_per_launch"]
    peaks = load_peaks()
    alg = ALG_BYTES[dom_name](nf) * n
    achieved = alg / (dom_t * 1e-3) / 1e9
    traffic = load_traffic(dom_name, n)
    roofline = {"bound": "hbm", "kernel": dom_name, "achieved": round(achieved, 1), "peak": peaks["hbm"],
                "unit": "GB/s", "frac": round(achieved / peaks["hbm"], 4), "traffic": traffic,
                "peak_source": peaks["src"], "alg_bytes_per_launch": int(alg)}
    step_alg = STEP_ALG_BYTES[w["kind"]](nf) * n
    mean_step = total_ms / args.steps

    # end to end through the C ABI with host buffers
    e2e = e2e_resident = None
    if not args.no_e2e:
        e2e = run_e2e(ctx, n, args.steps, torch)
        e2e_resident = run_e2e(ctx, n, args.steps, torch, full=False)

    cpu = None
    if rank == 0 and not args.no_cpu:
        cpu = cpu_baseline(args)

    surrogate = None
    if w["kind"] == "nn":
        surrogate = surrogate_report(ctx, w, x, v, lo, hi, device, args, torch)
    issue = issue_roof(dom_name, n, dom_t, torch, device)

    out = {
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": mean_step,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64" if w["kind"] == "lj" else "f32 forces, f64 integration",
        "data": "synthetic (seeded %s lattice, Gaussian displacements, Maxwell-Boltzmann velocities)" %
                ("diamond" if BASIS[w["kind"]] == 8 else "FCC"),
        "config": {"workload": desc, "atoms_per_gpu": n, "mean_neighbours": round(nf, 2),
                   "neighbour_rebuilds_in_timed_steps": rebuilds,
                   "replica_rebuilds": replica_rebuilds,
                   "l2": "flushed before every step (%d MB write, then read back so the write-back of its dirty "
                         "lines falls outside the step)" % args.flush_mb, "parallelism": "replicas only" if world > 1 else "single GPU",
                   "launch_shapes": ctx.launch_shapes()},
        "gpu_launches": launches,
        "clocks": clk,
        "roofline": roofline,
        "step_roofline": {"alg_bytes_per_step": int(step_alg), "achieved_GBps": round(step_alg / (mean_step * 1e-3)
                                                                                     / 1e9, 1),
                          "frac": round(step_alg / (mean_step * 1e-3) / 1e9 / peaks["hbm"], 4)},
        "kernels": {k: round(v_["ms_per_launch"] * 1e3, 2) for k, v_ in kernels.items()},
        "kernels_unit": "us per launch",
        "e2e": e2e,
        "e2e_state_resident": e2e_resident,
        "cpu_baseline": cpu,
        "energy": {"kinetic": led["kinetic"], "potential": led["potential"], "energy": led["energy"]},
        "surrogate": surrogate,
        "issue_roofline": issue,
        "wall_s_timed_loop": t_wall1 - t_wall0,
    }
    if "nn_mlp" in kernels:
        out["mlp_roofline"] = mlp_roof(kernels, n)
    # the other headline workloads, as sub-objects of the same line
    if args.workload == "eam_al_256k" and not args.ncell and not args.no_sub and world == 1:
        ctx.close()
        ctx = None
        subs = {}
        for name in ("tersoff_si_512k", "nn_si_512k", "sw_si_512k", "impact_256", "lj_ar_4000"):
            subs[name] = sub_workload(name, args, device, torch, flush_l2)
        out["workloads"] = subs
        out["fdtd"] = fdtd_report(device, torch)
        nn, ts = subs["nn_si_512k"], subs["tersoff_si_512k"]
        out["surrogate"] = {"nn_atom_steps_per_s": nn["value"], "tersoff_atom_steps_per_s": ts["value"],
                            "nn_over_tersoff": nn["value"] / ts["value"],
                            "force_rmse_eV_per_A": nn.get("surrogate", {}).get("after_md", {}).get(
                                "force_rmse_eV_per_A"),
                            "goal_eV_per_A": 0.030}
    if rank == 0:
        print(json.dumps(out), flush=True)
    if ctx is not None:
        ctx.close()
    if world > 1:
        torch.distributed.destroy_process_group()


SURROGATE_MD_STEPS = 500  # 0.5 ps of the surrogate's own MD before the "after_md" comparison


def surrogate_report(ctx, w, x0, v0, lo, hi, device, args, torch):
    """Force RMSE of the surrogate against plain Tersoff on the starting
    configuration and after SURROGATE_MD_STEPS more steps of the surrogate's
    own MD (the 1000 K start has equilibrated by then), the fallback count,
    and plain Tersoff's atom-steps/s on the same cell."""
    from objectmd_gb300 import inputs, omdg

    tersoff = os.path.join(SI_DIR, "tersoff.silicon27")

    def forces(x, use_nn):
        with omdg.Context(device) as c:
            c.set_box(lo, hi)
            c.set_atoms(x, np.zeros_like(x), masses=[inputs.md_mass("silicon")], znum=[14.0])
            if use_nn:
                c.add_nn(NN_MODEL, tersoff)
            else:
                c.add_tersoff(tersoff)
            c.set_neighbor(0.3, 0)
            c.compute_forces()
            return c.get_state()["f"], (c.nn_fallback_atoms() if use_nn else 0)

    rm = lambda a: float(np.sqrt(np.mean(a * a)))  # noqa: E731
    out = {"md_steps_before_after_md": SURROGATE_MD_STEPS}
    ctx.step(SURROGATE_MD_STEPS)
    for tag, xx in (("start", x0), ("after_md", ctx.get_state()["x"])):
        fn, nfb = forces(xx, True)
        ft, _ = forces(xx, False)
        out[tag] = {"force_rmse_eV_per_A": rm(fn - ft), "force_rms_eV_per_A": rm(ft), "fallback_atoms": nfb}
    # plain Tersoff on the same cell, graph-replayed steps
    tw = dict(WORKLOADS["tersoff_si_512k"])
    tc = make_context(tw, x0, v0, lo, hi, device=device, tune=not args.no_tune)
    tc.step(5)
    st = torch.cuda.ExternalStream(tc.stream(), device=device)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    k = max(20, min(args.steps, 200))
    with torch.cuda.stream(st):
        e0.record(st)
        tc.step_async(k)
        e1.record(st)
    tc.sync()
    torch.cuda.synchronize()
    out["tersoff_atom_steps_per_s"] = len(x0) * k / (e0.elapsed_time(e1) * 1e-3)
    tc.close()
    return out


def run_e2e(ctx, n, steps, torch, full=True):
    """Per step one omdg_step_io call from pinned host arrays, then the
    ledger.  full: H2D of x and v, one step, D2H of x, v and f (x and f while
    the step's last kernels run) -- a caller that hands its whole state over
    every step.  Otherwise the state stays on the device and only positions
    come back each step (a trajectory writer)."""
    pin = lambda: torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy()  # noqa: E731
    x, v, f = pin(), pin(), pin()
    ctx.get_state_into(x=x, v=v)
    io = dict(x_in=x, v_in=v, x_out=x, v_out=v, f_out=f) if full else dict(x_out=x)
    ctx.step_io(1, **io)  # captures the step with its downloads
    t0 = time.perf_counter()
    for k in range(steps):
        ctx.step_io(1, **io)
        ctx.ledger()
    t1 = time.perf_counter()
    return {"value": n * steps / (t1 - t0), "unit": UNIT, "h2d_bytes_per_step": (2 * 24 * n) if full else 0,
            "d2h_bytes_per_step": (3 * 24 * n if full else 24 * n) + 32,
            "transfers": ("x, v host to device and x, v, f back, every step" if full else
                          "state resident on the device; x back every step")}


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(p))
        return {"hbm": float(d["hbm_gbs"]), "src": "measured (MEASURED_PEAKS.json hbm_gbs)",
                "bf16_sustained": float(d.get("bf16_tflops_sustained", 0.0)) or None}
    except Exception:
        return {"hbm": 6800.0, "src": "fallback 6.8 TB/s", "bf16_sustained": 1700.0}


def load_traffic(kernel, n_atoms):
    """DRAM bytes per launch: the committed ncu per-atom figure x atoms."""
    p = os.path.join(ROOT, "profiles", "traffic_per_atom.txt")
    try:
        for line in open(p):
            f = line.split()
            if len(f) == 2 and f[0] == kernel:
                return int(float(f[1]) * n_atoms)
    except OSError:
        pass
    return None


# ------------------------------------------------------------------ CPU baselines
SW_PARAM = dict(eps=2.1683, A=7.049556277, B=0.6022245584, p=4, q=0, sigma=2.0951, a=1.80, lam=21.0, gamma=1.2,
                icos0=-3.0, usezbl=1, sx0=1.2107, sx1=1.8456, sa0=335.0594, sa1=-492.3905, sa2=244.5280,
                sa3=-41.2347, z1=14, z2=14)
TERSOFF_PARAM = dict(A=3264.7, B=95.373, lambda1=3.2394, lambda2=1.3258, lambda3=1.3258, beta=0.33675, n=22.956,
                     c=4.8381, d=2.0417, h=0.0, R=2.7, D=0.15)
BASIS = {"eam": 4, "lj": 4, "tersoff": 8, "sw": 8, "nn": 8, "impact": 8}
CPU_SAMPLE_NCELL = {"eam": 16, "lj": 10, "tersoff": 10, "sw": 10, "nn": 10, "impact": 9}
NN_MODEL = os.path.join(ROOT, "objectmd_gb300", "models", "nn_tersoff_si.nn")


def _cpu_worker(args_tuple):
    """The oracle's step (kick-drift, wrap, neighbour list rebuilt every
    `refresh` steps -- 1 is the reference's default comm.refresh, 10 its
    comm.refresh 10 -- forces, kick) on `threads` OpenMP threads."""
    name, ncell, steps, warm, refresh, threads = args_tuple
    os.environ["OMP_NUM_THREADS"] = str(threads)  # before the oracle library loads
    sys.path.insert(0, ROOT)
    from objectmd_gb300 import inputs
    from oracle import oracle as oc

    w, x, v, lo, hi = make_workload(name, ncell)
    kind = w["kind"]
    n = len(x)
    box = oc.make_box(lo, hi, (1, 1, 0) if kind == "impact" else (1, 1, 1))
    elem = {"eam": "aluminum", "lj": "argon"}.get(kind, "silicon")
    mass = np.full(n, inputs.md_mass(elem))
    if kind == "eam":
        phi, ed, em = (oc.Table.from_file(TABLE, sec) for sec in ("PAIR", "EDENS", "EMBED"))
        rv = phi.max_range() + 0.3
        force = lambda nb: oc.eam(box, x, nb, phi, ed, em)[0]  # noqa: E731
    elif kind == "lj":
        phi = oc.Table.from_file(os.path.join(SI_DIR, "pair.lj.argon"), "")
        rv = phi.max_range() + 0.3
        force = lambda nb: oc.pair_table(box, x, nb, phi)[0]  # noqa: E731
    elif kind in ("tersoff", "nn", "impact"):  # the surrogate's CPU baseline is the method it replaces
        tp = oc.TersoffParam(**TERSOFF_PARAM)
        rv = TERSOFF_PARAM["R"] + TERSOFF_PARAM["D"] + (1.0 if kind == "impact" else 0.3)
        force = lambda nb: oc.tersoff(box, x, nb, tp)[0]  # noqa: E731
    else:
        sp = oc.SWParam(**SW_PARAM)
        rv = SW_PARAM["sigma"] * SW_PARAM["a"] + 0.3
        force = lambda nb: oc.sw(box, x, nb, sp)[0]  # noqa: E731
    x = np.ascontiguousarray(x)
    v = np.ascontiguousarray(v)
    f = np.zeros((n, 3))
    dt = w["dt"]
    bufs = (np.zeros(n + 1, dtype=np.int32), np.zeros(n * 160, dtype=np.int32), np.zeros(n * 160, dtype=np.int32))
    state = {"nb": None, "k": 0}

    def one_step():
        oc.vv_kick_drift(x, v, f, mass, dt)
        if state["nb"] is None or state["k"] % refresh == 0:
            x[:] = oc.wrap(box, x)
            state["nb"] = oc.neighbors(box, x, rv, buffers=bufs)
        state["k"] += 1
        f[:] = force(state["nb"])
        oc.vv_kick(v, f, mass, dt)

    for _ in range(warm):
        one_step()
    t0 = time.perf_counter()
    for _ in range(steps):
        one_step()
    t1 = time.perf_counter()
    return n, steps, t1 - t0


def cpu_baseline(args):
    """Single-core oracle port on a bounded sample of the workload."""
    kind = WORKLOADS[args.workload]["kind"]
    nc = CPU_SAMPLE_NCELL[kind]
    ctx = mp.get_context("spawn")
    with ctx.Pool(1) as pool:
        n, steps, sec = pool.map(_cpu_worker, [(args.workload, nc, args.cpu_steps, 1, 1, 1)])[0]
    return {"value": n * steps / sec, "unit": UNIT, "cores": 1, "kind": "port",
            "sample": "%s, lattice %d^3 = %d atoms, %d steps (neighbour list rebuilt every step, as the reference's "
                      "default comm.refresh), oracle/omd_oracle.c on one host core" % (kind, nc, n, steps)}


def run_reference(args):
    """The reference's algorithm (the oracle port: oracle/omd_oracle.c, pinned
    to the reference's own outputs to 1e-12) on the same box as the GPU arm,
    all host threads, under both of the reference's rebuild policies: the list
    rebuilt every step (comm.refresh unset, its default) and every 10 steps
    (comm.refresh 10).  The line's value is the faster of the two."""
    rank, world, local = dist_env()
    if rank != 0:
        return
    cores = os.cpu_count() or 1
    w = WORKLOADS[args.workload]
    desc = w["desc"] if not args.ncell else "%s (ncell %d)" % (w["desc"], args.ncell)
    steps = max(10, args.steps)
    warm = max(1, min(args.warmup, 3))
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    policies = {}
    with ctx.Pool(1) as pool:
        for refresh in (1, 10):
            n, k, sec = pool.map(_cpu_worker, [(args.workload, args.ncell or None, steps, warm, refresh, cores)])[0]
            policies[refresh] = (n, k, sec)
    t1 = time.perf_counter()
    rates = {r: n * k / sec for r, (n, k, sec) in policies.items()}
    best = max(rates, key=rates.get)
    n, k, sec = policies[best]
    value = rates[best]
    out = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": k,
           "warmup": args.warmup, "ms_per_step": sec / k * 1e3, "higher_is_better": True,
           "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
           "config": {"workload": desc, "atoms_total": n, "host_threads": cores,
                      "rebuild_policy": "every %d steps (comm.refresh %d)" % (best, best) if best > 1 else
                      "every step (comm.refresh unset)"},
           "rebuild_policies": {"every_step": {"value": rates[1], "ms_per_step": policies[1][2] / k * 1e3},
                                "refresh_10": {"value": rates[10], "ms_per_step": policies[10][2] / k * 1e3}},
           "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                            "sample": "the GPU arm's box (%d atoms), %d steps per policy after %d warm-up, "
                                      "oracle/omd_oracle.c (the reference's algorithm restated and pinned to its "
                                      "outputs to 1e-12) in %d OpenMP threads" % (n, k, warm, cores)},
           "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
           "wall_s": t1 - t0}
    print(json.dumps(out), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=1000)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--workload", default="eam_al_256k", choices=sorted(WORKLOADS))
    ap.add_argument("--ncell", type=int, default=0)
    ap.add_argument("--flush-mb", type=int, default=512)
    ap.add_argument("--cpu-steps", type=int, default=8)
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-tune", action="store_true")
    ap.add_argument("--no-sub", action="store_true",
                    help="time only --workload (the default run adds Tersoff Si 512k and the NN surrogate)")
    ap.add_argument("--skin", type=float, default=None,
                    help="Verlet skin in A instead of the workload's (omdg_set_neighbor)")
    ap.add_argument("--launch", action="append", default=[], metavar="KEY=VALUE",
                    help="set a launch shape after tuning (omdg_set_launch), e.g. build_lanes=1")
    ap.add_argument("--eager", action="store_true",
                    help="launch the step kernels one by one instead of replaying the captured graph "
                         "(profilers cannot see kernels inside a graph with conditional nodes)")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_gpu(args)


if __name__ == "__main__":
    main()
