#!/usr/bin/env python3
"""The headline benchmark of the explicit FVM solve on B200.

Default workload (``--workload warm``): converged HR cases per second at
<= 0.5 % CD error, warm start vs plain. Geometry NACA2412, HR mesh h=0.025
(25,968 cells), LR mesh h=0.1; cases Mach ~ U[0.7, 3], alpha ~ U[-5, 5] deg
from default_rng(3): the first --n-train draws train the warm start (LR and
HR solves by the batched solver, BF16 MLP trained by the library's kernels;
untimed set-up), the next --n-eval draws per GPU are the held-out cases. Each
held-out case gets a reference CD from a long float64 solve of the same
kernels (untimed). One bench step is one pass of the warm pipeline over the
held-out cases: LR solve -> LR pressure gradients -> IDW + MLP -> HR solve
from the prediction (local CFL step, FP32), every case ending once its CD
stayed within 0.5 % of its reference for 8 checks 25 steps apart; a case
counts when it stopped that way on a steady reference.

value   converged held-out cases / device time of the passes (CUDA events
        bracketing each pass after a device-wide synchronisation).
e2e     the same pipeline through the public API with the final HR fields of
        every case read back into host memory (and the LR fields and warm
        starts crossing PCIe as the pipeline moves them), wall clock.
converged_cases_per_s  the same cases solved by the plain single-case solve
        (one case per launch, freestream, every case measured), the plain
        batched solve (freestream, retire/refill) and the IDW start, with
        the warm/plain ratios.
cell_updates, roofline  the batched throughput workload (NACA0012 h=0.025 x
        256 cases, 50-step chunks): cell-updates/s and the K2 flux kernel
        against the measured HBM copy bandwidth.

--impl reference: the reference's own CPU path is its JAX solver (absent on
these hosts); this arm times the C/OpenMP restatement of the oracle solving
the held-out cases one at a time from freestream with the same rule, on all
host threads (reference CDs from tests/golden/warm_bench_truth.json, which
``--make-truth`` writes from the float64 GPU solves).

--workload naca / ragged / diamond: the throughput workloads alone (NACA0012
h=0.025 x 256 cases, the 12-mesh ragged batch of 1,024 cases, one diamond case).

Under torchrun every rank runs its own held-out shard (weak scaling; cases
are independent, no data-path collective); times are the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "converged HR cases/s at ≤0.5% CD err, warm-start vs plain; cell-upd/s; GB/s"
UNIT = "cell-updates/s"


def get_mesh(geom: str, h: float):
    from eulersr_b200.meshing.generate import cached_mesh
    return cached_mesh(geom, h)


def batch_cases(n, seed=1):
    rng = np.random.default_rng(seed)
    mach = rng.uniform(0.7, 3.0, n)
    aoa = rng.choice(np.arange(-5, 5.01, 0.5), n)
    return mach, aoa


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi sampling of SM clocks and throttle reasons during a region."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.path = ROOT / ".bench_tmp" / f"clocks_{os.getpid()}.csv"

    def start(self):
        try:
            self.path.parent.mkdir(parents=True, exist_ok=True)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.dev}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        rows = []
        for line in self.path.read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace('.', '').isdigit()]
        smax = max(float(r[2]) for r in rows if r[2].replace('.', '').isdigit())
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower().startswith("active")})
        loaded = [x for x in sm if x > 0.5 * smax] or sm
        return {"sm_mhz": float(np.median(loaded)), "sm_max_mhz": smax, "reasons": reasons,
                "samples": len(rows)}


def cpu_oracle_sample(mesh, mach, aoa, seconds=12.0, dtype=np.float32):
    """Time the oracle's SRK2 step on one case of the workload mesh on the
    host: the C/OpenMP restatement on every host thread (the NumPy oracle,
    one thread, when the C build is unavailable). Returns (cell-updates/s,
    steps, seconds, threads, kind)."""
    try:
        from oracle.cport import CpuCase, threads
        cc = CpuCase(mesh, float(mach), float(aoa), dtype)
        W = cc.srk2(cc.W0, 2)               # warm-up (thread pool, caches)
        n, t0 = 0, time.perf_counter()
        step = 5
        while time.perf_counter() - t0 < seconds:
            W = cc.srk2(W, step)
            n += step
        el = time.perf_counter() - t0
        return mesh.n_cells * n / el, n, el, threads(), "C/OpenMP restatement of the oracle"
    except Exception:
        pass
    from oracle import euler_oracle as O
    om = O.build_oracle_mesh(mesh.points, mesh.tris, mesh.neighbors, mesh.faces, mesh.face_markers,
                             mesh.face_connectivity, dtype=dtype, metadata=mesh.metadata)
    cfg = dict(rho_inf=1.0, p_inf=1.0, gamma=1.4, Mach=float(mach), aoa=float(aoa), case=mesh.metadata['case'])
    W, inlet = O.initialize(mesh.n_cells, cfg, dtype)
    dt = O.get_dt(W, om, CFL=0.6)
    W = O.time_step_srk2(W, om, dt, inlet)   # warm-up
    n, t0 = 0, time.perf_counter()
    while time.perf_counter() - t0 < seconds:
        W = O.time_step_srk2(W, om, dt, inlet)
        n += 1
    el = time.perf_counter() - t0
    return mesh.n_cells * n / el, n, el, 1, "NumPy oracle"


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch
        import torch.distributed as dist
        from datetime import timedelta
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))
    return world, rank, local


def _allreduce(x: float, world: int, op: str) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX if op == "max" else dist.ReduceOp.SUM)
    return float(t.item())


def allreduce_max(x: float, world: int) -> float:
    """Max over ranks (the job's time is its slowest rank's)."""
    return _allreduce(x, world, "max")


def allreduce_sum(x: float, world: int) -> float:
    """Sum over ranks (work done by the whole job)."""
    return _allreduce(x, world, "sum")


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def run_reference(args, world, rank):
    if rank != 0:
        return 0
    dtype, prec = np.float32, "f32"
    if args.workload == "ragged":
        meshes, per = ragged_workload()
        cfg_mesh, mesh = (meshes, per), meshes[-1]
        mach = np.array([m for p in per for m, _ in p])
        aoa = np.array([a for p in per for _, a in p])
        config = workload_config(args, cfg_mesh)
    elif args.workload == "diamond":
        mesh = get_mesh("diamond", args.h)
        m_d, a_d, cfl = diamond_case(args.h)[:3]
        mach, aoa = np.array([m_d]), np.array([a_d])
        if args.precision == "f64":
            dtype, prec = np.float64, "f64"
        config = {"workload": f"diamond h={args.h} ({mesh.n_cells} cells), one case M={m_d} alpha={a_d} CFL {cfl}, "
                              f"SRK2 steps of the case", "cells": mesh.n_cells}
    else:
        mesh = get_mesh("naca0012", args.h)
        mach, aoa = batch_cases(args.cases)
        config = workload_config(args, mesh)
    ncores = os.cpu_count() or 1
    vals = []
    per_step = max(3.0, 40.0 / max(1, args.steps + args.warmup))
    for i in range(args.warmup + args.steps):
        v, n, el, thr, kind = cpu_oracle_sample(mesh, mach[i % len(mach)], aoa[i % len(aoa)], seconds=per_step,
                                                dtype=dtype)
        if i >= args.warmup:
            vals.append((v, n, el))
    value = float(np.mean([v for v, _, _ in vals]))
    sample = (f"{kind} (the reference's JAX CPU path needs JAX, not installed), {np.dtype(dtype).name}, one case "
              f"of the workload mesh ({mesh.n_cells} cells) per step, {vals[-1][1]} SRK2 steps in "
              f"{vals[-1][2]:.1f} s on {thr} threads")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": float(np.mean([e for _, _, e in vals]) * 1e3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": prec,
            "data": "synthetic (seeded Mach/alpha draws, freestream start)",
            "config": config,
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": thr, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "note": f"host has {ncores} cores"}
    print(json.dumps(line), flush=True)
    return 0


RAGGED_GEOMS = ("diamond", "naca0012", "naca2412", "naca23012")
RAGGED_H = (0.1, 0.05, 0.025)


def ragged_workload(n_cases=1024, seed=2, rank=0, world=1):
    """The 12 meshes and, per mesh, the (Mach, alpha) of the cases dealt to it."""
    meshes = [get_mesh(g, h) for g in RAGGED_GEOMS for h in RAGGED_H]
    rng = np.random.default_rng(seed)
    mach = rng.uniform(0.7, 3.0, n_cases * world)
    aoa = rng.uniform(-5.0, 5.0, n_cases * world)
    mach, aoa = mach[rank::world], aoa[rank::world]
    per = [[] for _ in meshes]
    for i in range(len(mach)):
        per[i % len(meshes)].append((float(mach[i]), float(aoa[i])))
    return meshes, per


LINE_MAX = 8000   # characters of the JSON line: a reader that keeps a few KB of output must get all of it
# What a longer line gives up, to a JSON line on standard error
DETAILS = (("converged_cases_per_s", "per_case"), ("converged_cases_per_s", "by_case_class"),
           ("converged_cases_per_s", "details"), ("converged_cases_per_s", "warm_passes"),
           ("converged_cases_per_s", "warm_mlp_streamed"), ("converged_cases_per_s", "warm_mlp_lr_longest_first_queue"),
           ("converged_cases_per_s", "unsteady_capped_protocol"), ("cell_updates", "config"), ("config", "training"),
           ("config", "tuning"))


def emit(line):
    """Print the bench's one JSON line on standard output. When it is too long
    its breakdowns go to standard error instead, as one JSON object."""
    if len(json.dumps(line)) > LINE_MAX:
        line, moved = dict(line), {}
        for group, key in DETAILS:
            if isinstance(line.get(group), dict) and key in line[group]:
                moved.setdefault(group, {})[key] = line[group][key]
                line[group] = {k: v for k, v in line[group].items() if k != key}
        print(json.dumps({"details": moved}), file=sys.stderr, flush=True)
        line["details"] = "standard error"
    print(json.dumps(line), flush=True)


def workload_config(args, mesh):
    if getattr(args, "workload", "naca") == "ragged":
        meshes, per = mesh
        cells = [m.n_cells for m in meshes]
        return {"workload": f"ragged batch: 12 meshes ({', '.join(RAGGED_GEOMS)} x h in 0.1/0.05/0.025, "
                            f"{min(cells)}-{max(cells)} cells) x {sum(len(p) for p in per)} cases "
                            f"(default_rng(2): Mach~U[0.7,3], alpha~U[-5,5], round-robin), SRK2 chunk of {args.chunk} steps",
                "cells": cells, "cases_per_mesh": [len(p) for p in per],
                "cases_per_gpu": sum(len(p) for p in per), "srk2_steps_per_bench_step": args.chunk,
                "scheme": "HLLC + MUSCL/Venkatakrishnan + SRK2, global dt, CFL 0.6 (0.45 transonic)",
                "l2": "working set > L2", "parallelism": "cases sharded per GPU, all meshes in one launch"}
    return {"workload": f"naca0012 h={args.h} HR ({mesh.n_cells} cells) x {args.cases} cases "
                        f"(Mach~U[0.7,3] seed 1, alpha in -5..5 step 0.5), SRK2 chunk of {args.chunk} steps",
            "cells": int(mesh.n_cells), "cases_per_gpu": args.cases, "srk2_steps_per_bench_step": args.chunk,
            "scheme": "HLLC + MUSCL/Venkatakrishnan + SRK2, global dt, CFL 0.6 (0.45 transonic)",
            "l2": "working set > L2 (state 3x of 16 B per cell and case)",
            "parallelism": f"cases sharded, {args.cases} per GPU"}


def diamond_case(h):
    """(Mach, alpha, CFL, stop rule, threshold, max steps) of the single-case diamond workloads."""
    if h >= 0.1:
        return 2.5, 5.0, 0.8, "density_l2", 1e-6, 40000
    return 2.0, 0.0, 0.6, "reference", 1e-5, 40000


def run_single(args, world, rank, local):
    """One case per GPU solved from freestream to its stop rule, K times."""
    from eulersr_b200.solver import Solver, FlowCase, DeviceMesh
    mesh = get_mesh("diamond", args.h)
    mach, aoa, cfl, rule, thr, cap = diamond_case(args.h)
    prec = args.precision
    case = FlowCase(mach=mach, aoa_deg=aoa, cfl=cfl, tf=1e9, max_steps=cap,
                    dtype=np.float64 if prec == "f64" else np.float32)
    s = Solver(DeviceMesh(mesh), 1, precision=prec, stop_rule=rule, threshold=thr, check_every=25,
               device=local if world > 1 else 0)
    N = mesh.n_cells

    def solve():
        s.set_case(0, case)
        return s.run()[0]
    for _ in range(args.warmup):
        r = solve()
    clocks = ClockSampler(local)
    barrier(world)
    s.synchronize()
    l0 = s.kernel_launches()
    clocks.start()
    ms, steps = 0.0, 0
    t0 = time.perf_counter()
    for _ in range(args.steps):
        r = solve()
        ms += s.elapsed_ms()             # device time of the run (CUDA events on the solver stream)
        steps += int(r["steps"])
    s.synchronize()
    wall = time.perf_counter() - t0
    clk = clocks.stop()
    launches = s.kernel_launches() - l0
    ms_max = allreduce_max(ms, world)
    cu = allreduce_sum(float(N * steps), world)
    value = cu / (ms_max * 1e-3)
    kt = s.profile_step(8)
    hbm, peak_kind = peaks()
    alg_k2 = (40 + 64) * N
    k2_gbs = alg_k2 / (kt["flux_ms"] * 1e-3) / 1e9
    roofline = {"bound": "hbm", "achieved": k2_gbs, "peak": hbm, "unit": "GB/s", "frac": k2_gbs / hbm,
                "traffic": None, "kernel": "k_stage (one fused stage)" if kt["recon_launches"] == 0 else "k_flux (K2)",
                "peak_source": peak_kind, "kernel_ms": kt["flux_ms"],
                "recon_ms": kt["recon_ms"], "alg_bytes_per_launch": alg_k2,
                "note": "one case: the state is L2-resident and the launches are latency-bound"}
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        cdt = np.float64 if prec == "f64" else np.float32
        v, n, el, thr_, kind = cpu_oracle_sample(mesh, mach, aoa, seconds=12.0, dtype=cdt)
        cpu = {"value": v, "unit": UNIT, "cores": thr_, "kind": "port",
               "sample": f"{kind}, {np.dtype(cdt).name}, {n} SRK2 steps of the case on the {N}-cell mesh ({el:.1f} s)"}
    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms_max / args.steps, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": prec,
                "data": "synthetic (diamond mesh generated by the package's mesher, freestream start)",
                "config": {"workload": f"diamond h={args.h} ({N} cells), one case M={mach} alpha={aoa} CFL {cfl}, "
                                       f"stop rule {rule} {thr}, one bench step = one full solve",
                           "cells": N, "steps_per_solve": int(r["steps"]), "converged": bool(r["converged"]),
                           "cd": r["cd"], "cl": r["cl"], "l2": "working set < L2 (one case)"},
                "converged_cases_per_s": args.steps * world / (ms_max * 1e-3),
                "e2e": {"value": cu / wall, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0,
                        "api": "esr_set_case (freestream) + esr_run, results read back; wall clock"},
                "roofline": roofline, "cpu_baseline": cpu, "clocks": clk, "gpu_launches": int(launches),
                "kernel_times_ms": kt}
        emit(line)
    barrier(world)
    s.close()
    return 0


def run_throughput(args, world, rank, local, report=True):
    """The batched throughput workloads (NACA0012 h=0.025 x 256 cases, the
    12-mesh ragged batch): cell-updates/s of fixed 50-step chunks, the K2 roofline and the
    end-to-end rate with host fields. Prints its own line when `report`, and
    returns the measurements."""
    from eulersr_b200.parallel import case_cost, shard_cases
    from eulersr_b200.solver import Solver, FlowCase, DeviceMesh
    if args.workload == "ragged":
        meshes, per = ragged_workload(rank=rank, world=world)
        cases = [FlowCase(mach=m, aoa_deg=a, mesh=k, cfl=0.6, tf=1e9, dtype=np.float32)
                 for k, p in enumerate(per) for m, a in p]
        s = Solver([DeviceMesh(m) for m in meshes], [len(p) for p in per], precision="f32",
                   device=local if world > 1 else 0, block_size=args.block)
        mesh = (meshes, per)
        items = sum(m.n_cells * len(p) for m, p in zip(meshes, per))
        B, N = len(cases), items / len(cases)       # N: mean cells per case
        mach, aoa = [c.mach for c in cases], [c.aoa_deg for c in cases]
        cpu_mesh = meshes[-1]
        shard_note = "round-robin over ranks"
    else:
        mesh = get_mesh("naca0012", args.h)
        mach_all, aoa_all = batch_cases(args.cases * world)
        # the product's scheduler: cost-balanced longest-processing-time shards
        mine = shard_cases(case_cost(mach_all, mesh.n_cells), world)[rank]
        mach, aoa = mach_all[mine], aoa_all[mine]
        cases = [FlowCase(mach=float(m), aoa_deg=float(a), cfl=0.6, tf=1e9, dtype=np.float32)
                 for m, a in zip(mach, aoa)]
        s = Solver(DeviceMesh(mesh), len(cases), precision="f32", device=local if world > 1 else 0,
                   block_size=args.block)
        B, N = len(cases), mesh.n_cells
        cpu_mesh = mesh
        shard_note = "parallel.shard_cases (cost-balanced LPT)"
    s.set_cases(list(range(B)), cases)
    s.synchronize()
    tuning = s.tuning()

    # warm-up (graph capture happens in the first chunk)
    for _ in range(args.warmup):
        s.step(args.chunk)
    clocks = ClockSampler(local)
    barrier(world)
    s.synchronize()
    l0 = s.kernel_launches()
    clocks.start()
    ms = 0.0
    for _ in range(args.steps):
        s.step(args.chunk)          # CUDA events on the solver stream around each chunk
        ms += s.elapsed_ms()
    s.synchronize()
    clk = clocks.stop()
    launches = s.kernel_launches() - l0
    barrier(world)
    ms_max = allreduce_max(ms, world)
    cu_total = allreduce_sum(float(N * B * args.chunk * args.steps), world)
    value = cu_total / (ms_max * 1e-3)
    # geometry is shared by the cases of a mesh: 128 B per cell-step per mesh
    B_eff = B if args.workload != "ragged" else B / len(mesh[0])
    alg_step_bytes = 80 + 128 / B_eff

    # dominant kernel: the fused stage (or K2 at a requested launch shape), timed per launch with events on its stream
    kt = s.profile_step(8)
    hbm, peak_kind = peaks()
    alg_k2 = (40 + 64 / B_eff) * N * B
    k2_gbs = alg_k2 / (kt["flux_ms"] * 1e-3) / 1e9
    # DRAM traffic per item of the K2 form in use, from its ncu summary
    traffic = None
    fused = kt["recon_launches"] == 0
    patches = bool(tuning.get("k2_patches"))
    k2_name = ("k_stage_pair (one fused stage)" if fused else
               "k_flux_patch (K2 by patches)" if patches else "k_flux (K2 per cell)")
    pf = ROOT / "profiles" / ("k_stage_pair_naca0012_h0.025_b96.md" if fused else
                              "k_flux_patch_naca0012_h0.025_b128.md" if patches else "k_flux_naca0012_h0.025_b128.md")
    if pf.exists():
        for line in pf.read_text().splitlines():
            if line.startswith("traffic_bytes_per_item_per_launch"):
                traffic = float(line.split("=")[1].split()[0]) * N * B
    roofline = {"bound": "hbm", "achieved": k2_gbs, "peak": hbm, "unit": "GB/s", "frac": k2_gbs / hbm,
                "traffic": traffic, "traffic_source": f"ncu capture in profiles/{pf.name}, per item, scaled by items",
                "kernel": k2_name, "peak_source": peak_kind, "kernel_ms": kt["flux_ms"],
                "recon_ms": kt["recon_ms"], "alg_bytes_per_launch": alg_k2,
                "workload": f"batched {args.workload} workload, {B} cases per GPU, one launch",
                "note": "issue-bound; see profiles/"}

    # end to end through the public API with host buffers
    e2e = None
    if not args.no_e2e:
        sizes = [s._n_cells(b) for b in range(B)]
        # float32 host fields for the float32 solver (the values it stores)
        import torch
        def host_block():
            # every case's field as a view of one pinned block, back to back
            # in slot order: the library moves them with one copy each way
            try:
                big = torch.empty((int(sum(sizes)), 4), dtype=torch.float32, pin_memory=True).numpy()
            except Exception:
                big = np.empty((int(sum(sizes)), 4), dtype=np.float32)
            offs = np.concatenate([[0], np.cumsum(sizes)])
            return [big[offs[i]:offs[i + 1]] for i in range(len(sizes))]
        pinned = host_block()
        from eulersr_b200.solver import freestream
        for b, c in enumerate(cases):
            pinned[b][:] = freestream(c.mach, c.aoa_deg, dtype=np.float32)[None, :]
        h2d = int(sum(p.nbytes for p in pinned))
        outs = host_block()
        e2e_steps = max(10, args.steps)   # a stream of batches: the first upload and last download stay exposed
        slots = list(range(B))
        # one untimed pass first: the staging buffers are allocated on first use
        s.stage_cases(slots, cases, pinned)
        s.apply_staged()
        s.step(args.chunk)
        s.fetch_states(slots, outs)
        s.wait_transfers()
        barrier(world)
        t0 = time.perf_counter()
        s.stage_cases(slots, cases, pinned)
        s.apply_staged()
        for i in range(e2e_steps):
            if i + 1 < e2e_steps:
                s.stage_cases(slots, cases, pinned)    # the next step's fields go up while this chunk runs
            s.step(args.chunk)
            s.fetch_states(slots, outs)                # this step's fields come down while the next runs
            if i + 1 < e2e_steps:
                s.apply_staged()
        s.wait_transfers()
        s.synchronize()
        el = time.perf_counter() - t0
        el = allreduce_max(el, world)
        e2e_val = allreduce_sum(float(N * B * args.chunk * e2e_steps), world) / el
        e2e = {"value": e2e_val, "unit": UNIT, "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": int(sum(o.nbytes for o in outs)),
               "api": "esr_stage_cases_f32 (pinned float32 init fields, copy stream) + esr_apply_staged + "
                      "esr_step + esr_fetch_states_f32 (pinned float32 outputs, copy stream): each step's upload "
                      "and the previous step's download overlap the chunk; wall clock"}
    cost_max = allreduce_max(float(np.sum(case_cost(np.asarray(mach), N))), world)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu and report:
        v, n, el, thr, kind = cpu_oracle_sample(cpu_mesh, mach[0], aoa[0], seconds=12.0)
        cpu = {"value": v, "unit": UNIT, "cores": thr, "kind": "port",
               "sample": f"{kind}, float32, 1 case x {n} SRK2 steps on the {cpu_mesh.n_cells}-cell mesh ({el:.1f} s)"}
    out = {"value": value, "unit": UNIT, "ms_per_step": ms_max / args.steps,
           "alg_gbs_per_step": value * alg_step_bytes / 1e9, "alg_bytes_per_cell_update": alg_step_bytes,
           "roofline": roofline, "e2e": e2e, "clocks": clk, "gpu_launches": int(launches), "kernel_times_ms": kt,
           "config": dict(workload_config(args, mesh), tuning=tuning, sharding=shard_note, cases_this_rank=B,
                          max_rank_estimated_cost=cost_max)}
    if report and rank == 0:
        line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms_max / args.steps, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic (seeded Mach/alpha draws on meshes generated by the package's mesher, "
                        "freestream start)",
                "config": out["config"], "alg_gbs_per_step": out["alg_gbs_per_step"],
                "alg_bytes_per_cell_update": alg_step_bytes,
                "roofline": roofline, "e2e": e2e, "cpu_baseline": cpu, "clocks": clk,
                "gpu_launches": int(launches), "kernel_times_ms": kt}
        emit(line)
    barrier(world)
    s.close()
    return out


# ------------------------------------------------------------ warm start
WARM_UNIT = "converged HR cases/s"
TRUTH_FILE = ROOT / "tests" / "golden" / "warm_bench_truth.json"


def warm_cases(args, world, rank):
    """This rank's held-out (Mach, alpha): the n_eval x world draws after the
    training draws of default_rng(3), dealt by the product's cost-balanced
    scheduler. Returns (indices into the held-out draws, mach, alpha)."""
    from eulersr_b200.parallel import case_cost, shard_cases
    from eulersr_b200.warmstart.pipeline import draw_cases
    _, (me, ae) = draw_cases(args.n_train, args.n_eval * world, seed=3)
    idx = shard_cases(case_cost(me), world)[rank]
    return idx, me[idx], ae[idx]


def _truth_table():
    if TRUTH_FILE.exists():
        return json.loads(TRUTH_FILE.read_text())
    return None


PLAIN_TRUTH_FILE = ROOT / "tests" / "golden" / "naca0012_bench_truth.json"


def run_plain_converged(args, world, rank, local, make_truth=False):
    """The throughput workload's batch solved to the stop rule: the 256 NACA0012 h=0.025
    cases of the throughput workload (per GPU), freestream starts, through
    esr_batch_solve with retire/refill (the warm pipeline's 32 HR slots), each
    stopped once its CD stayed within 0.5 % of its float64 reference for 8
    checks 25 steps apart (12,000-step cap). The references come from
    tests/golden/naca0012_bench_truth.json (written by --make-plain-truth
    from float64 solves of the same kernels, 30,000 + 5,000 steps) or, for
    cases not in it, are computed here. Returns the leg's record."""
    from eulersr_b200.parallel import case_cost, shard_cases
    from eulersr_b200.warmstart.workflow import WarmStartWorkflow
    mesh = get_mesh("naca0012", args.h)
    mach_all, aoa_all = batch_cases(args.cases * world)
    mine = shard_cases(case_cost(mach_all, mesh.n_cells), world)[rank]
    me, ae = mach_all[mine], aoa_all[mine]
    wf = WarmStartWorkflow(geom="naca0012", h_hr=args.h, slots=args.slots, max_steps=args.max_steps, device=local,
                           warm_budget=None)
    table = {}
    if PLAIN_TRUTH_FILE.exists() and not make_truth:
        for r in json.loads(PLAIN_TRUTH_FILE.read_text())["cases"]:
            table[(round(r["mach"], 12), round(r["aoa"], 12))] = (r["cd"], r["steady"])
    keys = [(round(float(m), 12), round(float(a), 12)) for m, a in zip(me, ae)]
    todo = [i for i, k in enumerate(keys) if k not in table]
    t0 = time.perf_counter()
    if todo:
        cd, st = wf.truth(me[todo], ae[todo])
        for j, i in enumerate(todo):
            table[keys[i]] = (float(cd[j]), bool(st[j]))
    truth_s = time.perf_counter() - t0
    truth = np.array([table[k][0] for k in keys])
    steady = np.array([table[k][1] for k in keys])
    if make_truth:
        if rank == 0 and world == 1:
            rows = [{"mach": float(m), "aoa": float(a), "cd": float(c), "steady": bool(s_)}
                    for m, a, c, s_ in zip(me, ae, truth, steady)]
            PLAIN_TRUTH_FILE.write_text(json.dumps({
                "about": "reference CD of the throughput workload's NACA0012 h=0.025 cases: float64 solves of the "
                         "library's kernels (local CFL step, 30,000 steps, then 5,000 more; steady when the CD "
                         "moved by <= 0.1 %), written by python bench.py --make-plain-truth",
                "cases": rows}, indent=1) + "\n")
        wf.close()
        return {"truth_written": str(PLAIN_TRUTH_FILE), "cases": len(me), "steady": int(steady.sum())}
    r = wf.solve(me, ae, truth, steady, "cold")
    wf.close()
    value = allreduce_sum(float(r.converged), world) / allreduce_max(r.seconds, world)
    return {"value": value, "unit": WARM_UNIT, "cases_per_gpu": len(me), "steady": int(steady.sum()),
            "converged": r.converged, "seconds": r.seconds, "slots": args.slots,
            "median_iterations": float(np.median(r.iterations)), "references_computed_here": len(todo),
            "references_s": truth_s,
            "workload": "the throughput workload's 256 NACA0012 h=0.025 cases (Mach~U[0.7,3] seed 1, alpha on the 0.5-degree grid) "
                        "from freestream through esr_batch_solve, 0.5 % CD rule, 12,000-step cap"}


def cpu_converged_sample(cases, seconds_cap, mesh, cd_tol=0.005, patience=8, check_every=25, max_steps=12000):
    """The reference's method on the host: each case solved alone from
    freestream by the C/OpenMP restatement of the oracle (float32, local CFL
    step) until its CD stayed within cd_tol of its reference for `patience`
    checks `check_every` steps apart (or max_steps). cases: dicts with mach,
    aoa, cd, steady. Returns (converged, seconds, per-case records, threads)."""
    from oracle import euler_oracle as O
    from oracle.cport import CpuCase, threads
    from eulersr_b200.solver import clamp_cfl
    conv, total, recs = 0, 0.0, []
    L = mesh.metadata.get("obstacle_length", 1.0)
    for c in cases:
        t0 = time.perf_counter()
        cc = CpuCase(mesh, c["mach"], c["aoa"], np.float32)
        cfl = clamp_cfl(c["mach"], 0.6)
        u_inf = c["mach"] * 1.4 ** 0.5
        W, step, streak, start, stopped, cd = cc.W0, 0, 0, 0, False, 0.0
        tgt = c["cd"]
        while True:
            cd = float(O.force_coefficients(W.astype(np.float64), cc.om, 1.0, u_inf, L)[0])
            ok = abs(cd - tgt) <= cd_tol * max(abs(tgt), 1e-8)
            if ok and streak == 0:
                start = step
            streak = streak + 1 if ok else 0
            if streak >= patience:
                stopped = True
                break
            if step >= max_steps:
                break
            n = min(check_every, max_steps - step)
            W = cc.srk2_local(W, n, cfl)
            step += n
        el = time.perf_counter() - t0
        good = stopped and c["steady"] and abs(cd - tgt) <= cd_tol * abs(tgt)
        conv += int(good)
        total += el
        recs.append({"mach": c["mach"], "aoa": c["aoa"], "steps": step, "stopping_step": start if stopped else step,
                     "converged": bool(good), "seconds": el})
        if total >= seconds_cap:
            break
    return conv, total, recs, threads()


def run_reference_warm(args, world, rank):
    """--impl reference for the headline: the held-out cases one per bench
    step, solved on the host by the C/OpenMP restatement (warm-up steps run
    200 steps of a case to start the thread pool)."""
    if rank != 0:
        return 0
    table = _truth_table()
    if table is None:
        print(json.dumps({"impl": "reference", "unavailable": f"reference CDs missing ({TRUTH_FILE.name})"}), flush=True)
        return 0
    mesh = get_mesh("naca2412", 0.025)
    cases = table["cases"]
    from oracle.cport import CpuCase
    from eulersr_b200.solver import clamp_cfl
    for i in range(args.warmup):
        c = cases[i % len(cases)]
        cc = CpuCase(mesh, c["mach"], c["aoa"], np.float32)
        cc.srk2_local(cc.W0, 200, clamp_cfl(c["mach"], 0.6))
    conv, sec, recs, thr = 0, 0.0, [], 1
    for i in range(args.steps):
        c = cases[i % len(cases)]
        n, t, r, thr = cpu_converged_sample([c], 1e9, mesh)
        conv += n
        sec += t
        recs += r
    value = conv / sec if sec > 0 else 0.0
    sample = (f"C/OpenMP restatement of the oracle (the reference's JAX CPU path needs JAX, not installed), "
              f"float32, local CFL step, {len(recs)} held-out NACA2412 h=0.025 cases ({mesh.n_cells} cells) solved "
              f"one at a time from freestream to the 0.5 % CD rule, {conv} converged in {sec:.1f} s on {thr} threads")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": WARM_UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec / max(1, len(recs)) * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded Mach/alpha draws, freestream start)",
            "config": {"workload": "plain single-case solve of the held-out NACA2412 cases on the host cores",
                       "cases": len(recs), "truth": TRUTH_FILE.name},
            "cpu_baseline": {"value": value, "unit": WARM_UNIT, "cores": thr, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": WARM_UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "per_case": recs, "note": f"host has {os.cpu_count()} cores"}
    emit(line)
    return 0


def run_warm(args, world, rank, local):
    import torch
    from eulersr_b200.warmstart.workflow import WarmStartWorkflow
    torch.cuda.set_device(local)
    t_setup = time.perf_counter()
    wf = WarmStartWorkflow(slots=args.slots, max_steps=args.max_steps, device=local, lr_steps=args.lr_steps,
                           warm_budget=args.warm_budget or None)
    info = {} if args.make_truth else wf.prepare(n_train=args.n_train, target_steps=args.target_steps,
                                                 train_steps=args.train_steps)
    idx, me, ae = warm_cases(args, world, rank)
    t0 = time.perf_counter()
    truth, steady = wf.truth(me, ae)
    truth_s = time.perf_counter() - t0
    if args.make_truth:
        if rank == 0 and world == 1:
            rows = [{"mach": float(m), "aoa": float(a), "cd": float(c), "steady": bool(s_)}
                    for m, a, c, s_ in zip(me, ae, truth, steady)]
            TRUTH_FILE.write_text(json.dumps({
                "about": "reference CD of the bench's held-out NACA2412 h=0.025 cases: float64 solves of the "
                         "library's kernels (local CFL step, 30,000 steps, then 5,000 more; steady when the CD "
                         "moved by <= 0.1 %), written by python bench.py --make-truth",
                "n_train": args.n_train, "n_eval": args.n_eval, "cases": rows}, indent=1) + "\n")
            print(json.dumps({"truth_written": str(TRUTH_FILE), "cases": len(rows), "steady": int(steady.sum())}))
        wf.close()
        return 0
    table = _truth_table()
    truth_check = None
    if table is not None:
        tab = {(round(r["mach"], 12), round(r["aoa"], 12)): r["cd"] for r in table["cases"]}
        d = [abs(c - tab[(round(float(m), 12), round(float(a), 12))]) / abs(c)
             for m, a, c in zip(me, ae, truth) if (round(float(m), 12), round(float(a), 12)) in tab]
        truth_check = {"cases": len(d), "max_rel_diff_vs_committed": float(max(d)) if d else None}
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=f"cuda:{local}")   # 256 MB > L2
    setup_s = time.perf_counter() - t_setup
    for _ in range(args.warmup):
        wf.solve(me, ae, truth, steady, "mlp")
        flush.add_(1.0)
    clocks = ClockSampler(local)
    barrier(world)
    torch.cuda.synchronize()
    l0 = wf.kernel_launches()
    clocks.start()
    passes = []
    for _ in range(args.steps):
        passes.append(wf.solve(me, ae, truth, steady, "mlp"))
        flush.add_(1.0)                 # overwrite more than L2 between passes
    torch.cuda.synchronize()
    clk = clocks.stop()
    launches = wf.kernel_launches() - l0
    barrier(world)
    sec = sum(p.seconds for p in passes)
    conv = sum(p.converged for p in passes)
    sec_max = allreduce_max(sec, world)
    value = allreduce_sum(float(conv), world) / sec_max
    # the same cases by the other starts, one pass each
    base = {}

    def case_record(res):
        ok = [bool(x["status"] == 2 and st and abs(x["cd"] - t) <= wf.cd_tol * abs(t))
              for x, t, st in zip(res, truth, steady)]
        return {"steps": [int(x["steps"]) for x in res], "status": [int(x["status"]) for x in res],
                "fallback": [bool(x.get("fallback", False)) for x in res], "converged": ok}

    per_case = {"mach": [float(m) for m in me], "aoa": [float(a) for a in ae], "steady": [bool(x) for x in steady],
                "mlp": case_record(passes[-1].results)}
    for start in ("single", "cold", "idw"):
        flush.add_(1.0)
        barrier(world)
        r = wf.solve(me, ae, truth, steady, start)
        per_case[start] = case_record(r.results)
        base[start] = allreduce_sum(float(r.converged), world) / allreduce_max(r.seconds, world)
        base[start + "_detail"] = {"converged": r.converged, "seconds": r.seconds,
                                   "median_iterations": float(np.median(r.iterations)), "parts_s": r.parts_s}
    # converged cases and steps by Mach band, per start (this rank's cases)
    bands = [(0.7, 0.9), (0.9, 1.2), (1.2, 1.6), (1.6, 2.2), (2.2, 3.01)]
    by_band = []
    for lo, hi in bands:
        sel = [i for i, m in enumerate(me) if lo <= m < hi]
        row = {"mach": [lo, min(hi, 3.0)], "cases": len(sel), "steady": int(sum(bool(steady[i]) for i in sel))}
        for name in ("mlp", "idw", "cold"):
            rec = per_case[name]
            row[name] = {"converged": int(sum(rec["converged"][i] for i in sel)),
                         "steps": int(sum(rec["steps"][i] for i in sel)),
                         "fallbacks": int(sum(rec["fallback"][i] for i in sel))}
        by_band.append(row)
    # by case class: the cases whose reference settles, alone (the cases that
    # never settle cost every start the whole step cap)
    cls = {}
    keep = np.nonzero(steady)[0]
    if len(keep):
        for start in ("mlp", "single"):
            flush.add_(1.0)
            barrier(world)
            r = wf.solve(me[keep], ae[keep], truth[keep], steady[keep], start)
            cls[start] = allreduce_sum(float(r.converged), world) / allreduce_max(r.seconds, world)
    steps_warm = np.array([x["steps"] for x in passes[-1].results])
    capped = steps_warm >= args.max_steps
    fallbacks = [x for x in passes[-1].results if x.get("fallback")]
    by_class = {"steady_cases": int(steady.sum()), "unsteady_cases": int((~steady).sum()),
                "warm_capped_cases": int(capped.sum()),
                "warm_fallbacks_to_freestream": len(fallbacks),
                "warm_fallbacks_converged": int(sum(1 for x in fallbacks if x["status"] == 2)),
                "warm_step_share_of_fallback_warm_phase": float(
                    sum(x["warm_steps"] for x in fallbacks) / max(steps_warm.sum(), 1)),
                "warm_step_share_of_capped_cases": float(steps_warm[capped].sum() / max(steps_warm.sum(), 1)),
                "steady_only_warm_mlp_batched": cls.get("mlp"), "steady_only_plain_single_case": cls.get("single"),
                "steady_only_ratio": (cls["mlp"] / cls["single"]) if cls.get("single") else None,
                "by_mach_band": by_band}
    # the same warm pass with the HR cases queued longest-first by their LR solve
    flush.add_(1.0)
    barrier(world)
    wf.schedule = "lr_longest_first"
    try:
        r = wf.solve(me, ae, truth, steady, "mlp")
    finally:
        wf.schedule = "fifo"
    lpt = {"value": allreduce_sum(float(r.converged), world) / allreduce_max(r.seconds, world),
           "converged": r.converged, "seconds": r.seconds, "parts_s": r.parts_s}
    # the protocol variant with unsteady-flagged cases capped at --unsteady-cap
    # steps for every start (they fail for every start whatever they do)
    capped_proto = None
    if args.unsteady_cap:
        wf.unsteady_cap = args.unsteady_cap
        try:
            cp = {}
            for start in ("mlp", "single"):
                flush.add_(1.0)
                barrier(world)
                r = wf.solve(me, ae, truth, steady, start)
                cp[start] = allreduce_sum(float(r.converged), world) / allreduce_max(r.seconds, world)
        finally:
            wf.unsteady_cap = None
        capped_proto = {"unsteady_cap_steps": args.unsteady_cap, "warm_mlp_batched": cp["mlp"],
                        "plain_single_case": cp["single"], "ratio": cp["mlp"] / cp["single"] if cp["single"] else None}
    # a stream of batches, as a campaign runs them: the next batch's LR solve
    # and prediction overlap this batch's HR solve
    flush.add_(1.0)
    barrier(world)
    sp, s_sec, s_wall = wf.solve_stream([(me, ae)] * args.steps, [truth] * args.steps, [steady] * args.steps)
    streamed = {"batches": args.steps, "seconds": s_sec, "wall_s": s_wall,
                "value": allreduce_sum(float(sum(p.converged for p in sp)), world) / allreduce_max(s_sec, world),
                "parts_s": [p.parts_s for p in sp[:3]]}
    # end to end: the pipeline with every case's final HR field read into host memory
    flush.add_(1.0)
    barrier(world)
    t0 = time.perf_counter()
    e = wf.solve(me, ae, truth, steady, "mlp", want_states=True)
    e2e_s = allreduce_max(time.perf_counter() - t0, world)
    n_hr, n_lr = wf.hr.n_cells, wf.lr.n_cells
    h2d = len(me) * n_hr * 4 * 8 + len(me) * n_lr * 4 * 8          # warm fields up, LR fields for the gradients
    d2h = len(me) * n_hr * 4 * 8 + len(me) * n_lr * 4 * 8 + len(me) * 8 * n_lr * 8
    e2e = {"value": allreduce_sum(float(e.converged), world) / e2e_s, "unit": WARM_UNIT,
           "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h),
           "api": "WarmStartWorkflow.solve(start='mlp', want_states=True): esr_batch_solve of the LR cases "
                  "(final fields to host), esr_gradients per case, IDW/MLP kernels, esr_batch_solve of the HR "
                  "cases from the host warm fields with every final field returned to host memory; wall clock"}
    hr_mesh = wf.hr
    wf.close()
    del flush
    torch.cuda.empty_cache()
    # the throughput workload's 256 NACA0012 cases solved to the same CD rule from freestream
    pargs = argparse.Namespace(**vars(args))
    pargs.cases = 256
    plain3 = run_plain_converged(pargs, world, rank, local)
    # the batched throughput workload: cell-updates/s and the K2 roofline
    targs = argparse.Namespace(**vars(args))
    targs.workload, targs.steps, targs.warmup = "naca", min(args.steps, 10), 3
    thr = run_throughput(targs, world, rank, local, report=False)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        cases = [{"mach": float(m), "aoa": float(a), "cd": float(c), "steady": bool(s_)}
                 for m, a, c, s_ in zip(me, ae, truth, steady)]
        n, t, recs, thr_n = cpu_converged_sample(cases, 20.0, hr_mesh)
        cpu = {"value": n / t if t > 0 else 0.0, "unit": WARM_UNIT, "cores": thr_n, "kind": "port",
               "sample": f"C/OpenMP restatement of the oracle, float32, local CFL step, {len(recs)} held-out cases "
                         f"solved one at a time from freestream to the 0.5 % CD rule, {n} converged in {t:.1f} s"}
    if rank == 0:
        ratio = {k: value / base[k] if base[k] > 0 else None for k in ("single", "cold", "idw")}
        line = {"metric": METRIC, "value": value, "unit": WARM_UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": sec_max / args.steps * 1e3, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic (seeded Mach/alpha draws on meshes generated by the package's mesher)",
                "config": {"workload": f"warm-start pipeline (LR solve + IDW + MLP + HR solve) over {len(me)} "
                                       f"held-out NACA2412 cases per GPU, HR h=0.025 ({hr_mesh.n_cells} cells), "
                                       f"LR h=0.1 ({n_lr} cells), {args.slots} HR slots with retire/refill",
                           "cases_per_gpu": len(me), "slots": args.slots, "cd_tolerance": 0.005,
                           "rule": "CD within 0.5 % of the case's float64 reference CD for 8 checks 25 steps apart",
                           "dt": "local CFL 0.6 (0.45 transonic)", "max_steps": args.max_steps,
                           "warm_budget": args.warm_budget or None,
                           "fallback": "a warm start the rule has not stopped within warm_budget steps restarts "
                                       "from freestream with the rest of max_steps (steps of both phases counted)",
                           "lr_steps": args.lr_steps, "training": info,
                           "reference_cd": f"float64 solves of the same kernels, 30,000 + 5,000 steps ({truth_s:.1f} s)",
                           "steady_cases": int(steady.sum()), "truth_check": truth_check,
                           "l2": "256 MB buffer overwritten between passes", "setup_s": setup_s,
                           "sharding": "parallel.shard_cases (cost-balanced LPT)",
                           "hr_queue": "submission order (the LR-informed longest-first order is reported beside "
                                       "it: no measurable gain)"},
                "converged_cases_per_s": {
                    "warm_mlp_batched": value, "warm_idw_batched": base["idw"], "plain_batched": base["cold"],
                    "plain_single_case": base["single"], "ratio_warm_vs_plain_single_case": ratio["single"],
                    "ratio_warm_vs_plain_batched": ratio["cold"], "ratio_warm_vs_idw": ratio["idw"],
                    "warm_passes": [{"converged": p.converged, "seconds": p.seconds, "parts_s": p.parts_s}
                                    for p in passes[:3]],
                    "median_iterations_warm": float(np.median(passes[-1].iterations)),
                    "details": {k: base[k + "_detail"] for k in ("single", "cold", "idw")},
                    "by_case_class": by_class, "warm_mlp_streamed": streamed,
                    "warm_mlp_lr_longest_first_queue": lpt, "unsteady_capped_protocol": capped_proto,
                    "plain_batched_naca0012_x256": plain3, "per_case": per_case},
                "e2e": e2e, "roofline": thr["roofline"],
                "cell_updates": {k: thr[k] for k in ("value", "unit", "ms_per_step", "alg_gbs_per_step",
                                                      "alg_bytes_per_cell_update", "e2e", "kernel_times_ms",
                                                      "config")},
                "cpu_baseline": cpu, "clocks": clk, "gpu_launches": int(launches),
                "gpu_launches_throughput_leg": thr["gpu_launches"]}
        emit(line)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cases", type=int, default=256)
    ap.add_argument("--chunk", type=int, default=50)
    ap.add_argument("--h", type=float, default=0.025)
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--workload", default="warm", choices=["warm", "naca", "ragged", "diamond"])
    ap.add_argument("--precision", default="f32", choices=["f32", "f64"], help="diamond workload only")
    ap.add_argument("--n-train", type=int, default=256, help="warm workload: training cases")
    ap.add_argument("--n-eval", type=int, default=128, help="warm workload: held-out cases per GPU")
    ap.add_argument("--slots", type=int, default=32, help="warm workload: HR case slots")
    ap.add_argument("--max-steps", type=int, default=12000, help="warm workload: step cap of an HR solve")
    ap.add_argument("--target-steps", type=int, default=12000, help="warm workload: steps of a training target")
    ap.add_argument("--train-steps", type=int, default=2000, help="warm workload: MLP training steps")
    ap.add_argument("--lr-steps", type=int, default=2000, help="warm workload: steps of each LR solve")
    ap.add_argument("--warm-budget", type=int, default=3000,
                    help="warm workload: steps after which an unstopped warm start restarts from freestream (0: never)")
    ap.add_argument("--unsteady-cap", type=int, default=3000,
                    help="warm workload: extra leg with unsteady-flagged cases capped at this many steps for every "
                         "start (0: skip the leg)")
    ap.add_argument("--make-truth", action="store_true", help="write the held-out cases' reference CDs and exit")
    ap.add_argument("--make-plain-truth", action="store_true",
                    help="write the reference CDs of the throughput workload's NACA0012 cases and exit")
    ap.add_argument("--block", default="0", help="throughput workloads: 0 (the solver's own choice), 64, 128, 256 or patches")
    args = ap.parse_args()
    args.block = args.block if args.block == "patches" else int(args.block)
    args.warmup = max(3, args.warmup)

    if args.impl == "reference":
        # the reference's CPU path: rank 0 alone times it; other ranks exit at once
        world = int(os.environ.get("WORLD_SIZE", "1"))
        rank = int(os.environ.get("RANK", "0"))
        if args.workload == "warm":
            return run_reference_warm(args, world, rank)
        return run_reference(args, world, rank)
    world, rank, local = dist_setup()
    try:
        if args.workload == "diamond":
            return run_single(args, world, rank, local)
        if args.make_plain_truth:
            import torch
            torch.cuda.set_device(local)
            print(json.dumps(run_plain_converged(args, world, rank, local, make_truth=True)), flush=True)
            return 0
        if args.workload == "warm":
            return run_warm(args, world, rank, local)
        run_throughput(args, world, rank, local, report=True)
        return 0
    finally:
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()


if __name__ == "__main__":
    sys.exit(main())
