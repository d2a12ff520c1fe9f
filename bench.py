"""Benchmark of the CUDA cloth step: sim steps/s on the floor-drape workload.

python bench.py --gpus N --steps K --warmup W [--impl cuda|reference]
                [--workload floor_drape|strip_pull|sphere_drape|batch_sheets|material_fit]
                [--skip S]   # untimed steps after the warm-up (default 17: the window spans the landing)
                [--budget converged|reference]

Default (floor drape, 64 x 64, 4,096 vertices): the mixed-precision path and
the FP64 path run the same steps under a stepper budget where both converge
(exact-Newton mode: 40 Newton iterations, 3000 PCG iterations, gradTol 1e-8);
the timed window is steps W+S .. W+S+K (steps 20..119 by default: free fall,
the landing near step 28 and resting contact). `value` is the mixed path's
steps/s when its positions stay within 1e-5 (relative) of the FP64 path's on
every timed step with no admitted intersection, else the FP64 path's (the line
then says which gate failed). The reference's own budget (10 Newton, 60 PCG
iterations, PCG tolerance 1e-3) is reported beside it.

One process per GPU (torchrun for N > 1); every rank steps its own replica of
the workload (a single sheet does not shard: "replicas only", weak scaling).
Timing: per step, L2 is flushed (a 256 MiB write on the solver's stream), then
the step is bracketed by CUDA events on the solver's stream; the reported
time is the max over ranks. rank 0 prints one JSON line.
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
sys.path.insert(0, ROOT)

HBM_FALLBACK_GBS = 6650.0


def max_over_ranks(values, device, world):
    """Max of each timing over all ranks (the job is as slow as its slowest
    replica); identity when world == 1."""
    import torch
    import torch.distributed as dist
    t = torch.tensor(list(values), dtype=torch.float64, device=device)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return t.tolist()


def replica_throughput(world, steps, ms):
    """Whole-job steps/s of `world` independent replicas that each ran `steps`
    steps, timed as the slowest rank's `ms`."""
    return world * steps / (ms / 1000.0)


def measured_peak():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            j = json.load(f)
        return float(j["hbm_gbs"]), "measured"
    except Exception:
        return HBM_FALLBACK_GBS, "fallback"


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 200 ms during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.lines = []
        self.thread = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "200", "-i", str(self.dev)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()
        # nvidia-smi's start-up (NVML initialization) can stall the GPU's
        # clients for tens of ms: wait for its first sample, so the start-up
        # falls before the warm-up steps that follow, not inside timed steps.
        t0 = time.time()
        while not self.lines and time.time() - t0 < 10 and self.proc.poll() is None:
            time.sleep(0.01)

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def workload(name: str, steps_hint: int):
    from closim_b200 import configs
    if name == "floor_drape":
        return configs.floor_drape()
    if name == "strip_pull":
        return configs.strip_pull()
    if name == "sphere_drape":
        return configs.sphere_drape()
    raise SystemExit(f"unknown workload {name}")


def cpu_baseline(cfg, budget_s: float, max_steps: int):
    """The oracle (single-threaded C++ port of the reference CpuSolver) on a
    bounded sample: the first steps of the same workload, up to budget_s."""
    from tests.helpers import oracle_scene, oracle_step_kwargs
    from closim_b200 import configs
    sc = oracle_scene(cfg)
    kw = oracle_step_kwargs(cfg)
    t0 = time.perf_counter()
    k = 0
    while k < max_steps:
        sc.set_pins(configs.pins_at(cfg, k))
        sc.step(cfg["h"], **kw)
        k += 1
        if time.perf_counter() - t0 > budget_s:
            break
    dt = time.perf_counter() - t0
    return {"value": k / dt, "unit": "steps/s", "cores": 1, "kind": "port",
            "sample": f"first {k} steps of {cfg['name']} ({dt:.1f} s, 1 thread)"}


def run_reference(args, rank):
    """The reference's CPU path (the oracle, a C++ restatement of CpuSolver;
    the TypeScript itself has no runtime here) on the same workload, built
    with the oracle's own grid builder, stepped from step 0 at the reference's
    budget; timed over the CUDA arm's window start (steps W+S ..), as many
    steps as fit a bounded sample."""
    if rank != 0:
        return 0
    from oracle import oracle as O
    from closim_b200 import configs
    configs.set_grid_builder(O.build_grid)
    cfg = workload(args.workload, args.steps)
    from tests.helpers import oracle_scene, oracle_step_kwargs
    O.lib()
    sc = oracle_scene(cfg)
    kw = oracle_step_kwargs(cfg)
    start = args.warmup + args.skip
    for k in range(start):
        sc.set_pins(configs.pins_at(cfg, k))
        sc.step(cfg["h"], **kw)
    t0 = time.perf_counter()
    k = 0
    while k < args.steps and (k == 0 or time.perf_counter() - t0 < 60.0):
        sc.set_pins(configs.pins_at(cfg, start + k))
        sc.step(cfg["h"], **kw)
        k += 1
    dt = time.perf_counter() - t0
    v = k / dt
    sample = f"steps {start}..{start + k - 1} of {cfg['name']} ({dt:.1f} s, 1 thread, after {start} untimed steps)"
    line = {"metric": "sim steps/s", "value": v, "unit": "steps/s", "n_gpus": args.gpus, "steps": k,
            "warmup": args.warmup, "higher_is_better": True, "impl": "reference", "scaling": "weak",
            "dtype": "f64", "data": "synthetic (seeded)",
            "config": {"workload": cfg["name"], "n": len(cfg["x"]) // 3, "h": cfg["h"],
                       "budget": "reference (10 Newton, 60 PCG iterations, PCG tolerance 1e-3)"},
            "cpu_baseline": {"value": v, "unit": "steps/s", "cores": 1, "kind": "port", "sample": sample},
            "e2e": {"value": v, "unit": "steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "vs_baseline": None}
    print(json.dumps(line), flush=True)
    return 0


def step_algorithmic_bytes(st, mesh, precision, cfg):
    """Algorithmic bytes of one step from its measured counts (Newton
    iterations, PCG iterations, Armijo trials, contacts): per Newton iteration a
    gradient pass, per PCG iteration an HVP and the vector updates, per trial an
    energy pass, and per broadphase query the boxes, sort passes and nodes; f is
    the PCG vector width (4 mixed, 8 FP64), constants 4 B, 64 B per frozen
    contact record, 48 B per CCD candidate primitive."""
    f = 4 if precision == "mixed" else 8
    n, m, hg = mesh.count, mesh.triCount, mesh.hinges.shape[0]
    c = st.contact["activePairs"] if st.contact else 0
    cand = st.contact["candidatePairs"] if st.contact else 0
    D = (n + 7) // 8 if cfg["options"]["precond"] == "schwarz" else 0
    b_grad = (9 * f + 4) * n + 32 * m + (16 + 3 * f) * hg + 64 * c
    b_e = (6 * f + 4) * n + 32 * m + (16 + 3 * f) * hg + 64 * c
    b_hvp = (9 * f + 4) * n + 32 * m + 64 * c
    b_vec = 24 * f * n + D * 300 * 4
    newton = max(st.newtonItersUsed, 1)
    trials = st.armijoTrials
    b = newton * b_grad + st.pcgIters * (b_hvp + b_vec) + trials * b_e
    if st.contact:
        queries = newton + trials + 2
        b += queries * (6 * f * n + 12 * m + 24 * m + 8 * m + 2 * 8 * m * 4 + 2 * m * 40) + trials * 48 * cand
    return float(b)


# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) of one launch of
# the PCG kernel on the 64 x 64 floor drape, from one ncu capture of that kernel
# on that workload (not measured by this run; reported as traffic_from_profile).
PCG_DRAM_BYTES = {"k_mx_pcg_cluster": 3.418e6}


CONVERGED = dict(newtonIters=40, pcgMaxIters=3000, gradTol=1e-8)
# Relative PCG tolerance of the exact-Newton solves, on both paths: the forcing
# term of an inexact Newton method. Newton still stops only at gradTol 1e-8,
# so the converged step does not depend on it; on the config-1 drape 3e-4 was
# the fastest setting with the same Newton iteration count (1e-6: 2.81 ms per
# step, 1e-4: 2.48, 3e-4: 2.28, 1e-3 (the reference's PCG tolerance, newton.ts:148):
# 2.40 with 5% more Newton iterations), gate 1e-9.
EXACT_TOL = 3e-4
GATE_REL_ERR = 1e-5


def budget_options(cfg, budget):
    o = dict(cfg["options"])
    if budget == "converged":
        o.update(CONVERGED)
    return o


def run_path(cfg, precision, local, args, flush, budget, mode="device", sampler=None, record=False,
             profile=False):
    """Steps 0 .. W+S+K of `cfg` on one solver; the last K are timed, each
    bracketed by CUDA events on the solver's stream after an L2 flush.

    mode "device": device-resident steps (cs_step_n); "e2e": CudaSolver.step
    with the scene's pinned host arrays uploaded before and read back after
    every step (the ClothSolver call a user makes). profile: the PCG kernel's
    launches timed with events (this runs the host-driven step). Returns a dict
    with the timed milliseconds, per-step positions and contact minima of the
    timed window (record), launches, and the solver."""
    import torch
    import closim_b200 as cb
    from closim_b200 import configs
    sc = configs.make_scene(cfg)
    solver = cb.CudaSolver(precision, device=local, **budget_options(cfg, budget))
    solver.initialize(sc)
    if budget == "converged":
        solver.setNewtonMode("exact", EXACT_TOL)
    if args.no_graph:
        solver.setGraphMode(False)
    ext = torch.cuda.ExternalStream(solver.stream(), device=local)
    n = len(cfg["x"]) // 3
    if mode == "e2e":
        px = torch.empty(n * 3, dtype=torch.float64).pin_memory()
        pv = torch.empty(n * 3, dtype=torch.float64).pin_memory()
        px.numpy()[:] = sc.positions
        pv.numpy()[:] = sc.velocities
        sc.positions = px.numpy()
        sc.velocities = pv.numpy()
        solver.syncFromScene = True
    k = [0]

    def one():
        sc.pinned.clear()
        sc.pinned.update(configs.pins_at(cfg, k[0] % cfg["steps"]))
        k[0] += 1
        if mode == "e2e":
            solver.step(cfg["h"])
        else:
            solver.advance(cfg["h"], 1)

    if sampler:
        sampler.start()  # before the warm-up steps (see ClockSampler.start)
    for _ in range(args.warmup + args.skip):
        one()
    torch.cuda.synchronize()
    launches0 = solver.kernelLaunches()
    graph0 = solver.graphInfo()
    if profile:
        solver.profile(True)
    if args.profiler_range and mode == "device" and not profile:
        torch.cuda.profiler.start()  # ncu --profile-from-start off captures the timed steps only
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    total = 0.0
    pos, mind, stats = [], [], []
    step_bytes = 0.0
    mesh = sc.mesh
    for _ in range(args.steps):
        with torch.cuda.stream(ext):
            flush.fill_(1.0)
        ev0.record(ext)
        one()
        ev1.record(ext)
        ev1.synchronize()
        total += ev0.elapsed_time(ev1)
        st = solver.lastStats
        stats.append(st)
        step_bytes += step_algorithmic_bytes(st, mesh, precision, cfg)
        if st.contact:
            mind.append(st.contact["minDistance"])
        if record:
            if mode != "e2e":
                solver.pull()
            pos.append(sc.positions.copy())
    torch.cuda.synchronize()
    if args.profiler_range and mode == "device" and not profile:
        torch.cuda.profiler.stop()
    out = dict(ms=total, launches=solver.kernelLaunches() - launches0, solver=solver, scene=sc, pos=pos, mind=mind,
               stats=stats, step_bytes=step_bytes, graph=solver.graphInfo(), graph0=graph0)
    if profile:
        out["prof"] = solver.profileRead()
        out["prof"]["launch_info"] = solver.launchInfo()
        solver.profile(False)
    return out


def run_batch(args, world, rank, local):
    """512 uneven sheets stepped by the batched solver: one persistent launch
    per step, K steps graph-replayed; value = whole-job sheet-steps/s."""
    import torch
    import torch.distributed as dist
    from closim_b200 import configs
    from closim_b200.batch import BatchSolver
    sheets = configs.batch_sheets(count=args.sheets)
    h = sheets[0]["h"]
    bs = BatchSolver(sheets, device=local)
    threads = bs.autotune(h)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=f"cuda:{local}")
    ext = torch.cuda.ExternalStream(bs.stream(), device=local)
    sampler = ClockSampler(local)
    sampler.start()  # before the warm-up steps (see ClockSampler.start)
    bs.step(h, args.warmup)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    total = 0.0
    if args.profiler_range:
        torch.cuda.profiler.start()  # ncu --profile-from-start off captures the timed steps only
    for _ in range(args.steps):
        with torch.cuda.stream(ext):
            flush.fill_(1.0)
        ev0.record(ext)
        bs.step(h)
        ev1.record(ext)
        ev1.synchronize()
        total += ev0.elapsed_time(ev1)
    if args.profiler_range:
        torch.cuda.profiler.stop()
    clocks = sampler.stop()
    # graph-replayed multi-step call (the production path)
    ev0.record(ext)
    bs.step(h, args.steps)
    ev1.record(ext)
    ev1.synchronize()
    graph_ms = ev0.elapsed_time(ev1)
    st = bs.stats()
    # the same sheets stepped one by one by the single-sheet mixed solver (a
    # sample of 8, scaled to the batch by triangle count)
    import closim_b200 as cb
    sample = sheets[:: max(1, len(sheets) // 8)][:8]
    single_ms, single_m = 0.0, 0
    for cfg in sample:
        sc = configs.make_scene(dict(cfg, contact=None))  # no self-contact search in the comparison
        so = cb.CudaSolver("mixed", device=local, **dict(cfg["options"], precond="jacobi"))
        so.initialize(sc)
        so.advance(h, 2)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        so.advance(h, 3)
        torch.cuda.synchronize()
        single_ms += (time.perf_counter() - t0) * 1000.0 / 3
        single_m += len(cfg["idx"]) // 3
        so.close()
    total_m = int(sum(len(c["idx"]) // 3 for c in sheets))
    single_est_ms = single_ms * total_m / max(single_m, 1)
    total, graph_ms = max_over_ranks([total, graph_ms], f"cuda:{local}", world)
    if rank == 0:
        S = len(sheets)
        line = {"metric": "sim steps/s", "value": replica_throughput(world, args.steps, total), "unit": "steps/s",
                "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": total / args.steps,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
                "data": "synthetic (seeded)", "impl": "cuda",
                "config": {"workload": "batch_sheets", "sheets": S, "n": bs.N,
                           "m": int(sum(len(c["idx"]) // 3 for c in sheets)), "h": h,
                           "parallelism": f"replicas x{world}", "threads_per_sheet": threads,
                           "resident_blocks": bs.launchShape()["blocks"],
                           "l2": "flushed between timed steps (256 MiB write)"},
                "sheet_steps_per_s": world * S * args.steps / (total / 1000.0),
                "graph_replay": {"steps": args.steps, "ms_per_step": graph_ms / args.steps},
                "converged_sheets_last_step": int(sum(1 for x in st if x["converged"] == 1)),
                "mean_newton_iters": float(np.mean([x["newtonIters"] for x in st])),
                "mean_pcg_iters": float(np.mean([x["pcgIters"] for x in st])),
                "single_sheet_solver_ms_per_batch_step": single_est_ms,
                "single_sheet_solver_note": "8 sheets stepped one by one by the single-sheet mixed solver (Jacobi, "
                                            "no contact), scaled to the batch by triangle count",
                "speedup_vs_single_sheet_solver": single_est_ms / (total / args.steps),
                "gpu_launches": 2 * args.steps, "clocks": clocks}
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def run_material_fit(args, world, rank, local):
    """Adjoint cost: a rollout of the material-fit sheet (96 x 96, exact-Newton
    forward, checkpoints every 20 steps) and its backward; value = forward
    sim steps/s, plus the backward / forward time ratio."""
    import torch
    import closim_b200 as cb
    from closim_b200 import configs
    cfg = configs.material_fit(steps=args.rollout_steps, grad_tol=1e-9)
    sc = configs.make_scene(cfg)
    s = cb.CudaSolver("fp64", device=local, **cfg["options"])
    s.initialize(sc)
    s.setNewtonMode("exact", 1e-8)
    s.setAdjointOptions(4000, 1e-10)
    x0 = sc.positions.copy()
    ext = torch.cuda.ExternalStream(s.stream(), device=local)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    ev[0].record(ext)
    xN = s.forward(cfg["h"], cfg["steps"], cfg["checkpoint_every"]).copy()
    ev[1].record(ext)
    fwd_conv = s.adjointStats()["forwardConverged"]
    gx = 2 * (xN - x0) / (len(x0) // 3)
    dth, dv0 = s.backward(gx)
    ev[2].record(ext)
    ev[2].synchronize()
    f_ms = ev[0].elapsed_time(ev[1])
    b_ms = ev[1].elapsed_time(ev[2])
    st = s.adjointStats()
    if rank == 0:
        line = {"metric": "sim steps/s", "value": cfg["steps"] / (f_ms / 1000.0), "unit": "steps/s", "n_gpus": 1,
                "steps": cfg["steps"], "warmup": 0, "ms_per_step": f_ms / cfg["steps"], "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)", "impl": "cuda",
                "config": {"workload": "material_fit", "n": len(x0) // 3, "m": len(cfg["idx"]) // 3,
                           "checkpoint_every": cfg["checkpoint_every"], "newton": "exact, gradTol 1e-9"},
                "adjoint": {"backward_ms": b_ms, "forward_ms": f_ms, "backward_over_forward": b_ms / f_ms,
                            "forward_converged_steps": fwd_conv, "adjoint_pcg_iters": st["pcgIters"],
                            "max_rel_residual": st["maxRelResidual"],
                            "dL_dtheta": [dth["C00"], dth["C11"], dth["G"], dth["kBend"]]}}
        print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="cuda", choices=["cuda", "reference"])
    ap.add_argument("--workload", default="floor_drape",
                    choices=["floor_drape", "strip_pull", "sphere_drape", "batch_sheets", "material_fit"])
    ap.add_argument("--rollout-steps", type=int, default=40, help="material_fit: steps of the timed rollout")
    ap.add_argument("--sheets", type=int, default=512, help="batch_sheets: number of sheets (512 in the workload)")
    ap.add_argument("--skip", type=int, default=17, help="extra untimed steps before the timed region")
    ap.add_argument("--budget", default="converged", choices=["converged", "reference"],
                    help="stepper budget of the timed paths (converged: exact-Newton, both paths converge)")
    ap.add_argument("--no-reference-budget", action="store_true", help="skip the reference-budget figure")
    ap.add_argument("--small", action="store_true", help="32x32 floor drape (for profiler captures)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--paths", default="fp64,mixed,e2e,profile,refbudget",
                    help="profiler captures: run only these device-resident paths (fp64 and/or mixed), no JSON line")
    ap.add_argument("--no-graph", action="store_true",
                    help="host-driven steps instead of the captured step graph (same kernels; profilers cannot "
                         "capture kernel nodes of graphs with conditional nodes)")
    ap.add_argument("--profiler-range", action="store_true",
                    help="mark the timed steps for ncu --profile-from-start off")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank)

    import torch
    import torch.distributed as dist
    import datetime
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))

    from closim_b200 import configs
    if args.workload == "batch_sheets":
        return run_batch(args, world, rank, local)
    if args.workload == "material_fit":
        return run_material_fit(args, world, rank, local)
    if args.small:
        cfg = configs.floor_drape(nx=31, ny=31, w=0.4, hgt=0.4)
    else:
        cfg = workload(args.workload, args.steps)
    n = len(cfg["x"]) // 3
    dev = f"cuda:{local}"
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=dev)  # 256 MiB > 126 MB L2

    paths = set(args.paths.split(","))
    if paths != {"fp64", "mixed", "e2e", "profile", "refbudget"}:
        # some of the paths only (profiler captures, secondary workloads): one
        # summary line per run, not the headline line
        res = {}
        for pth in ("fp64", "mixed"):
            if pth in paths:
                r = run_path(cfg, pth, local, args, flush, args.budget, record="fp64" in paths and "mixed" in paths)
                res[pth] = r
        if rank == 0 and not args.profiler_range:
            line = {"metric": "sim steps/s", "unit": "steps/s", "impl": "cuda", "n_gpus": world,
                    "config": {"workload": cfg["name"], "n": n, "budget": args.budget,
                               "timed_steps": [args.warmup + args.skip, args.warmup + args.skip + args.steps - 1]}}
            for pth, r in res.items():
                line[pth] = {"value": args.steps / (r["ms"] / 1000.0), "ms_per_step": r["ms"] / args.steps,
                             "converged_steps": sum(1 for st in r["stats"] if st.converged),
                             "gpu_launches": r["launches"],
                             "graph_steps": r["graph"]["graphSteps"] - r["graph0"]["graphSteps"],
                             "min_distance": min(r["mind"]) if r["mind"] else None}
            if len(res) == 2:
                line["mixed_vs_fp64_rel_pos_err_max"] = max(
                    float(np.max(np.abs(b - a)) / np.max(np.abs(a))) for a, b in zip(res["fp64"]["pos"],
                                                                                    res["mixed"]["pos"]))
            print(json.dumps(line), flush=True)
        return 0
    # the FP64 path and the mixed path over the same steps and budget
    fp64 = run_path(cfg, "fp64", local, args, flush, args.budget, record=True)
    sampler = ClockSampler(local)
    mixed = run_path(cfg, "mixed", local, args, flush, args.budget, sampler=sampler, record=True)
    clocks = sampler.stop()
    e2e = run_path(cfg, "mixed", local, args, flush, args.budget, mode="e2e")
    prof = run_path(cfg, "mixed", local, args, flush, args.budget, profile=True)["prof"]
    ref_budget = None
    if args.budget == "converged" and not args.no_reference_budget:
        ref_budget = run_path(cfg, "mixed", local, args, flush, "reference")
    errs = [float(np.max(np.abs(b - a)) / np.max(np.abs(a))) for a, b in zip(fp64["pos"], mixed["pos"])]
    dmin = cfg["contact"]["dMinM"] if cfg["contact"] else None
    min_dist = min(mixed["mind"]) if mixed["mind"] else None
    gate_err = max(errs) <= GATE_REL_ERR
    gate_contact = min_dist is None or min_dist >= dmin * (1 - 1e-9)
    conv = sum(1 for st in mixed["stats"] if st.converged), sum(1 for st in fp64["stats"] if st.converged)

    times = [mixed["ms"], e2e["ms"], fp64["ms"]] + ([ref_budget["ms"]] if ref_budget else [])
    times = max_over_ranks(times, dev, world)
    mixed_ms, e2e_ms, fp64_ms = times[:3]
    if world > 1:
        dist.barrier()
    mixed_value = replica_throughput(world, args.steps, mixed_ms)
    fp64_value = replica_throughput(world, args.steps, fp64_ms)
    gate_pass = gate_err and gate_contact
    head = "mixed" if gate_pass else "fp64"
    value = mixed_value if gate_pass else fp64_value
    head_ms = mixed_ms if gate_pass else fp64_ms

    if rank == 0:
        peak, peak_kind = measured_peak()
        achieved = prof["bytes"] / prof["launches"] / (prof["ms_per_launch"] / 1000.0) / 1e9 if prof.get("launches") \
            else 0.0
        kname = prof["launch_info"]["pcgKernel"]
        n_h2d = 2 * n * 3 * 8
        line = {
            "metric": "sim steps/s", "value": value, "unit": "steps/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": head_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64" if head == "mixed" else "f64",
            "data": "synthetic (seeded)", "impl": "cuda",
            "config": {"workload": cfg["name"] + ("_32x32" if args.small else ""), "n": n, "m": len(cfg["idx"]) // 3,
                       "h": cfg["h"], "headline_path": head, "precond": cfg["options"]["precond"],
                       "budget": args.budget + (" (exact-Newton: 40 Newton, 3000 PCG iterations, gradTol 1e-8, "
                                                "PCG rel. tol 3e-4 on both paths)" if args.budget == "converged"
                                                else " (10 Newton, 60 PCG, PCG tol 1e-3)"),
                       "timed_steps": [args.warmup + args.skip, args.warmup + args.skip + args.steps - 1],
                       "parallelism": f"replicas x{world}", "l2": "flushed between timed steps (256 MiB write)",
                       "graph_steps": mixed["graph"]["graphSteps"] - mixed["graph0"]["graphSteps"]},
            "gate": {"mixed_vs_fp64_rel_pos_err_max": max(errs), "mixed_vs_fp64_rel_pos_err_last": errs[-1],
                     "limit": GATE_REL_ERR, "steps_compared": len(errs), "min_distance": min_dist, "dmin": dmin,
                     "intersection_free": gate_contact, "pass": gate_pass,
                     "converged_steps": {"mixed": conv[0], "fp64": conv[1], "of": args.steps}},
            "mixed_path": {"value": mixed_value, "ms_per_step": mixed_ms / args.steps,
                           "gpu_launches": mixed["launches"]},
            "fp64_path": {"value": fp64_value, "ms_per_step": fp64_ms / args.steps, "gpu_launches": fp64["launches"]},
            "mixed_over_fp64": mixed_value / fp64_value,
            "roofline": {"bound": "hbm", "kernel": kname, "achieved": achieved, "peak": peak,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / peak, "traffic": None,
                         "traffic_from_profile": PCG_DRAM_BYTES.get(kname) if cfg["name"] == "floor_drape" else None,
                         "launches": prof.get("launches"), "ms_per_launch": prof.get("ms_per_launch"),
                         "pcg_iters": prof.get("iters"),
                         "alg_bytes_per_launch": prof["bytes"] / max(1, prof["launches"]),
                         "timing": "CUDA events around each launch, host-driven replay of the same steps"},
            "e2e": {"value": replica_throughput(world, args.steps, e2e_ms), "unit": "steps/s",
                    "h2d_bytes_per_step": n_h2d, "d2h_bytes_per_step": n_h2d,
                    "path": "mixed, CudaSolver.step with pinned host arrays, same steps as value"},
            "gpu_launches": mixed["launches"] if head == "mixed" else fp64["launches"],
            "clocks": clocks,
            "step_roofline": {"bound": "hbm", "alg_bytes_per_step": mixed["step_bytes"] / args.steps,
                              "achieved": mixed["step_bytes"] / (mixed_ms / 1000.0) / 1e9, "peak": peak,
                              "unit": "GB/s", "frac": mixed["step_bytes"] / (mixed_ms / 1000.0) / 1e9 / peak},
        }
        if ref_budget:
            rv = replica_throughput(world, args.steps, times[3])
            line["reference_budget"] = {"value": rv, "unit": "steps/s", "ms_per_step": times[3] / args.steps,
                                        "path": "mixed, the reference's stepper budget (10 Newton, 60 PCG, "
                                                "PCG tol 1e-3): steps do not converge, so no 1e-5 comparison"}
        if world == 1 and not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(cfg, budget_s=20.0, max_steps=cfg["steps"])
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
