"""Benchmark: IMEX-DG DoF-steps/s of the flow-over-hill dynamical core on GB300.

A "step" is one full 3-stage IMEX step (Picard loops, Schur solves, stage
combination, sponge) of one member, run by the library's time loop.
Default workload: 320x160 cells, Q4 (25 nodes/cell, 5.12 M DoFs), FP64,
acoustic CFL 5.  Headline (`value`, `e2e`): the reference's algorithm on the
GPU -- Schur GMRES + Jacobi with the parameter-file eps 1e-8 -- the same
algorithm and tolerance as the CPU reference arm, with the two arms' field
difference after one step (`cpu_baseline.rel_l2_gpu_vs_cpu_after_1_step`).
Also reported: FP64 flexible GMRES + FP64 multigrid (`fp64_multigrid`) and
the same with the V-cycle in FP32 (`mixed_precision`), both at Schur rtol
1e-11 on the true residual, with the mixed path's speed-up, its field error
against FP64 on the workload and against the FP64 oracle after 200 steps of
the 40x20 member, and the roofline of its FP32 level operators.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
                  [--nx 320 --nz 160 --degree 4]

One JSON line on stdout (rank 0).  ``--impl reference`` times the CPU FP64
restatement of the reference algorithm (the oracle; the deal.II reference
cannot be built here) on the host cores for the same workload and metric.
Under torchrun (N > 1) every rank runs its own independent member
(replicas; no collective on the data path) and the timing is the max over
ranks.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "IMEX-DG DoF-steps/s"
UNIT = "DoF-steps/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--nx", type=int, default=320)
    ap.add_argument("--nz", type=int, default=160)
    ap.add_argument("--degree", type=int, default=4)
    ap.add_argument("--cfl", type=float, default=5.0)
    ap.add_argument("--eps", type=float, default=1e-11,
                    help="relative Schur tolerance (true residual) of the FGMRES variants; "
                         "1e-11 keeps the mixed path within 1e-8 of the FP64 oracle over "
                         "200 steps, 1e-10 drifts to ~1.1e-8-1.9e-8 in u")
    ap.add_argument("--precision", default="fp64", choices=["fp64"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-serving-sample", action="store_true",
                    help="leave the bounded serving sample out of the main line")
    ap.add_argument("--only-headline", action="store_true",
                    help="skip the multigrid variants (short runs, profiling)")
    ap.add_argument("--serving", action="store_true",
                    help="run a bounded sample of the ensemble-serving workload and exit")
    ap.add_argument("--serving-compare", action="store_true",
                    help="serve one ensemble with FP64 and with mixed-precision multigrid "
                         "and compare throughput and fields")
    ap.add_argument("--serving-batch", type=int, default=1,
                    help="concatenate up to this many waiting same-mesh members per context")
    ap.add_argument("--serving-rates", default="",
                    help="comma-separated Poisson rates: serving latency sweep")
    ap.add_argument("--serving-requests", type=int, default=48)
    ap.add_argument("--serving-meshes", default="40x20,80x40,160x80,320x160")
    ap.add_argument("--serving-degrees", default="2,3,4,5")
    ap.add_argument("--serving-rate", type=float, default=8.0)
    ap.add_argument("--serving-steps-scale", type=float, default=0.05)
    ap.add_argument("--amr", action="store_true",
                    help="run a bounded sample of the adaptive-mesh workload and exit")
    ap.add_argument("--amr-steps", type=int, default=200)
    ap.add_argument("--amr-every", type=int, default=50)
    ap.add_argument("--amr-nx", type=int, default=160)
    ap.add_argument("--amr-nz", type=int, default=80)
    ap.add_argument("--amr-degree", type=int, default=3)
    ap.add_argument("--amr-precision", type=int, default=1, choices=[0, 1, 2],
                    help="Schur solver of the adaptive sample: 0 the reference's GMRES + "
                         "Jacobi, 1 FP32 multigrid (default), 2 FP64 multigrid")
    ap.add_argument("--vcycle", action="store_true",
                    help="time the multigrid V-cycle of the workload alone and exit")
    ap.add_argument("--vcycle-no-graphs", action="store_true")
    ap.add_argument("--vcycle-fp64", action="store_true")
    ap.add_argument("--mg-levels", type=int, default=3)
    ap.add_argument("--mg-coarse-degree", type=int, default=6)
    ap.add_argument("--mg-smoother-degree", type=int, default=4)
    ap.add_argument("--shell", action="store_true",
                    help="time IMEX steps of the 3D spherical shell (the reference's own case, "
                         "6144 cells, degree 1) and exit")
    ap.add_argument("--fma-probe", action="store_true",
                    help="print the measured FP64/FP32 FMA peaks and exit")
    return ap.parse_args()


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


class RankGroup:
    """Barrier and max-over-ranks of the timing, on an initialised process
    group (NCCL on the GPUs; any backend works).  With one rank both are
    local.  `device` is where the reduction tensor lives ("cuda" or "cpu");
    on "cuda" the barrier also synchronises the device on both sides."""

    def __init__(self, world_size, device="cuda"):
        self.ws = int(world_size)
        self.device = device

    def _sync(self):
        if self.device == "cuda":
            import torch

            torch.cuda.synchronize()

    def barrier(self):
        self._sync()
        if self.ws > 1:
            import torch.distributed as dist

            dist.barrier()
            self._sync()

    def max(self, x):
        if self.ws == 1:
            return x
        import torch
        import torch.distributed as dist

        t = torch.tensor([float(x)], dtype=torch.float64, device=self.device)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())


def aggregate_rate(world_size, units_per_rank_per_step, steps, max_ms):
    """Whole-job throughput: the units every rank processed over the slowest
    rank's time (weak scaling: each rank advances its own member)."""
    return world_size * units_per_rank_per_step * steps / (max_ms * 1e-3)


def workload(args):
    return {"workload": f"flow-over-hill {args.nx}x{args.nz} Q{args.degree} FP64, acoustic "
                        f"CFL {args.cfl:g}, reference solver (GMRES + Jacobi, eps 1e-8)",
            "nx": args.nx, "nz": args.nz, "degree": args.degree,
            "dofs": 4 * args.nx * args.nz * (args.degree + 1) ** 2,
            "l2_policy": "working set (state, stage vectors, geometry, cell inverses) "
                         "is larger than the 129 MB L2; no flush between steps",
            "parallelism": "one member per GPU (replicas)"}


def gpu_uuid(device):
    """nvidia-smi id ("GPU-<uuid>") of CUDA device `device` of this process."""
    try:
        import torch

        return "GPU-" + str(torch.cuda.get_device_properties(device).uuid)
    except Exception:
        return str(device)


class ClockSampler:
    """nvidia-smi clocks/throttle sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device=0):
        # nvidia-smi numbers GPUs physically and ignores CUDA_VISIBLE_DEVICES:
        # name the CUDA device in use by its UUID
        self.index = gpu_uuid(device)
        self.proc = None
        import tempfile

        self.path = os.path.join(tempfile.gettempdir(), f"atm_clocks_{os.getpid()}.csv")

    def __enter__(self):
        try:
            os.makedirs(os.path.dirname(self.path), exist_ok=True)
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.fh, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
            self.fh.close()

    def summary(self):
        if self.proc is None or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for name, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        try:
            os.remove(self.path)
        except OSError:
            pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax),
                "reasons": sorted(reasons), "samples": len(sm)}


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as fh:
            d = json.load(fh)
        return d.get("hbm_gbs", 6800.0), "measured"
    return 6800.0, "fallback"


# FP64 FMA throughput of the GB300 (1255 GFLOP/s, measured with the
# independent-chain DFMA probe of `bench.py --fma-probe`)
FP64_PEAK_TFLOPS = 1.255
# DRAM bytes (read + write) per cell and launch of the dominant kernel families,
# from single-kernel `ncu` captures of the S apply at 320x160 Q4: 207.4 MB per
# k_exact_face_C and k_exact_CD pair and 339.1 MB per k_exact_B<4,2> launch over
# 51,200 cells; the traffic grows in proportion to the cell count.
NCU_TRAFFIC_PER_CELL = {4: {"CD": 207.4e6 / 51200, "B": 339.1e6 / 51200}}


def cpu_baseline(case, eps, gpu_state=None):
    """FP64 CPU restatement (oracle) on all host cores: one IMEX step.  With
    `gpu_state` (the GPU's fields after one step from the same initial state
    and setting), also the relative L2 difference of the two arms."""
    from oracle.oracle import OracleSolver, num_threads

    s = OracleSolver(case, eps=eps, inner_tol=1e-12)
    t0 = time.perf_counter()
    s.run(1)
    dt = time.perf_counter() - t0
    out = {"value": case.n_dofs / dt, "unit": UNIT, "cores": num_threads(), "kind": "port",
           "sample": f"1 IMEX step of the same {case.params.nx}x{case.params.nz} "
                     f"Q{case.degree} member ({dt:.2f} s), CPU FP64 restatement of the "
                     f"reference algorithm (nested CG A^-1 in the Schur apply)"}
    if gpu_state is not None:
        out["rel_l2_gpu_vs_cpu_after_1_step"] = {
            name: float(np.linalg.norm(a - b) / np.linalg.norm(b))
            for name, a, b in zip(("rho", "u", "p"), gpu_state, s.get_state())}
    return out


def config1_accuracy(precision, eps):
    """Fields of the 40x20 Q4 member after 200 GPU steps against the FP64
    oracle's (the committed fixture tests/golden/oracle_hill_c1_k4.npz, Schur
    solves at a true residual of ~1e-13): relative L2 per field."""
    from atmospheric_flows_gb300.euler_solver import EulerSolver
    from atmospheric_flows_gb300.hill import HillParams, build_case

    path = os.path.join(ROOT, "tests", "golden", "oracle_hill_c1_k4.npz")
    if not os.path.exists(path):
        return {"note": "oracle fixture missing"}
    ref = np.load(path)
    case = build_case(HillParams(nx=40, nz=20, degree=4, cfl=5.0))
    g = EulerSolver(case, eps=eps, precision=precision, true_residual_check=precision != 0)
    g.run(int(ref["steps"]))
    err = {name: float(np.linalg.norm(a - ref[name]) / np.linalg.norm(ref[name]))
           for name, a in zip(("rho", "u", "p"), g.get_state())}
    g.close()
    return {"workload": "flow-over-hill 40x20 Q4, CFL 5, 200 steps, same solver and rtol",
            "rel_l2": err}


def level_roofline(case, eps):
    """Roofline of the multigrid level operators (the FP32 B + A^-1 and C/D
    pair of every smoothing step and residual) of the mixed path: one IMEX
    step with the V-cycle launched kernel by kernel (a captured graph hides
    its kernels from the per-launch timers), CUDA events on the library's
    stream; algorithmic bytes per pair as the library counts them."""
    from atmospheric_flows_gb300 import _lib
    from atmospheric_flows_gb300.euler_solver import EulerSolver

    fams = _lib.KERNEL_FAMILIES
    g = EulerSolver(case, eps=eps, precision=1, true_residual_check=True)
    g.op.set_mg_graphs(False)
    g.run(1)
    h = g.op.handle
    nfam = len(fams)
    _lib.call("atm_timing_enable", h, 1)
    g.run(1)
    ms = (ctypes.c_double * nfam)()
    cnt = (ctypes.c_long * nfam)()
    byt = (ctypes.c_double * nfam)()
    flp = (ctypes.c_double * nfam)()
    _lib.call("atm_timing_read", h, ms, cnt, byt, flp, nfam)
    g.close()
    i = fams.index("mg_level_apply")
    avg = ms[i] / max(cnt[i], 1)
    gbs = byt[i] / max(cnt[i], 1) / (avg * 1e-3) / 1e9
    peak, kind = measured_peaks()
    return {"bound": "hbm", "kernel": "mg_level_apply (FP32 k_exact_B<K,2,float> + k_exact_CD<K,1|4,float>, "
            "all levels)", "achieved": gbs, "peak": peak, "unit": "GB/s", "frac": gbs / peak,
            "peak_source": kind, "avg_pair_ms": avg, "pairs": int(cnt[i]),
            "algorithmic_bytes_per_pair": byt[i] / max(cnt[i], 1),
            "vcycle_ms": ms[fams.index("mg_vcycle")] / max(cnt[fams.index("mg_vcycle")], 1)}


def run_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0:
        return 0
    from atmospheric_flows_gb300.hill import HillParams, build_case
    from oracle.oracle import OracleSolver, num_threads

    case = build_case(HillParams(nx=args.nx, nz=args.nz, degree=args.degree, cfl=args.cfl))
    # the reference's algorithm with its parameter-file tolerance
    # (parameter-file.prm:23), as the CPU baseline of the GPU line
    s = OracleSolver(case, eps=1e-8, inner_tol=1e-12)
    for _ in range(args.warmup):
        s.run(1)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        s.run(1)
    el = time.perf_counter() - t0
    v = case.n_dofs * args.steps / el
    cores = num_threads()
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT,
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * el / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": workload(args),
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": f"{args.steps} IMEX steps of the workload after "
                                       f"{args.warmup} warm-up steps, CPU FP64 restatement "
                                       "of the reference (deal.II is not installable here)"},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def run_variant(case, precision, eps, check, steps, warmup, barrier, timing):
    """Warm up, then time `steps` IMEX steps of one solver variant."""
    import torch

    from atmospheric_flows_gb300 import _lib
    from atmospheric_flows_gb300.euler_solver import EulerSolver

    L = _lib.load()
    solver = EulerSolver(case, eps=eps, precision=precision, true_residual_check=check)
    h = solver.op.handle
    for _ in range(warmup):
        solver.run(1)
    start = solver.get_state()  # the end-to-end run repeats the timed steps from here
    barrier()
    nfam = len(_lib.KERNEL_FAMILIES)
    if timing:
        _lib.call("atm_timing_enable", h, 1)
    launches0 = L.atm_kernel_launches()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    barrier()
    ev0.record()
    solver.run(steps)
    ev1.record()
    barrier()
    out = {"el_ms": ev0.elapsed_time(ev1), "launches": L.atm_kernel_launches() - launches0,
           "solver": solver, "stats": solver.stats(), "state": solver.get_state(),
           "start_state": start}
    if timing:
        ms = (ctypes.c_double * nfam)()
        cnt = (ctypes.c_long * nfam)()
        byt = (ctypes.c_double * nfam)()
        flp = (ctypes.c_double * nfam)()
        _lib.call("atm_timing_read", h, ms, cnt, byt, flp, nfam)
        _lib.call("atm_timing_enable", h, 0)
        out.update(ms=list(ms), cnt=list(cnt), byt=list(byt), flp=list(flp))
    return out


def run_gb300(args):
    import torch

    ws, rank, local = dist_env()
    if ws > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    else:
        torch.cuda.set_device(0)
    from atmospheric_flows_gb300 import _lib
    from atmospheric_flows_gb300.hill import HillParams, build_case

    case = build_case(HillParams(nx=args.nx, nz=args.nz, degree=args.degree, cfl=args.cfl))

    group = RankGroup(ws, "cuda")
    barrier = group.barrier

    def rate(ms):
        return aggregate_rate(ws, case.n_dofs, args.steps, group.max(ms))

    # ---- headline: the reference's solver and tolerance on the GPU --------
    with ClockSampler(local) as clk:
        main = run_variant(case, 0, 1e-8, False, args.steps, args.warmup, barrier, True)
    value = rate(main["el_ms"])
    solver = main["solver"]
    h = solver.op.handle
    # ---- end-to-end through the ABI with pinned host buffers: the same K
    # steps as the device-timed run (from its post-warm-up state), each with
    # its state uploaded from and read back to the host
    ns = solver.n_scalar
    host = {k: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
            for k, n in (("rho", ns), ("u", 2 * ns), ("p", ns))}
    r0, u0, p0 = main["start_state"]
    host["rho"][:] = r0
    host["u"][:] = u0
    host["p"][:] = p0
    dp = ctypes.POINTER(ctypes.c_double)
    ptrs = [host[k].ctypes.data_as(dp) for k in ("rho", "u", "p")]
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        _lib.call("atm_solver_set_state", h, *ptrs)
        _lib.call("atm_solver_run", h, 1)
        _lib.call("atm_solver_get_state", h, *ptrs)
    barrier()
    e2e_s = group.max(time.perf_counter() - t0)
    # the copies alone (upload and read-back of one state), for the record
    t0 = time.perf_counter()
    for _ in range(args.steps):
        _lib.call("atm_solver_set_state", h, *ptrs)
        _lib.call("atm_solver_get_state", h, *ptrs)
    copy_s = time.perf_counter() - t0
    e2e = {"value": ws * case.n_dofs * args.steps / e2e_s, "unit": UNIT,
           "h2d_bytes_per_step": int(8 * 4 * ns), "d2h_bytes_per_step": int(8 * 4 * ns),
           "ms_per_step": e2e_s * 1e3 / args.steps,
           "copy_ms_per_step": copy_s * 1e3 / args.steps}
    solver.close()
    variants = {}
    if not args.only_headline:
        # ---- FP64 FGMRES + FP64 multigrid vs the same with an FP32 V-cycle,
        # both Schur rtol args.eps on the true residual, same start, same steps
        f64 = run_variant(case, 2, args.eps, True, args.steps, args.warmup, barrier, True)
        mix = run_variant(case, 1, args.eps, True, args.steps, args.warmup, barrier, True)
        f64["solver"].close()
        mix["solver"].close()
        errs = {}
        for name, a, b_ in zip(("rho", "u", "p"), mix["state"], f64["state"]):
            errs[name] = float(np.linalg.norm(a - b_) / np.linalg.norm(b_))
        for key, v in (("fp64_multigrid", f64), ("mixed_precision", mix)):
            st = v["stats"]
            variants[key] = {"value": rate(v["el_ms"]), "unit": UNIT,
                             "ms_per_step": v["el_ms"] / args.steps,
                             "picard_per_step": st["picard_total"] / max(st["steps"], 1),
                             "krylov_per_step": st["krylov_total"] / max(st["steps"], 1),
                             "vcycle_ms_per_step": v["ms"][10] / args.steps}
        variants["fp64_multigrid"]["scheme"] = (
            f"FP64 FGMRES(16) + FP64 multigrid V-cycle (Chebyshev 4), Schur rtol {args.eps:g} "
            "on the true residual")
        variants["mixed_precision"]["scheme"] = (
            f"FP64 FGMRES(16) + FP32 multigrid V-cycle (Chebyshev 4), Schur rtol {args.eps:g} "
            "on the true residual")
        variants["mixed_precision"]["speedup_vs_fp64_multigrid"] = (
            variants["mixed_precision"]["value"] / variants["fp64_multigrid"]["value"])
        variants["mixed_precision"]["rel_l2_vs_fp64_after_steps"] = errs
        variants["mixed_precision"]["steps_compared"] = args.steps + args.warmup
        if rank == 0:
            variants["mixed_precision"]["error_vs_fp64_oracle"] = config1_accuracy(1, args.eps)
            variants["mixed_precision"]["roofline"] = level_roofline(case, args.eps)
    if rank != 0:
        if ws > 1:
            torch.distributed.destroy_process_group()
        return 0
    # ---------------------------------------------------------- roofline --
    fams = _lib.KERNEL_FAMILIES
    ms, cnt, byt, flp = main["ms"], main["cnt"], main["byt"], main["flp"]
    cand = [i for i in range(len(fams)) if fams[i] != "mg_vcycle"]  # nested region
    dom = max(cand, key=lambda i: ms[i])
    avg_ms = ms[dom] / max(cnt[dom], 1)
    gbs = byt[dom] / max(cnt[dom], 1) / (avg_ms * 1e-3) / 1e9
    tflops = flp[dom] / max(cnt[dom], 1) / (avg_ms * 1e-3) / 1e12
    peak, peak_kind = measured_peaks()
    traffic = os.environ.get("ATM_NCU_TRAFFIC_BYTES")
    if traffic is None and args.degree in NCU_TRAFFIC_PER_CELL and \
            fams[dom] in NCU_TRAFFIC_PER_CELL[args.degree]:
        traffic = NCU_TRAFFIC_PER_CELL[args.degree][fams[dom]] * case.n_cells
    total_ms = sum(ms[i] for i in cand)
    roofline = {"bound": "hbm", "kernel": fams[dom], "achieved": gbs, "peak": peak,
                "unit": "GB/s", "frac": gbs / peak, "peak_source": peak_kind,
                "traffic": float(traffic) if traffic else None,
                "algorithmic_bytes_per_launch": byt[dom] / max(cnt[dom], 1),
                "avg_launch_ms": avg_ms, "launches": int(cnt[dom]),
                "fp64": {"achieved_tflops": tflops, "peak_tflops": FP64_PEAK_TFLOPS,
                         "frac": tflops / FP64_PEAK_TFLOPS,
                         "note": "FP64 FMA pipe is the binding limit on GB300"},
                "families": {fams[i]: {"ms": ms[i], "launches": int(cnt[i]),
                                       "share": ms[i] / max(total_ms, 1e-30),
                                       "gbs": byt[i] / max(ms[i] * 1e-3, 1e-30) / 1e9,
                                       "fp64_tflops": flp[i] / max(ms[i] * 1e-3, 1e-30) / 1e12}
                             for i in range(len(fams)) if cnt[i]}}
    cpu = None
    if not args.no_cpu_baseline:
        try:
            from atmospheric_flows_gb300.euler_solver import EulerSolver

            g1 = EulerSolver(case, eps=1e-8)  # the headline setting, one step
            g1.run(1)
            first = g1.get_state()
            g1.close()
            cpu = cpu_baseline(case, 1e-8, first)
        except Exception as exc:  # the baseline must not kill the GPU line
            cpu = {"value": None, "unit": UNIT, "cores": None, "kind": "port",
                   "sample": f"failed: {exc}"}
    serving_sub = None
    if not args.only_headline and not args.no_serving_sample:
        try:
            serving_sub = serving_sample()
        except Exception as exc:  # the sample must not kill the GPU line
            serving_sub = {"note": f"failed: {exc}"}
    st = main["stats"]
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": main["el_ms"] / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": workload(args), "e2e": e2e,
            "gpu_launches": int(main["launches"]), "roofline": roofline, "cpu_baseline": cpu,
            "autotune": [{k: r[k] for k in ("family", "mode", "cells_per_block")}
                         for r in _lib.autotune_table()
                         if r["degree"] == args.degree and r["bytes"] == 8 and not r["hanging"]
                         and r["log2_cells"] == int(np.log2(case.n_cells))],
            "clocks": clk.summary(),
            "solver": {"scheme": "the reference's Schur solver on the GPU: GMRES(28) + Jacobi on "
                                 "diag(D), eps 1e-8 (parameter-file.prm) on the Jacobi-scaled "
                                 "residual; mass-type systems solved exactly per cell",
                       "picard_per_step": st["picard_total"] / max(st["steps"], 1),
                       "krylov_per_step": st["krylov_total"] / max(st["steps"], 1),
                       "solve_fail": st["solve_fail"]},
            **variants}
    if serving_sub is not None:
        line["serving"] = serving_sub
    print(json.dumps(line), flush=True)
    if ws > 1:
        torch.distributed.destroy_process_group()
    return 0


def serving_sample():
    """A bounded sample of the ensemble-serving workload for the main line:
    16 Poisson requests at 4/s, meshes 40x20 and 80x40, degrees 2-3, 100-400
    steps scaled by 0.1, mixed-precision solver, batches of up to 4 waiting
    requests (member-wise solves).  p50/p95/p99 latency and aggregate
    DoF-steps/s."""
    from atmospheric_flows_gb300.serving import Server, make_requests, summarize

    reqs = make_requests(n=16, rate=4.0, seed=0, steps_scale=0.1, meshes=((40, 20), (80, 40)),
                         degrees=(2, 3))
    srv = Server(hbm_budget=150e9, max_running=32, batch_size=4)
    res = srv.run(reqs)
    out = summarize(res, srv.makespan)
    out.update({"sample": "16 requests, Poisson 4/s, meshes 40x20/80x40, k 2-3, steps 100-400 "
                          "x 0.1, FGMRES + FP32 multigrid rtol 1e-8, batches of up to 4",
                "batches": len(srv.batches),
                "members_per_batch_mean": float(np.mean(srv.batches)) if srv.batches else 0.0})
    return out


def vcycle_sample(args):
    """Time the multigrid V-cycle of the workload alone: the Schur operator of
    IMEX stage 1 with rho_fix and p_fix perturbed by 1e-3, `--warmup`
    V-cycles, then `--steps` timed ones (CUDA events), launched kernel by
    kernel with `--vcycle-no-graphs` (for per-launch profiles) or replayed as
    a captured graph.  Prints ms per V-cycle and the residual reduction of one
    V-cycle on S x = b for a random x."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage
    from atmospheric_flows_gb300.hill import HillParams, build_case, mg_hierarchy

    case = build_case(HillParams(nx=args.nx, nz=args.nz, degree=args.degree, cfl=args.cfl))
    op = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    levels = mg_hierarchy(case.params, max_levels=args.mg_levels)
    for lv in levels:
        op.add_mg_level(lv)
    op.set_mg_smoother(degree=args.mg_smoother_degree, coarse_degree=args.mg_coarse_degree)
    rng = np.random.default_rng(3)

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")

    op.set_rho_for_fixed(dev(case.rho * (1 + 1e-3 * rng.standard_normal(case.rho.shape))))
    op.set_pres_fixed(dev(case.p * (1 + 1e-3 * rng.standard_normal(case.p.shape))))
    op.set_HYPERBOLIC_stage(1)
    op.set_NS_stage(2)
    op.set_mg_graphs(not args.vcycle_no_graphs)
    prec = 2 if args.vcycle_fp64 else 1
    x = dev(rng.standard_normal(op.n_scalar))
    b = torch.empty_like(x)
    op.vmult(b, x)
    z = torch.empty_like(x)
    for _ in range(args.warmup):
        op.mg_vcycle(z, b, prec)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        op.mg_vcycle(z, b, prec)
    e1.record()
    torch.cuda.synchronize()
    r = torch.empty_like(x)
    op.vmult(r, z)
    print(json.dumps({"metric": "multigrid V-cycle time", "unit": "ms",
                      "value": e0.elapsed_time(e1) / args.steps,
                      "precision": "fp64" if prec == 2 else "fp32",
                      "graphs": not args.vcycle_no_graphs, "levels": len(levels) + 1,
                      "max_levels": args.mg_levels, "coarse_degree": args.mg_coarse_degree,
                      "smoother_degree": args.mg_smoother_degree,
                      "residual_reduction": ((b - r).norm() / b.norm()).item(),
                      "config": {"workload": f"Schur operator of {args.nx}x{args.nz} "
                                             f"Q{args.degree}"}}), flush=True)
    op.close()
    return 0


def fma_probe():
    import torch

    from atmospheric_flows_gb300 import _lib

    torch.cuda.set_device(0)
    f64, f32 = ctypes.c_double(), ctypes.c_double()
    _lib.call("atm_probe_fma_peak", ctypes.byref(f64), ctypes.byref(f32))
    print(json.dumps({"fp64_fma_gflops": f64.value, "fp32_fma_gflops": f32.value,
                      "ratio": f32.value / f64.value}), flush=True)
    return 0


def serving(args):
    """Ensemble-serving sample: Poisson arrivals, mesh/degree/parameter
    draws of the serving workload, continuous batching under an HBM budget."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300.serving import Server, make_requests, summarize

    meshes = tuple(tuple(int(v) for v in m.split("x")) for m in args.serving_meshes.split(","))
    degrees = tuple(int(k) for k in args.serving_degrees.split(","))
    reqs = make_requests(n=args.serving_requests, rate=args.serving_rate, seed=0,
                         steps_scale=args.serving_steps_scale, meshes=meshes, degrees=degrees)
    srv = Server(hbm_budget=150e9, max_running=32, batch_size=args.serving_batch)
    res = srv.run(reqs)
    s = summarize(res, srv.makespan)
    s.update({"metric": "ensemble serving latency / aggregate DoF-steps/s", "unit": "s",
              "batch_size": args.serving_batch, "batches": len(srv.batches),
              "members_per_batch_mean": float(np.mean(srv.batches)) if srv.batches else 0.0,
              "requests_sample": f"{args.serving_requests} requests, Poisson rate "
                                 f"{args.serving_rate}/s, steps 100-400 scaled by "
                                 f"{args.serving_steps_scale}, meshes {args.serving_meshes}, "
                                 f"k {args.serving_degrees}",
              "hbm_budget_gb": 150, "peak_running": srv.peak_running,
              "peak_reserved_gb": srv.peak_bytes / 1e9,
              "solver": "FP64 state, FGMRES + FP32 multigrid, rtol 1e-8 true residual"})
    print(json.dumps(s), flush=True)
    return 0


def serving_sweep(args):
    """The serving sample at several Poisson rates: p50/p95/p99 latency, mean
    queue wait and aggregate throughput per rate.  A rate is sustained when
    the server drains: its makespan ends within the lowest rate's p99 latency
    after the last arrival (admission never backs up here, so a backlog
    shows as members slowed by sharing the GPU).  The p99 at the highest
    sustained rate is the headline latency."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300.serving import Server, make_requests, summarize

    meshes = tuple(tuple(int(v) for v in m.split("x")) for m in args.serving_meshes.split(","))
    degrees = tuple(int(k) for k in args.serving_degrees.split(","))
    rows = []
    for rate in (float(r) for r in args.serving_rates.split(",")):
        reqs = make_requests(n=args.serving_requests, rate=rate, seed=0,
                             steps_scale=args.serving_steps_scale, meshes=meshes,
                             degrees=degrees)
        srv = Server(hbm_budget=150e9, max_running=32, batch_size=args.serving_batch)
        res = srv.run(reqs)
        s = summarize(res, srv.makespan)
        last = max(r.arrival for r in reqs)
        rows.append({"rate_per_s": rate, "last_arrival_s": last, **{k: s[k] for k in (
            "completed", "p50_latency_s", "p95_latency_s", "p99_latency_s", "mean_queue_wait_s",
            "aggregate_dof_steps_per_s", "makespan_s")}})
        print(json.dumps(rows[-1]), file=sys.stderr, flush=True)  # partial progress
    rows.sort(key=lambda r: r["rate_per_s"])
    ref_p99 = rows[0]["p99_latency_s"]
    kept = [r for r in rows if r["completed"] == args.serving_requests
            and r["makespan_s"] - r["last_arrival_s"] <= ref_p99]
    sustained = max(kept, key=lambda r: r["rate_per_s"]) if kept else None
    print(json.dumps({
        "metric": "ensemble serving latency by request rate", "unit": "s",
        "sustained_rate_per_s": sustained["rate_per_s"] if sustained else None,
        "p99_latency_at_sustained_s": sustained["p99_latency_s"] if sustained else None,
        "rates": rows,
        "sample": f"{args.serving_requests} requests per rate, steps 100-400 scaled by "
                  f"{args.serving_steps_scale}, meshes {args.serving_meshes}, k "
                  f"{args.serving_degrees}, mixed-precision solver rtol 1e-8, HBM budget "
                  f"150 GB, batch size {args.serving_batch}",
        "sustained_rule": "highest rate whose makespan ends within the lowest rate's p99 "
                          "after the last arrival, every request done"}),
          flush=True)
    return 0


def serving_compare(args):
    """The same ensemble served twice -- FP64 multigrid (precision 2) and the
    mixed-precision solver (FP32 V-cycle, precision 1), both at Schur rtol
    `--eps` on the true residual -- with aggregate throughput of each, the
    speed-up, and every member's final-field error of the mixed run against
    the FP64 run."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300.serving import Server, make_requests, summarize

    out = {}
    states = {}
    for prec in (2, 1):
        reqs = make_requests(n=args.serving_requests, rate=args.serving_rate, seed=1,
                             steps_scale=args.serving_steps_scale, precision=prec,
                             eps=args.eps)
        srv = Server(hbm_budget=150e9, max_running=32, keep_state=True)
        res = srv.run(reqs, time_scale=0.0)  # all requests present at t = 0
        s = summarize(res, srv.makespan)
        out["fp64_multigrid" if prec == 2 else "mixed_precision"] = {
            k: s[k] for k in ("completed", "failed", "aggregate_dof_steps_per_s", "makespan_s",
                              "p50_latency_s", "p99_latency_s")}
        states[prec] = {r.request_id: r.state for r in res if r.state is not None}
    errs = {"rho": [], "u": [], "p": []}
    for rid, st2 in states[2].items():
        st1 = states[1].get(rid)
        if st1 is None:
            continue
        for name, a, b in zip(("rho", "u", "p"), st1, st2):
            errs[name].append(float(np.linalg.norm(a - b) / np.linalg.norm(b)))
    out.update({
        "metric": "ensemble DoF-steps/s, mixed precision vs FP64 multigrid on the same members",
        "unit": UNIT,
        "speedup_mixed_vs_fp64": out["mixed_precision"]["aggregate_dof_steps_per_s"] /
        out["fp64_multigrid"]["aggregate_dof_steps_per_s"],
        "members_compared": len(errs["rho"]),
        "max_rel_l2_mixed_vs_fp64": {k: max(v) if v else None for k, v in errs.items()},
        "sample": f"{args.serving_requests} requests all present at t = 0, meshes 40x20..320x160, "
                  f"k 2-5, steps 100-400 scaled by {args.serving_steps_scale}, Schur rtol "
                  f"{args.eps:g} on the true residual"})
    print(json.dumps(out), flush=True)
    return 0


def adaptive(args):
    """Adaptive-mesh sample: a flow-over-hill member on a 2:1 mesh refined by
    |grad theta'| (top 10%, two levels) and re-adapted every `--amr-every`
    steps.  `value` is DoF-steps/s of the device steps (CUDA events around
    each chunk of steps, the DoFs of the mesh the chunk ran on); the host
    re-adaptation (indicator, quadtree, transfer, new context) is timed apart
    and folded into `wall_value`."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300 import amr
    from atmospheric_flows_gb300.hill import HillParams

    p = HillParams(nx=args.amr_nx, nz=args.amr_nz, degree=args.amr_degree, cfl=args.cfl,
                   theta_noise=0.1, seed=1000)
    ap = amr.AdaptParams(max_level=2, every=args.amr_every)
    prec = args.amr_precision
    eps = 1e-8 if prec == 0 else args.eps
    t0 = time.perf_counter()
    m = amr.AdaptiveMember(p, ap, eps=eps, precision=prec)
    setup_s = time.perf_counter() - t0
    m.solver.run(args.warmup)
    torch.cuda.synchronize()
    gpu_ms, work, host_s, cells, hang = 0.0, 0.0, [], [], []
    tot = {"picard_total": 0.0, "krylov_total": 0.0, "solve_fail": 0.0, "vcycles": 0.0,
           "steps": 0.0}
    st0 = m.solver.stats()
    left = args.amr_steps
    while left > 0:
        n = min(left, ap.every)
        cells.append(m.case.n_cells)
        hang.append(int(np.count_nonzero(m.case.inner_faces[:, 4])) // 2)
        a = torch.cuda.Event(enable_timing=True)
        b = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        m.solver.run(n)
        b.record()
        torch.cuda.synchronize()
        gpu_ms += a.elapsed_time(b)
        work += m.n_dofs * n
        left -= n
        st = m.solver.stats()
        for key in tot:
            tot[key] += st[key] - st0.get(key, 0.0)
        st0 = {}
        if left > 0:
            t1 = time.perf_counter()
            m.adapt()
            host_s.append(time.perf_counter() - t1)
            st0 = m.solver.stats()  # the new context starts from the clock only
            for key in tot:
                if key != "steps":
                    st0[key] = 0.0
    st = tot
    d = m.solver.diagnostics()
    m.close()
    wall = gpu_ms * 1e-3 + sum(host_s)
    print(json.dumps({
        "metric": "adaptive IMEX-DG DoF-steps/s", "value": work / (gpu_ms * 1e-3),
        "unit": UNIT, "wall_value": work / wall, "steps": args.amr_steps,
        "warmup": args.warmup, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"flow-over-hill {p.nx}x{p.nz} Q{p.degree} base mesh, 2 "
                               f"refinement levels (|grad theta'| above the 90% quantile), "
                               f"re-adapted every {ap.every} steps, "
                               + ("reference Schur solver eps 1e-8" if prec == 0 else
                                  f"FP64 FGMRES + {'FP32' if prec == 1 else 'FP64'} multigrid "
                                  f"on the adaptive hierarchy, rtol {eps:g} true residual")
                               + ", theta' noise 0.1 K",
                   "dt": m.dt, "dt_note": "acoustic CFL of the finest admissible level"},
        "cells_per_chunk": cells, "hanging_faces_per_chunk": hang,
        "adaptations": len(host_s), "adapt_host_s_mean": float(np.mean(host_s)) if host_s else 0.0,
        "setup_s": setup_s, "solve_fail": st["solve_fail"],
        "picard_per_step": st["picard_total"] / max(st["steps"], 1),
        "krylov_per_step": st["krylov_total"] / max(st["steps"], 1),
        "vcycles_per_step": st["vcycles"] / max(st["steps"], 1),
        "min_rho": d["min_rho"], "max_velocity": d["max_velocity"]}), flush=True)
    return 0


def shell_sample(args):
    """IMEX steps of the reference's own 3D case on the GPU: the cubed-sphere
    shell of 6 x 16 x 16 x 4 = 6144 cells (concentric_hyper_shells refined
    three times has as many), 10 km thick, FE_DGQ(1), dt 8.64 s, GMRES +
    Jacobi Schur solves to eps 1e-12 on the scaled rule with the true-residual
    check.  `--warmup` untimed steps, then `--steps` timed ones (the solver
    synchronises with the host inside every step, so the wall clock times
    them); DoFs = 5 fields x 8 vertex values per cell."""
    import torch

    torch.cuda.set_device(0)
    from atmospheric_flows_gb300.shell import EARTH_A, ShellParams, ShellSolver, build_shell

    case = build_shell(ShellParams(n=16, nr=4, r_in=EARTH_A, r_out=EARTH_A + 1.0e4))
    g = ShellSolver(case, eps=1e-12, scaled_tol=True, true_residual_check=True)
    g.run(args.warmup)
    s0 = g.stats()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    g.run(args.steps)
    torch.cuda.synchronize()
    el = time.perf_counter() - t0
    s1 = g.stats()
    g.close()
    dofs = 5 * 8 * case.n_cells
    print(json.dumps({"metric": "3D shell IMEX DoF-steps/s", "value": dofs * args.steps / el,
                      "unit": "DoF-steps/s", "s_per_step": el / args.steps, "steps": args.steps,
                      "warmup": args.warmup, "dtype": "f64", "data": "synthetic",
                      "krylov_per_step": (s1["krylov_total"] - s0["krylov_total"]) / args.steps,
                      "picard_per_step": (s1["picard_total"] - s0["picard_total"]) / args.steps,
                      "config": {"workload": "cubed-sphere shell 6x16x16x4 = 6144 cells, "
                                             "10 km, FE_DGQ(1), dt 8.64 s, GMRES + Jacobi "
                                             "eps 1e-12 (scaled rule, true residual)",
                                 "dofs": dofs}}), flush=True)
    return 0


def main():
    args = parse()
    if args.fma_probe:
        return fma_probe()
    if args.shell:
        return shell_sample(args)
    if args.vcycle:
        return vcycle_sample(args)
    if args.serving_compare:
        return serving_compare(args)
    if args.serving_rates:
        return serving_sweep(args)
    if args.serving:
        return serving(args)
    if args.amr:
        return adaptive(args)
    if args.impl == "reference":
        return run_reference(args)
    return run_gb300(args)


if __name__ == "__main__":
    sys.exit(main())
