#!/usr/bin/env python
"""Benchmark: CPR-GMRES time to FP64 relative residual 1e-6 on one B200,
mixed precision + learned settings against the plain FP64 GPU path.

Workload (the configuration the headline metric is quoted on): the 1.12M-cell
channelised two-phase reservoir Jacobian -- 60x220x85 grid, 2x2 BSR blocks,
7.78M stored blocks, seed 1 -- decoupled by ABF and solved by CPR-GMRES(30)
(AMG V(1,1) on pressure + 3 block-Gauss-Seidel sweeps).  The data are the
seeded synthetic system of jxpamg_all_b200.synth (the reference's SPE10 inputs
are not available).

One step = one solve from x0 = 0 to FP64 rel-res <= 1e-6 (GMRES confirms the
true residual b - A x in FP64 before it reports convergence).
  value : device-resident solve with the measured path (FP32 preconditioner,
          learned per-level strength thresholds and Chebyshev intervals, the
          stage-2 weights of the reference's mixed-precision driver, flexible
          FP64 GMRES run on the device as one CUDA graph with its Krylov basis
          stored in FP32), seconds;
          details.plain_fp64_s is the same measurement for the plain FP64 path
          (the reference's CPR weights, host-driven MGS GMRES) and
          details.speedup_vs_plain_fp64 their ratio; details.*same_driver* is
          the plain FP64 preconditioner under the measured path's weights and
          GMRES driver (what precision + learned settings alone gain), and
          details.hybrid_* the reference's hybrid form (FP32 stage 1, FP64
          stage-2 polish).
  e2e   : the measured path through the public C ABI from pinned host buffers,
          timed per step from the host->device upload of the matrix and b,
          through decoupling, CPR setup and solve, to the device->host read
          of x (the whole call a user makes).
The matrix, AMG hierarchy and Krylov basis (~2 GB) exceed L2 (126 MB), so no
explicit flush is needed between steps.

On one GPU the default run also measures the three-phase system (--config c4)
and the uneven batch (--config c3) in child processes and summarises their
lines in details.other_workloads.

--impl reference times the reference library (compiled from its own sources
into oracle/_ref) on the host cores: every timed step is one complete run to
FP64 rel-res 1e-6 (until REF_BUDGET_S has passed); value = its GMRES solve
phase (setup excluded, as our value), e2e = decoupling + setup + solve.  Our arm's cpu_baseline is a
bounded sample of the same library (decoupling + setup + GMRES runs of 2 and
4 iterations, scaled to the reference's iteration count) so that the default
run stays short.

Multi-GPU (torchrun): replicas -- every rank solves its own copy of the
system; value is the max over ranks of the mean solve time (weak scaling).
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "CPR-GMRES time to 1e-6 FP64 rel-res, mixed+learned vs plain FP64, 1xB200"
UNIT = "s"
# the reference arm's timed complete runs stop after this many seconds (at least one run)
REF_BUDGET_S = 120.0
# GMRES iterations the reference library needs (tol 1e-6), measured by running
# it to convergence: config 1 with ABF decoupling and GMRES(30), one thread (the
# device path in exact-order mode reproduces the same count); config 4 with
# True-IMPES decoupling and GMRES(60), 16 threads (253 s on a 16-core host of a B200 machine).
REF_ITERS = {"c1": 51, "c0": 23, "c4": 233}
WORKLOADS = {
    "c1": "config-1 system: 60x220x85 channelised two-phase Jacobian, 1,122,000 cells, 2x2 BSR, 7,780,000 blocks, seed 1",
    "c0": "config-0 system: 20x40x10 two-phase Jacobian, 8,000 cells, 2x2 BSR, 53,200 blocks, seed 0",
    "slab45": "60x220x45 slab of the channelised geometry, 594,000 cells, 2x2 BSR, seed 5 (profiling case)",
    "c4": "config-4 system: 60x220x85 channelised three-phase black-oil Jacobian (p, Sw, Sg), 1,122,000 cells, "
          "3x3 BSR, 7,780,000 blocks, seed 2",
    "c3": "config-3 batch: 64 independent two-phase 2x2 BSR systems built as config 0 (system k: seed k), grids "
          "drawn uniformly from 16x16x8 to 60x110x40 (sizes seeded separately), 3,182,220 cells / 6,364,440 "
          "unknowns in total",
}
# plain FP64 GPU path (the comparison): the reference's method in the throughput ordering
PLAIN_OPTS = dict(decouple=1, k_dim=30, max_iter=300, tol=1e-6, stage2_maxit=3, smoother_order=1, coarse_exact=0,
                  precision=0, fast_smoother=0)
# measured path: FP32 preconditioner + learned settings, the stage-2 weights of the reference's
# mixed-precision driver (1.0 / 0.8, src/test_bsr_cprgmres_hybrid.c:373-374; its plain CPR uses
# 0.7 / 0.9, jxf_cpr.c:547-548), flexible FP64 GMRES run on the device as one CUDA graph with its
# Krylov basis stored in FP32 (products, norms, rotations and x in FP64)
SOLVER_OPTS = dict(PLAIN_OPTS, precision=1, fast_smoother=2, flexible=1, stage2_relax_weight=1.0, stage2_omega=0.8,
                   graph_gmres=1, krylov_fp32=1)
# ablation: the plain FP64 preconditioner with the measured path's stage-2 weights and GMRES driver,
# so that what precision + learned settings alone gain is visible
PLAIN_SAME_DRIVER_OPTS = dict(PLAIN_OPTS, flexible=1, stage2_relax_weight=1.0, stage2_omega=0.8, graph_gmres=1)
# the reference's hybrid form (src/test_bsr_cprgmres_hybrid.c:217-439): FP32 stage 1, FP64 stage-2 polish
# with weights 1.0 / 0.8, on the plain smoothers
HYBRID_OPTS = dict(PLAIN_OPTS, precision=3, flexible=1, stage2_relax_weight=1.0, stage2_omega=0.8)
BATCH_METRIC = "batched CPR-GMRES solves per second to 1e-6 FP64 rel-res (64 uneven systems), 1xB200"
# batched solves: mixed precision (FP32 preconditioner), Chebyshev-3 on the dense levels, flexible FP64 GMRES
BATCH_OPTS = dict(PLAIN_OPTS, precision=1, fast_smoother=1, flexible=1, stage2_relax_weight=1.0, stage2_omega=0.8)


# the kernel the `roofline` object reports for each workload: the one with the largest share of the
# measured solve in its launch list (profiles/launches_*): "cheb_level1" or "stage2"
DOMINANT = {"c1": "cheb_level1", "c4": "stage2"}

# per-workload method choices: the three-phase system is decoupled by True-IMPES and solved with
# GMRES(60) (with ABF, or with GMRES(30), the reference itself is still short of 1e-6 after 300
# iterations; GMRES(30) + True-IMPES needs ~1,550 on the GPU, GMRES(60) ~250)
CONFIG_OPTS = {"c4": dict(decouple=5, k_dim=60, max_iter=1000)}
# the three-phase system under the measured path's driver: the stage-2 weights of the reference's
# mixed-precision driver (1.0 / 0.8) leave GMRES(60) near 5e-5 after 1,000 iterations there, its
# plain CPR weights (0.7 / 0.9) converge in ~250; the learned settings (a network trained on two- and
# three-phase systems) are kept: 0.387 s against 0.404 s with the default Chebyshev intervals
DRIVER_CONFIG_OPTS = {"c4": dict(stage2_relax_weight=0.7, stage2_omega=0.9)}
MEASURED_CONFIG_OPTS = {"c4": dict(DRIVER_CONFIG_OPTS["c4"], fast_smoother=2)}


def measured_path_text(opts, learned):
    w, om = opts.get("stage2_relax_weight", 0.7), opts.get("stage2_omega", 0.9)
    src = ("the reference mixed driver's" if (w, om) == (1.0, 0.8) else "the reference plain CPR's")
    if opts.get("fast_smoother") == 2:
        tuned = ("learned per-level strength thresholds and Chebyshev-3 intervals (" +
                 ("kept" if learned["learned_used"] else "rejected by the probe: plain smoothers") + ")")
    else:
        tuned = "default strength threshold, Chebyshev-3 on the dense levels (no learned settings)"
    return (f"mixed: FP32 preconditioner storage/arithmetic (AMG levels, transfers, stage 2 with {src} weights "
            f"{w}/{om}), FP64 flexible GMRES run on the device as one CUDA graph"
            f"{' (Krylov basis stored in FP32)' if opts.get('krylov_fp32') else ''} / SpMV / true residual / "
            f"coarsest solve; {tuned}; the plain FP64 path is the reference's CPR (weights 0.7/0.9) with its host-driven "
            "MGS GMRES")


def plain_opts(args):
    return dict(PLAIN_OPTS, **CONFIG_OPTS.get(args.config, {}))


def solver_opts(args):
    opts = dict(SOLVER_OPTS, **CONFIG_OPTS.get(args.config, {}), **MEASURED_CONFIG_OPTS.get(args.config, {}))
    for kv in getattr(args, "opt", []) or []:
        k, v = kv.split("=", 1)
        opts[k] = float(v) if ("." in v or "e" in v.lower()) else int(v)
    return opts


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (FileNotFoundError, OSError):
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                rows.append(dict(sm=float(parts[1]), smax=float(parts[2]), power=float(parts[3]),
                                 hw=parts[5], hwt=parts[6], swt=parts[7], swp=parts[8]))
            except ValueError:
                continue
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        loaded = [r for r in rows if r["power"] > 200] or rows
        reasons = set()
        for r in rows:
            for key, name in (("hw", "hw_slowdown"), ("hwt", "hw_thermal_slowdown"), ("swt", "sw_thermal_slowdown"),
                              ("swp", "sw_power_cap")):
                if r[key].lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(r["sm"] for r in loaded), "sm_max_mhz": max(r["smax"] for r in rows),
                "reasons": sorted(reasons), "samples": len(rows)}


# ---------------------------------------------------------------------------
# reference arm / CPU baseline
# ---------------------------------------------------------------------------
def reference_sample(s, threads, cfg):
    """Reference library on the host, bounded sample: decouple + CPR setup + 2 and 4 GMRES iterations.

    Returns (estimated seconds of the solve phase to 1e-6, measured sample seconds,
    description, kind)."""
    os.environ["OMP_NUM_THREADS"] = str(threads)
    import oracle

    iters_full = REF_ITERS[cfg]
    if oracle.ref_available():
        # two bounded runs (2 and 4 GMRES iterations) isolate the per-iteration cost
        t0 = time.perf_counter()
        dec = CONFIG_OPTS.get(cfg, {}).get("decouple", 1)
        kd = CONFIG_OPTS.get(cfg, {}).get("k_dim", 30)
        r2 = oracle.ref_gmres(s.ia, s.ja, s.a, s.block_size, s.b, decouple=dec, tol=1e-6, max_iter=2, k_dim=kd)
        r4 = oracle.ref_gmres(s.ia, s.ja, s.a, s.block_size, s.b, decouple=dec, tol=1e-6, max_iter=4, k_dim=kd)
        wall = time.perf_counter() - t0
        t_dec, t_setup = r2["times"][0], r2["times"][1]
        per_iter = max(0.0, (r4["times"][2] - r2["times"][2]) / 2.0)
        est = r2["times"][2] + per_iter * max(0, iters_full - 2)
        desc = (f"reference JXFPAMG built from source (FP64), {threads} OpenMP threads: decoupling + CPR setup + "
                f"GMRES runs of 2 and 4 iterations ({wall:.1f} s in total); the solve phase (setup excluded, as "
                f"value) is the 2-iteration run's plus the per-iteration time (difference / 2) scaled to the "
                f"{iters_full} iterations the reference needs on this system (decoupling {t_dec:.2f} s and setup "
                f"{t_setup:.2f} s come on top)")
        return est, wall, desc, "reference"
    # fallback: the oracle restatement (single thread)
    sample_iters = 4
    t0 = time.perf_counter()
    a, b = oracle.bsr_decouple(s.ia, s.ja, s.a, s.block_size, s.b, CONFIG_OPTS.get(cfg, {}).get("decouple", 1))
    C = oracle.OracleCPR(s.ia, s.ja, a, s.block_size)
    t1 = time.perf_counter()
    oracle.gmres(s.ia, s.ja, a, s.block_size, b, tol=1e-6, max_iter=sample_iters, cpr=C,
                 k_dim=CONFIG_OPTS.get(cfg, {}).get("k_dim", 30))
    t2 = time.perf_counter()
    est = (t2 - t1) / sample_iters * iters_full
    desc = (f"oracle C restatement (1 thread): decoupling + CPR setup + {sample_iters} GMRES iterations "
            f"({t2 - t0:.1f} s); the solve phase scaled to {iters_full} iterations")
    return est, t2 - t0, desc, "port"


def common_config(cfg, opts):
    """The `config` object both arms print (identical keys and values for one workload)."""
    return {"workload": WORKLOADS[cfg],
            "decoupling": "True-IMPES" if opts.get("decouple") == 5 else "ABF",
            "tol": 1e-6, "k_dim": opts.get("k_dim", 30),
            "l2_flush": "not needed: matrix + hierarchy + Krylov basis > 126 MB L2"}


def reference_full_solve(s, threads, cfg):
    """One complete run of the reference library on the host: decoupling, CPR setup and GMRES to
    FP64 rel-res 1e-6.  Returns (seconds per phase [decouple, setup, solve], iterations)."""
    os.environ["OMP_NUM_THREADS"] = str(threads)
    import oracle

    dec = CONFIG_OPTS.get(cfg, {}).get("decouple", 1)
    kd = CONFIG_OPTS.get(cfg, {}).get("k_dim", 30)
    mi = CONFIG_OPTS.get(cfg, {}).get("max_iter", 300)
    r = oracle.ref_gmres(s.ia, s.ja, s.a, s.block_size, s.b, decouple=dec, tol=1e-6, max_iter=mi, k_dim=kd)
    if not r["converged"]:
        raise RuntimeError(f"reference solve did not converge (rel {r['rel']})")
    return [float(r["times"][0]), float(r["times"][1]), float(r["times"][2])], r["iters"]


def reference_unavailable():
    """Prints the reference arm's line and returns True where the reference library is not built: the arm
    runs the reference or nothing."""
    import oracle

    if oracle.ref_available():
        return False
    print(json.dumps({"impl": "reference",
                      "unavailable": "the reference library is not built: no source tree to compile it from"}),
          flush=True)
    return True


def run_reference(args):
    """--impl reference: the reference's own CPU implementation of the path (compiled from its sources
    into oracle/_ref; where it is absent the line says "unavailable") on all host threads.  Each timed step is
    one complete run to convergence; value = the GMRES solve phase (setup excluded, as in our arm's
    value), e2e = decoupling + CPR setup + solve (as our arm's e2e, which also includes the uploads).
    Warm-up steps are short runs (two GMRES iterations) that page the library and the system in.  A
    complete run takes about 35 s on C1 and 250 s on C4, so the timed runs stop once REF_BUDGET_S
    has passed (at least one): the line's `steps` is the number of runs made."""
    ws, rank, _ = dist_env()
    if rank != 0 or reference_unavailable():
        return 0
    from jxpamg_all_b200 import synth

    s = synth.config_system(args.config)
    threads = os.cpu_count() or 1
    os.environ["OMP_NUM_THREADS"] = str(threads)
    import oracle

    dec = CONFIG_OPTS.get(args.config, {}).get("decouple", 1)
    kd = CONFIG_OPTS.get(args.config, {}).get("k_dim", 30)
    for _ in range(args.warmup):
        oracle.ref_gmres(s.ia, s.ja, s.a, s.block_size, s.b, decouple=dec, tol=1e-6, max_iter=2, k_dim=kd)
    phases, iters = [], []
    w0 = time.perf_counter()
    for _ in range(args.steps):
        t, it = reference_full_solve(s, threads, args.config)
        phases.append(t)
        iters.append(it)
        if time.perf_counter() - w0 > REF_BUDGET_S:
            break
    wall = time.perf_counter() - w0
    ph = np.array(phases)
    value = float(ph[:, 2].mean())
    total = float(ph.sum(axis=1).mean())
    desc = (f"reference JXFPAMG built from source (FP64), {threads} OpenMP threads, {len(phases)} complete runs to FP64 rel-res 1e-6 "
            f"({iters[0]} GMRES iterations; decoupling {ph[:, 0].mean():.2f} s, CPR setup {ph[:, 1].mean():.2f} s, "
            f"solve {value:.2f} s per run; {wall:.0f} s in all)")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": len(phases), "steps_requested": args.steps, "warmup": args.warmup, "ms_per_step": total * 1e3,
        "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": common_config(args.config, plain_opts(args)),
        "parallelism": f"1 host process, {threads} OpenMP threads",
        "details": {"value_definition": "GMRES solve phase of a complete run (decoupling and CPR setup excluded, "
                                        "reported in e2e)",
                    "iterations": iters[0], "decouple_s": float(ph[:, 0].mean()), "setup_s": float(ph[:, 1].mean()),
                    "solve_s": value, "ms_per_step_definition": "one complete run (decoupling + setup + solve)"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "reference", "sample": desc},
        "e2e": {"value": total, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def run_ours(args):
    import torch
    import torch.distributed as dist

    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    if ws > 1:
        import datetime

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600), device_id=torch.device("cuda", local))
    from jxpamg_all_b200 import lib, synth
    from jxpamg_all_b200.solver import CprGmres

    so = lib.load()
    s = synth.config_system(args.config)
    n = s.n
    stream = torch.cuda.current_stream()
    dev = lambda arr: torch.from_numpy(np.ascontiguousarray(arr)).cuda()  # noqa: E731
    d_ia, d_ja, d_a, d_b = dev(s.ia), dev(s.ja), dev(s.a), dev(s.b)
    d_x = torch.zeros(n, dtype=torch.float64, device="cuda")

    def make(opts):
        G = CprGmres(**opts)
        G.set_stream(stream.cuda_stream)
        G.setup(d_ia.data_ptr(), d_ja.data_ptr(), d_a.data_ptr(), s.block_size, nb=s.num_block_rows, nnzb=s.nnzb,
                device=True)
        return G

    def solve_device(G):
        d_x.zero_()
        return G.solve(d_b.data_ptr(), d_x.data_ptr(), device=True)

    measured_opts = solver_opts(args)
    if args.profile_kernels:
        # the roofline kernels alone inside a profiler range (ncu --profile-from-start off): one stage-2
        # sweep, two level-1 Chebyshev steps, one FP64 BSR SpMV, the dense inverse of a seeded 1,024 x
        # 1,024 diagonally dominant matrix (the coarse-level kernel) and, on the measured path, one
        # device-GMRES orthogonalisation step at the mid-cycle basis size after a solve; --path bilu: one
        # exact block-ILU(0) application (level-scheduled substitutions) of the plain FP64 path instead
        if args.path == "bilu":
            G = make(dict(plain_opts(args), stage2_solver_type=5, bilu_exact=1, bilu_ir_iters=1))
        else:
            G = make(plain_opts(args) if args.path == "plain" else measured_opts)
        x1 = torch.ones(s.n, dtype=torch.float64, device="cuda")
        y1 = torch.zeros(s.n, dtype=torch.float64, device="cuda")
        gen = torch.Generator(device="cuda").manual_seed(3)
        nd = 1024
        dm = -torch.rand((nd, nd), dtype=torch.float64, device="cuda", generator=gen) * 0.01
        dm += torch.diag(dm.abs().sum(dim=1) + 1.0)
        dinv = torch.empty_like(dm)

        def kernels():
            if args.path == "bilu":
                lib.check(so.jxcpr_solver_bilu_apply(G.h, ctypes.c_void_p(x1.data_ptr()),
                                                     ctypes.c_void_p(y1.data_ptr()), 1))
                return
            lib.check(so.jxcpr_solver_stage2_native(G.h, 1))
            if G.num_levels() > 2:
                lib.check(so.jxcpr_solver_level_native(G.h, 1, 1, 2))
            lib.check(so.jxcpr_bsr_matvec_dev(s.num_block_rows, s.block_size, s.nnzb, d_ia.data_ptr(),
                                              d_ja.data_ptr(), d_a.data_ptr(), 1.0, x1.data_ptr(), 0.0,
                                              y1.data_ptr(), 0, ctypes.c_void_p(stream.cuda_stream)))
            lib.check(so.jxcpr_dense_inverse_dev(nd, dm.data_ptr(), dinv.data_ptr(),
                                                 ctypes.c_void_p(stream.cuda_stream)))

        if args.path == "mixed" and measured_opts.get("graph_gmres"):
            solve_device(G)  # the orthogonalisation kernels run on the basis a solve leaves
            m_kry = (measured_opts.get("k_dim", 30) + 1) // 2
            base_kernels = kernels

            def kernels():
                base_kernels()
                lib.check(so.jxcpr_solver_krylov_native(G.h, m_kry, 1))

        kernels()  # warm
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        kernels()
        torch.cuda.synchronize()
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_kernels": args.config, "path": args.path}))
        G.close()
        return 0
    if args.profile_solve:
        # one solve inside a profiler range (ncu --profile-from-start off), nothing else
        G = make(plain_opts(args) if args.path == "plain" else measured_opts)
        for _ in range(args.warmup):
            solve_device(G)
        torch.cuda.synchronize()
        torch.cuda.profiler.start()
        _, it, rel, conv = solve_device(G)
        torch.cuda.synchronize()
        torch.cuda.profiler.stop()
        print(json.dumps({"profile_solve": args.config, "path": args.path, "iterations": it, "rel": rel,
                          "converged": conv}))
        G.close()
        return 0 if conv else 1

    def timed(G, clk_name):
        """Device-resident solves: W warm-up, K timed between barriers (CUDA events, max over ranks)."""
        for _ in range(args.warmup):
            solve_device(G)
        torch.cuda.synchronize()
        if ws > 1:
            dist.barrier()
        torch.cuda.synchronize()
        l0 = so.jxcpr_launch_count()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        iters, rels = [], []
        with ClockSampler(local) as clk:
            e0.record(stream)
            for _ in range(args.steps):
                _, it, rel, conv = solve_device(G)
                iters.append(it)
                rels.append(rel)
                if not conv:
                    raise RuntimeError(f"{clk_name}: solve did not converge (rel {rel})")
            e1.record(stream)
            torch.cuda.synchronize()
        launches = so.jxcpr_launch_count() - l0
        t = torch.tensor([e0.elapsed_time(e1) / 1e3], dtype=torch.float64, device="cuda")
        if ws > 1:
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item()) / args.steps, int(np.median(iters)), float(rels[-1]), launches, clk.summary()

    # ---- plain FP64 path (the comparison) ----------------------------------------
    P = make(plain_opts(args))
    plain_setup = P.stats()
    plain_t, plain_it, plain_rel, _, clk_p = timed(P, "plain FP64")
    x_plain = d_x.cpu().numpy().copy()
    roof_plain = roofline_stage2(P, s, stream, 8, args.config)
    plain_gbs = iteration_bytes(P, s, plain_opts(args)) * plain_it / plain_t / 1e9
    P.close()

    # ---- the reference's hybrid form (FP32 stage 1 + FP64 polish), for comparison ------
    Hy = make(dict(HYBRID_OPTS, **CONFIG_OPTS.get(args.config, {}), **DRIVER_CONFIG_OPTS.get(args.config, {})))
    hybrid_t, hybrid_it, hybrid_rel, _, _ = timed(Hy, "hybrid FP32/FP64")
    Hy.close()
    # ---- ablation: plain FP64 preconditioner, measured path's weights and GMRES driver ----
    Pd = make(dict(PLAIN_SAME_DRIVER_OPTS, **CONFIG_OPTS.get(args.config, {}),
                   **DRIVER_CONFIG_OPTS.get(args.config, {})))
    plain_d_t, plain_d_it, _, _, _ = timed(Pd, "plain FP64, same driver")
    Pd.close()

    # ---- measured path: mixed precision + learned settings ------------------------
    G = make(measured_opts)
    setup_stats = G.stats()
    learned = G.learned_status()
    per_solve, it_m, rel_m, launches, clocks = timed(G, "mixed+learned")
    x_mixed = d_x.cpu().numpy().copy()
    err_vs_fp64 = float(np.linalg.norm(x_mixed - x_plain) / np.linalg.norm(x_plain))
    vb = 8 if measured_opts.get("precision", 0) == 0 else 4
    roof_st2 = roofline_stage2(G, s, stream, 8 if measured_opts.get("precision", 0) in (0, 3) else 4, args.config)
    roof_lvl = roofline_level(G, stream, 1, 1, vb, vb, args.config) if G.num_levels() > 2 else None
    solve_gbs = iteration_bytes(G, s, measured_opts) * it_m / per_solve / 1e9
    roof_kry = roofline_krylov(G, s, stream, measured_opts, args.config) if measured_opts.get("graph_gmres") else None
    G.close()
    roof_spmv = roofline_bsr_spmv(d_ia, d_ja, d_a, s, stream, args.config)
    roof_spmv_tma = roofline_bsr_spmv(d_ia, d_ja, d_a, s, stream, args.config, staged=1)
    # the roofline line names the kernel with the largest share of the measured solve (launch list in
    # profiles/): the level-1 Chebyshev pass where the level has one, else the stage-2 sweep
    roof = roof_lvl if (roof_lvl is not None and DOMINANT.get(args.config) == "cheb_level1") else roof_st2
    if clk_p.get("reasons"):
        clocks["reasons"] = sorted(set(clocks.get("reasons", [])) | set(clk_p["reasons"]))

    # ---- e2e: public C ABI with pinned host buffers, setup included --------------
    pin = lambda arr: torch.from_numpy(np.ascontiguousarray(arr)).pin_memory()  # noqa: E731
    h_ia, h_ja, h_a, h_b = pin(s.ia), pin(s.ja), pin(s.a), pin(s.b)
    h_x = torch.zeros(n, dtype=torch.float64).pin_memory()
    h2d = (h_ia.numel() * 4 + h_ja.numel() * 4 + h_a.numel() * 8 + h_b.numel() * 8 + h_x.numel() * 8)
    d2h = h_x.numel() * 8

    def e2e_step():
        E = CprGmres(**measured_opts)
        E.set_stream(stream.cuda_stream)
        E.nb, E.bs = s.num_block_rows, s.block_size
        lib.check(E._so.jxcpr_solver_setup(E.h, s.num_block_rows, s.block_size, s.nnzb,
                                           ctypes.c_void_p(h_ia.data_ptr()), ctypes.c_void_p(h_ja.data_ptr()),
                                           ctypes.c_void_p(h_a.data_ptr()), 0))
        h_x.zero_()
        itv = np.zeros(1, np.int32)
        relv = np.zeros(1)
        st = E._so.jxcpr_solver_solve(E.h, ctypes.c_void_p(h_b.data_ptr()), ctypes.c_void_p(h_x.data_ptr()), 0,
                                      itv.ctypes.data_as(ctypes.c_void_p), relv.ctypes.data_as(ctypes.c_void_p))
        lib.check(st)
        E.close()

    e2e_steps = max(1, min(args.steps, 3))
    e2e_step()  # warm
    torch.cuda.synchronize()
    if ws > 1:
        dist.barrier()
    f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(e2e_steps):
        e2e_step()
    f1.record(stream)
    torch.cuda.synchronize()
    e2e_t = torch.tensor([f0.elapsed_time(f1) / 1e3 / e2e_steps], dtype=torch.float64, device="cuda")
    if ws > 1:
        dist.all_reduce(e2e_t, op=dist.ReduceOp.MAX)

    line = None
    if rank == 0:
        cpu = None
        if ws == 1 and not args.no_cpu_baseline:
            est, wall, desc, kind = reference_sample(s, os.cpu_count() or 1, args.config)
            cpu = {"value": est, "unit": UNIT, "cores": os.cpu_count() or 1, "kind": kind, "sample": desc}
        line = {
            "metric": METRIC, "value": per_solve, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": per_solve * 1e3, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
            "config": common_config(args.config, measured_opts),
            "parallelism": f"replicas x{ws}" if ws > 1 else "1 GPU",
            "details": {"method": f"CPR-GMRES({measured_opts.get('k_dim', 30)}) to FP64 true rel-res 1e-6, " +
                                  ("True-IMPES" if measured_opts.get("decouple") == 5 else "ABF") +
                                  " decoupling, AMG V(1,1) (HMIS, ext+i) + 3 block-GS stage-2 sweeps",
                        "measured_path": measured_path_text(measured_opts, learned),
                        "options": measured_opts,
                        "iterations": it_m, "final_rel_res": rel_m,
                        "solve_gbs": solve_gbs,
                        "solve_gbs_definition": "modelled bytes per GMRES iteration (preconditioner traffic at its "
                                                "storage precision + FP64 BSR SpMV + orthogonalisation: three "
                                                "CGS2 passes over the basis at its storage precision, or one MGS "
                                                "pass per vector on the host-driven path) x iterations / solve time",
                        "plain_fp64_s": plain_t, "plain_fp64_iterations": plain_it, "plain_fp64_rel_res": plain_rel,
                        "plain_fp64_solve_gbs": plain_gbs,
                        "speedup_vs_plain_fp64": plain_t / per_solve,
                        "hybrid_fp32_fp64_s": hybrid_t, "hybrid_iterations": hybrid_it,
                        "plain_fp64_same_driver_s": plain_d_t, "plain_fp64_same_driver_iterations": plain_d_it,
                        "speedup_vs_plain_fp64_same_driver": plain_d_t / per_solve,
                        "hybrid_speedup_vs_plain_fp64": plain_t / hybrid_t,
                        "x_rel_diff_vs_plain_fp64": err_vs_fp64,
                        "learned": learned,
                        "setup_s": setup_stats["setup_ms"] / 1e3, "plain_setup_s": plain_setup["setup_ms"] / 1e3,
                        "amg_levels": setup_stats["levels"],
                        "roofline_bsr_spmv": roof_spmv,
                        "roofline_bsr_spmv_tma_staged": roof_spmv_tma,
                        "roofline_krylov_step": roof_kry,
                        "roofline_stage2": roof_st2,
                        "roofline_cheb_level1": roof_lvl,
                        "roofline_plain_fp64_stage2": roof_plain},
            "roofline": roof,
            "cpu_baseline": cpu,
            "e2e": {"value": float(e2e_t.item()), "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h),
                    "note": "public C ABI from pinned host memory, mixed+learned path: upload + decoupling + CPR setup "
                            "(incl. the learned-settings probe) + solve + x download"},
            "gpu_launches": int(launches),
            "clocks": clocks,
        }
        if ws == 1 and args.config == "c1" and not args.no_extras:
            line["details"]["other_workloads"] = other_workloads(args)
        print(json.dumps(line), flush=True)
    if ws > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def other_workloads(args):
    """The three-phase system (config 4) and the uneven batch (config 3) measured by this same run, one
    child process each after the config-1 measurement (their own JSON lines, summarised): the default
    bench line then carries every workload's device-timed result."""
    out = {}
    for cfg in ("c4", "c3"):
        cmd = [sys.executable, os.path.abspath(__file__), "--config", cfg, "--steps", str(min(args.steps, 3)),
               "--warmup", "2", "--no-cpu-baseline", "--no-extras"]
        t0 = time.perf_counter()
        p = subprocess.run(cmd, capture_output=True, text=True, timeout=900)
        lines = [ln for ln in p.stdout.splitlines() if ln.startswith("{")]
        if p.returncode != 0 or not lines:
            out[cfg] = {"error": f"exit {p.returncode}: {p.stderr.strip().splitlines()[-1:]}"}
            continue
        d = json.loads(lines[-1])
        t = d.get("details", {})
        c = d.get("config", {})
        keep = {"workload": c.get("workload"), "metric": d["metric"], "value": d["value"], "unit": d["unit"],
                "steps": d["steps"], "ms_per_step": d["ms_per_step"], "e2e": d.get("e2e", {}).get("value"),
                "roofline_frac": (d.get("roofline") or {}).get("frac"), "clocks": d.get("clocks"),
                "wall_s": time.perf_counter() - t0}
        if cfg == "c4":
            keep.update({"iterations": t.get("iterations"), "plain_fp64_s": t.get("plain_fp64_s"),
                         "plain_fp64_iterations": t.get("plain_fp64_iterations"),
                         "speedup_vs_plain_fp64": t.get("speedup_vs_plain_fp64"),
                         "learned_used": (t.get("learned") or {}).get("learned_used")})
        else:
            keep.update({k: c.get(k) for k in ("latency_ms_p50", "latency_ms_p99", "last_finish_ms")})
        out[cfg] = keep
    return out


# DRAM traffic of the roofline kernels per timed unit (a stage-2 sweep = its colour launches, a Chebyshev
# step, one SpMV), from an ncu capture of `bench.py --profile-kernels` (dram__bytes_read.sum +
# dram__bytes_write.sum; layouts reused through JXCPR_TUNE_CACHE), each summarised in profiles/:
# (workload, kernel key) -> bytes.  None where not captured.
TRAFFIC_BYTES = {
    ("c1", "stage2/4/chunk4"): 207_780_864,    # hgs_chunk<2,4,float>: 99,497,984 + 108,282,880 (2 colours)
    ("c1", "cheb/A1/4/csr/4"): 103_513_600,    # row_kernel<CsrFmt<4,float>, OpCheb>: mean of 2 launches
    ("c1", "cheb/A1/4/sell"): 108_742_144,     # row_kernel<SellFmt<float>, OpCheb>: mean of 2 launches
    ("c1", "cheb/A1/4/sell/near"): 82_076_416,  # row_kernel<SellFmt<float, 16-bit columns>, OpCheb>: mean of 2
    ("c1", "bsr_spmv/8"): 317_666_304,         # bsr_spmv_slab_kernel<double, NoKeep, true>
    ("c4", "stage2/4/chunk4"): 389_371_648,    # hgs_chunk<3,4,float>: 189,119,232 + 200,252,416 (2 colours)
}


def hbm_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    peaks = json.load(open(p)) if os.path.exists(p) else {}
    if peaks.get("hbm_gbs"):
        return float(peaks["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def _event_time(stream, body, reps):
    """Mean device seconds of body() (which queues `reps` launches) between events on `stream`."""
    import torch

    body(3)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    body(reps)
    e1.record(stream)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / 1e3 / reps


def _roof(kernel, alg, sec, cfg, key, extra=None):
    peak, src = hbm_peak()
    achieved = alg / sec / 1e9
    out = {"bound": "hbm", "kernel": kernel, "achieved": achieved, "peak": peak, "unit": "GB/s",
           "frac": achieved / peak, "peak_source": src, "traffic": TRAFFIC_BYTES.get((cfg, key)),
           "algorithmic_bytes": int(alg), "launch_ms": sec * 1e3}
    out.update(extra or {})
    return out


def _layout(G, name):
    for line in G.setup_report().splitlines():
        if line.startswith("tuned " + name + " ") and " layout " in line:
            return line.split(" layout ")[1].split()[0]
    return "?"


def roofline_stage2(G, s, stream, value_bytes, cfg="c1"):
    """Stage-2 block Gauss-Seidel sweep (one launch per colour) in the path's own storage precision:
    algorithmic bytes of one sweep / mean sweep time (CUDA events on the solver's stream)."""
    from jxpamg_all_b200 import lib

    so = lib.load()
    reps = 20
    sec = _event_time(stream, lambda r: lib.check(so.jxcpr_solver_stage2_native(G.h, r)), reps)
    bs, nb, nnzb, n = s.block_size, s.num_block_rows, s.nnzb, s.n
    # values + column indices + row pointers; b read, x read and written, the start values of the
    # colours before the last written to vt and read back by their neighbours (about n in all)
    alg = nnzb * (bs * bs * value_bytes + 4) + (nb + 1) * 4 + n * value_bytes * 5
    layout = _layout(G, "stage2")
    kname = {"sell": f"hgs_sell<{bs}>"}.get(layout, f"hgs_chunk<{bs}>" if layout.startswith("chunk")
                                               else f"hgs_color<{bs}> ({layout})")
    return _roof(f"stage-2 block hybrid Gauss-Seidel sweep ({kname}, {'FP64' if value_bytes == 8 else 'FP32'} "
                 "values, one launch per colour)", alg, sec, cfg, f"stage2/{value_bytes}/{layout}",
                 {"sweep_ms": sec * 1e3})


def level_format(layout, near, value_bytes):
    """(kernel format, key) of a level operator's layout as the setup report names it: "sell" (one lane per
    row), "sell/P" (P lanes) or "csr/V"; near: 16-bit columns."""
    ty = {8: "double", 4: "float", 2: "bf16"}[value_bytes]
    kind, _, lanes = layout.partition("/")
    args = [ty] + ([lanes] if lanes else []) if kind == "sell" else [lanes, ty]
    fmt = "SellFmt" if kind == "sell" else "CsrFmt"
    return (f"{fmt}<{', '.join(args + (['16-bit columns'] if near else []))}>",
            layout + ("/near" if near else ""))


def roofline_level(G, stream, level, op, value_bytes, vec_bytes, cfg="c1"):
    """One pass over AMG level `level` (op 1: a Chebyshev step y = c z + D^-1 A x) in the path's storage
    precision and layout: algorithmic bytes nnz (p_v + 4; 2 where the columns are 16-bit) + (n + 1) 4 +
    4 n p_x (x, z, D^-1 read, y written) / mean launch time (CUDA events on the solver's stream)."""
    from jxpamg_all_b200 import lib

    so = lib.load()
    n, _, nnz = G.level_sizes(level, 0)
    sec = _event_time(stream, lambda r: lib.check(so.jxcpr_solver_level_native(G.h, level, op, r)), 20)
    near = any(line.startswith(f"tuned A{level} ") and "16-bit columns" in line
               for line in G.setup_report().splitlines())
    alg = nnz * (value_bytes + (2 if near else 4)) + (n + 1) * 4 + 4 * n * vec_bytes
    fmt, layout = level_format(_layout(G, f"A{level}"), near, value_bytes)
    return _roof(f"AMG level {level} Chebyshev step (row_kernel<{fmt}, OpCheb>, {n} rows, {nnz} entries)",
                 alg, sec, cfg, f"cheb/A{level}/{value_bytes}/{layout}", {"level": level})


def roofline_bsr_spmv(d_ia, d_ja, d_a, s, stream, cfg="c1", staged=0):
    """The FP64 BSR SpMV y = A x on the workload's matrix: bsr_spmv_slab_kernel (3x3 blocks:
    bsr_spmv_direct_kernel), the solve's kernels, in the form for a product alone; or with staged = 1 the
    TMA-staged bsr_spmv_tma_kernel for comparison."""
    import torch

    from jxpamg_all_b200 import lib

    so = lib.load()
    x = torch.ones(s.n, dtype=torch.float64, device="cuda")
    y = torch.zeros(s.n, dtype=torch.float64, device="cuda")

    def body(r):
        for _ in range(r):
            lib.check(so.jxcpr_bsr_matvec_dev(s.num_block_rows, s.block_size, s.nnzb, d_ia.data_ptr(),
                                              d_ja.data_ptr(), d_a.data_ptr(), 1.0, x.data_ptr(), 0.0,
                                              y.data_ptr(), staged, ctypes.c_void_p(stream.cuda_stream)))

    sec = _event_time(stream, body, 20)
    bs, nb, nnzb, n = s.block_size, s.num_block_rows, s.nnzb, s.n
    alg = nnzb * (bs * bs * 8 + 4) + (nb + 1) * 4 + 2 * n * 8
    kname = (f"bsr_spmv_tma_kernel<{bs}>" if staged else "bsr_spmv_slab_kernel<double, NoKeep, true>" if bs == 2
             else f"bsr_spmv_direct_kernel<{bs}, double>")
    return _roof(f"BSR SpMV y = A x ({kname}, FP64)", alg, sec, cfg, "bsr_spmv_tma/8" if staged else "bsr_spmv/8")


def roofline_krylov(G, s, stream, opts, cfg="c1"):
    """One device-GMRES orthogonalisation step at the mid-cycle basis size m = (k + 1) // 2: the first
    Gram products, the fused update + second products and the final update (four launches, one of them a
    one-block reduction), timed together with CUDA events on the solver's stream after a solve.
    Algorithmic bytes: three passes over m basis vectors at p_b bytes an entry, w read three times and
    written once, v_m written: (3 m p_b + 32 + p_b) n."""
    from jxpamg_all_b200 import lib

    so = lib.load()
    m = (opts.get("k_dim", 30) + 1) // 2
    pb = 4 if opts.get("krylov_fp32", 0) else 8
    sec = _event_time(stream, lambda r: lib.check(so.jxcpr_solver_krylov_native(G.h, m, r)), 20)
    alg = (3 * m * pb + 32 + pb) * s.n
    ty = "float" if pb == 4 else "double"
    return _roof(f"CGS2 orthogonalisation step, m = {m} (dots_kernel<{ty}> + update_dots_kernel<{ty}> + "
                 f"final_kernel<{ty}>, basis in {'FP32' if pb == 4 else 'FP64'})", alg, sec, cfg,
                 f"krylov/{pb}/{m}", {"m": m})


def iteration_bytes(G, s, opts):
    """Modelled bytes of one GMRES iteration: the preconditioner application (its modelled traffic), the
    FP64 BSR SpMV, and the orthogonalisation at the mean basis size m = (k + 1) / 2 of a cycle.
    - Device GMRES (graph_gmres 1, CGS2), with p_b bytes per basis entry (8, or 4 with krylov_fp32):
      three passes over the basis (first products; the first update fused with the second products;
      the final update) plus w, the new vector, and the copies in and out of the preconditioner. That
      is (3 m p_b + 48 + 3 p_b) n bytes, and 8 n more when an FP32 basis rounds the direction in place.
    - Host GMRES (modified Gram-Schmidt): one pass per basis vector. Each pass reads w and v_j and
      writes w, giving (32 m + 16) n bytes."""
    from jxpamg_all_b200 import lib

    so = lib.load()
    ab = np.zeros(1)
    lib.check(so.jxcpr_solver_apply_bytes(G.h, ab.ctypes.data_as(ctypes.c_void_p)))
    spmv = s.nnzb * (s.block_size ** 2 * 8 + 4) + (s.num_block_rows + 1) * 4 + 2 * s.n * 8
    m = (opts.get("k_dim", 30) + 1) / 2.0
    if opts.get("graph_gmres", 0):
        pb = 4 if opts.get("krylov_fp32", 0) else 8
        orth = (3 * m * pb + 48 + 3 * pb + (8 if pb == 4 else 0)) * s.n
    else:
        orth = (32 * m + 16) * s.n
    return float(ab[0]) + spmv + orth


# ---------------------------------------------------------------------------
# batched solves (config 3)
# ---------------------------------------------------------------------------
def batch_partition(cells, ws):
    """Whole systems per rank, balanced by cell count (largest first to the least-loaded rank)."""
    parts = [[] for _ in range(ws)]
    load = [0] * ws
    for k in sorted(range(len(cells)), key=lambda k: -cells[k]):
        r = load.index(min(load))
        parts[r].append(k)
        load[r] += cells[k]
    return [sorted(p) for p in parts]


def batch_reference_sample(systems, threads):
    """Reference library on the host, run to convergence on every 9th system in size order
    (smallest to largest), one after another; the batch time is scaled by the cell-count ratio.
    Returns (systems/s, sample seconds, description, kind)."""
    os.environ["OMP_NUM_THREADS"] = str(threads)
    import oracle

    cells = [s.num_block_rows for s in systems]
    order = sorted(range(len(systems)), key=lambda k: cells[k])
    sample = order[::9]
    t0 = time.perf_counter()
    iters = []
    kind = "reference" if oracle.ref_available() else "port"
    for k in sample:
        s = systems[k]
        if kind == "reference":
            r = oracle.ref_gmres(s.ia, s.ja, s.a, s.block_size, s.b, decouple=1, tol=1e-6, max_iter=300)
        else:
            a, b = oracle.bsr_decouple(s.ia, s.ja, s.a, s.block_size, s.b, 1)
            C = oracle.OracleCPR(s.ia, s.ja, a, s.block_size)
            r = oracle.gmres(s.ia, s.ja, a, s.block_size, b, tol=1e-6, max_iter=300, cpr=C)
        iters.append(int(r["iters"]))
    wall = time.perf_counter() - t0
    frac = sum(cells[k] for k in sample) / sum(cells)
    est = wall / frac
    what = "reference JXFPAMG built from source (FP64)" if kind == "reference" else "oracle C restatement"
    desc = (f"{what}, {threads} OpenMP threads, one system after another (decoupling + CPR setup + GMRES to 1e-6) "
            f"on {len(sample)} of the {len(systems)} systems (every 9th by size, {100 * frac:.0f}% of the cells, "
            f"{wall:.1f} s, iterations {iters}); batch time scaled by the cell-count ratio")
    return len(systems) / est, wall, desc, kind


def run_batch_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0 or reference_unavailable():
        return 0
    from jxpamg_all_b200 import synth

    systems = synth.batch_systems()
    threads = os.cpu_count() or 1
    vals = []
    desc = kind = None
    for _ in range(max(1, min(args.steps, 2))):
        v, _, desc, kind = batch_reference_sample(systems, threads)
        vals.append(v)
    value = float(np.mean(vals))
    line = {
        "impl": "reference", "metric": BATCH_METRIC, "value": value, "unit": "systems/s", "n_gpus": args.gpus,
        "steps": len(vals), "warmup": 0, "ms_per_step": 1e3 * len(systems) / value, "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": WORKLOADS["c3"], "decoupling": "ABF", "tol": 1e-6, "k_dim": 30,
                   "includes": "decoupling + CPR setup + GMRES solve of every system"},
        "cpu_baseline": {"value": value, "unit": "systems/s", "cores": threads, "kind": kind, "sample": desc},
        "e2e": {"value": value, "unit": "systems/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


def run_batch(args):
    """One step = every system of the batch solved from x0 = 0 by ONE graph launch per rank
    (ranks: whole systems, balanced by cells, no collective on the data path)."""
    import torch
    import torch.distributed as dist

    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    if ws > 1:
        import datetime

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600), device_id=torch.device("cuda", local))
    from jxpamg_all_b200 import lib, synth
    from jxpamg_all_b200.solver import CprGmres, CprGmresBatch, setup_many

    so = lib.load()
    opts = dict(BATCH_OPTS)
    for kv in args.opt or []:
        k, v = kv.split("=", 1)
        opts[k] = float(v) if ("." in v or "e" in v.lower()) else int(v)
    grids = synth.batch_grids()
    nsys = len(grids)
    cells_all = [nx * ny * nz for nx, ny, nz in grids]
    mine = batch_partition(cells_all, ws)[rank]
    systems = {k: synth.reservoir_system(*grids[k], k) for k in mine}

    threads = os.cpu_count() or 1
    t_setup = time.perf_counter()
    solvers = setup_many([CprGmres(**opts) for _ in mine], [systems[k] for k in mine], threads=threads)
    t_setup = time.perf_counter() - t_setup
    t_create = time.perf_counter()
    B = CprGmresBatch(solvers)
    t_create = time.perf_counter() - t_create
    d_b = [torch.from_numpy(systems[k].b).cuda() for k in mine]
    d_x = [torch.zeros(systems[k].n, dtype=torch.float64, device="cuda") for k in mine]
    bp = [t.data_ptr() for t in d_b]
    xp = [t.data_ptr() for t in d_x]

    def step():
        for t in d_x:
            t.zero_()
        torch.cuda.synchronize()
        return B.solve_ptrs(bp, xp, True)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    if ws > 1:
        dist.barrier()
    torch.cuda.synchronize()
    l0 = so.jxcpr_launch_count()
    times, out = [], None
    with ClockSampler(local) as clk:
        for _ in range(args.steps):
            out = step()
            times.append(B.last_ms() / 1e3)
            if not np.all(out["status"] == 0):
                raise RuntimeError(f"batch: systems did not converge: {out['status']}")
    launches = so.jxcpr_launch_count() - l0
    clocks = clk.summary()
    t = torch.tensor([float(np.mean(times))], dtype=torch.float64, device="cuda")
    if ws > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    step_s = float(t.item())
    # true FP64 residuals of the decoupled systems, recomputed on the host
    import oracle

    rels = []
    for j, k in enumerate(mine):
        s = systems[k]
        a, b = oracle.bsr_decouple(s.ia, s.ja, s.a, s.block_size, s.b, 1)
        xk = d_x[j].cpu().numpy()
        r = b - synth.bsr_matvec_np(s.ia, s.ja, a, s.block_size, xk)
        rels.append(float(np.linalg.norm(r) / np.linalg.norm(b)))
    worst = float(np.max(rels))  # NaN propagates
    lat, fin = out["latency_ms"], out["finish_ms"]
    B.close()
    for G in solvers:
        G.close()

    # e2e: from pinned host arrays (matrices, b, x0) through the C ABI: setup of every system,
    # the batch graph, one solve call for the batch, solutions back
    pin = lambda arr: torch.from_numpy(np.ascontiguousarray(arr)).pin_memory()  # noqa: E731
    hm = {k: (pin(systems[k].ia), pin(systems[k].ja), pin(systems[k].a), pin(systems[k].b),
              torch.zeros(systems[k].n, dtype=torch.float64).pin_memory()) for k in mine}
    h2d = sum(v[0].numel() * 4 + v[1].numel() * 4 + v[2].numel() * 8 + v[3].numel() * 8 + v[4].numel() * 8
              for v in hm.values())
    d2h = sum(v[4].numel() * 8 for v in hm.values())

    m = len(mine)
    arr = lambda vals: (ctypes.c_void_p * m)(*vals)  # noqa: E731
    e_nb = np.array([systems[k].num_block_rows for k in mine], np.int32)
    e_bs = np.array([systems[k].block_size for k in mine], np.int32)
    e_nnzb = np.array([systems[k].nnzb for k in mine], np.int64)
    e_ia = arr([hm[k][0].data_ptr() for k in mine])
    e_ja = arr([hm[k][1].data_ptr() for k in mine])
    e_a = arr([hm[k][2].data_ptr() for k in mine])
    P = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731

    def e2e_step():
        Ss = [CprGmres(**opts) for _ in mine]
        for E, k in zip(Ss, mine):
            E.nb, E.bs = systems[k].num_block_rows, systems[k].block_size
        lib.check(so.jxcpr_batch_setup(m, arr([E.h.value for E in Ss]), P(e_nb), P(e_bs), P(e_nnzb), e_ia, e_ja,
                                       e_a, 0, threads, None))
        EB = CprGmresBatch(Ss)
        for k in mine:
            hm[k][4].zero_()
        res = EB.solve_ptrs([hm[k][3].data_ptr() for k in mine], [hm[k][4].data_ptr() for k in mine], False)
        EB.close()
        for E in Ss:
            E.close()
        return res

    e2e_step()  # warm
    e2e_steps = max(1, min(args.steps, 2))
    torch.cuda.synchronize()
    if ws > 1:
        dist.barrier()
    w0 = time.perf_counter()
    for _ in range(e2e_steps):
        res = e2e_step()
        if not np.all(res["status"] == 0):
            raise RuntimeError("batch e2e: systems did not converge")
    torch.cuda.synchronize()
    e2e_s = torch.tensor([(time.perf_counter() - w0) / e2e_steps], dtype=torch.float64, device="cuda")
    if ws > 1:
        dist.all_reduce(e2e_s, op=dist.ReduceOp.MAX)
    stats = torch.tensor([np.percentile(lat, 50), np.percentile(lat, 99), float(lat.max()), float(fin.max()),
                          worst, float(out["iterations"].sum()), t_setup, t_create], dtype=torch.float64,
                         device="cuda")
    if ws > 1:
        gathered = [torch.zeros_like(stats) for _ in range(ws)]
        dist.all_gather(gathered, stats)
    else:
        gathered = [stats]
    if rank == 0:
        g = torch.stack(gathered).cpu().numpy()
        value = nsys / step_s
        cpu = None
        if ws == 1 and not args.no_cpu_baseline:
            v, _, desc, kind = batch_reference_sample([systems[k] for k in range(nsys)], os.cpu_count() or 1)
            cpu = {"value": v, "unit": "systems/s", "cores": os.cpu_count() or 1, "kind": kind, "sample": desc}
        line = {
            "metric": BATCH_METRIC, "value": value, "unit": "systems/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": step_s * 1e3, "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
            "config": {"workload": WORKLOADS["c3"],
                       "method": "per system: CPR-GMRES(30) to FP64 true rel-res 1e-6, ABF decoupling, AMG V(1,1) "
                                 "(HMIS, ext+i) + 3 block-GS stage-2 sweeps; FP32 preconditioner with Chebyshev-3 on "
                                 "the dense levels, flexible FP64 GMRES on the device (conditional graph nodes, CGS2); "
                                 "operator layouts autotuned per system; all systems of a rank in one graph launch",
                       "options": opts,
                       "value_definition": "systems / device time of one batch solve (input copies, the one graph "
                                           "launch, output copies; hierarchies set up beforehand)",
                       "latency_ms_p50": float(np.median(g[:, 0])), "latency_ms_p99": float(g[:, 1].max()),
                       "latency_ms_max": float(g[:, 2].max()), "last_finish_ms": float(g[:, 3].max()),
                       "latency_definition": "per system: device global timer from the start of its branch to its "
                                             "convergence, inside the one launch",
                       "worst_true_rel_res": float(g[:, 4].max()), "total_iterations": int(g[:, 5].sum()),
                       "setup_s_all_systems": float(g[:, 6].max()), "batch_graph_build_s": float(g[:, 7].max()),
                       "l2_flush": "not needed: the 64 matrices, hierarchies and Krylov bases (~9 GB) exceed L2",
                       "parallelism": f"{ws} GPUs, whole systems per rank (cell-balanced)" if ws > 1 else "1 GPU"},
            "cpu_baseline": cpu,
            "e2e": {"value": nsys / float(e2e_s.item()), "unit": "systems/s", "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h),
                    "note": f"C ABI from pinned host arrays: jxcpr_batch_setup of every system on {threads} host "
                            "threads (upload, decoupling, CPR setup), jxcpr_batch_create, one jxcpr_batch_solve "
                            "(b / x0 uploads, one graph launch, x downloads); the reference arm's time also covers "
                            "decoupling + setup + solve"},
            "gpu_launches": int(launches),
            "clocks": clocks,
        }
        print(json.dumps(line), flush=True)
    if ws > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="c1", choices=sorted(WORKLOADS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-extras", action="store_true",
                    help="config 1 on one GPU: skip the config-4 and config-3 runs summarised in the line")
    ap.add_argument("--opt", action="append", default=[], metavar="KEY=VALUE",
                    help="override a solver option of the measured path (repeatable)")
    ap.add_argument("--path", default="mixed", choices=["mixed", "plain", "bilu"],
                    help="path --profile-solve / --profile-kernels runs (bilu: --profile-kernels only)")
    ap.add_argument("--profile-solve", action="store_true",
                    help="set up, run --warmup solves, then one solve inside a profiler range, and exit")
    ap.add_argument("--profile-kernels", action="store_true",
                    help="set up, then the roofline kernels (stage-2 sweep, level-1 Chebyshev steps, BSR SpMV) "
                         "once inside a profiler range, and exit")
    args = ap.parse_args()
    if args.config == "c3":
        return run_batch_reference(args) if args.impl == "reference" else run_batch(args)
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
