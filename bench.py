"""Benchmark of the clSPARSE hot path on B200: CSR-Adaptive SpMV on the
irregular 2M-row workload (log-normal row lengths mu=2.5 sigma=1.2 plus 50 rows
of 200k nonzeros, columns uniform without replacement, values U[-1,1]; seeded
synthetic input), FP64 (the precision of the reference's published SpM-dV
numbers).

One step = one y = A*x SpMV (alpha=1, beta=0) through clsparseDcsrmv. The
metric is achieved HBM GB/s over the reference's algorithmic byte count
(src/benchmarks/clsparse-bench/functions/clfunc_xSpMdV.hpp:91):
4*(nnz+nrows) + 8*(nnz+ncols+nrows). The matrix (~760 MB) is far larger than
L2 (126 MB), so every step streams it from HBM.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

After the SpMV line's timing, rank 0 (N=1) also measures CG time-to-solution
(key "cg": C1 against the CPU oracle, C3 mixed FP32 vs FP64, C5 learned+mixed
and mixed vs FP64 Jacobi-CG); --no-cg skips it.

N>1 (torchrun): the same matrix is split into nnz-balanced row blocks, one per
rank; a step is every rank's SpMV of its rows followed by an NCCL all-gather of
y (the exchange an iterative method needs before the next product); strong
scaling, timing = max over ranks of device events.
--impl reference times the reference algorithm's CPU restatement (the oracle
port; the reference's OpenCL path cannot run on this machine) on all host cores.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "CG time-to-1e-10 rel. residual, learned+mixed vs plain FP64; SpMV HBM GB/s"
WORKLOAD = "irregular SpMV, n=2,000,000, log-normal(2.5,1.2) rows + 50 rows of 200k nnz, FP64 CSR"


def measured_peak():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def ncu_traffic():
    """dram bytes per launch of the SpMV kernel from the committed ncu summary."""
    p = ROOT / "profiles" / "spmv_irregular_fp64_traffic.json"
    if p.exists():
        return json.loads(p.read_text())
    return None


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=self.f, stderr=subprocess.DEVNULL)
        except (FileNotFoundError, OSError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.f.flush()
        self.f.seek(0)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.f.read().splitlines():
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        os.unlink(self.f.name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# CPU timing protocol of the reference's benchmark client
# (src/benchmarks/clsparse-bench/functions/clfunc_xSpMdV.hpp:208-215 with
# src/benchmarks/clsparse-bench/src/statisticalTimer.cpp:270-293): SAMPLES
# host-timed samples, each the mean of CALLS back-to-back calls; samples
# further than 3 standard deviations from the mean are pruned; the mean of
# the rest is reported.
CPU_SAMPLES = 20
CPU_CALLS = 20


def cpu_spmv_protocol(rp, col, val, samples=CPU_SAMPLES, calls=CPU_CALLS):
    """The oracle port of the reference SpMV (FP64, alpha 1, beta 0) on all
    host cores through a thread pool created once, timed by the protocol
    above. One function serves both the repo arm's cpu_baseline and the
    --impl reference arm, so the two report the same measurement."""
    import oracle
    n = len(rp) - 1
    threads = os.cpu_count() or 1
    x = np.random.default_rng(3).uniform(-1, 1, n)
    y = np.zeros(n)
    nbytes = 4 * (len(col) + n) + 8 * (len(col) + 2 * n)
    for _ in range(3):  # warm: pool start-up, page faults, caches
        oracle.dcsrmv_mt(rp, col, val, 1.0, x, 0.0, y, threads)
    per_call = []
    for _ in range(samples):
        t0 = time.perf_counter()
        for _ in range(calls):
            oracle.dcsrmv_mt(rp, col, val, 1.0, x, 0.0, y, threads)
        per_call.append((time.perf_counter() - t0) / calls)
    mean = statistics.fmean(per_call)
    sd = statistics.pstdev(per_call)
    kept = [t for t in per_call if abs(t - mean) <= 3.0 * sd] or per_call
    t = statistics.fmean(kept)
    gbs = nbytes / t / 1e9
    return {"value": round(gbs, 3), "unit": "GB/s", "cores": threads, "kind": "port",
            "seconds_per_call": t,
            "sample": f"{samples} samples x {calls} full FP64 SpMVs of the same 2M-row matrix, 3-sigma pruning "
                      f"({len(per_call) - len(kept)} pruned); row ranges balanced by nnz over a pool of "
                      f"{threads} host threads created once"}


def cpu_baseline(rp, col, val):
    """Oracle port of the reference SpMV on all host cores (the protocol above)."""
    r = cpu_spmv_protocol(rp, col, val)
    r.pop("seconds_per_call")
    return r


def _timed(fn, reps=2):
    """Device-synchronised wall time of the last of `reps` calls (the first
    builds the cached solver graph)."""
    import torch
    r = None
    t = 0.0
    for _ in range(reps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r = fn()
        torch.cuda.synchronize()
        t = time.perf_counter() - t0
    return t, r


# Inner tolerance of the refinement: each inner solve (continued across
# refinements) reduces its residual by this factor before the FP64 residual
# is recomputed and replaced.
INNER_TOL = 0.3


def cg_profile(iters: int):
    """A short FP64 Jacobi-CG on the C5 matrix with the solver loop in host
    chunks (loop mode 1), so every kernel of an iteration is an ordinary
    stream launch a profiler lists (graph nodes of the default loop are not)."""
    import torch
    from clsparse_b200 import _lib as L
    from clsparse_b200 import api, matgen
    api.setup()
    ctrl = api.Control()
    ctrl.set_solver_loop_mode(1)
    os.environ["CLSPARSE_B200_DIA"] = "0"  # the graph engine's kernels, not the banded engine's one launch
    A = api.CsrMatrix.from_numpy(*matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005))
    A.create_meta(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    sc = api.SolverControl(L.DIAGONAL, iters, 0.0, 0.0)
    sc.set_norm(2)
    info = api.solve("cg", x, A, b, sc, ctrl)
    sc.release()
    print(json.dumps({"cg_profile_iterations": info["nIters"]}), flush=True)
    ctrl.release()


def dia_cg_profile(iters: int):
    """Two FP64 Jacobi-CG calls of ITERS iterations on the C5 matrix through
    the banded drop-in engine (solver loop mode 3): per call the offset
    detection, the diagonal-layout fill, the symmetry check and one launch
    of the cooperative CG kernel."""
    import torch
    from clsparse_b200 import _lib as L
    from clsparse_b200 import api, matgen
    api.setup()
    ctrl = api.Control()
    ctrl.set_solver_loop_mode(3)
    A = api.CsrMatrix.from_numpy(*matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005))
    A.create_meta(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    for _ in range(2):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, iters, 0.0, 0.0)
        sc.set_norm(2)
        info = api.solve("cg", x, A, b, sc, ctrl)
        sc.release()
    torch.cuda.synchronize()
    print(json.dumps({"dia_cg_profile_iterations": info["nIters"]}), flush=True)
    ctrl.release()


def batched_profile(nsys: int):
    """Two batched FP32 Jacobi-CG solves (clsparseScsrcgBatched) over the
    first `nsys` systems of the C4 family (same generator and seed), for a
    profiler: per call the offset detection, the diagonal layout and one
    persistent solver launch."""
    import torch
    from clsparse_b200 import _lib as L
    from clsparse_b200 import api, matgen
    api.setup()
    ctrl = api.Control()
    rp, col, val, off, _ = matgen.batched_systems(nsys, 500, 50_000, sigma=1.0, seed=11)
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=torch.float32)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), dtype=torch.float32, device="cuda")
    for _ in range(2):
        x = torch.zeros(n, dtype=torch.float32, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 20000, 1e-5, 0.0)
        r = api.cg_batched(x, A, b, off, sc, ctrl)
        sc.release()
    torch.cuda.synchronize()
    print(json.dumps({"batched_profile_systems": nsys, "converged": int(r["converged"])}), flush=True)
    ctrl.release()


def gnn_profile(builds: int):
    """BF16 factor builds of the learned preconditioner on the C5 matrix
    (1,048,576 rows): the network's forward pass with its dense layers on the
    tcgen05 tensor cores (linear_fwd_umma), then the factor export. Prints the
    median build time; for profiler launch lists and captures."""
    import torch
    from clsparse_b200 import api, matgen
    api.setup()
    ctrl = api.Control()
    A = api.CsrMatrix.from_numpy(*matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005))
    spai = api.Spai(3)
    spai.set_matrix(A, ctrl)
    ts = []
    for _ in range(builds):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        spai.build(ctrl)
        torch.cuda.synchronize()
        ts.append(time.perf_counter() - t0)
    spai.release()
    ctrl.release()
    print(json.dumps({"gnn_profile_builds": builds, "median_build_ms": round(1e3 * float(np.median(ts)), 3)}),
          flush=True)


def learned_profile(iters: int):
    """A short learned + mixed FP32 solve on the C5 matrix (network trained
    briefly on 32^2 members of the family) with the solver loop in host chunks
    (loop mode 1), so every kernel of a learned inner iteration is an ordinary
    stream launch a profiler lists; ITERS bounds the inner iterations."""
    import torch
    from clsparse_b200 import _lib as L
    from clsparse_b200 import api, learn, matgen
    api.setup()
    ctrl = api.Control()
    spai, _ = learn.train(ctrl, sizes=(32,), seeds=range(2), steps=20, lr=3e-3)
    ctrl.set_solver_loop_mode(1)
    A = api.CsrMatrix.from_numpy(*matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005))
    A.create_meta(ctrl)
    spai.set_matrix(A, ctrl)
    spai.build(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    sc = api.SolverControl(L.DIAGONAL, iters, 1e-10, 0.0)
    info = api.cg_learned(x, A, b, sc, spai, ctrl, inner="fp32", inner_tol=0.3)
    sc.release()
    spai.release()
    print(json.dumps({"learned_profile_inner_iterations": info["innerIterations"]}), flush=True)
    ctrl.release()


def dist_cg_section(rank: int, world: int):
    """Row-partitioned FP64 Jacobi-CG (clsparseB200DistCg*) on the C3 matrix
    (128^3 log-normal diffusion, 2,097,152 rows) over the ranks of this run:
    nnz-balanced row blocks, a halo exchange of boundary planes (NCCL
    send/recv) and one all-reduce of three FP64 sums per iteration, the
    reference's L1 stop test at 1e-10. Every rank calls it; the time is the
    max over ranks of the device time of a whole solve (best of two after one
    warm-up solve). At one rank the same kernels run without collectives."""
    import torch
    import torch.distributed as dist

    from clsparse_b200 import api, matgen
    from clsparse_b200 import distributed as D
    rp, col, val = matgen.diffusion3d_lognormal(128, sigma=1.5, seed=3)
    n = len(rp) - 1
    b = np.random.default_rng(1).uniform(-1, 1, n)
    parts = D.row_partition(rp, world)
    r0, r1 = parts[rank]
    _, lcol, _ = D.local_rows(rp, col, val, r0, r1)
    if world > 1:
        plan = D.plan_for_rank(lcol, parts, rank)
        comm = D.TorchComm()
    else:
        plan = D.make_plans([D.needed_columns(lcol, r0, r1)], parts)[0]
        comm = D.LocalComm()
    ctrl = api.Control()
    rk = D.DeviceRank(plan, *D.setup_local(rp, col, val, parts, rank, plan), 1, ctrl)
    bl = torch.tensor(b[r0:r1], device="cuda")
    times, info = [], None
    for _ in range(3):
        x = torch.zeros(r1 - r0, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(1, 20000, 1e-10, 0.0)
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        info = D.dist_cg([rk], comm, [x], [bl], [sc])
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
        sc.release()
    rk.release()
    t = torch.tensor([min(times[1:])], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ctrl.release()
    ms = float(t.item())
    halo = sum(cnt for _, cnt in plan.recv.values()) if plan.mode == D.HALO else plan.ext_len - plan.chunk
    return {"workload": "3D 7-point log-normal diffusion 128^3 (n=2,097,152, sigma 1.5), FP64 Jacobi-CG, "
                        "L1 stop test 1e-10, rows partitioned over the ranks",
            "ranks": world, "exchange": plan.mode, "iterations": info["nIters"],
            "relative_residual": info["currentResidual"], "s": round(ms * 1e-3, 5),
            "us_per_iteration": round(1e3 * ms / max(info["nIters"] + 1, 1), 2),
            "remote_entries_per_exchange_rank0": int(halo),
            "collectives_per_iteration": "1 exchange + 1 all-reduce of 3 FP64" if world > 1 else "none (one rank)"}


def cg_section(ctrl, with_cpu: bool):
    """Time-to-solution of the solver configurations the headline metric names.

    C1  2D Poisson 512^2, FP64 Jacobi-CG with the reference's L1 stop test at
        1e-10 (clsparseDcsrcg) -- beside it the oracle restatement of the
        reference CG on one host core.
    C3  3D 7-point log-normal diffusion 128^3 (sigma 1.5): FP64 Jacobi-CG vs
        the FP64 refinement around FP32 CG (clsparseDcsrcgMixed), both to a
        relative L2 true residual of 1e-10.
    C5  2D GRF diffusion 1024^2 (corr 0.05, sigma 2): FP64 Jacobi-CG vs
        mixed FP32 and vs learned (G^T G, BF16 factor) + mixed FP32
        (clsparseDcsrcgLearned); the network is trained on the GPU by the
        library's kernels on 128^2 matrices of the family (different seeds)
        before the timed solves; training time is reported separately.
    Beside each FP64 Jacobi-CG entry, banded_loop_mode3 times the same
    clsparseDcsrcg call with solver loop mode 3 (the banded drop-in engine).
    (The default mode runs these matrices on the same engine.)
    Each solve is timed on its second call (the first captures the graph).
    Every solution's error against the FP64 oracle solution is stated
    (error_vs_fp64_oracle, relative 2-norm): C1 against the serial oracle
    restatement of the reference CG at the same stop test, C3 / C5 against the
    oracle's threaded FP64 Jacobi-PCG run to a relative residual of 1e-12,
    computed on the host after all GPU timings."""
    import torch
    from clsparse_b200 import _lib as L
    from clsparse_b200 import api, learn, matgen

    out = {}
    solutions = {}  # config -> {entry: x on the host}, compared with the oracle at the end

    def fp64_cg(A, b, x, l2=True, max_iters=200000, loop_mode=0):
        def run():
            x.zero_()
            sc = api.SolverControl(L.DIAGONAL, max_iters, 1e-10, 0.0)
            if l2:
                sc.set_norm(2)
            info = api.solve("cg", x, A, b, sc, ctrl)
            sc.release()
            return info
        ctrl.set_solver_loop_mode(loop_mode)
        try:
            return _timed(run)
        finally:
            ctrl.set_solver_loop_mode(0)

    # The same drop-in clsparseDcsrcg call with the banded engine (solver loop
    # mode 3): one cooperative launch over a diagonal-storage copy rebuilt at
    # every call (inside the timing), rows in the reference's CSR-Adaptive
    # order; its x against the default engine's.
    def banded_entry(A, b, x, l2, t_default):
        x_default = x.clone()
        t, info = fp64_cg(A, b, x, l2=l2, loop_mode=3)
        d = float((x - x_default).abs().max() / x_default.abs().max())
        return {"s": round(t, 5), "iterations": info["nIters"] + (1 if l2 else 0),
                "speedup_vs_default_engine": round(t_default / t, 3), "max_rel_diff_vs_default_engine": d}

    def true_res(np_mat, x, b):
        import scipy.sparse as sp
        rp, col, val = np_mat
        n = len(rp) - 1
        M = sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))
        bb = b.cpu().numpy()
        return float(np.linalg.norm(bb - M @ x.cpu().numpy()) / np.linalg.norm(bb))

    # C1
    c1 = matgen.poisson2d(512)
    A = api.CsrMatrix.from_numpy(*c1)
    A.create_meta(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    t, info = fp64_cg(A, b, x, l2=False)
    c1_out = {"workload": "2D Poisson 512x512 (n=262,144), FP64 Jacobi-CG, L1 stop test 1e-10",
              "gpu_s": round(t, 5), "iterations": info["nIters"]}
    if with_cpu:
        import oracle
        rp, col, val = c1
        t0 = time.perf_counter()
        xo, oi = oracle.solve("cg", np.float64, rp, col, val, np.zeros(n), b.cpu().numpy(), 1, 200000, 1e-10, 0.0)
        tc = time.perf_counter() - t0
        c1_out["cpu_baseline"] = {"s": round(tc, 3), "iterations": oi.nIters, "cores": 1, "kind": "port",
                                  "sample": "the whole solve, oracle restatement of the reference CG"}
        c1_out["speedup_vs_cpu"] = round(tc / t, 1)
        xg = x.cpu().numpy()
        c1_out["error_vs_fp64_oracle"] = float(np.linalg.norm(xg - xo) / np.linalg.norm(xo))
    c1_banded = banded_entry(A, b, x, False, t)
    if with_cpu:
        c1_banded["speedup_vs_cpu"] = round(tc / c1_banded["s"], 1)
    c1_out["banded_loop_mode3"] = c1_banded
    out["C1"] = c1_out
    del A

    # C3
    c3 = matgen.diffusion3d_lognormal(128, sigma=1.5, seed=3)
    A = api.CsrMatrix.from_numpy(*c3)
    A.create_meta(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    t64, i64 = fp64_cg(A, b, x)
    r64 = true_res(c3, x, b)
    solutions["C3"] = {"fp64_jacobi": x.cpu().numpy()}
    c3_banded = banded_entry(A, b, x, True, t64)

    def mixed():
        x.zero_()
        sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
        r = api.cg_mixed(x, A, b, sc, ctrl, inner="fp32", inner_tol=INNER_TOL)
        sc.release()
        return r
    tm, im = _timed(mixed)
    solutions["C3"]["mixed_fp32"] = x.cpu().numpy()
    r3 = true_res(c3, x, b)

    # BF16 matrix values (FP32 vectors) in the same refinement: the
    # refinement contracts only while ||A_bf16^-1 (A - A_bf16)|| < 1; the
    # entry records whether it converged and the measured contraction per
    # refinement step, (final / initial FP64 residual)^(1 / steps).
    def mixed_bf16():
        x.zero_()
        sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
        r = api.cg_mixed(x, A, b, sc, ctrl, inner="bf16", inner_tol=INNER_TOL)
        sc.release()
        return r
    tbf, ibf = _timed(mixed_bf16)
    steps = max(1, ibf["outerIterations"])
    contraction = (ibf["trueResidual"] / ibf["initialTrueResidual"]) ** (1.0 / steps) \
        if ibf["initialTrueResidual"] > 0 and ibf["trueResidual"] > 0 else 0.0
    bf16_out = {"s": round(tbf, 5), "converged": int(ibf["converged"]), "inner_iterations": ibf["innerIterations"],
                "refinements": ibf["outerIterations"], "true_residual": ibf["trueResidual"],
                "contraction_per_refinement": round(contraction, 4)}
    if ibf["converged"]:
        solutions["C3"]["mixed_bf16"] = x.cpu().numpy()
    out["C3"] = {"workload": "3D 7-point log-normal diffusion 128^3 (n=2,097,152, sigma 1.5), rel. L2 residual 1e-10",
                 "fp64_jacobi": {"s": round(t64, 5), "iterations": i64["nIters"] + 1, "true_residual": r64,
                                 "banded_loop_mode3": c3_banded},
                 "mixed_fp32": {"s": round(tm, 5), "inner_iterations": im["innerIterations"],
                                "refinements": im["outerIterations"], "true_residual": r3},
                 "mixed_bf16": bf16_out,
                 "speedup": round(t64 / tm, 3)}
    del A

    # C4: 4096 SPD systems in one persistent launch (FP32 CG, FP64 residual
    # check). Tolerance 1e-5: FP32 storage of x limits the reachable relative
    # residual near 1e-6 on the worse-conditioned systems.
    rp4, col4, val4, off4, _ = matgen.batched_systems(4096, 500, 50_000, sigma=1.0, seed=11)
    A = api.CsrMatrix.from_numpy(rp4, col4, val4, dtype=torch.float32)
    n = A.num_rows
    b4 = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), dtype=torch.float32, device="cuda")
    x4 = torch.zeros(n, dtype=torch.float32, device="cuda")

    def batched():
        x4.zero_()
        sc = api.SolverControl(L.DIAGONAL, 20000, 1e-5, 0.0)
        r = api.cg_batched(x4, A, b4, off4, sc, ctrl)
        sc.release()
        return r
    tb, rb = _timed(batched)
    out["C4"] = {"workload": "4096 SPD stencil systems, n log-uniform in [500, 50000] (sum n = %d, nnz = %d), "
                             "log-normal coefficients sigma 1.0, FP32 Jacobi-CG, FP64 residual check, rel. 1e-5"
                             % (n, len(val4)),
                 "s": round(tb, 4), "systems_per_s": round(4096 / tb, 1), "converged": int(rb["converged"]),
                 "max_iterations": int(rb["max_iterations"]), "worst_fp64_residual": float(rb["worst_residual"])}
    del A, x4, b4

    # C5
    t0 = time.perf_counter()
    spai, hist = learn.train(ctrl, sizes=(128,), seeds=range(6), steps=300, lr=3e-3)
    torch.cuda.synchronize()
    train_s = time.perf_counter() - t0
    c5 = matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005)
    A = api.CsrMatrix.from_numpy(*c5)
    A.create_meta(ctrl)
    n = A.num_rows
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda")
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    t64, i64 = fp64_cg(A, b, x)
    r64 = true_res(c5, x, b)
    solutions["C5"] = {"fp64_jacobi": x.cpu().numpy()}
    c5_banded = banded_entry(A, b, x, True, t64)

    def mixed5():
        x.zero_()
        sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
        r = api.cg_mixed(x, A, b, sc, ctrl, inner="fp32", inner_tol=INNER_TOL)
        sc.release()
        return r
    tm, im = _timed(mixed5)
    rm = true_res(c5, x, b)
    solutions["C5"]["mixed_fp32"] = x.cpu().numpy()
    # Factor build = graph of A + network forward + export of G and G^T. The
    # first build for a matrix size allocates the network's buffers; the
    # second (timed, what every new matrix of that size costs) rebuilds the
    # graph and the factor into them.
    tb0 = time.perf_counter()
    spai.set_matrix(A, ctrl)
    spai.build(ctrl)
    torch.cuda.synchronize()
    build_cold_s = time.perf_counter() - tb0
    tb0 = time.perf_counter()
    spai.set_matrix(A, ctrl)
    spai.build(ctrl)
    torch.cuda.synchronize()
    build_s = time.perf_counter() - tb0

    def learned():
        x.zero_()
        sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
        r = api.cg_learned(x, A, b, sc, spai, ctrl, inner="fp32", inner_tol=INNER_TOL)
        sc.release()
        return r
    tl, il = _timed(learned)
    rl = true_res(c5, x, b)
    solutions["C5"]["learned_mixed_fp32"] = x.cpu().numpy()
    spai.release()
    out["C5"] = {"workload": "2D GRF diffusion 1024^2 (n=1,048,576, corr 0.05, sigma 2), rel. L2 residual 1e-10",
                 "fp64_jacobi": {"s": round(t64, 5), "iterations": i64["nIters"] + 1, "true_residual": r64,
                                 "banded_loop_mode3": c5_banded},
                 "mixed_fp32": {"s": round(tm, 5), "inner_iterations": im["innerIterations"],
                                "refinements": im["outerIterations"], "true_residual": rm,
                                "speedup": round(t64 / tm, 3)},
                 "learned_mixed_fp32": {"s": round(tl, 5), "inner_iterations": il["innerIterations"],
                                        "refinements": il["outerIterations"], "true_residual": rl,
                                        "fell_back_to_jacobi": il["fell_back"],
                                        "factor_build_s": round(build_s, 4),
                                        "factor_build_first_s": round(build_cold_s, 4),
                                        "speedup": round(t64 / tl, 3),
                                        "speedup_with_factor_build": round(t64 / (tl + build_s), 3)},
                 "train_s": round(train_s, 2), "train_loss_first_last": [hist[0], hist[-1]]}
    # errors against the FP64 oracle solutions (host, after every GPU timing)
    import oracle
    for name, mat in (("C3", c3), ("C5", c5)):
        rp, col, val = mat
        bh = np.random.default_rng(1).uniform(-1, 1, len(rp) - 1)
        xo, _, _ = oracle.reference_solution(rp, col, val, bh, rel_tol=1e-12)
        for entry, xs in solutions[name].items():
            out[name][entry]["error_vs_fp64_oracle"] = float(np.linalg.norm(xs - xo) / np.linalg.norm(xo))
    return out


def e2e_pipelined(api, ctrl, A, stream, hx, n, one, zero, steps, y_resident):
    """End-to-end SpMV stream from host memory: every step copies x from
    pinned host memory, runs clsparseDcsrmv on the control's stream and copies
    y back. Two device buffers of x and y and two copy streams let step k's
    SpMV overlap step k+1's host-to-device and step k-1's device-to-host copy
    (PCIe is full duplex); events order every buffer reuse. Returns the device
    time from the first copy's start to the last copy's end (ms)."""
    import torch
    s_in = torch.cuda.Stream()
    s_out = torch.cuda.Stream()
    xb = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    yb = [torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    hy = [torch.empty(n, dtype=torch.float64, pin_memory=True) for _ in range(2)]
    copied = [torch.cuda.Event() for _ in range(2)]
    computed = [torch.cuda.Event() for _ in range(2)]
    drained = [torch.cuda.Event() for _ in range(2)]

    def run(count, t0=None, t1=None):
        if t0 is not None:
            t0.record(s_in)
        for k in range(count):
            b = k & 1
            if k >= 2:
                s_in.wait_event(computed[b])  # SpMV k-2 has read xb[b]
            with torch.cuda.stream(s_in):
                xb[b].copy_(hx, non_blocking=True)
            copied[b].record(s_in)
            stream.wait_event(copied[b])
            if k >= 2:
                stream.wait_event(drained[b])  # D2H k-2 has read yb[b]
            api.csrmv(one, A, xb[b], zero, yb[b], ctrl)
            computed[b].record(stream)
            s_out.wait_event(computed[b])
            with torch.cuda.stream(s_out):
                hy[b].copy_(yb[b], non_blocking=True)
            drained[b].record(s_out)
        if t1 is not None:
            s_out.wait_stream(s_in)
            t1.record(s_out)

    run(4)
    torch.cuda.synchronize()
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    s_in.wait_stream(stream)
    run(steps, t0, t1)
    torch.cuda.synchronize()
    # the streamed result is the device-resident one, bit for bit
    if not torch.equal(hy[(steps - 1) & 1], y_resident.cpu()):
        raise RuntimeError("pipelined end-to-end SpMV result differs from the device-resident one")
    return t0.elapsed_time(t1)


def spmv_fp32(api, ctrl, stream, rp, col, val, steps, peak):
    """The same irregular matrix with FP32 values and vectors
    (clsparseScsrmv): per-launch CUDA-event time, GB/s over the FP32 byte
    count 4*(nnz + nrows) + 4*(nnz + 2*nrows)."""
    import torch
    n = len(rp) - 1
    nbytes = 4 * (len(col) + n) + 4 * (len(col) + 2 * n)
    with torch.cuda.stream(stream):
        A = api.CsrMatrix.from_numpy(rp, col, val, dtype=torch.float32)
        A.create_meta(ctrl)
        x = torch.tensor(np.random.default_rng(3).uniform(-1, 1, n), dtype=torch.float32, device="cuda")
        y = torch.zeros(n, dtype=torch.float32, device="cuda")
        one = torch.ones(1, dtype=torch.float32, device="cuda")
        zero = torch.zeros(1, dtype=torch.float32, device="cuda")
        for _ in range(5):
            api.csrmv(one, A, x, zero, y, ctrl)
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        for s, e in ev:
            s.record(stream)
            api.csrmv(one, A, x, zero, y, ctrl)
            e.record(stream)
        torch.cuda.synchronize()
    ms = float(np.mean([s.elapsed_time(e) for s, e in ev]))
    gbs = nbytes / (ms * 1e-3) / 1e9
    return {"value": round(gbs, 2), "unit": "GB/s", "us_per_launch": round(1e3 * ms, 2), "bytes_per_step": nbytes,
            "roofline_frac": round(gbs / peak, 4), "kernel": "csr_adaptive_kernel<float,false,0>"}


def make_matrix():
    from clsparse_b200 import matgen
    return matgen.irregular(2_000_000, mu=2.5, sigma=1.2, n_dense=50, dense_len=200_000, seed=7)


def run_reference(args, rank, world):
    """The reference arm: the oracle port of the reference SpMV on all host
    cores, by the same protocol and function as the repo arm's cpu_baseline:
    each step is one sample of CPU_CALLS SpMVs (fewer calls per sample above
    20 steps, so that about 400 SpMVs are timed whatever --steps is)."""
    if rank != 0:
        return
    rp, col, val = make_matrix()
    n = len(rp) - 1
    nbytes = 4 * (len(col) + n) + 8 * (len(col) + 2 * n)
    samples = max(args.steps, 3)
    calls = CPU_CALLS if samples <= CPU_SAMPLES else max(2, (CPU_SAMPLES * CPU_CALLS) // samples)
    r = cpu_spmv_protocol(rp, col, val, samples=samples, calls=calls)
    gbs = r["value"]
    line = {
        "impl": "reference", "metric": METRIC, "value": gbs, "unit": "GB/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(1e3 * r["seconds_per_call"], 4), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
        "config": {"workload": WORKLOAD, "nnz": int(len(col)), "rows": n, "bytes_per_step": nbytes},
        "cpu_baseline": {"value": gbs, "unit": "GB/s", "cores": r["cores"], "kind": "port",
                         "sample": r["sample"] + " (oracle restatement of the reference algorithm; the "
                                                 "reference's OpenCL path has no runtime here)"},
        "e2e": {"value": gbs, "unit": "GB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_ours(args, rank, world, local_rank):
    import torch
    import torch.distributed as dist

    from clsparse_b200 import api

    from clsparse_b200 import distributed as D

    torch.cuda.set_device(local_rank)
    rp, col, val = make_matrix()
    n = len(rp) - 1
    nnz = len(col)
    nbytes = 4 * (nnz + n) + 8 * (nnz + n + n)
    # N > 1: this rank's nnz-balanced block of rows (global column indices)
    parts = D.row_partition(rp, world)
    r0, r1 = parts[rank]
    lrp, lcol, lval = D.local_rows(rp, col, val, r0, r1) if world > 1 else (rp, col, val)
    m = max(b - a for a, b in parts)

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctrl = api.Control(stream)
        A = api.CsrMatrix.from_numpy(lrp, lcol, lval, num_cols=n, dtype=torch.float64)
        A.create_meta(ctrl)
        ctrl.enable_async(True)
        x = torch.tensor(np.random.default_rng(3).uniform(-1, 1, n), device="cuda")
        ybuf = torch.zeros(m, dtype=torch.float64, device="cuda")
        y = ybuf[: r1 - r0]
        yfull = torch.zeros(world * m, dtype=torch.float64, device="cuda")
        one = torch.ones(1, dtype=torch.float64, device="cuda")
        zero = torch.zeros(1, dtype=torch.float64, device="cuda")

        def step():
            api.csrmv(one, A, x, zero, y, ctrl)
            if world > 1:
                # the exchange an iterative method needs: every rank gets all of y
                dist.all_gather_into_tensor(yfull, ybuf)

        for _ in range(args.warmup):
            step()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        sampler = ClockSampler(local_rank)
        sampler.start()
        time.sleep(0.3)
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
              for _ in range(args.steps)]
        t_all0 = torch.cuda.Event(enable_timing=True)
        t_all1 = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        t_all0.record(stream)
        for s, e in ev:
            s.record(stream)
            step()
            e.record(stream)
        t_all1.record(stream)
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        per = [s.elapsed_time(e) for s, e in ev]
        total_ms = t_all0.elapsed_time(t_all1)

        # end to end through the C ABI with host buffers: H2D x, SpMV, D2H y
        hx = torch.empty(n, dtype=torch.float64, pin_memory=True)
        hx.copy_(x.cpu())
        hy = torch.empty(r1 - r0, dtype=torch.float64, pin_memory=True)
        for _ in range(3):
            x.copy_(hx, non_blocking=True)
            step()
            hy.copy_(y, non_blocking=True)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(args.steps):
            x.copy_(hx, non_blocking=True)
            step()
            hy.copy_(y, non_blocking=True)
        e1.record(stream)
        torch.cuda.synchronize()
        e2e_ms = e0.elapsed_time(e1)
        e2e_serial_ms = e2e_ms
        if world == 1:
            e2e_ms = e2e_pipelined(api, ctrl, A, stream, hx, n, one, zero, args.steps, y)
        clocks = sampler.stop()

    t = torch.tensor([total_ms, e2e_ms, float(np.mean(per)), e2e_serial_ms], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    total_ms, e2e_ms, avg_launch_ms, e2e_serial_ms = t.tolist()
    dcg = None
    if not args.no_cg:
        # every rank takes part; an error (raised alike on every rank: the
        # ranks run the same stages) is reported instead of the entry
        try:
            dcg = dist_cg_section(rank, world)
        except Exception as exc:  # noqa: BLE001
            dcg = {"error": f"{type(exc).__name__}: {exc}"[:300]}
    if rank != 0:
        ctrl.release()
        return
    value = nbytes * args.steps / (total_ms * 1e-3) / 1e9
    e2e_val = nbytes * args.steps / (e2e_ms * 1e-3) / 1e9
    # the kernel's own bytes: this rank's share of the matrix and vectors
    achieved = (nbytes / world) / (avg_launch_ms * 1e-3) / 1e9
    peak, peak_kind = measured_peak()
    tr = ncu_traffic()
    line = {
        "metric": METRIC, "value": round(value, 2), "unit": "GB/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(total_ms / args.steps, 5), "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
        "config": {"workload": WORKLOAD, "rows": n, "nnz": nnz, "bytes_per_step": nbytes,
                   "l2": "inputs larger than L2 (~760 MB streamed per step)",
                   "parallelism": (f"row-sharded x{world} (nnz-balanced row blocks), y all-gathered over NCCL "
                                   "every step") if world > 1 else "single GPU"},
        "roofline": {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                     "frac": round(achieved / peak, 4), "peak_kind": peak_kind,
                     "traffic": (tr or {}).get("dram_bytes_per_launch"),
                     "algorithmic_bytes_per_launch": nbytes,
                     "kernel": "csr_adaptive_kernel<double,false,0>"},
        "e2e": {"value": round(e2e_val, 2), "unit": "GB/s", "h2d_bytes_per_step": 8 * n * world,
                "d2h_bytes_per_step": 8 * n,
                "mode": ("pipelined: every step copies its x in and its y out, double-buffered on two copy "
                         "streams so step k's SpMV overlaps step k+1's H2D and step k-1's D2H")
                if world == 1 else "serial: H2D x, SpMV + all-gather, D2H y on one stream",
                "serial_value": round(nbytes * args.steps / (e2e_serial_ms * 1e-3) / 1e9, 2)},
        "gpu_launches": args.steps,
        "clocks": clocks,
        "gflops": round(2 * nnz * args.steps / (total_ms * 1e-3) / 1e9, 2),
    }
    if dcg is not None:
        line["dist_cg"] = dcg
    if world == 1:
        line["fp32"] = spmv_fp32(api, ctrl, stream, rp, col, val, args.steps, peak)
    if world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline(rp, col, val)
    if world == 1 and not args.no_cg:
        del A
        with torch.cuda.stream(stream):
            ctrl.enable_async(False)
            line["cg"] = cg_section(ctrl, with_cpu=not args.no_cpu_baseline)
    print(json.dumps(line), flush=True)
    ctrl.release()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-cg", action="store_true", help="skip the CG time-to-solution section")
    ap.add_argument("--gnn-profile", type=int, default=0, metavar="BUILDS",
                    help="only run BUILDS learned-factor builds on the C5 matrix (profiling)")
    ap.add_argument("--learned-profile", type=int, default=0, metavar="ITERS",
                    help="only run a learned + mixed solve of at most ITERS inner iterations in loop mode 1 "
                         "(profiling)")
    ap.add_argument("--cg-profile", type=int, default=0, metavar="ITERS",
                    help="only run ITERS iterations of FP64 Jacobi-CG on the C5 matrix with directly launched "
                         "kernels (for a profiler's launch list), then exit")
    ap.add_argument("--batched-profile", type=int, default=0, metavar="NSYS",
                    help="only run two batched solves over the first NSYS systems of the C4 family, then exit")
    ap.add_argument("--dia-cg-profile", type=int, default=0, metavar="ITERS",
                    help="only run two FP64 Jacobi-CG calls of ITERS iterations on the C5 matrix through the "
                         "banded drop-in engine (loop mode 3), then exit")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.dia_cg_profile:
        dia_cg_profile(args.dia_cg_profile)
        return
    if args.batched_profile:
        batched_profile(args.batched_profile)
        return
    if args.gnn_profile:
        gnn_profile(args.gnn_profile)
        return
    if args.cg_profile:
        cg_profile(args.cg_profile)
        return
    if args.learned_profile:
        learned_profile(args.learned_profile)
        return
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return
    import torch.distributed as dist
    if world > 1:
        import datetime
        import torch
        torch.cuda.set_device(local_rank)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    try:
        run_ours(args, rank, world, local_rank)
    finally:
        if world > 1:
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
