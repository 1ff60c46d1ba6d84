"""Solvers at the full configured sizes, through the C ABI, against the CPU
oracle.

* C1 -- 2D Poisson 512x512 (262,144 rows), FP64 Jacobi-CG with the
  reference's L1 stop test at 1e-10 (clsparseDcsrcg), against the serial
  oracle restatement of the reference CG (conjugate-gradients.hpp:47-228):
  the same stop decision within 1% of the iterations, the same initial
  residual, and the same solution -- on the graph engine and on the banded
  drop-in engine (solver loop mode 3; the default, too, at these sizes), as
  the FP64 Jacobi-CG of C3 and C5.
* C3 -- 3D 7-point log-normal diffusion 128^3 (2,097,152 rows, sigma 1.5)
  and C5 -- 2D Gaussian-random-field diffusion 1024^2 (1,048,576 rows,
  correlation length 0.05, sigma 2): FP64 Jacobi-CG, the mixed-precision
  refinement and (C5) the learned factor with the refinement, each to a
  relative L2 residual of 1e-10, recomputed here in FP64 on the host, and
  each solution's error against the FP64 oracle solution (the oracle's
  threaded Jacobi-PCG run to 1e-12).

Error bar: 1e-7 relative in the 2-norm. Two FP64 CG solutions at residual
1e-10 and 1e-12 of these matrices differ by about 1e-9 (C3) and 1e-10 (C5),
measured with the oracle alone, so the bar leaves two orders of magnitude for
rounding-order differences while still catching a wrong answer."""
from __future__ import annotations

import functools

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api, learn, matgen

pytestmark = pytest.mark.gpu

ERR_BAR = 1e-7


@functools.lru_cache(maxsize=None)
def config(name):
    if name == "C1":
        return matgen.poisson2d(512)
    if name == "C3":
        return matgen.diffusion3d_lognormal(128, sigma=1.5, seed=3)
    if name == "C5":
        return matgen.diffusion2d_grf(1024, corr_len=0.05, sigma=2.0, seed=1005)
    raise KeyError(name)


def rhs(n):
    return np.random.default_rng(1).uniform(-1, 1, n)


@functools.lru_cache(maxsize=None)
def fp64_oracle_solution(name):
    import oracle
    rp, col, val = config(name)
    x, it, res = oracle.reference_solution(rp, col, val, rhs(len(rp) - 1), rel_tol=1e-12)
    assert res <= 1e-12
    return x


@functools.lru_cache(maxsize=None)
def oracle_iterations_1e10(name):
    import oracle
    rp, col, val = config(name)
    return oracle.reference_solution(rp, col, val, rhs(len(rp) - 1), rel_tol=1e-10)[1]


def scipy_matrix(name):
    rp, col, val = config(name)
    n = len(rp) - 1
    return sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))


def l2_residual(name, x):
    b = rhs(len(config(name)[0]) - 1)
    return float(np.linalg.norm(b - scipy_matrix(name) @ x) / np.linalg.norm(b))


def error_vs_oracle(name, x):
    xo = fp64_oracle_solution(name)
    return float(np.linalg.norm(x - xo) / np.linalg.norm(xo))


def device_problem(ctrl, name):
    A = api.CsrMatrix.from_numpy(*config(name))
    A.create_meta(ctrl)
    b = torch.tensor(rhs(A.num_rows), device="cuda")
    x = torch.zeros(A.num_rows, dtype=torch.float64, device="cuda")
    return A, b, x


@functools.lru_cache(maxsize=None)
def c1_oracle_cg():
    import oracle
    rp, col, val = config("C1")
    n = len(rp) - 1
    return oracle.solve("cg", np.float64, rp, col, val, np.zeros(n), rhs(n), L.DIAGONAL, 200000, 1e-10, 0.0)


def engine_for(monkeypatch, loop_mode):
    """The graph engine for loop mode 0 (the banded one switched off)."""
    if loop_mode == 0:
        monkeypatch.setenv("CLSPARSE_B200_DIA", "0")


@pytest.mark.parametrize("loop_mode", [0, 3], ids=["graph", "banded"])
def test_c1_poisson512_cg_matches_oracle(ctrl, orc, monkeypatch, loop_mode):
    engine_for(monkeypatch, loop_mode)
    rp, col, val = config("C1")
    n = len(rp) - 1
    b = rhs(n)
    A, bt, x = device_problem(ctrl, "C1")
    ctrl.set_solver_loop_mode(loop_mode)
    sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
    info = api.solve("cg", x, A, bt, sc, ctrl)
    sc.release()
    ctrl.set_solver_loop_mode(0)
    assert ctrl.solver_engine() == ("graph" if loop_mode == 0 else "banded-on-chip")
    xo, oi = c1_oracle_cg()
    assert oi.nIters > 1000
    assert abs(info["nIters"] - oi.nIters) <= max(3, int(0.01 * oi.nIters)), (info, oi.nIters)
    assert info["initialResidual"] == pytest.approx(oi.initialResidual, rel=1e-9)
    assert info["currentResidual"] <= 1e-10
    xs = x.cpu().numpy()
    l1 = np.abs(b - scipy_matrix("C1") @ xs).sum() / np.abs(b).sum()
    assert l1 <= 1.1e-10, l1
    assert np.linalg.norm(xs - xo) / np.linalg.norm(xo) <= ERR_BAR


def _fp64_cg(ctrl, name, loop_mode=0):
    A, b, x = device_problem(ctrl, name)
    ctrl.set_solver_loop_mode(loop_mode)
    sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
    sc.set_norm(2)
    info = api.solve("cg", x, A, b, sc, ctrl)
    sc.release()
    ctrl.set_solver_loop_mode(0)
    return x.cpu().numpy(), info


@pytest.mark.parametrize("loop_mode", [0, 3], ids=["graph", "banded"])
@pytest.mark.parametrize("name", ["C3", "C5"])
def test_fp64_jacobi_cg_at_config_matches_oracle(ctrl, orc, monkeypatch, name, loop_mode):
    engine_for(monkeypatch, loop_mode)
    xs, info = _fp64_cg(ctrl, name, loop_mode)
    assert ctrl.solver_engine() == ("graph" if loop_mode == 0 else "banded-on-chip" if name == "C5" else "banded")
    # the oracle's threaded CG to the same L2 tolerance: same iteration count
    # up to reduction order
    it_o = oracle_iterations_1e10(name)
    assert abs(info["nIters"] + 1 - it_o) <= max(3, int(0.02 * it_o)), (info, it_o)
    assert l2_residual(name, xs) <= 1.5e-10
    assert error_vs_oracle(name, xs) <= ERR_BAR


@pytest.mark.parametrize("name", ["C3", "C5"])
def test_mixed_fp32_at_config_reaches_fp64_oracle(ctrl, name):
    A, b, x = device_problem(ctrl, name)
    sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
    info = api.cg_mixed(x, A, b, sc, ctrl, inner="fp32", inner_tol=0.3)
    sc.release()
    xs = x.cpu().numpy()
    assert info["converged"] == 1, info
    assert l2_residual(name, xs) <= 1.5e-10
    assert error_vs_oracle(name, xs) <= ERR_BAR


def test_c5_learned_mixed_reaches_fp64_oracle_in_fewer_iterations(ctrl):
    """The network trained on 128^2 members of the family (as the benchmark
    does), its factor built for the 1024^2 matrix, then the FP64 refinement
    around FP32 G^T G-PCG: FP64 residual 1e-10, the oracle's solution, and
    fewer inner iterations than FP64 Jacobi-CG needs."""
    spai, hist = learn.train(ctrl, sizes=(128,), seeds=range(6), steps=300, lr=3e-3)
    assert np.mean(hist[-20:]) < np.mean(hist[:8])
    A, b, x = device_problem(ctrl, "C5")
    spai.set_matrix(A, ctrl)
    spai.build(ctrl)
    sc = api.SolverControl(L.DIAGONAL, 200000, 1e-10, 0.0)
    info = api.cg_learned(x, A, b, sc, spai, ctrl, inner="fp32", inner_tol=0.3)
    sc.release()
    spai.release()
    xs = x.cpu().numpy()
    assert info["converged"] == 1 and info["fell_back"] == 0, info
    assert l2_residual("C5", xs) <= 1.5e-10
    assert error_vs_oracle("C5", xs) <= ERR_BAR
    _, jac = _fp64_cg(ctrl, "C5")
    assert info["innerIterations"] < 0.85 * (jac["nIters"] + 1), (info, jac)
