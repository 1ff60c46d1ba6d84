"""Which engine a CG or BiCGStab solve runs on (clsparseB200GetSolverEngine),
and that a solve whose banded engine cannot have its memory or its launch runs
on the next engine instead of failing: on chip, then streaming, then the graph.
The failures are made on the host (CLSPARSE_B200_TEST_FAIL names the step that
reports failure without being tried)."""
from __future__ import annotations

import time

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api, matgen

pytestmark = pytest.mark.gpu

MATS = {"poisson": lambda: matgen.poisson2d(60, 50), "wide3d": lambda: matgen.diffusion((30, 30, 6), np.ones(5400))}


def solve(ctrl, kind, mat, mode=0, dtype=torch.float64, meta=True, precond=L.DIAGONAL):
    ctrl.set_solver_loop_mode(mode)
    A = api.CsrMatrix.from_numpy(*mat, dtype=dtype)
    if meta:
        A.create_meta(ctrl)
    n = len(mat[0]) - 1
    b = np.random.default_rng(3).uniform(-1, 1, n)
    x = torch.zeros(n, dtype=dtype, device="cuda")
    sc = api.SolverControl(precond, 3000, 1e-9 if dtype == torch.float64 else 1e-4, 0.0)
    info = api.solve(kind, x, A, torch.tensor(b, dtype=dtype, device="cuda"), sc, ctrl)
    status = sc.device_status()
    sc.release()
    ctrl.set_solver_loop_mode(0)
    M = sp.csr_matrix((mat[2], mat[1].astype(np.int64), mat[0].astype(np.int64)), shape=(n, n))
    res = np.abs(b - M @ x.double().cpu().numpy()).sum() / np.abs(b).sum()
    assert status & ~8 == 0 and res <= (1e-8 if dtype == torch.float64 else 5e-3)
    return info["nIters"], ctrl.solver_engine()


@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
def test_engine_of_a_solve(ctrl, kind, monkeypatch):
    mat = MATS["poisson"]()
    assert ctrl.solver_engine() == "none"
    for mode in (0, 1, 3):
        assert solve(ctrl, kind, mat, mode)[1] == "banded-on-chip"
        assert solve(ctrl, kind, mat, mode, meta=False)[1] == ("chunks" if mode == 1 else "graph")
    assert solve(ctrl, kind, mat, 2)[1] == ("persistent" if kind == "cg" else "graph")
    monkeypatch.setenv("CLSPARSE_B200_DIA_RESIDENT", "0")
    assert solve(ctrl, kind, mat)[1] == "banded"
    monkeypatch.setenv("CLSPARSE_B200_DIA", "0")
    assert solve(ctrl, kind, mat)[1] == "graph"


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("precond", [L.DIAGONAL, L.NOPRECOND], ids=["jacobi", "none"])
@pytest.mark.parametrize("mode", [0, 1, 3])
@pytest.mark.parametrize("mat", sorted(MATS))
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
def test_solve_falls_back_when_the_banded_engine_is_refused(ctrl, monkeypatch, kind, mat, mode, precond, dtype):
    graph = "chunks" if mode == 1 else "graph"
    m = MATS[mat]()
    k, engine = solve(ctrl, kind, m, mode, dtype, precond=precond)
    assert engine == "banded-on-chip"
    for steps, want in (("onchip-alloc", "banded"), ("onchip-launch", "banded"), ("onchip-alloc,banded-alloc", graph),
                        ("onchip-launch,banded-launch", graph), ("banded-copy", graph)):
        monkeypatch.setenv("CLSPARSE_B200_TEST_FAIL", steps)
        kf, engine = solve(ctrl, kind, m, mode, dtype, precond=precond)
        assert engine == want, steps
        assert abs(kf - k) <= max(8, 0.25 * k)
    monkeypatch.delenv("CLSPARSE_B200_TEST_FAIL")
    assert solve(ctrl, kind, m, mode, dtype, precond=precond) == (k, "banded-on-chip")


@pytest.mark.parametrize("resident", [True, False], ids=["onchip", "streamed"])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("mode", [0, 1])
def test_wait_that_runs_out_in_a_default_mode_is_not_an_error(ctrl, monkeypatch, mode, kind, resident):
    """With one CTA never releasing its exchange every wait runs out (2 ms):
    the default modes solve on the graph engine from the same initial guess, bit
    for bit what that engine alone gives; loop mode 3 reports it (the other
    tests)."""
    mat = MATS["poisson"]()
    n = len(mat[0]) - 1
    rng = np.random.default_rng(8)
    b, x0 = (torch.tensor(rng.uniform(-1, 1, n), device="cuda") for _ in range(2))
    A = api.CsrMatrix.from_numpy(*mat)
    A.create_meta(ctrl)
    ctrl.set_solver_loop_mode(mode)

    def run():
        x = x0.clone()
        sc = api.SolverControl(L.DIAGONAL, 3000, 1e-9, 0.0)
        info = api.solve(kind, x, A, b, sc, ctrl)
        status = sc.device_status()
        sc.release()
        return x, info, status

    monkeypatch.setenv("CLSPARSE_B200_DIA", "0")
    xg, ig, sg = run()
    monkeypatch.delenv("CLSPARSE_B200_DIA")
    if not resident:
        monkeypatch.setenv("CLSPARSE_B200_DIA_RESIDENT", "0")
    monkeypatch.setenv("CLSPARSE_B200_TEST_BARRIER_NEVER_RELEASE", "1")
    monkeypatch.setenv("CLSPARSE_B200_BARRIER_WAIT_NS", "2000000")
    x, i, s = run()
    assert ctrl.solver_engine() == ("chunks" if mode == 1 else "graph")
    assert torch.equal(x, xg) and i == ig and s == sg
    monkeypatch.delenv("CLSPARSE_B200_TEST_BARRIER_NEVER_RELEASE")
    run()
    assert ctrl.solver_engine() == ("banded-on-chip" if resident else "banded")
    ctrl.set_solver_loop_mode(0)


@pytest.mark.parametrize("inner", ["fp32", "bf16"])
def test_inner_solves_stream_when_the_chip_is_refused(ctrl, monkeypatch, inner):
    """The refinement's inner solves: without the on-chip form's exchange area
    or its launch they stream, with the same refinements."""
    mat = MATS["poisson"]()
    n = len(mat[0]) - 1
    A = api.CsrMatrix.from_numpy(*mat)
    A.create_meta(ctrl)
    b = torch.tensor(np.random.default_rng(4).uniform(-1, 1, n), device="cuda")

    def run():
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 5000, 1e-10, 0.0)
        info = api.cg_mixed(x, A, b, sc, ctrl, inner=inner, inner_tol=0.1)
        sc.release()
        assert info["converged"] == 1
        return info, ctrl.solver_engine()

    ref, engine = run()
    assert engine == "banded-on-chip"
    for step in ("onchip-alloc", "onchip-launch"):
        monkeypatch.setenv("CLSPARSE_B200_TEST_FAIL", step)
        info, engine = run()
        assert engine == "banded"
        assert abs(info["outerIterations"] - ref["outerIterations"]) <= 1
    monkeypatch.delenv("CLSPARSE_B200_TEST_FAIL")
    monkeypatch.setenv("CLSPARSE_B200_DIA", "0")
    assert run()[1] == "graph"


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("reach,rows,want", [(7168, 40000, "banded-on-chip"), (7169, 40000, "banded"),
                                             (8100, 48600, "banded"), (9000, 444000, "banded-on-chip"),
                                             (9001, 444000, "banded")])
def test_wide_halo_streams(ctrl, reach, rows, want, dtype):
    """A stencil that reaches further than its halo is worth on chip streams its
    vectors: at most 14,336 halo rows, or six times a CTA's own (444,000
    rows on 148 SMs: 3000)."""
    n = rows
    v = np.full(n, 4.1)
    A = sp.diags([np.full(n - reach, -1.0), np.full(n - 1, -1.0), v, np.full(n - 1, -1.0), np.full(n - reach, -1.0)],
                 [-reach, -1, 0, 1, reach]).tocsr()
    A.sort_indices()
    mat = (A.indptr.astype(np.uint32), A.indices.astype(np.uint32), A.data)
    assert solve(ctrl, "cg", mat, dtype=dtype)[1] == want


@pytest.mark.parametrize("kind,dtype", [("cg", torch.float64), ("cg", torch.float32), ("bicgstab", torch.float64)],
                         ids=["cg-f64", "cg-f32", "bicgstab-f64"])
def test_large_solves_run_on_the_faster_engine(ctrl, kind, dtype):
    """The default modes leave a CG whose diagonals and vectors are more than
    L2 bytes / 3.2 values, and a BiCGStab whose are more than L2, to the graph
    engine, which is faster there; loop mode 3 streams the CG at any size. A
    tridiagonal matrix on both sides of the line."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    n = l2 * 5 // 160 if kind == "cg" else l2 // (14 * 8)
    for rows, want in ((n, "banded"), (n + 1, "graph")):
        A = sp.diags([np.full(rows - 1, -1.0), np.full(rows, 4.1), np.full(rows - 1, -1.0)], [-1, 0, 1]).tocsr()
        mat = (A.indptr.astype(np.uint32), A.indices.astype(np.uint32), A.data)
        assert solve(ctrl, kind, mat, dtype=dtype)[1] == want
        if kind == "cg":
            assert solve(ctrl, kind, mat, mode=3, dtype=dtype)[1] == "banded"


def test_solves_of_matrices_that_are_not_banded_pay_nothing(ctrl, monkeypatch):
    """A matrix of short rows with more column offsets than the banded engine
    takes is known from its meta: a solve of one iteration takes no longer than with
    that engine off (with a search at every solve: 140 us instead of 100)."""
    rng = np.random.default_rng(3)
    n = 20000
    S = sp.csr_matrix((n, n))
    for o in np.unique(rng.integers(1, n // 3, 15)):
        S = S + sp.diags([-rng.uniform(0.1, 1, n - o) * (rng.uniform(size=n - o) < 0.2)], [o], shape=(n, n))
    S = S + S.T
    S = (S + sp.diags([np.asarray(abs(S).sum(axis=1)).ravel() + 0.3], [0])).tocsr()
    S.eliminate_zeros()
    S.sort_indices()
    assert np.diff(S.indptr).max() <= 16
    A = api.CsrMatrix.from_numpy(S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)
    A.create_meta(ctrl)
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)

    def best():
        times = []
        for _ in range(40):
            sc = api.SolverControl(L.DIAGONAL, 1, 0.0, 0.0)
            torch.cuda.synchronize()
            t = time.perf_counter()
            api.solve("cg", x, A, b, sc, ctrl)
            times.append(time.perf_counter() - t)
            sc.release()
        return min(times)

    default = best()
    assert ctrl.solver_engine() == "graph"
    monkeypatch.setenv("CLSPARSE_B200_DIA", "0")
    assert default <= 1.15 * best()
