"""The banded solves with their vectors on chip against the same solves
streaming their vectors through L2 (CLSPARSE_B200_DIA_RESIDENT=0), which
test_dia_cg_gpu.py and test_banded_gpu.py hold to the oracle and to CSR. Both form every
row and vector entry with the same operations; only the FP64 sums of the dot
products run in another order. A fixed, small number of iterations from the
same start therefore agrees to rounding: the scalars differ by a few 1e-16 (FP64
sums of products whose absolute sum is within 1e3 of the sum), each iteration
carries that over with a factor below ten for these matrices (condition below
1e3), and 12 iterations stay below 1e-9; in FP32 the scalars are rounded to
2^-24 after the sum, so an iterate moves by at most a few 1e-6.

Sizes: one row to a few, around one CTA's share (1024 rows), around the
register arrays (2, 4 and 14 rows per thread of 512 on 148 SMs), odd splits;
stencils within a CTA, across neighbours, and across several CTAs (the plain
exchange of z); 3 to 9 diagonals and padded counts. Just beyond what the chip
takes (rows, halo, shared memory) both sides stream, as asserted."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api, learn, matgen

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed=0, skew=0.0):
    rng = np.random.default_rng(seed)
    diags, offs = [], []
    total = np.zeros(n)
    for o in offsets:
        if o >= n:
            continue
        v = -rng.uniform(0.1, 1.0, n - o)
        w = v * (1.0 + skew * rng.uniform(0, 1, n - o))
        diags += [v, w]
        offs += [o, -o]
        total[: n - o] += np.abs(v)
        total[o:] += np.abs(w)
    diags.append(total + rng.uniform(0.05, 0.5, n))
    offs.append(0)
    A = sp.diags(diags, offs, shape=(n, n)).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.uint32), A.indices.astype(np.uint32), A.data


def both(monkeypatch, fn):
    got = fn()
    monkeypatch.setenv("CLSPARSE_B200_DIA_RESIDENT", "0")
    ref = fn()
    monkeypatch.delenv("CLSPARSE_B200_DIA_RESIDENT")
    return got, ref


SMALL = [(1, [1]), (2, [1]), (3, [1, 2]), (40, [1, 7]), (1023, [1, 31]), (1024, [1, 32]), (1025, [1, 32, 900]),
         (2049, [1, 2, 3, 4]), (5000, [1, 2100]), (12345, [1, 20, 400]), (30011, [1, 7000]), (30011, [1, 9000])]
LARGE = [(303104, [1, 551]), (303105, [1, 551]), (200001, [1, 60, 3600]), (262144, [1, 512])]
HUGE = [(1060864, [1, 1030]), (1060865, [1, 1030]), (1000000, [1, 100, 10000])]


def _case_id(c):
    return f"n{c[0]}o{c[1][-1]}"


def expected_engine(kind, case, dtype):
    """On chip, but for a halo wider than it pays (18,000 rows), more than 7168
    (CG) or 2048 (BiCGStab) rows a CTA, and BiCGStab halos beyond the shared
    memory (five words a halo row). A single row is no STREAM block of its
    meta: the graph engine's."""
    n, offs = case
    if n == 1:
        return "graph"
    if offs[-1] == 9000 or n > 1060864:
        return "banded"
    wide = 5 * 2 * offs[-1] * (8 if dtype == torch.float64 else 4) > 220000
    return "banded" if kind == "bicgstab" and (n > 303104 or wide) else "banded-on-chip"


@pytest.mark.parametrize("precond", [L.DIAGONAL, L.NOPRECOND], ids=["jacobi", "none"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("case", SMALL + LARGE + HUGE, ids=_case_id)
def test_dropin_solves(ctrl, monkeypatch, case, kind, dtype, precond):
    n, offs = case
    if n > 250000 and (precond == L.NOPRECOND or (n > 400000 and kind == "bicgstab")):
        pytest.skip("the same split as the Jacobi case / beyond the on-chip BiCGStab")
    rp, col, val = banded(n, offs, seed=n, skew=0.5 if kind == "bicgstab" else 0.0)
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=dtype)
    A.create_meta(ctrl)
    rng = np.random.default_rng(7)
    b = torch.tensor(rng.uniform(-1, 1, n), dtype=dtype, device="cuda")
    x0 = torch.tensor(rng.uniform(-1, 1, n), dtype=dtype, device="cuda")
    ctrl.set_solver_loop_mode(3)

    def solve(iters, tol):
        x = x0.clone()
        sc = api.SolverControl(precond, iters, tol, 0.0)
        info = api.solve(kind, x, A, b, sc, ctrl)
        sc.release()
        engines.append(ctrl.solver_engine())
        return x.double().cpu().numpy(), info

    engines = []
    (x, i), (xr, ir) = both(monkeypatch, lambda: solve(12 if n > 64 else 2, 0.0))
    assert engines == [expected_engine(kind, case, dtype), "graph" if n == 1 else "banded"]
    tol = 1e-9 if dtype == torch.float64 else 2e-4
    if n > 64:
        assert i["nIters"] == ir["nIters"]
        assert np.linalg.norm(x - xr) <= tol * np.linalg.norm(xr)
        assert i["currentResidual"] == pytest.approx(ir["currentResidual"], rel=1e-6 if dtype == torch.float64 else 1e-2)
    # to a tolerance: the stop test is met on a fresh FP64 check
    rel = 1e-9 if dtype == torch.float64 else 1e-4
    x, i = solve(4000, rel)
    M = sp.csr_matrix((np.asarray(A.val.double().cpu()), col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))
    bb = b.double().cpu().numpy()
    assert np.abs(bb - M @ x).sum() <= (10 if dtype == torch.float64 else 50) * rel * np.abs(bb).sum()
    ctrl.set_solver_loop_mode(0)


@pytest.mark.parametrize("inner", ["fp32", "bf16"])
@pytest.mark.parametrize("case", [(50, [1, 7]), (1025, [1, 32]), (30011, [1, 6000]), (30011, [1, 9000]),
                                  (20000, [1, 2, 3, 4]), (303105, [1, 551]), (1060864, [1, 80, 6400]),
                                  (1060865, [1, 80, 6400]), (2121728, [1, 128, 16384]), (2121729, [1, 1456])],
                         ids=_case_id)
def test_inner_solves(ctrl, monkeypatch, case, inner):
    """The refinement's inner PCG: the same number of refinements, and the FP64
    true residual recomputed here meets the tolerance on both."""
    n, offs = case
    rp, col, val = banded(n, offs, seed=n)
    A = api.CsrMatrix.from_numpy(rp, col, val)
    A.create_meta(ctrl)
    b = torch.tensor(np.random.default_rng(3).uniform(-1, 1, n), device="cuda")

    def solve():
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 20000, 1e-10, 0.0)
        info = api.cg_mixed(x, A, b, sc, ctrl, inner=inner, inner_tol=0.1)
        sc.release()
        engines.append(ctrl.solver_engine())
        return x.cpu().numpy(), info

    engines = []
    M = sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))
    bb = b.cpu().numpy()
    (x, i), (xr, ir) = both(monkeypatch, solve)
    assert engines == [expected_engine("cg", case, torch.float32), "banded"]
    for v, info in ((x, i), (xr, ir)):
        assert info["converged"] == 1
        assert np.linalg.norm(bb - M @ v) <= 1.5e-10 * np.linalg.norm(bb)
    assert abs(i["outerIterations"] - ir["outerIterations"]) <= 1
    assert abs(i["innerIterations"] - ir["innerIterations"]) <= max(3, 0.05 * ir["innerIterations"])
    assert np.linalg.norm(x - xr) <= 1e-7 * np.linalg.norm(xr)


@pytest.mark.parametrize("shape", [(31,), (64,), (300,), (1029,), (24, 24, 24)], ids=str)
def test_learned_inner_solves(ctrl, monkeypatch, shape):
    """The learned factor's inner PCG on grids of 961 to 1,058,841 rows and on a
    3D stencil (four diagonals in G, seven in A; a network that has seen only
    2D matrices need not converge there, so it runs 200 iterations): the same
    iterations and refinements, and the true residual recomputed here."""
    rng = np.random.default_rng(5)
    if len(shape) == 1:
        rp, col, val = matgen.diffusion2d_grf(shape[0], corr_len=0.2, sigma=1.0, seed=3)
    else:
        rp, col, val = matgen.diffusion(shape, np.exp(0.3 * rng.normal(0, 1, int(np.prod(shape)))))
    n = len(rp) - 1
    A = api.CsrMatrix.from_numpy(rp, col, val)
    A.create_meta(ctrl)
    spai, _ = learn.train(ctrl, sizes=(24,), seeds=range(2), steps=20, lr=3e-3)
    spai.set_matrix(A, ctrl)
    spai.build(ctrl)
    b = torch.tensor(rng.uniform(-1, 1, n), device="cuda")

    def solve():
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 60000 if len(shape) == 1 else 200, 1e-9, 0.0)
        info = api.cg_learned(x, A, b, sc, spai, ctrl, inner="fp32", inner_tol=0.3)
        sc.release()
        engines.append(ctrl.solver_engine())
        return x.cpu().numpy(), info

    engines = []
    (x, i), (xr, ir) = both(monkeypatch, solve)
    assert engines == ["banded-on-chip", "banded"]
    spai.release()
    M = sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))
    bb = b.cpu().numpy()
    for v, info in ((x, i), (xr, ir)):
        res = np.linalg.norm(bb - M @ v) / np.linalg.norm(bb)
        assert res == pytest.approx(info["trueResidual"], rel=1e-3, abs=1e-12)
        assert info["converged"] == (1 if len(shape) == 1 else 0)
    assert i["fell_back"] == ir["fell_back"] and abs(i["outerIterations"] - ir["outerIterations"]) <= 1
    assert abs(i["innerIterations"] - ir["innerIterations"]) <= max(5, 0.1 * ir["innerIterations"])


def test_default_mode_takes_the_banded_engine_with_its_results(ctrl, orc):
    """Loop mode 0 on a banded matrix: the same iterates as loop mode 3, bit
    for bit, and the oracle's stop decision; without a meta, with history or
    in extended precision the graph engine runs and agrees to rounding."""
    rp, col, val = matgen.poisson2d(90, 71)
    n = len(rp) - 1
    b = np.random.default_rng(2).uniform(-1, 1, n)
    bt = torch.tensor(b, device="cuda")

    def solve(kind, mode, meta=True, history=False, ext=False):
        ctrl.set_solver_loop_mode(mode)
        ctrl.enable_extended_precision(ext)
        A = api.CsrMatrix.from_numpy(rp, col, val)
        if meta:
            A.create_meta(ctrl)
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 3000, 1e-9, 0.0)
        if history:
            sc.set_history(torch.zeros(4000, dtype=torch.float64, device="cuda"))
        info = api.solve(kind, x, A, bt, sc, ctrl)
        sc.release()
        ctrl.set_solver_loop_mode(0)
        ctrl.enable_extended_precision(False)
        return x.cpu().numpy(), info["nIters"]

    for kind in ("cg", "bicgstab"):
        x3, k3 = solve(kind, 3)
        x0, k0 = solve(kind, 0)
        assert k0 == k3 and np.array_equal(x0, x3)
        _, oi = orc.solve(kind, np.float64, rp, col, val, np.zeros(n), b, 1, 3000, 1e-9, 0.0)
        assert abs(k0 - oi.nIters) <= max(3, 0.05 * oi.nIters)
        for other in (dict(meta=False), dict(history=True), dict(ext=True)):
            xg, kg = solve(kind, 0, **other)
            assert abs(kg - k0) <= max(3, 0.1 * k0)
            assert np.linalg.norm(xg - x0) <= 1e-6 * np.linalg.norm(x0)


def test_threads_with_different_plans(ctrl):
    """Two threads with a control each on one stream, whose matrices need the
    same kernel with different amounts of shared memory: every launch is taken
    (the limit is the kernel's, shared by the threads: set to each launch's own
    amount, one thread's smaller value came between the other's two calls)."""
    errors = []

    def work(offs):
        c = api.Control(stream)
        try:
            n = 1500
            A = api.CsrMatrix.from_numpy(*banded(n, offs))
            A.create_meta(c)
            b = torch.ones(n, dtype=torch.float64, device="cuda")
            x = torch.zeros(n, dtype=torch.float64, device="cuda")
            for _ in range(1500):
                sc = api.SolverControl(L.DIAGONAL, 1, 0.0, 0.0)
                api.solve("cg", x, A, b, sc, c)
                sc.release()
        except Exception as e:  # noqa: BLE001
            errors.append(e)
        finally:
            c.release()

    stream = torch.cuda.current_stream()
    threads = [threading.Thread(target=work, args=(o,)) for o in ([1, 20], [1, 700])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("case", [(1000000, [1, 1000]), (1060864, [1, 1030]), (700001, [1, 60, 3000]), (20000, [1, 150])],
                         ids=_case_id)
def test_lower_diagonals_from_the_upper_ones(ctrl, monkeypatch, case, dtype):
    """CLSPARSE_B200_DIA_SYM on chip: never (0), wherever possible (1) and the
    default (where not every diagonal fits) give the same x bit for bit."""
    n, offs = case
    rp, col, val = banded(n, offs, seed=n)
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=dtype)
    A.create_meta(ctrl)
    b = torch.tensor(np.random.default_rng(7).uniform(-1, 1, n), dtype=dtype, device="cuda")

    def solve(mode):
        if mode is None:
            monkeypatch.delenv("CLSPARSE_B200_DIA_SYM", raising=False)
        else:
            monkeypatch.setenv("CLSPARSE_B200_DIA_SYM", mode)
        x = torch.zeros_like(b)
        sc = api.SolverControl(L.DIAGONAL, 25, 0.0, 0.0)
        api.solve("cg", x, A, b, sc, ctrl)
        sc.release()
        assert ctrl.solver_engine() == "banded-on-chip"
        return x

    x0, x1, xd = solve("0"), solve("1"), solve(None)
    assert torch.equal(x0, x1) and torch.equal(x0, xd)
