"""Batched FP32 Jacobi-CG (clsparseScsrcgBatched) through the C ABI: every
system's solution against an FP64 direct solve of that system, and the FP64
residual each system reports against one recomputed here -- from diagonal
storage (banded systems, the default) and from CSR."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api, matgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["diagonal", "csr"])
@pytest.mark.parametrize("lanes", [None, 1, 4])
def test_batched_cg_matches_direct_solves(ctrl, lanes, storage, monkeypatch):
    """Banded systems run from diagonal storage by default;
    CLSPARSE_B200_BATCH_DIA=0 keeps them on CSR (the lanes-per-row path)."""
    if storage == "csr":
        monkeypatch.setenv("CLSPARSE_B200_BATCH_DIA", "0")
    rp, col, val, off, dims = matgen.batched_systems(48, 40, 4000, sigma=1.0, seed=3)
    n = len(rp) - 1
    A64 = sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(n, n))
    b = np.random.default_rng(5).uniform(-1, 1, n).astype(np.float32)
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=torch.float32)
    x = torch.zeros(n, dtype=torch.float32, device="cuda")
    sc = api.SolverControl(L.DIAGONAL, 20000, 1e-6, 0.0)
    ln = None if lanes is None else np.full(48, lanes)
    out = api.cg_batched(x, A, torch.tensor(b, device="cuda"), off, sc, ctrl, lanes=ln)
    sc.release()
    assert out["converged"] == 48, out
    xs = x.cpu().numpy().astype(np.float64)
    A32 = sp.csr_matrix((val.astype(np.float32).astype(np.float64), col.astype(np.int64), rp.astype(np.int64)),
                        shape=(n, n))
    for s in range(48):
        a, e = int(off[s]), int(off[s + 1])
        bs = b[a:e].astype(np.float64)
        rres = np.linalg.norm(bs - A32[a:e, a:e] @ xs[a:e]) / np.linalg.norm(bs)
        assert rres <= 1.05e-6, (s, rres)
        assert abs(out["residuals"][s] - rres) <= 1e-9 + 1e-3 * rres
        xd = spla.spsolve(A64[a:e, a:e].tocsc(), bs)
        cond_bound = 1e-6 * 1e4
        assert np.linalg.norm(xs[a:e] - xd) / np.linalg.norm(xd) <= cond_bound


def test_batched_cg_repeat_is_deterministic(ctrl):
    rp, col, val, off, _ = matgen.batched_systems(16, 100, 2000, seed=9)
    n = len(rp) - 1
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=torch.float32)
    b = torch.tensor(np.random.default_rng(1).uniform(-1, 1, n), dtype=torch.float32, device="cuda")
    outs = []
    for _ in range(2):
        x = torch.zeros(n, dtype=torch.float32, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 5000, 1e-6, 0.0)
        api.cg_batched(x, A, b, off, sc, ctrl)
        sc.release()
        outs.append(x.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])


def test_batched_rejects_bad_offsets(ctrl):
    rp, col, val, off, _ = matgen.batched_systems(4, 50, 200, seed=2)
    n = len(rp) - 1
    A = api.CsrMatrix.from_numpy(rp, col, val, dtype=torch.float32)
    x = torch.zeros(n, dtype=torch.float32, device="cuda")
    sc = api.SolverControl(L.DIAGONAL, 100, 1e-6, 0.0)
    bad = off.copy()
    bad[-1] += 1
    with pytest.raises(api.ClsparseError):
        api.cg_batched(x, A, x, bad, sc, ctrl)
    sc.release()


def test_batch_with_a_non_banded_system_runs_on_csr(ctrl):
    """One system with more column offsets than diagonal storage takes: the
    batch runs from CSR, and every system still meets the tolerance."""
    rp, col, val, off, _ = matgen.batched_systems(12, 200, 3000, sigma=1.0, seed=4)
    S = sp.csr_matrix((val, col.astype(np.int64), rp.astype(np.int64)), shape=(len(rp) - 1,) * 2)
    rrp, rcol, rval = matgen.random_spd(1500, seed=8)
    R = sp.csr_matrix((rval, rcol.astype(np.int64), rrp.astype(np.int64)), shape=(1500, 1500))
    M = sp.block_diag([S, R], format="csr")
    M.sort_indices()
    offs = np.concatenate([off, [off[-1] + 1500]]).astype(np.uint32)
    n = M.shape[0]
    b = np.random.default_rng(6).uniform(-1, 1, n).astype(np.float32)
    A = api.CsrMatrix.from_numpy(M.indptr.astype(np.uint32), M.indices.astype(np.uint32), M.data,
                                 dtype=torch.float32)
    x = torch.zeros(n, dtype=torch.float32, device="cuda")
    sc = api.SolverControl(L.DIAGONAL, 20000, 1e-6, 0.0)
    out = api.cg_batched(x, A, torch.tensor(b, device="cuda"), offs, sc, ctrl)
    sc.release()
    assert out["converged"] == 13, out
    M32 = sp.csr_matrix((M.data.astype(np.float32).astype(np.float64), M.indices, M.indptr), shape=M.shape)
    xs = x.cpu().numpy().astype(np.float64)
    for s in range(13):
        a, e = int(offs[s]), int(offs[s + 1])
        bs = b[a:e].astype(np.float64)
        assert np.linalg.norm(bs - M32[a:e, a:e] @ xs[a:e]) / np.linalg.norm(bs) <= 1.05e-6


def _banded_spd(n, offsets, seed):
    """Symmetric, strictly diagonally dominant matrix with the given upper
    offsets, some entries missing (boundaries inside the system)."""
    rng = np.random.default_rng(seed)
    M = sp.csr_matrix((n, n))
    for o in offsets:
        if o < n:
            v = -rng.uniform(0.1, 1.0, n - o) * (rng.uniform(size=n - o) < 0.9)
            U = sp.diags([v], [o], shape=(n, n))
            M = M + U + U.T
    M = M + sp.diags([np.asarray(abs(M).sum(axis=1)).ravel() + rng.uniform(0.01, 0.2, n)], [0])
    M = M.tocsr()
    M.eliminate_zeros()
    M.sort_indices()
    return M


# Rows at the edges of a CTA's registers (14 per thread: 1792, 7168), of the
# cluster sizes 2, 4 and 8, past the largest, and of uneven splits; diagonals
# 1 to 8; stencils that reach one row short of, exactly and past the
# neighbouring CTA of the split.
RESIDENT = [
    [(1, [1]), (2, [1]), (33, [1, 5]), (128, [1, 16]), (129, [1, 2, 3])],
    [(1791, [1]), (1792, [1, 40]), (1793, [1, 40]), (1800, [1, 899]), (1900, [1, 2, 1899])],
    [(7167, [1, 80]), (7168, [1, 19, 361]), (7169, [1, 19, 361]), (14336, [1, 119]), (14337, [1, 24, 7168])],
    [(28672, [1, 30, 900]), (28673, [1, 169]), (20000, [1, 4999]), (20000, [1, 5001]), (9000, [1, 2, 4])],
    [(50001, [1, 37, 1369]), (57343, [1, 239]), (300, [1])],
    [(57345, [1, 239]), (500, [1, 22]), (40000, [1, 30000])],
]


@pytest.mark.parametrize("case", range(len(RESIDENT)))
def test_resident_sizes_against_csr(ctrl, case, monkeypatch):
    """Systems held on chip against the general kernel's CSR path: every
    residual recomputed here in FP64 meets the tolerance and is the reported
    one, and the two solutions agree to the tolerance times the condition of
    these matrices (row sums at least 1 % of the diagonal: below 1e3)."""
    mats = [_banded_spd(n, o, seed=100 * case + k) for k, (n, o) in enumerate(RESIDENT[case])]
    M = sp.block_diag(mats, format="csr")
    M.sort_indices()
    off = np.concatenate([[0], np.cumsum([m.shape[0] for m in mats])]).astype(np.uint32)
    n = M.shape[0]
    A = api.CsrMatrix.from_numpy(M.indptr.astype(np.uint32), M.indices.astype(np.uint32), M.data, dtype=torch.float32)
    M32 = sp.csr_matrix((M.data.astype(np.float32).astype(np.float64), M.indices, M.indptr), shape=M.shape)
    b = np.random.default_rng(case).uniform(-1, 1, n).astype(np.float32)
    x0 = np.random.default_rng(case + 50).uniform(-1, 1, n).astype(np.float32)
    xs = {}
    for storage in ("resident", "csr"):
        if storage == "csr":
            monkeypatch.setenv("CLSPARSE_B200_BATCH_DIA", "0")
        x = torch.tensor(x0, device="cuda")
        sc = api.SolverControl(L.DIAGONAL, 5000, 1e-6, 0.0)
        out = api.cg_batched(x, A, torch.tensor(b, device="cuda"), off, sc, ctrl)
        # the iteration budget ends a solve between two exchanges alike
        few = torch.tensor(x0, device="cuda")
        sc3 = api.SolverControl(L.DIAGONAL, 3, 1e-6, 0.0)
        out3 = api.cg_batched(few, A, torch.tensor(b, device="cuda"), off, sc3, ctrl)
        sc.release()
        sc3.release()
        assert out["converged"] == len(mats), out
        xs[storage] = x.cpu().numpy().astype(np.float64), few.cpu().numpy().astype(np.float64), out3["residuals"]
        for s in range(len(mats)):
            a, e = int(off[s]), int(off[s + 1])
            bs = b[a:e].astype(np.float64)
            res = np.linalg.norm(bs - M32[a:e, a:e] @ xs[storage][0][a:e]) / np.linalg.norm(bs)
            assert res <= 1.05e-6 and abs(out["residuals"][s] - res) <= 1e-9 + 1e-3 * res, (storage, s, res)
    for s in range(len(mats)):
        a, e = int(off[s]), int(off[s + 1])
        for k in (0, 1):
            u, v = xs["resident"][k][a:e], xs["csr"][k][a:e]
            assert np.linalg.norm(u - v) <= 1e-3 * np.linalg.norm(v), (s, k)
        assert abs(xs["resident"][2][s] - xs["csr"][2][s]) <= 1e-3 * xs["csr"][2][s] + 1e-6


def test_batch_without_memory_leaves_x_and_a_refused_launch_is_solved_anyway(ctrl, monkeypatch):
    """A batch with systems for the chip and one too large for it. When the
    general kernel's memory cannot be had the call says so before anything has
    run: x is as it was. When the on-chip launches are not taken, their systems
    run in the general kernel. (The failures are made on the host.)"""
    mats = [_banded_spd(n, o, seed=n) for n, o in ((60000, [1, 240]), (9000, [1, 90]), (500, [1, 22]), (700, [1]))]
    M = sp.block_diag(mats, format="csr")
    M.sort_indices()
    off = np.concatenate([[0], np.cumsum([m.shape[0] for m in mats])]).astype(np.uint32)
    n = M.shape[0]
    A = api.CsrMatrix.from_numpy(M.indptr.astype(np.uint32), M.indices.astype(np.uint32), M.data, dtype=torch.float32)
    rng = np.random.default_rng(5)
    b, x0 = (torch.tensor(rng.uniform(-1, 1, n).astype(np.float32), device="cuda") for _ in range(2))

    def solve():
        x = x0.clone()
        sc = api.SolverControl(L.DIAGONAL, 5000, 1e-6, 0.0)
        try:
            return x, api.cg_batched(x, A, b, off, sc, ctrl)
        except api.ClsparseError as e:
            return x, e.status
        finally:
            sc.release()

    x, out = solve()
    assert out["converged"] == len(mats)
    monkeypatch.setenv("CLSPARSE_B200_TEST_FAIL", "batched-alloc")
    xf, status = solve()
    assert status == L.clsparseOutOfResources and torch.equal(xf, x0)
    monkeypatch.setenv("CLSPARSE_B200_TEST_FAIL", "batched-launch")
    xl, out = solve()
    assert out["converged"] == len(mats) and out["worst_residual"] <= 1e-6
    assert float((xl - x).norm()) <= 1e-3 * float(x.norm())
    monkeypatch.delenv("CLSPARSE_B200_TEST_FAIL")
    assert torch.equal(solve()[0], x)


def test_one_small_system_is_not_spread_over_a_cluster(ctrl):
    """A hundred rows alone take no longer than in a batch of 148 (which has no
    idle SMs to give them): 2.5 us an iteration, 4.0 on a cluster of eight."""
    m = _banded_spd(100, [1, 10], seed=3)

    def best(count):
        M = sp.block_diag([m] * count, format="csr")
        M.sort_indices()
        A = api.CsrMatrix.from_numpy(M.indptr.astype(np.uint32), M.indices.astype(np.uint32), M.data,
                                     dtype=torch.float32)
        off = (np.arange(count + 1) * 100).astype(np.uint32)
        b = torch.ones(100 * count, dtype=torch.float32, device="cuda")
        x = torch.zeros_like(b)
        times = []
        for _ in range(8):
            x.zero_()
            sc = api.SolverControl(L.DIAGONAL, 2000, 1e-30, 0.0)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            api.cg_batched(x, A, b, off, sc, ctrl)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
            sc.release()
        return min(times)

    assert best(1) <= 1.2 * best(148)
