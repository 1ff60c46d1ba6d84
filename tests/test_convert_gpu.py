"""Format conversions (clsparse{S,D}coo2csr, csr2coo, csr2dense, dense2csr;
reference src/library/transform/) through the C ABI against scipy, including
empty rows, more rows than one scan block, row- and column-major dense
matrices with padded leading dimensions, and round trips."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api

pytestmark = pytest.mark.gpu
DT = {"f64": torch.float64, "f32": torch.float32}
NPT = {"f64": np.float64, "f32": np.float32}


def random_csr(rows, cols, density, seed, empty_every=7):
    M = sp.random(rows, cols, density=density, random_state=seed, format="csr")
    M = M.tolil()
    for r in range(0, rows, empty_every):
        M[r, :] = 0
    M = M.tocsr()
    M.eliminate_zeros()
    M.sort_indices()
    return M


def coo_struct(ri, ci, vv, rows, cols):
    m = L.clsparseCooMatrix()
    api.lib().clsparseInitCooMatrix(C.byref(m))
    m.num_rows, m.num_cols, m.num_nonzeros = rows, cols, vv.numel()
    m.values, m.col_indices, m.row_indices = vv.data_ptr(), ci.data_ptr(), ri.data_ptr()
    return m


def dense_struct(t, rows, cols, ld, major):
    d = L.cldenseMatrix()
    d.num_rows, d.num_cols, d.lead_dim, d.major = rows, cols, ld, major
    d.values = C.c_void_p(t.data_ptr())
    d.off_values = 0
    return d


@pytest.mark.parametrize("dt", ["f64", "f32"])
def test_coo2csr_and_back(ctrl, dt):
    dtype, t = DT[dt], NPT[dt]
    M = random_csr(3000, 700, 0.01, 3)
    coo = M.tocoo()
    order = np.lexsort((coo.col, coo.row))
    ri = torch.tensor(coo.row[order].astype(np.int32), device="cuda")
    ci = torch.tensor(coo.col[order].astype(np.int32), device="cuda")
    vv = torch.tensor(coo.data[order].astype(t), device="cuda")
    cm = coo_struct(ri, ci, vv, 3000, 700)
    out = api.CsrMatrix(torch.zeros(3001, dtype=torch.int32, device="cuda"),
                        torch.zeros(M.nnz, dtype=torch.int32, device="cuda"),
                        torch.zeros(M.nnz, dtype=dtype, device="cuda"), 700)
    fn = api.lib().clsparseDcoo2csr if dt == "f64" else api.lib().clsparseScoo2csr
    assert fn(C.byref(cm), C.byref(out.s), ctrl.handle) == 0
    assert (out.s.num_rows, out.s.num_cols, out.s.num_nonzeros) == (3000, 700, M.nnz)
    np.testing.assert_array_equal(out.row_ptr.cpu().numpy(), M.indptr)
    np.testing.assert_array_equal(out.col.cpu().numpy(), M.indices)
    np.testing.assert_array_equal(out.val.cpu().numpy(), M.data.astype(t))
    # and back
    ri2 = torch.zeros_like(ri)
    ci2 = torch.zeros_like(ci)
    vv2 = torch.zeros_like(vv)
    cm2 = coo_struct(ri2, ci2, vv2, 0, 0)
    fn2 = api.lib().clsparseDcsr2coo if dt == "f64" else api.lib().clsparseScsr2coo
    assert fn2(C.byref(out.s), C.byref(cm2), ctrl.handle) == 0
    assert cm2.num_nonzeros == M.nnz and cm2.num_rows == 3000
    np.testing.assert_array_equal(ri2.cpu().numpy(), coo.row[order])
    np.testing.assert_array_equal(ci2.cpu().numpy(), coo.col[order])
    np.testing.assert_array_equal(vv2.cpu().numpy(), coo.data[order].astype(t))


@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("major", ["row", "col"])
def test_csr2dense_and_dense2csr(ctrl, dt, major):
    dtype, t = DT[dt], NPT[dt]
    mj = L.rowMajor if major == "row" else L.columnMajor
    rows, cols = 2500, 90
    M = random_csr(rows, cols, 0.05, 5, empty_every=5)
    A = api.CsrMatrix.from_numpy(M.indptr, M.indices, M.data, num_cols=cols, dtype=dtype)
    ld = (cols if mj == L.rowMajor else rows) + 3
    buf = torch.full(((rows if mj == L.rowMajor else cols) * ld,), 7.0, dtype=dtype, device="cuda")
    d = dense_struct(buf, rows, cols, ld, mj)
    fn = api.lib().clsparseDcsr2dense if dt == "f64" else api.lib().clsparseScsr2dense
    assert fn(C.byref(A.s), C.byref(d), ctrl.handle) == 0
    full = buf.cpu().numpy()
    dense = full.reshape(rows, ld)[:, :cols] if mj == L.rowMajor else full.reshape(cols, ld)[:, :rows].T
    np.testing.assert_array_equal(dense, M.toarray().astype(t))
    # padding untouched
    pad = full.reshape(-1, ld)[:, -3:]
    assert np.all(pad == 7.0)
    # back to CSR
    out = api.CsrMatrix(torch.zeros(rows + 1, dtype=torch.int32, device="cuda"),
                        torch.zeros(rows * cols, dtype=torch.int32, device="cuda"),
                        torch.zeros(rows * cols, dtype=dtype, device="cuda"), cols)
    fn2 = api.lib().clsparseDdense2csr if dt == "f64" else api.lib().clsparseSdense2csr
    assert fn2(C.byref(d), C.byref(out.s), ctrl.handle) == 0
    assert (out.s.num_rows, out.s.num_cols, out.s.num_nonzeros) == (rows, cols, M.nnz)
    np.testing.assert_array_equal(out.row_ptr.cpu().numpy(), M.indptr)
    np.testing.assert_array_equal(out.col.cpu().numpy()[: M.nnz], M.indices)
    np.testing.assert_array_equal(out.val.cpu().numpy()[: M.nnz], M.data.astype(t))


def test_dense2csr_all_zero_and_reductions_after(ctrl):
    """An all-zero dense matrix gives an empty CSR, and the shared reduction
    scratch still works afterwards."""
    buf = torch.zeros(1500 * 4, dtype=torch.float64, device="cuda")
    d = dense_struct(buf, 1500, 4, 4, L.rowMajor)
    out = api.CsrMatrix(torch.zeros(1501, dtype=torch.int32, device="cuda"),
                        torch.zeros(8, dtype=torch.int32, device="cuda"),
                        torch.zeros(8, dtype=torch.float64, device="cuda"), 4)
    assert api.lib().clsparseDdense2csr(C.byref(d), C.byref(out.s), ctrl.handle) == 0
    assert out.s.num_nonzeros == 0 and int(out.row_ptr.abs().sum()) == 0
    x = torch.arange(1, 5001, dtype=torch.float64, device="cuda")
    r = torch.zeros(1, dtype=torch.float64, device="cuda")
    api.blas1("cldenseDreduce", ("s", r), x, ctrl=ctrl)
    assert float(r) == 5000 * 5001 / 2


@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-2.0, 0.5)])
def test_coomv_sorted_with_duplicates(ctrl, dt, alpha, beta):
    dtype, t = DT[dt], NPT[dt]
    rng = np.random.default_rng(11)
    M = random_csr(4001, 3000, 0.004, 8).tocoo()  # a row count that leaves idle groups
    # duplicate some entries (kept, summed by the product) and keep row order
    dup = rng.choice(M.nnz, 300, replace=False)
    rows = np.concatenate([M.row, M.row[dup]])
    cols = np.concatenate([M.col, M.col[dup]])
    vals = np.concatenate([M.data, rng.uniform(-1, 1, 300)])
    order = np.argsort(rows, kind="stable")
    rows, cols, vals = rows[order], cols[order], vals[order]
    # the struct holds raw pointers: keep the tensors alive
    keep = (torch.tensor(rows.astype(np.int32), device="cuda"), torch.tensor(cols.astype(np.int32), device="cuda"),
            torch.tensor(vals.astype(t), device="cuda"))
    cm = coo_struct(*keep, 4001, 3000)
    x = rng.uniform(-1, 1, 3000)
    y0 = rng.uniform(-1, 1, 4001)
    xt = torch.tensor(x.astype(t), device="cuda")
    yt = torch.tensor(y0.astype(t), device="cuda")
    a = torch.tensor([alpha], dtype=dtype, device="cuda")
    b = torch.tensor([beta], dtype=dtype, device="cuda")
    fn = api.lib().clsparseDcoomv if dt == "f64" else api.lib().clsparseScoomv
    assert fn(C.byref(api.scalar(a)), C.byref(cm), C.byref(api.vector(xt)), C.byref(api.scalar(b)),
              C.byref(api.vector(yt)), ctrl.handle) == 0
    A = sp.csr_matrix((vals.astype(t).astype(np.float64), (rows, cols)), shape=(4001, 3000))
    ref = alpha * (A @ x.astype(t).astype(np.float64)) + beta * y0.astype(t).astype(np.float64)
    scale = abs(alpha) * (abs(A) @ abs(x.astype(t).astype(np.float64))) + abs(beta * y0) + 1e-300
    tol = 1e-12 if dt == "f64" else 1e-5
    assert np.max(np.abs(yt.cpu().numpy() - ref) / scale) <= 10 * tol


@pytest.mark.parametrize("off", [0, 1, 3])
@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("rows,nnz", [(1, 1), (5, 0), (40, 2047), (40, 2048), (40, 2049), (9000, 4096), (100000, 3),
                                      (30000, 20000), (3, 10000)])
def test_coo_csr_runs(ctrl, dt, rows, nnz, off):
    """Both directions around a CTA's run of 2048 nonzeros, with short and
    long gaps of empty rows before, between and behind the nonzeros, and
    arrays that do not start on 16 bytes: exact."""
    dtype, t = DT[dt], NPT[dt]
    rng = np.random.default_rng(rows + nnz)
    r = np.sort(rng.choice(max(rows // 3, 1), nnz) + (rows // 3 if rows > 3 else 0)) if nnz else np.zeros(0, np.int64)
    c = rng.integers(0, 777, nnz)
    v = rng.uniform(-1, 1, nnz).astype(t)

    def dev(a, d):
        return torch.cat([torch.full((off,), 77, dtype=d, device="cuda"), torch.tensor(a, device="cuda").to(d),
                          torch.full((4,), 78, dtype=d, device="cuda")])

    ri, ci, vv = dev(r, torch.int32), dev(c, torch.int32), dev(v, dtype)
    cm = coo_struct(ri, ci, vv, rows, 777)
    cm.num_nonzeros = nnz
    cm.off_values = cm.off_col_indices = cm.off_row_indices = off
    rp, co, vo = (torch.full((off + k + 4,), 99, dtype=d, device="cuda") for k, d in
                  ((rows + 1, torch.int32), (nnz, torch.int32), (nnz, dtype)))
    out = api.CsrMatrix(rp, co, vo, 777)
    out.s.off_values = out.s.off_col_indices = out.s.off_row_pointer = off
    p = "D" if dt == "f64" else "S"
    assert getattr(api.lib(), f"clsparse{p}coo2csr")(C.byref(cm), C.byref(out.s), ctrl.handle) == 0
    want = np.searchsorted(r, np.arange(rows + 1), side="left")
    for got, ref in ((rp, want), (co, c), (vo, v)):
        g = got.cpu().numpy()
        np.testing.assert_array_equal(g[off:off + len(ref)], ref)
        assert (g[:off] == 99).all() and (g[off + len(ref):] == 99).all()
    r2, c2, v2 = (torch.full((off + nnz + 4,), 55, dtype=d, device="cuda") for d in (torch.int32, torch.int32, dtype))
    cm2 = coo_struct(r2, c2, v2, 0, 0)
    cm2.off_values = cm2.off_col_indices = cm2.off_row_indices = off
    assert getattr(api.lib(), f"clsparse{p}csr2coo")(C.byref(out.s), C.byref(cm2), ctrl.handle) == 0
    for got, ref in ((r2, r), (c2, c), (v2, v)):
        g = got.cpu().numpy()
        np.testing.assert_array_equal(g[off:off + nnz], ref)
        assert (g[:off] == 55).all() and (g[off + nnz:] == 55).all()


def conversions(ctrl, rows, r):
    """coo2csr and csr2coo of sorted row indices r (FP64) as two closures, and
    what they write."""
    nnz = len(r)
    ri = torch.tensor(np.asarray(r, dtype=np.int32), device="cuda")
    ci = torch.arange(nnz, dtype=torch.int32, device="cuda") % 777
    vv = torch.rand(nnz, dtype=torch.float64, device="cuda")
    cm = coo_struct(ri, ci, vv, rows, 777)
    out = api.CsrMatrix(*(torch.full((k,), -7, dtype=d, device="cuda") for k, d in
                          ((rows + 1, torch.int32), (nnz, torch.int32), (nnz, torch.float64))), 777)
    back = [torch.full_like(a, -5) for a in (ri, ci, vv)]
    cm2 = coo_struct(*back, 0, 0)
    to_csr = lambda: api.check(api.lib().clsparseDcoo2csr(C.byref(cm), C.byref(out.s), ctrl.handle), "coo2csr")
    to_coo = lambda: api.check(api.lib().clsparseDcsr2coo(C.byref(out.s), C.byref(cm2), ctrl.handle), "csr2coo")
    return to_csr, to_coo, (ri, ci, vv), out, back


# gaps between two occupied rows, around a lane's and a warp's share of a gap (16), a chunk of
# row pointers (32) and a gap CTA's share (32 x 256)
GAPS = [15, 16, 17, 18, 31, 32, 33, 34, 62, 63, 64, 65, 95, 96, 97, 8191, 8192, 8193, 40000]


@pytest.mark.parametrize("first", [0, 1, 31, 32, 200])
def test_coo_csr_gaps_of_empty_rows(ctrl, first):
    """Every gap length at every place within a chunk, several within one run
    of nonzeros, rows with several nonzeros among them, and gaps before and
    behind: exact."""
    rows_at = first + np.cumsum([0] + [g for g in GAPS for _ in range(3)])
    r = np.repeat(rows_at, 1 + np.arange(len(rows_at)) % 3)
    for tail in (0, 1, 31, 32, 33, 20000):
        rows = int(r[-1]) + 1 + tail
        to_csr, to_coo, src, out, back = conversions(ctrl, rows, r)
        to_csr()
        want = np.searchsorted(r, np.arange(rows + 1), side="left")
        np.testing.assert_array_equal(out.row_ptr.cpu().numpy(), want)
        to_coo()
        for a, b in zip(src, back):
            assert torch.equal(a, b)


@pytest.mark.parametrize("rows_in_run", [8191, 8192, 8193, 8194, 30000, 3000000])
@pytest.mark.parametrize("nnz", [2, 2048, 2049, 5000])
def test_csr2coo_runs_among_many_empty_rows(ctrl, rows_in_run, nnz):
    """A run's rows found by walking the row pointers or by looking its
    positions up (beyond 8192 rows between its first and last): exact."""
    r = np.sort(np.concatenate([[0, rows_in_run], np.random.default_rng(nnz).integers(0, rows_in_run + 1, nnz - 2)]))
    to_csr, to_coo, src, out, back = conversions(ctrl, rows_in_run + 5, r)
    to_csr()
    np.testing.assert_array_equal(out.row_ptr.cpu().numpy(), np.searchsorted(r, np.arange(rows_in_run + 6), side="left"))
    to_coo()
    for a, b in zip(src, back):
        assert torch.equal(a, b)


@pytest.mark.parametrize("case", ["spread", "two_blocks", "even"])
def test_conversions_spread_empty_rows_over_the_device(ctrl, case):
    """Many empty rows are not left to one CTA: each direction within the time
    of moving its arrays at a thirtieth of HBM's rate, and 60 us for launches
    and dependent loads (one CTA took 640 and 6100 us on `spread`, 660 and
    8700 on `two_blocks`; coo2csr 370 on `even`)."""
    rng = np.random.default_rng(1)
    rows, r = {"spread": (10_000_000, np.sort(rng.integers(0, 10_000_000, 3000))),
               "two_blocks": (10_000_000, np.sort(np.concatenate([rng.integers(0, 50_000, 500_000),
                                                                  9_950_000 + rng.integers(0, 50_000, 500_000)]))),
               "even": (1_000_000, np.linspace(0, 999_999, 16_000).astype(np.int64))}[case]
    to_csr, to_coo, src, out, back = conversions(ctrl, rows, r)
    bar = 60.0 + (4 * rows + 2 * 16 * len(r)) / 2.0e5  # us; 200 GB/s
    for fn in (to_csr, to_coo):
        times = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1) * 1e3)
        assert min(times) <= bar, (times, bar)
    assert torch.equal(src[0], back[0])
