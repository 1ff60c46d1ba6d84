"""Performance cases of the library, each through its public Python entry
points (clsparse_b200.api, thin calls through the C ABI).

A case names a kind of work (a sparse product, a conversion, vector steps, a
solve, a training step), its sizes and its options. The listed cases are:

  spmv_small_f64        y = A x inside a caller's own iteration on a small
                        unstructured system: call and launch latency count
  spmv_irregular_f64    the library's benchmark matrix: 2,000,000 rows of
                        log-normal lengths and 50 long rows, 60 M nonzeros
  spmv_stencil3d_f32    a residual r = b - A x on a 128^3 seven-point stencil
                        (short rows, alpha and beta in use)
  csrmm_f32             sparse times a block of 40 vectors, row-major (several
                        right-hand sides, feature aggregation on a graph)
  coo_csr_f64           a matrix read as COO turned into CSR and back
  blas1_f64             the vector steps of a caller's own Krylov loop: dot,
                        axpy, axpby, nrm2 on an odd length
  cg_poisson2d_f64      clsparseDcsrcg with Jacobi on the 512^2 Poisson problem
                        at the library's default settings, to 1e-10
  bicgstab_convdiff_f64 clsparseDcsrbicgStab on an upwind convection-diffusion
                        operator (nonsymmetric), to 1e-10
  cg_mixed_diff3d_f32   FP64 refinement around FP32 CG on a 128^3 log-normal
                        diffusion operator, to 1e-10
  cg_batched_f32        1024 independent stencil systems of 500 to 50,000 rows
                        in one call
  cg_learned_grf2d_f32  a new 1024^2 diffusion matrix end to end with a trained
                        network: graph, factor build, preconditioned solve
  spai_grad_f32         loss and gradient of that network on a 128^2 matrix,
                        four probes (the body of a training step)

draw() gives further cases of the same kinds over their whole ranges.

Inputs are made on the GPU from the seed alone. Matrices are the families the
library is tested on: Poisson, variable-coefficient diffusion (log-normal and
Gaussian-random-field coefficients, harmonic means on the faces), upwind
convection-diffusion, log-normal row lengths with uniform columns.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from clsparse_b200 import _lib as L
from clsparse_b200 import api, learn

DEV = "cuda"
DT = {"f64": torch.float64, "f32": torch.float32}
SIZE = {"f64": 8, "f32": 4}


# ---------------------------------------------------------------- the cases


def listed():
    return [
        {"name": "spmv_small_f64", "kind": "spmv", "pattern": "irregular", "n": 20011, "dense_rows": 0, "dtype": "f64",
         "alpha": 1.0, "beta": 0.0, "ext": False, "meta": True},
        {"name": "spmv_irregular_f64", "kind": "spmv", "pattern": "irregular", "n": 2000000, "dense_rows": 50,
         "dtype": "f64", "alpha": 1.0, "beta": 0.0, "ext": False, "meta": True},
        {"name": "spmv_stencil3d_f32", "kind": "spmv", "pattern": "diff3d", "n": 128, "dense_rows": 0, "dtype": "f32",
         "alpha": -1.0, "beta": 1.0, "ext": False, "meta": True},
        {"name": "csrmm_f32", "kind": "csrmm", "pattern": "irregular", "n": 200003, "dense_rows": 0, "dtype": "f32",
         "columns": 40, "alpha": 1.0, "beta": 0.0},
        {"name": "coo_csr_f64", "kind": "coo_csr", "pattern": "irregular", "n": 400009, "dense_rows": 0,
         "dtype": "f64"},
        {"name": "blas1_f64", "kind": "blas1", "n": 3000001, "dtype": "f64"},
        {"name": "cg_poisson2d_f64", "kind": "cg", "pattern": "poisson2d", "n": 512, "dtype": "f64", "tol": 1e-10,
         "loop_mode": 0},
        {"name": "bicgstab_convdiff_f64", "kind": "bicgstab", "pattern": "convdiff2d", "n": 300, "dtype": "f64",
         "tol": 1e-10, "loop_mode": 0},
        {"name": "cg_mixed_diff3d_f32", "kind": "mixed", "pattern": "diff3d", "n": 128, "dtype": "f64",
         "inner": "fp32", "tol": 1e-10},
        {"name": "cg_batched_f32", "kind": "batched", "systems": 1024, "n_min": 500, "n_max": 50000, "dtype": "f32",
         "tol": 1e-5},
        {"name": "cg_learned_grf2d_f32", "kind": "learned", "pattern": "grf2d", "n": 1024, "dtype": "f64",
         "inner": "fp32", "tol": 1e-10},
        {"name": "spai_grad_f32", "kind": "spai_grad", "pattern": "grf2d", "n": 128, "dtype": "f64", "probes": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "csrmm", "coo_csr", "blas1", "cg", "cg", "bicgstab", "mixed", "batched",
                       "learned", "spai_grad"])
    if kind == "spmv":
        pattern = rng.choice(["irregular", "irregular", "diff3d", "grf2d"])
        n = {"irregular": lambda: _log_int(rng, 1000, 1500000), "diff3d": lambda: _log_int(rng, 20, 128),
             "grf2d": lambda: _log_int(rng, 60, 1024)}[pattern]()
        alpha, beta = rng.choice([(1.0, 0.0), (1.0, 0.0), (-1.0, 1.0), (0.75, -0.5)])
        dense = rng.choice([0, 0, 7, 30]) if pattern == "irregular" and n > 500000 else 0
        return {"kind": kind, "pattern": pattern, "n": n, "dense_rows": dense, "dtype": rng.choice(["f64", "f32"]),
                "alpha": alpha, "beta": beta, "ext": rng.random() < 0.2, "meta": rng.random() < 0.75}
    if kind == "csrmm":
        alpha, beta = rng.choice([(1.0, 0.0), (-0.5, 1.0)])
        pattern = rng.choice(["irregular", "diff3d"])
        n = _log_int(rng, 2000, 300000) if pattern == "irregular" else _log_int(rng, 16, 80)
        return {"kind": kind, "pattern": pattern, "n": n, "dense_rows": 0, "dtype": rng.choice(["f64", "f32"]),
                "columns": _log_int(rng, 2, 64), "alpha": alpha, "beta": beta}
    if kind == "coo_csr":
        pattern = rng.choice(["irregular", "diff3d"])
        n = _log_int(rng, 5000, 800000) if pattern == "irregular" else _log_int(rng, 24, 128)
        return {"kind": kind, "pattern": pattern, "n": n, "dense_rows": 0, "dtype": rng.choice(["f64", "f32"])}
    if kind == "blas1":
        return {"kind": kind, "n": _log_int(rng, 5000, 20000000), "dtype": rng.choice(["f64", "f32"])}
    if kind == "cg":
        pattern = rng.choice(["poisson2d", "diff3d", "grf2d", "unstructured"])
        n = _log_int(rng, 20, 100) if pattern == "diff3d" else _log_int(rng, 60, 512)
        # (FP32 on the ill-conditioned random fields has no accurate digits to compare)
        dtype = "f64" if pattern == "grf2d" else rng.choice(["f64", "f64", "f32"])
        return {"kind": kind, "pattern": pattern, "n": n, "dtype": dtype, "tol": 1e-10 if dtype == "f64" else 1e-4,
                "loop_mode": rng.choice([0, 0, 0, 3])}
    if kind == "bicgstab":
        return {"kind": kind, "pattern": "convdiff2d", "n": _log_int(rng, 60, 512), "dtype": "f64", "tol": 1e-10,
                "loop_mode": rng.choice([0, 0, 3])}
    if kind == "mixed":
        pattern = rng.choice(["diff3d", "grf2d", "poisson2d"])
        n = _log_int(rng, 24, 128) if pattern == "diff3d" else _log_int(rng, 80, 700)
        inner = rng.choice(["fp32", "bf16"]) if pattern == "diff3d" else "fp32"
        return {"kind": kind, "pattern": pattern, "n": n, "dtype": "f64", "inner": inner, "tol": 1e-10}
    if kind == "batched":
        n_min = _log_int(rng, 100, 2000)
        return {"kind": kind, "systems": _log_int(rng, 48, 1024), "n_min": n_min,
                "n_max": n_min * _log_int(rng, 2, 25), "dtype": "f32", "tol": 1e-5}
    if kind == "learned":
        return {"kind": kind, "pattern": "grf2d", "n": _log_int(rng, 128, 1024), "dtype": "f64", "inner": "fp32",
                "tol": 1e-10}
    return {"kind": "spai_grad", "pattern": "grf2d", "n": _log_int(rng, 48, 160), "dtype": "f64",
            "probes": rng.choice([0, 2, 4])}


# ------------------------------------------------------------- the matrices


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) % (2 ** 62))
    return g


def _uniform(g, *size, dtype=torch.float64):
    return torch.rand(*size, generator=g, device=DEV, dtype=torch.float64).mul_(2).sub_(1).to(dtype)


def _from_diagonals(offsets, values, valid):
    """CSR (rp, col, val) from per-row diagonal values (lists over increasing
    column offsets of [n] tensors) and validity masks."""
    n = values[0].numel()
    rows = torch.arange(n, device=DEV)
    v = torch.stack(values, dim=1)
    m = torch.stack(valid, dim=1)
    c = torch.stack([rows + o for o in offsets], dim=1)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(m.sum(dim=1), 0, out=rp[1:])
    return rp, c[m], v[m]


def _harmonic(a, b):
    return 2.0 * a * b / (a + b)


def _diffusion(shape, k):
    """Cell-centred diffusion on a grid, first axis fastest, Dirichlet walls."""
    n = int(np.prod(shape))
    idx = torch.arange(n, device=DEV)
    rem, coords, strides, s = idx, [], [], 1
    for m in shape:
        coords.append(rem % m)
        rem = rem // m
        strides.append(s)
        s *= m
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    low, high = [], []
    for m, st, c in zip(shape, strides, coords):
        for d, out in ((-1, low), (1, high)):
            ok = (c + d >= 0) & (c + d < m)
            nb = torch.where(ok, idx + d * st, idx)
            kf = torch.where(ok, _harmonic(k, k[nb]), k)
            diag += kf
            out.append((d * st, -kf, ok))
    entries = sorted(low + high + [(0, diag, torch.ones_like(idx, dtype=torch.bool))], key=lambda e: e[0])
    return _from_diagonals([e[0] for e in entries], [e[1] for e in entries], [e[2] for e in entries])


def _grf2d(m, g, corr_len=0.05, sigma=2.0):
    f = torch.fft.fftfreq(m, d=1.0 / m, device=DEV, dtype=torch.float64)
    k2 = (2 * math.pi) ** 2 * (f[:, None] ** 2 + f[None, :] ** 2)
    spec = torch.exp(-k2 * corr_len ** 2 / 4.0)
    noise = torch.complex(torch.randn(m, m, generator=g, device=DEV, dtype=torch.float64),
                          torch.randn(m, m, generator=g, device=DEV, dtype=torch.float64))
    x = torch.fft.ifft2(torch.sqrt(spec) * noise).real
    return (x - x.mean()) / x.std() * sigma


def _convdiff2d(m, g):
    """Upwind convection-diffusion, velocity drawn per row and positive."""
    n = m * m
    idx = torch.arange(n, device=DEV)
    i, j = idx % m, idx // m
    cx = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    cy = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    return _from_diagonals([-m, -1, 0, 1, m], [-one - cy, -one - cx, 4 * one + cx + cy, -one, -one],
                           [j > 0, i > 0, i >= 0, i < m - 1, j < m - 1])


def _renumber(rp, col, val, g, window=512):
    """Symmetric renumbering at random inside windows of rows: the operator of
    an unstructured mesh with a bandwidth-reducing order."""
    n = rp.numel() - 1
    idx = torch.arange(n, device=DEV)
    key = (idx // window).double() + torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    new_of = torch.empty(n, dtype=torch.int64, device=DEV)
    new_of[torch.argsort(key)] = idx
    rows = new_of[torch.repeat_interleave(idx, rp[1:] - rp[:-1])]
    cols = new_of[col]
    order = torch.argsort(rows * n + cols)
    out = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(rows, minlength=n), 0, out=out[1:])
    return out, cols[order], val[order]


def _irregular(n, dense_rows, g):
    """Log-normal(2.5, 1.2) row lengths (of n alone, so that every seed has as
    many nonzeros), `dense_rows` rows of n / 10; each row's columns uniform,
    one in each of as many equal strata (distinct and sorted); values U[-1, 1]."""
    shape = _generator(n)
    lens = torch.exp(torch.randn(n, generator=shape, device=DEV, dtype=torch.float64) * 1.2 + 2.5).round().long()
    lens = lens.clamp(1, max(1, n // 4))
    if dense_rows:
        lens[torch.randperm(n, generator=shape, device=DEV)[:dense_rows]] = n // 10
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(lens, 0, out=rp[1:])
    nnz = int(rp[-1])
    k = torch.arange(nnz, device=DEV) - torch.repeat_interleave(rp[:-1], lens)
    width = torch.repeat_interleave(lens, lens)
    lo, hi = k * n // width, (k + 1) * n // width
    cols = lo + (torch.rand(nnz, generator=g, device=DEV, dtype=torch.float64) * (hi - lo)).long()
    return rp, torch.minimum(cols, hi - 1), _uniform(g, nnz)


def _matrix(case, g):
    """(row pointers, columns, values) as int64 / int64 / float64 tensors."""
    p, n = case["pattern"], case["n"]
    if p == "irregular":
        return _irregular(n, case["dense_rows"], g)
    if p == "poisson2d":
        return _diffusion((n, n), torch.ones(n * n, dtype=torch.float64, device=DEV))
    if p == "diff3d":
        k = torch.exp(1.5 * torch.randn(n ** 3, generator=g, device=DEV, dtype=torch.float64))
        return _diffusion((n, n, n), k)
    if p == "grf2d":
        return _diffusion((n, n), torch.exp(_grf2d(n, g)).reshape(-1))
    if p == "convdiff2d":
        return _convdiff2d(n, g)
    if p == "unstructured":
        k = torch.exp(torch.randn(n * n, generator=g, device=DEV, dtype=torch.float64))
        return _renumber(*_diffusion((n, n), k), g)
    raise ValueError(p)


def _batch(case, g):
    """Independent 2D / 3D diffusion systems stacked block-diagonally, sizes
    log-uniform (of the case alone, the coefficients of the seed): system s is
    the first n_s cells of a grid just large enough."""
    nsys = case["systems"]
    shape = _generator(nsys)
    u = torch.rand(nsys, generator=shape, device=DEV, dtype=torch.float64)
    ns = torch.exp(math.log(case["n_min"]) + u * (math.log(case["n_max"]) - math.log(case["n_min"]))).round().long()
    three = torch.rand(nsys, generator=shape, device=DEV) < 0.5
    side = torch.where(three, ns.double().pow(1 / 3), ns.double().sqrt()).ceil().long() + 1
    cells = torch.where(three, side ** 3, side ** 2)
    off = torch.zeros(nsys + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(ns, 0, out=off[1:])
    coff = torch.zeros(nsys + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(cells, 0, out=coff[1:])
    k = torch.exp(torch.randn(int(coff[-1]), generator=g, device=DEV, dtype=torch.float64))
    n = int(off[-1])
    sys = torch.repeat_interleave(torch.arange(nsys, device=DEV), ns)
    row = torch.arange(n, device=DEV)
    local = row - off[sys]
    m, t, cbase, nloc = side[sys], three[sys], coff[sys], ns[sys]
    kc = k[cbase + local]
    coords = [local % m, torch.where(t, (local // m) % m, local // m), torch.where(t, local // (m * m), 0)]
    strides = [torch.ones_like(m), m, m * m]
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    cols, vals, keep = [], [], []
    for d in (-1, 1):
        for ax in (2, 1, 0) if d < 0 else (0, 1, 2):
            used = t if ax == 2 else torch.ones_like(t)
            ok = used & (coords[ax] + d >= 0) & (coords[ax] + d < m)
            nb = torch.where(ok, local + d * strides[ax], local)
            kf = torch.where(ok, _harmonic(kc, k[cbase + nb]), kc)
            diag += torch.where(used, kf, 0.0)
            cols.append(row + (nb - local))
            vals.append(-kf)
            keep.append(ok & (nb < nloc))
        if d < 0:
            at = len(cols)
    cols.insert(at, row)
    vals.insert(at, diag)
    keep.insert(at, torch.ones_like(t))
    mask = torch.stack(keep, dim=1)
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(mask.sum(dim=1), 0, out=rp[1:])
    return rp, torch.stack(cols, dim=1)[mask], torch.stack(vals, dim=1)[mask], off


# ------------------------------------------------------------- prepare, run


class State:
    """What a caller's program keeps between calls; the library's handles are
    given back with it."""

    def __init__(self):
        self.ctrl = api.Control()
        self.spai = None

    def __del__(self):
        try:
            if self.spai is not None:
                self.spai.release()
            self.ctrl.release()
        except Exception:
            pass


def _csr(rp, col, val, dtype, ncols=None):
    return api.CsrMatrix(rp.to(torch.int32), col.to(torch.int32), val.to(dtype),
                         rp.numel() - 1 if ncols is None else ncols)


def _trained(ctrl):
    """A network trained briefly on two small members of the family."""
    spai, _ = learn.train(ctrl, sizes=(32,), seeds=range(2), steps=20, lr=3e-3)
    return spai


def _dense_struct(t, rows, cols):
    return L.cldenseMatrix(rows, cols, cols, L.rowMajor, C.c_void_p(t.data_ptr()), 0)


def _coo_struct(n, nnz, val, col, row):
    return L.clsparseCooMatrix(n, n, nnz, C.c_void_p(val.data_ptr()), C.c_void_p(col.data_ptr()),
                               C.c_void_p(row.data_ptr()), 0, 0, 0)


def prepare(case, seed):
    g = _generator(seed)
    kind, dt = case["kind"], DT[case["dtype"]]
    st = State()
    st.case = case
    ctrl = st.ctrl
    if kind in ("spmv", "csrmm", "coo_csr", "blas1"):
        ctrl.enable_async(True)  # the caller's loop is ordered by its stream
    if kind == "blas1":
        st.x, st.y = _uniform(g, case["n"], dtype=dt), _uniform(g, case["n"], dtype=dt)
        st.r, st.w = torch.empty_like(st.x), torch.empty_like(st.x)
        st.a, st.b = torch.full((1,), 0.375, dtype=dt, device=DEV), torch.full((1,), -0.75, dtype=dt, device=DEV)
        st.dot, st.nrm = torch.zeros(1, dtype=dt, device=DEV), torch.zeros(1, dtype=dt, device=DEV)
        return st
    if kind == "batched":
        rp, col, val, off = _batch(case, g)
        st.off = off.cpu().numpy().astype(np.uint32)
    else:
        rp, col, val = _matrix(case, g)
    n = rp.numel() - 1
    st.A = A = _csr(rp, col, val, dt)
    if kind == "spmv":
        if case["meta"]:
            A.create_meta(ctrl)
        if case["ext"]:
            ctrl.enable_extended_precision(True)
        st.x, st.b = _uniform(g, n, dtype=dt), _uniform(g, n, dtype=dt)
        st.y = torch.empty_like(st.b)
        st.alpha = torch.full((1,), case["alpha"], dtype=dt, device=DEV)
        st.beta = torch.full((1,), case["beta"], dtype=dt, device=DEV)
    elif kind == "csrmm":
        k = case["columns"]
        st.B, st.C0 = _uniform(g, n, k, dtype=dt), _uniform(g, n, k, dtype=dt)
        st.C = torch.empty_like(st.C0)
        st.alpha = torch.full((1,), case["alpha"], dtype=dt, device=DEV)
        st.beta = torch.full((1,), case["beta"], dtype=dt, device=DEV)
    elif kind == "coo_csr":
        st.row = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1]).to(torch.int32)
        st.col, st.val, st.n, st.nnz = A.col, A.val, n, A.nnz
        st.A = None
        st.rp2 = torch.empty(n + 1, dtype=torch.int32, device=DEV)
        st.col2, st.val2 = torch.empty_like(st.col), torch.empty_like(st.val)
        st.row3, st.col3, st.val3 = torch.empty_like(st.row), torch.empty_like(st.col), torch.empty_like(st.val)
    elif kind == "spai_grad":
        st.spai = _trained(ctrl)
        st.spai.set_matrix(A, ctrl)
        st.probes = None
        if case["probes"]:
            p = torch.randn(case["probes"], n, generator=g, device=DEV, dtype=torch.float64)
            st.probes = (p / p.norm(dim=1, keepdim=True)).float()
    else:
        if kind in ("cg", "bicgstab", "mixed", "learned"):
            A.create_meta(ctrl)
        if kind in ("cg", "bicgstab"):
            ctrl.set_solver_loop_mode(case["loop_mode"])
        if kind == "learned":
            st.spai = _trained(ctrl)
        st.b = _uniform(g, n, dtype=dt)
        st.x = torch.zeros_like(st.b)
    return st


def run(st):
    case, ctrl = st.case, st.ctrl
    kind = case["kind"]
    pre = "D" if case["dtype"] == "f64" else "S"
    if kind == "spmv":
        if case["beta"] != 0.0:
            st.y.copy_(st.b)
        api.csrmv(st.alpha, st.A, st.x, st.beta, st.y, ctrl)
        return st.y
    if kind == "csrmm":
        n, k = st.C.shape
        if case["beta"] != 0.0:
            st.C.copy_(st.C0)
        b, c = _dense_struct(st.B, n, k), _dense_struct(st.C, n, k)
        api.check(getattr(api.lib(), f"clsparse{pre}csrmm")(
            C.byref(api.scalar(st.alpha)), C.byref(st.A.s), C.byref(b), C.byref(api.scalar(st.beta)), C.byref(c),
            ctrl.handle), "csrmm")
        return st.C
    if kind == "coo_csr":
        coo = _coo_struct(st.n, st.nnz, st.val, st.col, st.row)
        csr = api.CsrMatrix(st.rp2, st.col2, st.val2, st.n)
        api.check(getattr(api.lib(), f"clsparse{pre}coo2csr")(C.byref(coo), C.byref(csr.s), ctrl.handle), "coo2csr")
        back = _coo_struct(st.n, st.nnz, st.val3, st.col3, st.row3)
        api.check(getattr(api.lib(), f"clsparse{pre}csr2coo")(C.byref(csr.s), C.byref(back), ctrl.handle), "csr2coo")
        return st.rp2, st.col2, st.val2, st.row3, st.col3, st.val3
    if kind == "blas1":
        api.blas1(f"cldense{pre}dot", ("s", st.dot), st.x, st.y, ctrl=ctrl)
        api.blas1(f"cldense{pre}axpy", st.r, ("s", st.a), st.x, st.y, ctrl=ctrl)
        api.blas1(f"cldense{pre}axpby", st.w, ("s", st.a), st.r, ("s", st.b), st.y, ctrl=ctrl)
        api.blas1(f"cldense{pre}nrm2", ("s", st.nrm), st.w, ctrl=ctrl)
        return st.dot, st.r, st.w, st.nrm
    if kind == "spai_grad":
        loss = st.spai.loss_grad_device(ctrl, st.probes, 0.2 if st.probes is not None else 0.0)
        return loss, st.spai.grad_buffer().clone()  # the buffer itself goes with the network
    st.x.zero_()
    sc = api.SolverControl(L.DIAGONAL, 100000, case["tol"], 0.0)
    if kind == "learned":
        st.spai.set_matrix(st.A, ctrl)
        st.spai.build(ctrl)
        api.cg_learned(st.x, st.A, st.b, sc, st.spai, ctrl, inner=case["inner"], inner_tol=0.3)
    elif kind == "mixed":
        api.cg_mixed(st.x, st.A, st.b, sc, ctrl, inner=case["inner"], inner_tol=0.3)
    elif kind == "batched":
        api.cg_batched(st.x, st.A, st.b, st.off, sc, ctrl)
    else:
        api.solve(kind, st.x, st.A, st.b, sc, ctrl)
    sc.release()
    return st.x


# --------------------------------------------------- work, tolerance, exact


def _sizes(case):
    """(rows, nonzeros), expected."""
    if case["kind"] == "batched":
        lo, hi = case["n_min"], case["n_max"]
        n = case["systems"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        return n, 5.9 * n
    p, m = case["pattern"], case["n"]
    if p == "irregular":
        return m, 25.03 * m + case["dense_rows"] * (m // 10)
    if p == "diff3d":
        return m ** 3, 7 * m ** 3 - 6 * m ** 2
    return m ** 2, 5 * m ** 2 - 4 * m


def work(case):
    """Inputs read once, outputs written once. A solve's iterations are not in
    the bytes (what they move depends on where the system is kept) nor in the
    operations (their number is the method's)."""
    kind, s = case["kind"], SIZE[case["dtype"]]
    if kind == "blas1":
        n = case["n"]  # x, y in; r, w out
        return {"bytes": 4 * n * s, "flops": 9 * n}
    n, nnz = _sizes(case)
    matrix = (4 + s) * nnz + 4 * (n + 1)
    if kind == "spmv":
        return {"bytes": matrix + (3 if case["beta"] else 2) * n * s, "flops": 2 * nnz}
    if kind == "csrmm":
        k = case["columns"]
        return {"bytes": matrix + (3 if case["beta"] else 2) * n * k * s, "flops": 2 * nnz * k}
    if kind == "coo_csr":
        # COO in, CSR out; CSR in, COO out
        return {"bytes": 2 * (matrix + (8 + s) * nnz), "flops": 0}
    if kind == "spai_grad":
        # per node and layer two dense products (64x64, 64x128), forward and
        # twice that backward; the output layer's two 32x64
        dense = 4 * (64 * 64 + 64 * 128) + 2 * 32 * 64
        return {"bytes": matrix + case["probes"] * n * 4 + 4 * 54000, "flops": 2 * n * dense * 3}
    if kind == "learned":
        dense = 4 * (64 * 64 + 64 * 128) + 2 * 32 * 64
        return {"bytes": matrix + 2 * n * s, "flops": 2 * n * dense}
    return {"bytes": matrix + 2 * n * s, "flops": 2 * nnz}


def tolerance(case):
    kind = case["kind"]
    if kind == "coo_csr":
        return "exact"
    if kind in ("spmv", "csrmm", "blas1"):
        return {"rel": 1e-13, "max": 1e-11} if case["dtype"] == "f64" else {"rel": 2e-6, "max": 2e-4}
    if kind == "spai_grad":
        return {"rel": 2e-3, "max": 0.1}
    if kind == "batched" or case["dtype"] == "f32":
        return {"rel": 1e-2, "max": 0.9}  # x of an FP32 solve that stops at 1e-4 or 1e-5
    return {"rel": 1e-7, "max": 1e-5}  # x of a solve that stops at 1e-10


def _apply(rows, col, val, x, n):
    y = torch.zeros((n,) + x.shape[1:], dtype=torch.float64, device=DEV)
    for k0 in range(0, col.numel(), 4 << 20):  # in pieces: x may have many columns
        k1 = min(col.numel(), k0 + (4 << 20))
        v = val[k0:k1]
        y.index_add_(0, rows[k0:k1], (v if x.dim() == 1 else v[:, None]) * x[col[k0:k1]])
    return y


def _solve64(rp, col, val, b, max_iters=60000):
    """x with ||b - A x|| <= 1e-13 ||b||, or as far as FP64 goes: Jacobi-
    preconditioned BiCGStab for a nonsymmetric A is not needed beyond the
    operators here, whose normal equations are avoided by restarting."""
    n = b.numel()
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    M = torch.sparse_csr_tensor(rp, col, val, (n, n))
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    on = rows == col
    diag[rows[on]] = val[on]
    inv = 1.0 / diag
    x = torch.zeros(n, dtype=torch.float64, device=DEV)
    bn = b.norm()
    left = max_iters
    for _ in range(6):  # restarted on the true residual
        r = b - M @ x
        if r.norm() <= 1e-13 * bn or left <= 0:
            break
        z = inv * r
        p = z.clone()
        rz = torch.dot(r, z)
        stop = 1e-13 * bn
        while left > 0:
            for _ in range(50):
                q = M @ p
                alpha = rz / torch.dot(p, q)
                x += alpha * p
                r -= alpha * q
                z = inv * r
                new = torch.dot(r, z)
                p = z + (new / rz) * p
                rz = new
            left -= 50
            if not bool(r.norm() > stop):
                break
        x = torch.nan_to_num(x)
    return x


def _solve64_nonsym(rp, col, val, b, max_iters=20000):
    n = b.numel()
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    M = torch.sparse_csr_tensor(rp, col, val, (n, n))
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    on = rows == col
    diag[rows[on]] = val[on]
    inv = 1.0 / diag
    best = x = torch.zeros(n, dtype=torch.float64, device=DEV)
    bn = b.norm()
    best_res, left = math.inf, max_iters
    for _ in range(12):
        r = b - M @ x
        res = float(r.norm() / bn)
        if res < best_res:
            best, best_res = x.clone(), res
        if best_res <= 1e-13 or left <= 0:
            break
        x = best.clone()
        r = b - M @ x
        rs, p = r.clone(), r.clone()
        rho = torch.dot(rs, r)
        for it in range(left):
            ph = inv * p
            v = M @ ph
            alpha = rho / torch.dot(rs, v)
            s = r - alpha * v
            sh = inv * s
            t = M @ sh
            w = torch.dot(t, s) / torch.dot(t, t)
            x = x + alpha * ph + w * sh
            r = s - w * t
            new = torch.dot(rs, r)
            p = r + (new / rho) * (alpha / w) * (p - w * v)
            rho = new
            left -= 1
            if it % 10 == 9 and not bool(r.norm() > 2e-14 * bn):
                break
        x = torch.nan_to_num(x)
    return best


def _exact_grad(st):
    """Loss and gradient of the network in 64 bits (weights rounded to BF16 as
    the library uses them), by automatic differentiation."""
    H, HO, NF, NL = 64, 32, 4, 4
    rp, col, val = st.A.row_ptr.long(), st.A.col.long(), st.A.val
    n = rp.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    on = rows == col
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    diag[rows[on]] = val[on]
    dinv = diag.rsqrt()
    e = val * dinv[rows] * dinv[col]
    w = torch.tensor(st.spai.params(), device=DEV).bfloat16().double().requires_grad_(True)
    at = 0

    def take(*shape):
        nonlocal at
        size = int(np.prod(shape))
        out = w[at:at + size].reshape(*shape)
        at += size
        return out

    w_in, b_in = take(H, NF), take(H)
    layers = [(take(H, H), take(H), take(H), take(H, 2 * H), take(H)) for _ in range(NL)]
    P, Q, rr, tt, w_o, b_o, w_d, b_d = take(HO, H), take(HO, H), take(HO), take(HO), take(HO), take(1), take(H), take(1)
    ro, co, eo = rows[~on], col[~on], e[~on]
    zero = torch.zeros(n, dtype=torch.float64, device=DEV)
    F = torch.stack([zero + 1, zero.index_add(0, ro, eo.abs()), zero.index_add(0, ro, torch.ones_like(eo)) / 8, zero],
                    dim=1)
    h = torch.relu(F @ w_in.T + b_in)
    for U, wl, cl, V, dl in layers:
        msg = torch.relu((h @ U.T)[co] + eo[:, None] * wl + cl)
        s = torch.zeros(n, H, dtype=torch.float64, device=DEV).index_add(0, ro, msg)
        h = h + torch.relu(torch.cat([h, s], dim=1) @ V.T + dl)
    low = col < rows
    li, lj, le = rows[low], col[low], e[low]
    g = torch.relu((h @ P.T)[li] + (h @ Q.T)[lj] + le[:, None] * rr + tt) @ w_o + b_o
    gd = torch.nn.functional.softplus(h @ w_d + b_d, threshold=40)
    # <g_i, A[P_i, P_i] g_i>: on a five-point grid a row's lower neighbours
    # are not adjacent to one another, and the scaled diagonal is 1
    tr = (gd ** 2).sum() + (g ** 2).sum() + 2 * (gd[li] * g * le).sum()
    loss = torch.log(tr / n) - 2 * torch.log(gd).sum() / n
    if st.probes is not None:
        def lower(v):
            return (gd * v).index_add(0, li, g * v[lj])

        def upper(v):
            return (gd * v).index_add(0, lj, g * v[li])

        for r in st.probes.double():
            d = upper(lower(zero.index_add(0, rows, e * r[col]))) - r
            loss = loss + 0.2 * (d @ d) / (len(st.probes) * (r @ r))
    grad = torch.autograd.grad(loss, w)[0]
    return float(loss), grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "coo_csr":
        return None
    st = prepare(case, seed)
    if kind == "blas1":
        x, y, a, b = st.x.double(), st.y.double(), st.a.double(), st.b.double()
        r = y + a * x
        # the second step reads the first one's stored (rounded) result
        w = a * r.to(st.r.dtype).double() + b * y
        nrm = w.to(st.w.dtype).double().square().sum().sqrt()
        return (x * y).sum().reshape(1), r, w, nrm.reshape(1)
    if kind == "spai_grad":
        return _exact_grad(st)
    rp, col, val = st.A.row_ptr.long(), st.A.col.long(), st.A.val.double()
    n = rp.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), rp[1:] - rp[:-1])
    if kind == "spmv":
        y = st.alpha.double() * _apply(rows, col, val, st.x.double(), n)
        return y + st.beta.double() * st.b.double() if case["beta"] else y
    if kind == "csrmm":
        y = st.alpha.double() * _apply(rows, col, val, st.B.double(), n)
        return y + st.beta.double() * st.C0.double() if case["beta"] else y
    if kind == "bicgstab":
        return _solve64_nonsym(rp, col, val, st.b.double())
    return _solve64(rp, col, val, st.b.double())
