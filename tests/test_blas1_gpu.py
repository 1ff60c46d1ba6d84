"""cldense* BLAS-1 entry points through the C ABI against numpy (float64
references), the semantics of src/library/blas1/*.cpp. Tolerances: FP64 1e-12
relative, FP32 1e-5 relative (the reference's own test uses absolute 1e-14 /
1e-7 on constant vectors, src/tests/test-blas1.cpp:146-148)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from clsparse_b200 import api

pytestmark = pytest.mark.gpu

TOL = {torch.float64: 1e-12, torch.float32: 1e-5}
SIZES = [1, 7, 1000, 1_048_579]


def t(a, dtype):
    return torch.tensor(np.asarray(a), dtype=dtype, device="cuda")


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("n", SIZES)
def test_reductions(ctrl, dtype, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, n)
    y = rng.uniform(-1, 1, n)
    p = "D" if dtype == torch.float64 else "S"
    xt, yt = t(x, dtype), t(y, dtype)
    xd = xt.double().cpu().numpy()
    yd = yt.double().cpu().numpy()
    s = torch.zeros(1, dtype=dtype, device="cuda")
    cases = {
        f"cldense{p}reduce": (xd.sum(), np.abs(xd).sum()),
        f"cldense{p}nrm1": (np.abs(xd).sum(), np.abs(xd).sum()),
        f"cldense{p}nrm2": (np.sqrt((xd * xd).sum()), np.sqrt((xd * xd).sum())),
    }
    for name, (ref, scale) in cases.items():
        api.blas1(name, ("s", s), xt, ctrl=ctrl)
        assert abs(float(s) - ref) <= TOL[dtype] * scale + 1e-300, name
    api.blas1(f"cldense{p}dot", ("s", s), xt, yt, ctrl=ctrl)
    assert abs(float(s) - (xd * yd).sum()) <= TOL[dtype] * np.abs(xd * yd).sum() + 1e-300


def test_int_reduce(ctrl):
    x = torch.arange(-500, 100_000, dtype=torch.int32, device="cuda")
    s = torch.zeros(1, dtype=torch.int32, device="cuda")
    api.blas1("cldenseIreduce", ("s", s), x, ctrl=ctrl)
    # 32-bit two's-complement wraparound, as an int accumulation would give
    total = int(np.arange(-500, 100_000, dtype=np.int64).sum())
    assert int(s) == ((total + 2 ** 31) % 2 ** 32) - 2 ** 31


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("n", SIZES)
def test_elementwise_and_axpy(ctrl, dtype, n):
    rng = np.random.default_rng(n + 1)
    x = rng.uniform(-1, 1, n)
    y = rng.uniform(0.5, 1.5, n)
    p = "D" if dtype == torch.float64 else "S"
    xt, yt = t(x, dtype), t(y, dtype)
    xd, yd = xt.double().cpu().numpy(), yt.double().cpu().numpy()
    r = torch.empty(n, dtype=dtype, device="cuda")
    for name, ref in (("add", xd + yd), ("sub", xd - yd), ("mul", xd * yd), ("div", xd / yd)):
        api.blas1(f"cldense{p}{name}", r, xt, yt, ctrl=ctrl)
        np.testing.assert_allclose(r.double().cpu().numpy(), ref, rtol=TOL[dtype] * 10, atol=1e-30)
    a = t([1.75], dtype)
    bb = t([-0.5], dtype)
    api.blas1(f"cldense{p}scale", r, ("s", a), yt, ctrl=ctrl)
    np.testing.assert_allclose(r.double().cpu().numpy(), 1.75 * yd, rtol=TOL[dtype] * 10)
    api.blas1(f"cldense{p}axpy", r, ("s", a), xt, yt, ctrl=ctrl)
    np.testing.assert_allclose(r.double().cpu().numpy(), yd + 1.75 * xd, rtol=TOL[dtype] * 10, atol=TOL[dtype])
    api.blas1(f"cldense{p}axpby", r, ("s", a), xt, ("s", bb), yt, ctrl=ctrl)
    np.testing.assert_allclose(r.double().cpu().numpy(), 1.75 * xd - 0.5 * yd, rtol=TOL[dtype] * 10,
                               atol=TOL[dtype])


def test_alpha_zero_shortcuts(ctrl):
    """alpha == 0: scale fills zeros, axpy copies y (cldense-scale.cpp:41-53,
    cldense-axpy.cpp:50-63) -- even when x holds NaN."""
    n = 1000
    x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
    y = torch.arange(n, dtype=torch.float64, device="cuda")
    r = torch.empty(n, dtype=torch.float64, device="cuda")
    z = torch.zeros(1, dtype=torch.float64, device="cuda")
    api.blas1("cldenseDscale", r, ("s", z), x, ctrl=ctrl)
    assert float(r.abs().sum()) == 0.0
    api.blas1("cldenseDaxpy", r, ("s", z), x, y, ctrl=ctrl)
    assert torch.equal(r, y)


def test_empty_vectors(ctrl):
    e = torch.empty(0, dtype=torch.float64, device="cuda")
    s = torch.full((1,), 5.0, dtype=torch.float64, device="cuda")
    api.blas1("cldenseDnrm1", ("s", s), e, ctrl=ctrl)
    assert float(s) == 0.0
    api.blas1("cldenseDadd", e, e, e, ctrl=ctrl)


def test_size_mismatch(ctrl):
    a = torch.zeros(5, dtype=torch.float64, device="cuda")
    b = torch.zeros(6, dtype=torch.float64, device="cuda")
    with pytest.raises(api.ClsparseError):
        api.blas1("cldenseDadd", a, a, b, ctrl=ctrl)


def test_async_mode_and_event(ctrl):
    ctrl.enable_async(True)
    n = 1 << 20
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    s = torch.zeros(1, dtype=torch.float64, device="cuda")
    api.blas1("cldenseDnrm1", ("s", s), x, ctrl=ctrl)
    ev = api.lib().clsparseGetEvent(ctrl.handle)
    assert ev.status == 0 and ev.event
    torch.cuda.synchronize()
    assert float(s) == n


@pytest.mark.parametrize("offs", [(0, 0, 0), (1, 1, 1), (3, 3, 3), (0, 1, 0), (2, 0, 2)], ids=str)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("n", [1, 2, 5, 17, 4095, 4096, 4099, 606_208, 606_213, 3_000_001])
def test_vector_runs(ctrl, dtype, n, offs):
    """Elementwise results and reductions around a vector, a CTA's pass, one
    wave of reduction CTAs and beyond, with operands that start alike or
    differently off a 16-byte boundary: the elementwise ops differ from FP64 by
    the roundings of one multiply and one add, the sums by the bars above."""
    rng = np.random.default_rng(n)
    ox, oy, orr = offs
    px, py = t(rng.uniform(-1, 1, n + ox + 3), dtype), t(rng.uniform(0.5, 1, n + oy + 3), dtype)
    pr = torch.full((n + orr + 3,), 9.0, dtype=dtype, device="cuda")
    x, y, r = px[ox:ox + n], py[oy:oy + n], pr[orr:orr + n]
    xd, yd = x.double().cpu().numpy(), y.double().cpu().numpy()
    a, b = t([0.375], dtype), t([-0.75], dtype)
    p = "D" if dtype == torch.float64 else "S"
    eps = np.finfo(np.float64 if dtype == torch.float64 else np.float32).eps
    for name, args, ref in ((f"cldense{p}axpy", (("s", a), x, y), yd + 0.375 * xd),
                            (f"cldense{p}axpby", (("s", a), x, ("s", b), y), 0.375 * xd - 0.75 * yd),
                            (f"cldense{p}scale", (("s", a), x), 0.375 * xd),
                            (f"cldense{p}div", (x, y), xd / yd)):
        api.blas1(name, r, *args, ctrl=ctrl)
        got = pr.double().cpu().numpy()
        assert np.all(np.abs(got[orr:orr + n] - ref) <= 2 * eps * (np.abs(xd) + np.abs(yd) + np.abs(ref))), name
        assert (got[:orr] == 9).all() and (got[orr + n:] == 9).all(), name
    api.blas1(f"cldense{p}mul", x, x, y, ctrl=ctrl)  # in place
    assert np.all(np.abs(x.double().cpu().numpy() - xd * yd) <= eps * np.abs(xd))
    xd = x.double().cpu().numpy()
    s = torch.zeros(1, dtype=dtype, device="cuda")
    for name, args, ref, scale in ((f"cldense{p}dot", (x, y), (xd * yd).sum(), np.abs(xd * yd).sum()),
                                   (f"cldense{p}nrm1", (x,), np.abs(xd).sum(), np.abs(xd).sum()),
                                   (f"cldense{p}nrm2", (y,), np.linalg.norm(yd), np.linalg.norm(yd))):
        api.blas1(name, ("s", s), *args, ctrl=ctrl)
        assert abs(float(s) - ref) <= TOL[dtype] * scale + 1e-300, name


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("op", ["dot", "axpy"])
def test_operands_aligned_differently_are_not_much_slower(ctrl, op, dtype):
    """Operands that start differently off a 16-byte boundary go element by
    element, with as many bytes in flight: at most 1.35 times the time of
    aligned ones on 20 million elements (the element-by-element form with one
    load in flight per thread took 1.5 to 2.6 times as long)."""
    n = 20_000_000
    x, y, r = (torch.rand(n + 4, dtype=dtype, device="cuda") for _ in range(3))
    a, s = t([0.5], dtype), torch.zeros(1, dtype=dtype, device="cuda")
    p = "D" if dtype == torch.float64 else "S"

    def best(shift):
        xs, ys, rs = x[:n], y[shift:shift + n], r[:n]
        times = []
        for _ in range(12):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(4):
                if op == "dot":
                    api.blas1(f"cldense{p}dot", ("s", s), xs, ys, ctrl=ctrl)
                else:
                    api.blas1(f"cldense{p}axpy", rs, ("s", a), xs, ys, ctrl=ctrl)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    ctrl.enable_async(True)
    aligned, shifted = best(0), best(1)
    ctrl.enable_async(False)
    assert shifted <= 1.35 * aligned, (shifted, aligned)
