// Dense BLAS-1 entry points cldense{S,D,I}* (reference src/library/blas1/*):
// scale, axpy, axpby, add/sub/mul/div, reduce, nrm1, nrm2 and dot.
//
// Every op is one launch over 16-byte vectors (scalar where the operands are
// not aligned alike). Reductions are one launch as well: each CTA stores a partial
// in the control's scratch area and the last CTA to arrive adds the partials in
// index order (deterministic, no second kernel, no spin-wait), applies the final
// operation (sqrt for nrm2) and writes the device scalar. The reference used two
// launches with a CAS-loop atomic for the second (src/library/blas1/reduce.hpp:102-168,
// src/library/kernels/atomic_reduce.cl:95-113).
//
// Scalars alpha/beta are read from device memory by the kernels, as in the
// reference (src/library/kernels/blas1.cl:59-127). The reference's host-side
// shortcuts for alpha == 0 in scale and axpy (cldense-scale.cpp:41-53,
// cldense-axpy.cpp:50-63, both blocking reads of alpha) are evaluated on the
// device instead, with the same results.
#include <algorithm>
#include <cmath>

#include "device_common.cuh"
#include "internal.h"

namespace clsp {
namespace {

constexpr int kThreads = 256;     // elementwise CTAs
constexpr int kRedThreads = 512;  // reduction CTAs

// Vectors of each operand a thread has in flight: 16 bytes each, or (W = 1) single
// elements, where the operands are not aligned alike. (20 M FP32 elements, axpy: 93
// us element by element with one load of each operand in flight, 41 with eight,
// 39 as 16-byte vectors.)
template <int W>
constexpr int kUnroll = W > 1 ? 4 : 8;

enum class Ew : int { Add, Sub, Mul, Div };
enum class Red : int { Plus, Abs, Sqr, Dot };

// A run of elements in 16-byte vectors: `head` elements up to the first
// 16-byte boundary, `vecs` vectors, then the rest. An operand at another
// distance from its boundary leaves everything to the scalar ends (vecs 0; the
// launches below then take the elements one by one as vectors of one).
struct Runs {
    size_t head, vecs;
};

template <typename T>
Runs runs_of(size_t n, const T* a, const T* b, const T* c) {
    const auto off = [](const T* p) { return reinterpret_cast<uintptr_t>(p) & 15u; };
    const size_t o = off(a);
    if ((b && off(b) != o) || (c && off(c) != o) || o % sizeof(T) != 0) return Runs{n, 0};
    const size_t head = ((16 - o) & 15u) / sizeof(T);
    if (head >= n) return Runs{n, 0};
    return Runs{head, (n - head) * sizeof(T) / 16};
}

template <typename T, int WIDTH>
struct alignas(WIDTH * sizeof(T)) Vec {
    static constexpr int W = WIDTH;
    T v[W];
};

uint32_t grid_of(size_t work, size_t per_cta, size_t cap) {
    size_t ctas = (work + per_cta - 1) / per_cta;
    if (ctas > cap) ctas = cap;
    return static_cast<uint32_t>(ctas ? ctas : 1);
}

// r[i] = f(x[i], y[i]) (NX 1: f(x[i], .)): one pass of kUnroll vectors of W
// elements of each operand per thread, all loaded before the first store (r may be
// x or y). Bound by HBM: 3,000,001 FP64 elements (72 MB) take 11.3 us, 6.4
// TB/s, from DRAM either way; the vectors pay where the operands come from L2.
template <typename T, int W, int NX, typename F>
__global__ void __launch_bounds__(kThreads)
    map_kernel(size_t n, Runs runs, T* r, const T* x, const T* y, const T* __restrict__ alpha_p,
               const T* __restrict__ beta_p, F f) {
    const T a = alpha_p ? *alpha_p : T(0);
    const T b = beta_p ? *beta_p : T(0);
    using V = Vec<T, W>;
    constexpr int U = kUnroll<W>;
    const size_t stride = static_cast<size_t>(gridDim.x) * kThreads;
    const size_t tid = static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x;
    const V* xv = reinterpret_cast<const V*>(x + runs.head);
    const V* yv = reinterpret_cast<const V*>(y + runs.head);
    V* rv = reinterpret_cast<V*>(r + runs.head);
    for (size_t i0 = tid; i0 < runs.vecs; i0 += stride * U) {
        V p[U], q[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * stride < runs.vecs) {
                p[u] = xv[i0 + u * stride];
                if constexpr (NX == 2) q[u] = yv[i0 + u * stride];
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i0 + u * stride < runs.vecs) {
                V o;
#pragma unroll
                for (int w = 0; w < V::W; ++w) o.v[w] = f(p[u].v[w], NX == 2 ? q[u].v[w] : T(0), a, b);
                rv[i0 + u * stride] = o;
            }
    }
    const size_t done = runs.head + runs.vecs * V::W;
    for (size_t i = tid; i < runs.head; i += stride) r[i] = f(x[i], NX == 2 ? y[i] : T(0), a, b);
    for (size_t i = done + tid; i < n; i += stride) r[i] = f(x[i], NX == 2 ? y[i] : T(0), a, b);
}

struct ScaleOp {
    template <typename T>
    __device__ __forceinline__ T operator()(T y, T, T a, T) const {
        return (a == T(0)) ? T(0) : y * a;
    }
};
// r = y + alpha * x  (alpha == 0: r = y)
struct AxpyOp {
    template <typename T>
    __device__ __forceinline__ T operator()(T x, T y, T a, T) const {
        return (a == T(0)) ? y : y + a * x;
    }
};
// r = alpha * x + beta * y
struct AxpbyOp {
    template <typename T>
    __device__ __forceinline__ T operator()(T x, T y, T a, T b) const {
        return a * x + b * y;
    }
};
template <Ew OP>
struct EwOp {
    template <typename T>
    __device__ __forceinline__ T operator()(T a, T b, T, T) const {
        if constexpr (OP == Ew::Add) return a + b;
        if constexpr (OP == Ew::Sub) return a - b;
        if constexpr (OP == Ew::Mul) return a * b;
        return a / b;
    }
};

template <typename T, int NX, typename F>
void launch_map(size_t n, T* r, const T* x, const T* y, const T* alpha, const T* beta, F f, clsparseControl c) {
    constexpr int W = 16 / sizeof(T);
    const Runs runs = runs_of<T>(n, r, x, NX == 2 ? y : nullptr);
    const size_t cap = static_cast<size_t>(c->sm_count) * 64;
    if (runs.vecs)
        map_kernel<T, W, NX, F><<<grid_of(runs.vecs, kThreads * kUnroll<W>, cap), kThreads, 0, c->stream>>>(
            n, runs, r, x, y, alpha, beta, f);
    else
        map_kernel<T, 1, NX, F><<<grid_of(n, kThreads * kUnroll<1>, cap), kThreads, 0, c->stream>>>(
            n, Runs{0, n}, r, x, y, alpha, beta, f);
}

// Accumulator type of a reduction: double for floating point, 64-bit integer
// for cldenseIreduce (wraps to 32 bits when stored, as an int sum would).
template <typename T>
struct RedAcc {
    using type = double;
};
template <>
struct RedAcc<int> {
    using type = long long;
};

// Sum over x (and y): kUnroll vectors of each operand in flight per thread, two
// CTAs of 512 threads per SM at most -- every CTA's partial and its arrival on
// one counter are serial work at the end of the call. 3,000,001 FP64 elements:
// the 2-norm (24 MB) 10.5 us with 1184 CTAs of scalar loads, 8.9 here, the dot
// product (48 MB, from DRAM) 12.8 and 12.6; dot, axpy, axpby and 2-norm in a row
// 43.4 -> 40.4 us.
// Element by element (W = 1), 20 M elements, operands aligned differently: FP64 82
// us with one load of each operand in flight on two CTAs per SM, 58 with eight, 57
// with four on three CTAs; FP32 77, 31 and 48.
template <typename T, int W>
constexpr int kRedUnroll = W > 1 || sizeof(T) == 8 ? 4 : 8;
template <typename T, int W>
constexpr int kRedCtas = W > 1 || sizeof(T) == 4 ? 2 : 3;
template <typename T, int W, Red OP>
__global__ void __launch_bounds__(kRedThreads, kRedCtas<T, W>)
    reduce_kernel(size_t n, Runs runs, const T* __restrict__ x, const T* __restrict__ y, T* out,
                  typename RedAcc<T>::type* partials, uint32_t* ticket) {
    using U = typename RedAcc<T>::type;
    using V = Vec<T, W>;
    constexpr int N = kRedUnroll<T, W>;
    U acc[1] = {U(0)};
    auto add = [&](T xi, T yi) {
        const U v = static_cast<U>(xi);
        if constexpr (OP == Red::Plus) acc[0] += v;
        if constexpr (OP == Red::Abs) acc[0] += v < U(0) ? -v : v;
        if constexpr (OP == Red::Sqr) acc[0] += v * v;
        if constexpr (OP == Red::Dot) acc[0] += v * static_cast<U>(yi);
    };
    const size_t stride = static_cast<size_t>(gridDim.x) * kRedThreads;
    const size_t tid = static_cast<size_t>(blockIdx.x) * kRedThreads + threadIdx.x;
    const V* xv = reinterpret_cast<const V*>(x + runs.head);
    const V* yv = reinterpret_cast<const V*>(OP == Red::Dot ? y + runs.head : x);
    for (size_t i0 = tid; i0 < runs.vecs; i0 += stride * N) {
        V p[N], q[N];
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (i0 + u * stride < runs.vecs) {
                p[u] = xv[i0 + u * stride];
                if constexpr (OP == Red::Dot) q[u] = yv[i0 + u * stride];
            }
#pragma unroll
        for (int u = 0; u < N; ++u)
            if (i0 + u * stride < runs.vecs) {
#pragma unroll
                for (int w = 0; w < V::W; ++w) add(p[u].v[w], OP == Red::Dot ? q[u].v[w] : T(0));
            }
    }
    const size_t done = runs.head + runs.vecs * V::W;
    for (size_t i = tid; i < runs.head; i += stride) add(x[i], OP == Red::Dot ? y[i] : T(0));
    for (size_t i = done + tid; i < n; i += stride) add(x[i], OP == Red::Dot ? y[i] : T(0));
    U tot[1];
    if (dev::grid_reduce_last<1, U>(acc, partials, ticket, tot)) {
        if (threadIdx.x == 0) {
            if constexpr (OP == Red::Sqr) {
                *out = static_cast<T>(sqrt(static_cast<double>(tot[0])));
            } else {
                *out = static_cast<T>(tot[0]);
            }
        }
    }
}

bool sizes_ok(const cldenseVector* a, const cldenseVector* b) {
    return a->num_values == b->num_values;
}

template <typename T>
clsparseStatus do_scale(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* y,
                        clsparseControl c) {
    clsparseStatus st = check_entry(c);
    if (st != clsparseSuccess) return st;
    if (!r || !alpha || !y) return clsparseInvalidValue;
    if (!sizes_ok(r, y)) return clsparseInvalidSize;
    const size_t n = r->num_values;
    if (n == 0) return clsparseSuccess;
    DeviceGuard g(c->device);
    launch_map<T, 1>(n, dev_ptr<T>(r->values, r->off_values), dev_ptr<const T>(y->values, y->off_values),
                     static_cast<const T*>(nullptr), dev_ptr<const T>(alpha->value, alpha->off_value),
                     static_cast<const T*>(nullptr), ScaleOp{}, c);
    return finish_call(c);
}

template <typename T>
clsparseStatus do_axpy(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                       const cldenseVector* y, clsparseControl c) {
    clsparseStatus st = check_entry(c);
    if (st != clsparseSuccess) return st;
    if (!r || !alpha || !x || !y) return clsparseInvalidValue;
    if (!sizes_ok(r, y) || !sizes_ok(r, x)) return clsparseInvalidSize;
    const size_t n = r->num_values;
    if (n == 0) return clsparseSuccess;
    DeviceGuard g(c->device);
    launch_map<T, 2>(n, dev_ptr<T>(r->values, r->off_values), dev_ptr<const T>(x->values, x->off_values),
                     dev_ptr<const T>(y->values, y->off_values), dev_ptr<const T>(alpha->value, alpha->off_value),
                     static_cast<const T*>(nullptr), AxpyOp{}, c);
    return finish_call(c);
}

template <typename T>
clsparseStatus do_axpby(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                        const clsparseScalar* beta, const cldenseVector* y, clsparseControl c) {
    clsparseStatus st = check_entry(c);
    if (st != clsparseSuccess) return st;
    if (!r || !alpha || !x || !beta || !y) return clsparseInvalidValue;
    if (!sizes_ok(r, y) || !sizes_ok(r, x)) return clsparseInvalidSize;
    const size_t n = r->num_values;
    if (n == 0) return clsparseSuccess;
    DeviceGuard g(c->device);
    launch_map<T, 2>(n, dev_ptr<T>(r->values, r->off_values), dev_ptr<const T>(x->values, x->off_values),
                     dev_ptr<const T>(y->values, y->off_values), dev_ptr<const T>(alpha->value, alpha->off_value),
                     dev_ptr<const T>(beta->value, beta->off_value), AxpbyOp{}, c);
    return finish_call(c);
}

template <typename T, Ew OP>
clsparseStatus do_ew(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                     clsparseControl c) {
    clsparseStatus st = check_entry(c);
    if (st != clsparseSuccess) return st;
    if (!r || !x || !y) return clsparseInvalidValue;
    if (!sizes_ok(x, y) || !sizes_ok(r, x)) return clsparseInvalidSize;
    const size_t n = x->num_values;
    if (n == 0) return clsparseSuccess;
    DeviceGuard g(c->device);
    launch_map<T, 2>(n, dev_ptr<T>(r->values, r->off_values), dev_ptr<const T>(x->values, x->off_values),
                     dev_ptr<const T>(y->values, y->off_values), static_cast<const T*>(nullptr),
                     static_cast<const T*>(nullptr), EwOp<OP>{}, c);
    return finish_call(c);
}

template <typename T, Red OP>
clsparseStatus do_reduce(clsparseScalar* s, const cldenseVector* x, const cldenseVector* y,
                         clsparseControl c) {
    using U = typename RedAcc<T>::type;
    clsparseStatus st = check_entry(c);
    if (st != clsparseSuccess) return st;
    if (!s || !x || (OP == Red::Dot && !y)) return clsparseInvalidValue;
    if (OP == Red::Dot && !sizes_ok(x, y)) return clsparseInvalidSize;
    const size_t n = x->num_values;
    DeviceGuard g(c->device);
    U* partials = static_cast<U*>(c->reduce_scratch.ptr);
    uint32_t* ticket = reinterpret_cast<uint32_t*>(static_cast<char*>(c->reduce_scratch.ptr) +
                                                   sizeof(double) * 4 * kMaxReduceCtas);
    const T* yp = (OP == Red::Dot) ? dev_ptr<const T>(y->values, y->off_values) : nullptr;
    const T* xp = dev_ptr<const T>(x->values, x->off_values);
    const Runs runs = runs_of<T>(n, xp, yp, static_cast<const T*>(nullptr));
    const size_t sms = static_cast<size_t>(c->sm_count);
    const auto cap = [&](int per_sm) { return std::min<size_t>(sms * per_sm, kMaxReduceCtas); };
    constexpr int W = 16 / sizeof(T);
    T* out = dev_ptr<T>(s->value, s->off_value);
    if (runs.vecs)
        reduce_kernel<T, W, OP><<<grid_of(runs.vecs, kRedThreads * kRedUnroll<T, W>, cap(kRedCtas<T, W>)), kRedThreads, 0, c->stream>>>(
            n, runs, xp, yp, out, partials, ticket);
    else
        reduce_kernel<T, 1, OP><<<grid_of(n, kRedThreads * kRedUnroll<T, 1>, cap(kRedCtas<T, 1>)), kRedThreads, 0, c->stream>>>(
            n, Runs{0, n}, xp, yp, out, partials, ticket);
    return finish_call(c);
}

}  // namespace
}  // namespace clsp

using namespace clsp;

extern "C" {

clsparseStatus cldenseSscale(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* y,
                             const clsparseControl control) {
    return do_scale<float>(r, alpha, y, control);
}
clsparseStatus cldenseDscale(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* y,
                             const clsparseControl control) {
    return do_scale<double>(r, alpha, y, control);
}
clsparseStatus cldenseSaxpy(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                            const cldenseVector* y, const clsparseControl control) {
    return do_axpy<float>(r, alpha, x, y, control);
}
clsparseStatus cldenseDaxpy(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                            const cldenseVector* y, const clsparseControl control) {
    return do_axpy<double>(r, alpha, x, y, control);
}
clsparseStatus cldenseSaxpby(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                             const clsparseScalar* beta, const cldenseVector* y,
                             const clsparseControl control) {
    return do_axpby<float>(r, alpha, x, beta, y, control);
}
clsparseStatus cldenseDaxpby(cldenseVector* r, const clsparseScalar* alpha, const cldenseVector* x,
                             const clsparseScalar* beta, const cldenseVector* y,
                             const clsparseControl control) {
    return do_axpby<double>(r, alpha, x, beta, y, control);
}
clsparseStatus cldenseIreduce(clsparseScalar* s, const cldenseVector* x,
                              const clsparseControl control) {
    return do_reduce<int, Red::Plus>(s, x, nullptr, control);
}
clsparseStatus cldenseSreduce(clsparseScalar* s, const cldenseVector* x,
                              const clsparseControl control) {
    return do_reduce<float, Red::Plus>(s, x, nullptr, control);
}
clsparseStatus cldenseDreduce(clsparseScalar* s, const cldenseVector* x,
                              const clsparseControl control) {
    return do_reduce<double, Red::Plus>(s, x, nullptr, control);
}
clsparseStatus cldenseSnrm1(clsparseScalar* s, const cldenseVector* x, const clsparseControl control) {
    return do_reduce<float, Red::Abs>(s, x, nullptr, control);
}
clsparseStatus cldenseDnrm1(clsparseScalar* s, const cldenseVector* x, const clsparseControl control) {
    return do_reduce<double, Red::Abs>(s, x, nullptr, control);
}
clsparseStatus cldenseSnrm2(clsparseScalar* s, const cldenseVector* x, const clsparseControl control) {
    return do_reduce<float, Red::Sqr>(s, x, nullptr, control);
}
clsparseStatus cldenseDnrm2(clsparseScalar* s, const cldenseVector* x, const clsparseControl control) {
    return do_reduce<double, Red::Sqr>(s, x, nullptr, control);
}
clsparseStatus cldenseSdot(clsparseScalar* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_reduce<float, Red::Dot>(r, x, y, control);
}
clsparseStatus cldenseDdot(clsparseScalar* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_reduce<double, Red::Dot>(r, x, y, control);
}
clsparseStatus cldenseSadd(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<float, Ew::Add>(r, x, y, control);
}
clsparseStatus cldenseDadd(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<double, Ew::Add>(r, x, y, control);
}
clsparseStatus cldenseSsub(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<float, Ew::Sub>(r, x, y, control);
}
clsparseStatus cldenseDsub(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<double, Ew::Sub>(r, x, y, control);
}
clsparseStatus cldenseSmul(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<float, Ew::Mul>(r, x, y, control);
}
clsparseStatus cldenseDmul(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<double, Ew::Mul>(r, x, y, control);
}
clsparseStatus cldenseSdiv(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<float, Ew::Div>(r, x, y, control);
}
clsparseStatus cldenseDdiv(cldenseVector* r, const cldenseVector* x, const cldenseVector* y,
                           const clsparseControl control) {
    return do_ew<double, Ew::Div>(r, x, y, control);
}

}  // extern "C"
