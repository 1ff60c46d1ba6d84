// Sparse x dense product C = alpha * A * B + beta * C (clsparseScsrmm /
// clsparseDcsrmm) for sm_100a.
//
// The reference runs it as a batched SpMV: one csrmv pass per column of C
// (src/library/blas3/clsparse-csrmm.hpp:28-118, kernel
// src/library/kernels/csrmm_general.cl:60-167), re-reading A once per
// column. Here A is read once per tile of columns: a group of G lanes owns a
// row of A and a tile of L vectors of VW consecutive columns. The lanes load
// G nonzeros of the row at a time (coalesced); S = G / L of them are in work
// at once, lane s * L + v multiplying nonzero s by vector v of its row of B
// (one 16-byte load where the layout allows), four such steps' loads in
// flight; the S partial sums of a vector are added by shuffles at the end of
// the row. Short rows have a form of their own (SHORT). alpha multiplies each product and beta == 0 overwrites C without
// reading it, as in the reference (csrmm_general.cl:96-126).
//
// What bounds it: the gathered rows of B (a random row per nonzero, from L2),
// then the loads in flight. Measured, 200,003 rows of log-normal lengths
// (5.0 M nonzeros, uniform columns), FP32, 40 columns: 934 us with one lane
// per column and one dependent load per nonzero (40 columns were a tile of 32
// and one of 8), 237 us in this form (3.4 TB/s of gathered rows).
//
// Layouts: the reference indexes B and C row-major through lead_dim whatever
// their `major` field says; here row-major is the same, and column-major
// matrices are indexed as column-major.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "device_common.cuh"
#include "internal.h"

namespace clsp {
namespace {

// Two warps a CTA: a CTA's slots come free when its longest row is done, and row
// lengths differ widely (284 us with 256 threads on the matrix above, 237 with 64).
constexpr int kThreads = 64;

// Rows of fewer than kShortRow nonzeros on average, where the columns go one by
// one or all in one vector: four steps at once are mostly empty ones there, and a
// CTA of two warps is more to start than its few rows are work, so that as many
// steps are in flight as are left (4, 2, 1), in eight warps a CTA and a grid of at
// most kShortCtas per SM. 300^2 five-point, row-major, device time of the form
// above / this one: FP64, 1 column 40 / 8.5 us, 2 columns 39 / 9.4, 65 columns 144 /
// 113; FP32, 1 column 28 / 6.0, 33 columns 64 / 52. Wider vectors (32, 40, 64
// columns) measured the same in both, rows of 8 to 40 nonzeros slower here; five rows
// of 20,000 among 60,000 short ones, 33 columns, take 3.0 ms here, 2.3 above and 4.6
// with a lane per column. (No look at a meta: this call takes matrices whose meta was
// never set.)
constexpr uint32_t kShortRow = 8;
constexpr int kThreadsShort = 256;
constexpr uint32_t kShortCtas = 32;

// Element (r, c) of a dense matrix is at r * rs + c * cs.
struct DenseView {
    size_t rs, cs;
};

template <typename T, int VW>
struct alignas(VW * sizeof(T)) Vec {
    T v[VW];
};

constexpr int kSteps = 4;  // steps of S nonzeros whose loads of B are in flight

// VW > 1: cs == 1 on both matrices, rows VW-aligned and ncols a multiple of VW.
template <typename T, int VW, int G, bool SHORT>
__global__ void __launch_bounds__(SHORT ? kThreadsShort : kThreads)
    csrmm_kernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ cols, const T* __restrict__ vals,
                 uint32_t nrows, uint32_t nvec, uint32_t L, uint32_t tiles, const T* __restrict__ alpha_p,
                 const T* __restrict__ beta_p, const T* __restrict__ B, DenseView bv, T* __restrict__ C,
                 DenseView cv) {
    using V = Vec<T, VW>;
    constexpr uint32_t NT = SHORT ? kThreadsShort : kThreads;
    if constexpr (SHORT && G == 1) L = 1;
    const T alpha = *alpha_p, beta = *beta_p;
    const uint32_t lane = threadIdx.x & (G - 1);
    // Groups of one warp may be at different rows and iterations: shuffles
    // name only this group's lanes.
    const unsigned mask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << ((threadIdx.x & 31u) & ~(G - 1u)));
    const uint32_t S = G / L;  // >= 1: L <= G
    const uint32_t slot = lane / L, v = lane - slot * L;
    const uint64_t group = (static_cast<uint64_t>(blockIdx.x) * NT + threadIdx.x) / G;
    const uint64_t ngroups = static_cast<uint64_t>(gridDim.x) * NT / G;
    const uint64_t work = static_cast<uint64_t>(nrows) * tiles;
    for (uint64_t w = group; w < work; w += ngroups) {
        // (short rows: one tile, the usual case, without the division)
        const bool one = SHORT && tiles == 1;
        const uint32_t row = static_cast<uint32_t>(one ? w : w / tiles);
        const uint32_t vec = one ? v : static_cast<uint32_t>(w - static_cast<uint64_t>(row) * tiles) * L + v;
        const bool on = slot < S && vec < nvec;
        const T* Bc = B + static_cast<size_t>(vec) * VW * bv.cs;
        const uint32_t rb = dev::ld_ro(rp + row), re = dev::ld_ro(rp + row + 1);
        V acc;
#pragma unroll
        for (int c = 0; c < VW; ++c) acc.v[c] = T(0);
        auto load = [&](uint32_t k, V& b) {
            const T* p = Bc + static_cast<size_t>(k) * bv.rs;
            if constexpr (VW * sizeof(T) == 16) {
                const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
                memcpy(&b, &q, 16);
            } else if constexpr (VW * sizeof(T) == 8) {
                const uint2 q = __ldg(reinterpret_cast<const uint2*>(p));
                memcpy(&b, &q, 8);
            } else {
                b.v[0] = dev::ld_ro(p);
            }
        };
        auto add = [&](T a, const V& b) {
#pragma unroll
            for (int c = 0; c < VW; ++c) acc.v[c] = dev::fma_rn(a, b.v[c], acc.v[c]);
        };
        for (uint32_t base = rb; base < re; base += G) {
            uint32_t kc = 0;
            T kv = T(0);
            if (base + lane < re) {
                kc = dev::ld_stream(cols + base + lane);
                kv = alpha * dev::ld_stream(vals + base + lane);
            }
            if constexpr (SHORT && G == 1) {
                V b;
                load(kc, b);
                add(kv, b);
                continue;
            }
            const uint32_t cnt = min(static_cast<uint32_t>(G), re - base);
            if constexpr (SHORT) {
                // N steps, all of their nonzeros there
                uint32_t j = 0;
                auto steps = [&](auto n) {
                    constexpr int N = decltype(n)::value;
                    V b[N];
                    T a[N];
#pragma unroll
                    for (int u = 0; u < N; ++u) {
                        const uint32_t e = j + u * S + slot;
                        const uint32_t k = __shfl_sync(mask, kc, e & (G - 1), G);
                        a[u] = __shfl_sync(mask, kv, e & (G - 1), G);
                        if (on) load(k, b[u]);
                    }
                    if (on) {
#pragma unroll
                        for (int u = 0; u < N; ++u) add(a[u], b[u]);
                    }
                    j += N * S;
                };
                while (j + 4 * S <= cnt) steps(std::integral_constant<int, 4>{});
                if (j + 2 * S <= cnt) steps(std::integral_constant<int, 2>{});
                for (; j < cnt; j += S) {
                    const uint32_t e = j + slot;
                    const uint32_t k = __shfl_sync(mask, kc, e & (G - 1), G);
                    const T a = __shfl_sync(mask, kv, e & (G - 1), G);
                    if (on && e < cnt) {
                        V b;
                        load(k, b);
                        add(a, b);
                    }
                }
            } else {
                for (uint32_t j = 0; j < cnt; j += S * kSteps) {
                    V b[kSteps];
                    T a[kSteps];
#pragma unroll
                    for (int u = 0; u < kSteps; ++u) {
                        const uint32_t e = j + u * S + slot;
                        const uint32_t k = __shfl_sync(mask, kc, e & (G - 1), G);
                        a[u] = __shfl_sync(mask, kv, e & (G - 1), G);
                        if (on && e < cnt) {
                            load(k, b[u]);
                        } else {
                            a[u] = T(0);
#pragma unroll
                            for (int c = 0; c < VW; ++c) b[u].v[c] = T(0);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kSteps; ++u)
#pragma unroll
                        for (int c = 0; c < VW; ++c) acc.v[c] = dev::fma_rn(a[u], b[u].v[c], acc.v[c]);
                }
            }
        }
        // add the slots' sums onto slot 0: halves, the middle one of an odd count waiting
        for (uint32_t left = S; left > 1;) {
            const uint32_t half = (left + 1) / 2;
            const uint32_t from = min(lane + half * L, static_cast<uint32_t>(G - 1));
#pragma unroll
            for (int c = 0; c < VW; ++c) {
                const T o = __shfl_sync(mask, acc.v[c], from, G);
                if (slot + half < left) acc.v[c] += o;
            }
            left = half;
        }
        if (on && slot == 0) {
            T* dst = C + static_cast<size_t>(row) * cv.rs + static_cast<size_t>(vec) * VW * cv.cs;
            V* d = reinterpret_cast<V*>(dst);
            if (beta != T(0)) {
                const V old = *d;
#pragma unroll
                for (int c = 0; c < VW; ++c)
                    acc.v[c] = beta == T(1) ? acc.v[c] + old.v[c] : acc.v[c] + beta * old.v[c];
            }
            *d = acc;
        }
    }
}

struct MmArgs {
    const uint32_t* rp;
    const uint32_t* cols;
    uint32_t nrows, ncols, nnz;
    DenseView bv, cv;
    uint32_t sms;
    cudaStream_t stream;
};

template <typename T, int VW>
void launch_csrmm(const MmArgs& m, const T* vals, const T* alpha, const T* beta, const T* B, T* C) {
    const uint32_t nvec = m.ncols / VW;
    const uint32_t tiles = (nvec + 31) / 32;
    const uint32_t per_row = m.nnz / std::max(1u, m.nrows);
    // Tiles of equal width; for short rows full ones where no two slots fit side
    // by side (aligned, the last one narrow).
    uint32_t L = (nvec + tiles - 1) / tiles;
    const bool rows_short = per_row < kShortRow && (VW == 1 || L == 1);
    if (rows_short && tiles > 1 && L > 16) L = 32;
    // Lanes per row: enough for about a quarter of an average row's nonzeros
    // at a time (four steps in flight then cover the row); at least L, and two
    // where one vector holds several columns of short rows.
    const uint64_t want = std::min<uint64_t>(32, static_cast<uint64_t>(L) * std::max(1u, per_row / 4u));
    uint32_t G = 1;
    while (G < want || G < L || (rows_short && VW > 1 && G < 2)) G *= 2;
    const uint64_t groups = static_cast<uint64_t>(m.nrows) * tiles;
    const uint32_t threads = rows_short ? kThreadsShort : kThreads;
    const uint64_t cap = rows_short ? static_cast<uint64_t>(m.sms) * kShortCtas : 0x7fffffffull;
    const uint64_t ctas = std::min(std::max<uint64_t>((groups * G + threads - 1) / threads, 1), cap);
    auto launch = [&](auto kernel) {
        kernel<<<static_cast<uint32_t>(ctas), threads, 0, m.stream>>>(m.rp, m.cols, vals, m.nrows, nvec, L, tiles, alpha,
                                                                      beta, B, m.bv, C, m.cv);
    };
#define CLSP_MM(GW) \
    rows_short ? launch(csrmm_kernel<T, VW, GW, true>) : launch(csrmm_kernel<T, VW, GW, false>)
    switch (G) {
        case 1: CLSP_MM(1); break;
        case 2: CLSP_MM(2); break;
        case 4: CLSP_MM(4); break;
        case 8: CLSP_MM(8); break;
        case 16: CLSP_MM(16); break;
        default: CLSP_MM(32); break;
    }
#undef CLSP_MM
}

template <typename T>
clsparseStatus csrmm_entry(const clsparseScalar* alpha, const clsparseCsrMatrix* A, const cldenseMatrix* B,
                           const clsparseScalar* beta, cldenseMatrix* C, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!alpha || !A || !B || !beta || !C) return clsparseInvalidValue;
    if (B->num_rows < A->num_cols || C->num_rows < A->num_rows || B->num_cols < C->num_cols) return clsparseInvalidSize;
    const bool bcm = B->major == columnMajor, ccm = C->major == columnMajor;
    if (B->lead_dim < (bcm ? B->num_rows : B->num_cols) || C->lead_dim < (ccm ? C->num_rows : C->num_cols))
        return clsparseInvalidSize;
    if (A->num_rows == 0 || C->num_cols == 0) return clsparseSuccess;
    if (!alpha->value || !beta->value || !B->values || !C->values || !A->row_pointer ||
        (A->num_nonzeros > 0 && (!A->values || !A->col_indices)))
        return clsparseInvalidMemObject;
    DeviceGuard g(control->device);
    const uint32_t ncols = C->num_cols;
    const T* va = dev_ptr<const T>(A->values, A->off_values);
    const T* a = dev_ptr<const T>(alpha->value, alpha->off_value);
    const T* b = dev_ptr<const T>(beta->value, beta->off_value);
    const T* Bp = dev_ptr<const T>(B->values, B->off_values);
    T* Cp = dev_ptr<T>(C->values, C->off_values);
    MmArgs m;
    m.rp = dev_ptr<const uint32_t>(A->row_pointer, A->off_row_pointer);
    m.cols = dev_ptr<const uint32_t>(A->col_indices, A->off_col_indices);
    m.nrows = A->num_rows;
    m.ncols = ncols;
    m.nnz = A->num_nonzeros;
    m.bv = bcm ? DenseView{1, B->lead_dim} : DenseView{B->lead_dim, 1};
    m.cv = ccm ? DenseView{1, C->lead_dim} : DenseView{C->lead_dim, 1};
    m.sms = static_cast<uint32_t>(std::max(1, control->sm_count));
    m.stream = control->stream;
    // The widest vector (up to 16 bytes) that both row-major matrices' rows
    // start on and that divides the column count (no vector then crosses the
    // last column, so nothing outside the matrices is touched).
    auto fits = [&](size_t vw) {
        const size_t bytes = vw * sizeof(T);
        return !bcm && !ccm && ncols % vw == 0 && B->lead_dim % vw == 0 && C->lead_dim % vw == 0 &&
               reinterpret_cast<uintptr_t>(Bp) % bytes == 0 && reinterpret_cast<uintptr_t>(Cp) % bytes == 0;
    };
    constexpr int kWide = 16 / sizeof(T);
    if (fits(kWide))
        launch_csrmm<T, kWide>(m, va, a, b, Bp, Cp);
    else if (sizeof(T) == 4 && fits(2))
        launch_csrmm<T, 2>(m, va, a, b, Bp, Cp);
    else
        launch_csrmm<T, 1>(m, va, a, b, Bp, Cp);
    if (cudaGetLastError() != cudaSuccess) return clsparseInvalidKernelExecution;
    return finish_call(control);
}

}  // namespace
}  // namespace clsp

extern "C" {

clsparseStatus clsparseScsrmm(const clsparseScalar* alpha, const clsparseCsrMatrix* sparseMatA,
                              const cldenseMatrix* denseMatB, const clsparseScalar* beta, cldenseMatrix* denseMatC,
                              const clsparseControl control) {
    clsp::TraceRange trace_("clsparseScsrmm");
    return clsp::csrmm_entry<float>(alpha, sparseMatA, denseMatB, beta, denseMatC, control);
}

clsparseStatus clsparseDcsrmm(const clsparseScalar* alpha, const clsparseCsrMatrix* sparseMatA,
                              const cldenseMatrix* denseMatB, const clsparseScalar* beta, cldenseMatrix* denseMatC,
                              const clsparseControl control) {
    clsp::TraceRange trace_("clsparseDcsrmm");
    return clsp::csrmm_entry<double>(alpha, sparseMatA, denseMatB, beta, denseMatC, control);
}

}  // extern "C"
