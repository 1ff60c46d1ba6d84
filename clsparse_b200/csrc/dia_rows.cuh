// Drop-in banded solves: argument blocks, and the rows of a product in the
// reference's order and rounding, shared by the streaming kernels (dia.cu) and
// the on-chip ones (dia_resident.cu).
#pragma once

#include "device_common.cuh"
#include "dia.h"

namespace clsp {

// In/out block of one drop-in solve.
struct DiaCgState {
    // in: the solver control
    double rel_tol = 0.0, abs_tol = 0.0;
    int max_iters = 0;
    int n_iters_in = 0;  // nIters the control held before the solve (the first stop test sees it)
    int l2 = 0;          // 0: ||.||_1 stop test as the reference, 1: ||.||_2
    int stop_nonfinite = 0;
    // out
    int n_iters = 0;
    int zero_b = 0;      // ||b|| == 0: x = b, nothing else done
    int zero_diag = 0;   // Jacobi with a zero on the main diagonal: nothing written to x
    int status = 0;      // kStatusCurvature / kStatusNonFinite / kStatusBarrierTimeout
    double init_res = 0.0, cur_res = 0.0;
};

// Rows [r0, r1) whose CSR-Adaptive block reduces a row over g > 1 lanes.
struct LaneRange {
    uint32_t r0, r1, g;
};
constexpr int kMaxLaneRanges = 8;

template <typename T>
struct DiaCgArgs {
    using value_type = T;
    DiaMat<T> A;
    // CSR arrays of A, for the rows of lane ranges
    const uint32_t* rp;
    const uint32_t* cols;
    const T* vals;
    LaneRange lanes[kMaxLaneRanges];
    int nlanes;
    // A symmetric bit for bit with its offsets symmetric and no padding
    // diagonals (the kernel's SYM form): the value of lower diagonal d at row
    // i is read as A[j][i] from its upper partner ND - 1 - d at row
    // j = i + off[d], and the lower diagonals are not read at all
    int nd_real;
    int d0;         // index of the main diagonal (Jacobi)
    T* invD;        // Jacobi: 1 / a_ii, formed in the prologue; nullptr: no preconditioner
    const T* b;
    T* x;           // initial guess in, solution out
    T* r;
    T* p[2];        // direction of iteration k in p[k & 1]
    T* q;           // A p
    T* z;           // M r (== r without preconditioner)
    uint32_t n;
    FusedSync sync;
    DiaCgState* st;
};

template <typename T>
struct DiaBicgArgs {
    using value_type = T;
    DiaMat<T> A;
    const uint32_t* rp;
    const uint32_t* cols;
    const T* vals;
    LaneRange lanes[kMaxLaneRanges];
    int nlanes;
    int nd_real;
    int d0;
    T* invD;        // Jacobi: 1 / a_ii, formed in the prologue; nullptr: no preconditioner
    const T* b;
    T* x;
    T* r;
    T* rs;          // r*
    T* p[2];        // direction of iteration k in p[k & 1]
    T* AMp[2];      // A M p_k in AMp[k & 1]
    T* Mp;          // M p_k (== p_k without preconditioner)
    T* s;
    T* Ms;          // M s (== s without preconditioner)
    T* AMs;
    uint32_t n;
    FusedSync sync;
    DiaCgState* st;
};

namespace {

// Separately rounded products and sums (no contraction into FMAs): the
// arithmetic of the reference's kernels as compiled for its CPU runs.
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
using dev::mul_rn;

// sum_d A[d][i] * xf(i + off[d]) in T: products rounded, then summed one by
// one in increasing column order from zero -- the order of a CSR-Adaptive
// STREAM block that reduces each row on one lane
// (src/library/kernels/csrmv_adaptive.cl:312-420); the zeros of entries a
// CSR row does not hold add nothing. Loads are unconditional with
// out-of-matrix columns clamped and their products zero; a mirrored
// diagonal's value is read from the upper one at the column's row.
template <int ND, bool SYM, typename Args, typename XF>
__device__ __forceinline__ typename Args::value_type dia_row_seq(const Args& a, uint32_t i, XF xf) {
    using T = typename Args::value_type;
    const uint32_t n = a.n;
    T av[ND], xv[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int64_t j = static_cast<int64_t>(i) + a.A.off[d];
        const bool in = j >= 0 && j < static_cast<int64_t>(n);
        const uint32_t jc = in ? static_cast<uint32_t>(j) : i;
        T v;
        if (SYM && a.A.off[d] < 0)
            v = __ldg(a.A.vals + static_cast<size_t>(ND - 1 - d) * n + jc);
        else
            v = __ldg(a.A.vals + static_cast<size_t>(d) * n + i);
        const T xj = xf(jc);
        av[d] = in ? v : T(0);
        xv[d] = in ? xj : T(0);
    }
    T s = T(0);
#pragma unroll
    for (int d = 0; d < ND; ++d) s = add_rn(s, mul_rn(av[d], xv[d]));
    return s;
}

// Row i of a CSR-Adaptive STREAM block that reduces a row over g lanes (g a
// power of two): lane l sums the row's products l, l + g, ... one by one,
// then the lanes combine pairwise at distances g/2, ..., 1. A banded row
// holds at most kMaxDiags entries, so lanes from kMaxDiags on hold zero.
template <typename T, typename XF>
__device__ __noinline__ T csr_row_lanes(const uint32_t* rp, const uint32_t* cols, const T* vals, uint32_t i,
                                        uint32_t g, XF xf) {
    T v[kMaxDiags];
#pragma unroll
    for (int l = 0; l < kMaxDiags; ++l) v[l] = T(0);
    g = g > static_cast<uint32_t>(kMaxDiags) ? static_cast<uint32_t>(kMaxDiags) : g;
    const uint32_t b = rp[i], e = rp[i + 1];
    for (uint32_t k = b; k < e; ++k) {
        const uint32_t l = (k - b) & (g - 1);
        v[l] = add_rn(v[l], mul_rn(__ldg(vals + k), xf(cols[k])));
    }
    for (uint32_t off = g / 2; off > 0; off >>= 1)
        for (uint32_t l = 0; l < off; ++l) v[l] = add_rn(v[l], v[l + off]);
    return v[0];
}

// q_i = (A xf)_i in the reference's order for row i.
template <int ND, bool SYM, typename Args, typename XF>
__device__ __forceinline__ typename Args::value_type cg_row(const Args& a, uint32_t i, XF xf) {
    for (int k = 0; k < a.nlanes; ++k)
        if (i >= a.lanes[k].r0 && i < a.lanes[k].r1) return csr_row_lanes(a.rp, a.cols, a.vals, i, a.lanes[k].g, xf);
    return dia_row_seq<ND, SYM>(a, i, xf);
}

}  // namespace
}  // namespace clsp
