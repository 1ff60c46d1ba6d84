// Format conversions (reference src/library/transform/): clsparse{S,D}coo2csr,
// csr2coo, csr2dense and dense2csr; and the COO SpMV clsparse{S,D}coomv, which
// the reference declares (src/include/clSPARSE.h:1106-1132) but never defines.
//
// * coo2csr (clsparse-coo2csr.cpp:20-100): the COO must be sorted by row
//   (the reference's precondition); columns and values are copied and
//   row_pointer[r] is the first position whose row index is >= r, written where
//   the row index steps (no atomics, no scan; empty rows come out right,
//   which the reference's reduce-by-key of present keys does not guarantee).
// * csr2coo (clsparse-csr2coo.cpp): columns and values copied, each row's
//   positions get its row index (a running maximum over a CTA's positions).
// * csr2dense (clsparse-csr2dense.cpp): the dense matrix is zeroed, then every
//   entry is written at its (row, column); duplicates: the last one wins.
// * dense2csr (clsparse-dense2csr.cpp): every non-zero of the dense matrix,
//   row by row and column by column; counts per row (warp ballots), an
//   exclusive scan into the row pointer, then an ordered per-row compaction.
//   The CSR buffers must hold the non-zeros (at most rows x columns); the
//   struct's sizes are set.
// Dense matrices: row-major as the reference reads them, column-major
// honoured, lead_dim as given (0 means packed).
#include "device_common.cuh"
#include "scan.cuh"
#include "internal.h"

namespace clsp {
namespace {

constexpr int kThreads = 256;

uint32_t grid_for(uint64_t work, int sms) {
    uint64_t g = (work + kThreads - 1) / kThreads;
    const uint64_t cap = static_cast<uint64_t>(sms) * 32;
    if (g > cap) g = cap;
    return static_cast<uint32_t>(g ? g : 1);
}

struct Dense {
    size_t ld;
    bool cm;
    __device__ __forceinline__ size_t at(size_t r, size_t c) const { return cm ? c * ld + r : r * ld + c; }
};

Dense dense_view(const cldenseMatrix* D) {
    const bool cm = D->major == columnMajor;
    size_t ld = D->lead_dim;
    if (ld == 0) ld = cm ? D->num_rows : D->num_cols;
    return Dense{ld, cm};
}

bool dense_ok(const cldenseMatrix* D) {
    const Dense v = dense_view(D);
    return v.ld >= (v.cm ? D->num_rows : D->num_cols);
}

// ---- COO <-> CSR in one pass over the nonzeros: every CTA copies a run of
// kChunk columns and values (16-byte loads and stores) and turns the run's row
// indices into row pointers or the other way round. Bound by HBM (one read of
// the input, one write of the output). Measured, 10.0 M FP64 nonzeros, both
// directions: 159 us as two copies and a kernel each (a binary search per row,
// 22 us; a warp per row, 31 us), 109 us here (5.2 TB/s; 128 with the columns and
// values copied in loops instead of all loaded before the first store).
constexpr uint32_t kChunk = 2048;

// A run's columns and values on their way through the registers: load() starts
// every 16-byte load of a full run whose arrays lie on 16 bytes, store() writes
// them out; other runs are copied element by element in store().
template <typename T>
struct Run {
    static constexpr uint32_t NC = kChunk * 4 / 16 / kThreads, NV = kChunk * sizeof(T) / 16 / kThreads;
    uint4 c[NC], v[NV];
    bool wide;
    __device__ __forceinline__ void load(const uint32_t* __restrict__ ci, const T* __restrict__ vi,
                                         const uint32_t* co, const T* vo, uint32_t b, uint32_t e) {
        wide = e - b == kChunk && ((reinterpret_cast<uintptr_t>(ci) | reinterpret_cast<uintptr_t>(vi) |
                                    reinterpret_cast<uintptr_t>(co) | reinterpret_cast<uintptr_t>(vo)) & 15u) == 0;
        if (!wide) return;
        const uint4* cs = reinterpret_cast<const uint4*>(ci + b);
        const uint4* vs = reinterpret_cast<const uint4*>(vi + b);
#pragma unroll
        for (uint32_t u = 0; u < NC; ++u) c[u] = __ldcs(cs + u * kThreads + threadIdx.x);
#pragma unroll
        for (uint32_t u = 0; u < NV; ++u) v[u] = __ldcs(vs + u * kThreads + threadIdx.x);
    }
    __device__ __forceinline__ void store(const uint32_t* __restrict__ ci, const T* __restrict__ vi,
                                          uint32_t* __restrict__ co, T* __restrict__ vo, uint32_t b, uint32_t e) {
        if (wide) {
            uint4* cd = reinterpret_cast<uint4*>(co + b);
            uint4* vd = reinterpret_cast<uint4*>(vo + b);
#pragma unroll
            for (uint32_t u = 0; u < NC; ++u) __stcs(cd + u * kThreads + threadIdx.x, c[u]);
#pragma unroll
            for (uint32_t u = 0; u < NV; ++u) __stcs(vd + u * kThreads + threadIdx.x, v[u]);
        } else {
            for (uint32_t i = b + threadIdx.x; i < e; i += kThreads) {
                co[i] = ci[i];
                vo[i] = vi[i];
            }
        }
    }
};

// First position of ri[0, n) whose row index is >= r.
__device__ __forceinline__ uint32_t first_at_least(const uint32_t* __restrict__ ri, uint32_t n, uint64_t r) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (__ldg(ri + mid) < r)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// rp[r] = first position whose row index is >= r (sorted row indices). The
// first `runs` CTAs copy a run each, and the thread of position k, whose row is
// above its predecessor's, has the pointers in between to write; the last
// position's also those behind its row. More than kShortGap of them are written
// by its warp, a lane each. Whole chunks [c kGapRows, (c + 1) kGapRows) without a step,
// as long runs of empty rows hold, are left to the CTAs before the runs, a
// thread per chunk to look it up and a warp to write it: the pointers are
// spread over the device however the nonzeros lie. Both ends of the rule
// measured, coo2csr with its wait: 10 M rows with 3000 nonzeros 644 us with every
// gap written by the CTA of the position behind it, 39 in this form; 400,000 rows with
// 10 M nonzeros 69 and 71.
constexpr uint32_t kShortGap = 16;
constexpr uint32_t kGapRows = 32;
constexpr uint32_t kGapCta = kGapRows * kThreads;  // row pointers of one gap CTA

__device__ __forceinline__ void fill_gap_chunks(const uint32_t* __restrict__ ri, uint32_t nnz, uint32_t nrows,
                                                uint32_t cta, uint32_t* __restrict__ rp) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t w0 = static_cast<uint64_t>(cta) * kGapCta + (threadIdx.x - lane) * kGapRows;  // the warp's first
    const uint64_t r0 = w0 + lane * kGapRows;
    uint32_t at = 0;
    bool empty = false;
    if (r0 + kGapRows <= nrows) {
        // no step inside: the row index behind the chunk's start is no smaller
        // than the chunk's last row
        at = first_at_least(ri, nnz, r0);
        empty = at == nnz || __ldg(ri + at) >= r0 + kGapRows - 1;
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, empty); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const uint32_t v = __shfl_sync(0xffffffffu, at, l);
        uint32_t* const out = rp + w0 + l * kGapRows;
        out[lane] = v;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    coo_to_csr_kernel(const uint32_t* __restrict__ ri, const uint32_t* __restrict__ ci, const T* __restrict__ vi,
                      uint32_t nnz, uint32_t nrows, uint32_t gap_ctas, uint32_t* __restrict__ rp,
                      uint32_t* __restrict__ co, T* __restrict__ vo) {
    constexpr uint32_t PER = kChunk / kThreads;
    if (blockIdx.x < gap_ctas) {  // (first: their look-ups are chains of loads)
        fill_gap_chunks(ri, nnz, nrows, blockIdx.x, rp);
        return;
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t b = (blockIdx.x - gap_ctas) * kChunk;
    const uint32_t e = static_cast<uint32_t>(min(static_cast<uint64_t>(nnz), static_cast<uint64_t>(b) + kChunk));
    uint32_t row[PER], prev[PER];
#pragma unroll
    for (uint32_t u = 0; u < PER; ++u) {
        const uint32_t k = b + u * kThreads + threadIdx.x;
        row[u] = k < e ? __ldcs(ri + k) : 0;
        prev[u] = k < e && k > 0 ? __ldg(ri + k - 1) : 0;
    }
    Run<T> run;
    run.load(ci, vi, co, vo, b, e);
    run.store(ci, vi, co, vo, b, e);
    // the pointers [from, to) of position k, and the last one's [row + 1, nrows)
    auto from_of = [&](uint32_t u, uint32_t k) { return k > 0 ? (prev[u] < nrows ? prev[u] + 1 : nrows) : 0; };
    auto to_of = [&](uint32_t u) { return row[u] < nrows ? row[u] + 1 : nrows; };
    bool any_long = e == nnz;
#pragma unroll
    for (uint32_t u = 0; u < PER; ++u) {
        const uint32_t k = b + u * kThreads + threadIdx.x;
        if (k >= e) continue;
        const uint32_t from = from_of(u, k), to = to_of(u);
        if (to > from && to - from > kShortGap)
            any_long = true;
        else
            for (uint32_t r = from; r < to; ++r) rp[r] = k;
    }
    if (!__any_sync(0xffffffffu, any_long)) return;
    // long ones, by every lane of the warp, but for the whole chunks inside
    auto fill = [&](bool lng, uint32_t from, uint32_t to, uint32_t at) {
        for (unsigned todo = __ballot_sync(0xffffffffu, lng); todo;) {
            // four gaps at a time (the last one again where fewer are left)
            int l = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                l = todo ? __ffs(todo) - 1 : l;
                todo &= todo - 1;
                const uint32_t f = __shfl_sync(0xffffffffu, from, l), t = __shfl_sync(0xffffffffu, to, l);
                const uint32_t v = __shfl_sync(0xffffffffu, at, l);
                // chunks [c0, c1) stay out: two pieces of less than a chunk each
                const uint64_t c0 = (static_cast<uint64_t>(f) + kGapRows - 1) / kGapRows * kGapRows;
                const uint64_t c1 = t / kGapRows * kGapRows;
                const uint64_t first = static_cast<uint64_t>(f) + lane, second = (c0 < c1 ? c1 : f + 32ull) + lane;
                if (first < (c0 < c1 ? c0 : t)) rp[first] = v;
                if (second < t) rp[second] = v;
            }
        }
    };
#pragma unroll 1
    for (uint32_t u = 0; u < PER; ++u) {  // (not unrolled, the rows read again: no code or registers more for runs without gaps)
        const uint32_t k = b + u * kThreads + threadIdx.x;
        const bool on = k < e;
        const uint32_t rk = on ? __ldg(ri + k) : 0, pk = on && k > 0 ? __ldg(ri + k - 1) : 0;
        const uint32_t from = on && k > 0 ? (pk < nrows ? pk + 1 : nrows) : 0;
        const uint32_t to = on ? (rk < nrows ? rk + 1 : nrows) : 0;
        fill(to > from && to - from > kShortGap, from, to, k);
        if (e == nnz) {
            const bool last = on && k == nnz - 1;
            fill(last && to < nrows, to, nrows, nnz);
            if (last) rp[nrows] = nnz;
        }
    }
}

// Row index of every position of a run: the rows that start inside it mark
// their first position, and a running maximum over the run spreads them. A run
// among so many empty rows that its CTA would walk more than kWalkRows row
// pointers looks its positions' rows up instead (a dependent load per halving,
// eight positions a thread side by side: about as long as walking 32 row
// pointers a thread). 10 M rows with 3000 nonzeros: 6.1 ms walking, 44 us here.
constexpr uint32_t kWalkRows = 4 * kChunk;
template <typename T>
__global__ void __launch_bounds__(kThreads, 8)  // (32 registers: the looking up, rare, may spill)
    csr_to_coo_kernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci, const T* __restrict__ vi,
                      uint32_t nnz, uint32_t nrows, uint32_t* __restrict__ ro, uint32_t* __restrict__ co,
                      T* __restrict__ vo) {
    constexpr uint32_t PER = kChunk / kThreads;  // consecutive positions of a thread in the scan
    __shared__ uint32_t mark[kChunk];
    __shared__ uint32_t warp_max[kThreads / 32];
    __shared__ uint32_t first;
    const uint32_t b = blockIdx.x * kChunk;
    const uint32_t e = static_cast<uint32_t>(min(static_cast<uint64_t>(nnz), static_cast<uint64_t>(b) + kChunk));
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t rows_b = __ldg(rp), rows_e = __ldg(rp + nrows);  // positions outside the rows stay as they are
    Run<T> run;
    run.load(ci, vi, co, vo, b, e);
    if (t == 0) {
        // the row of position b: the last with rp[row] <= b
        uint32_t lo = 0, hi = nrows;
        while (hi - lo > 1) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (__ldg(rp + mid) <= b)
                lo = mid;
            else
                hi = mid;
        }
        first = lo;
    }
    for (uint32_t i = t; i < kChunk; i += kThreads) mark[i] = 0;
    run.store(ci, vi, co, vo, b, e);
    __syncthreads();
    const uint32_t r0 = first;
    // rows after the first that start inside the run (empty ones share a
    // position with the next: the largest stays)
    const bool far = nrows - r0 > kWalkRows && __ldg(rp + r0 + kWalkRows) < e;  // (the same in every thread)
    if (!far) {
        for (uint32_t r = r0 + 1 + t; r < nrows; r += kThreads) {
            const uint32_t at = __ldg(rp + r);
            if (at >= e) break;
            if (at >= b) atomicMax(&mark[at - b], r);
        }
    } else {
        uint32_t lo[PER], hi[PER];
#pragma unroll
        for (uint32_t u = 0; u < PER; ++u) {
            lo[u] = r0;
            hi[u] = nrows;
        }
        for (uint32_t w = nrows - r0; w > 0; w >>= 1)  // (one halving more than nrows - r0 rows need at most)
#pragma unroll
            for (uint32_t u = 0; u < PER; ++u)
                if (hi[u] - lo[u] > 1) {
                    const uint32_t mid = lo[u] + (hi[u] - lo[u]) / 2;
                    if (__ldg(rp + mid) <= b + u * kThreads + t)
                        lo[u] = mid;
                    else
                        hi[u] = mid;
                }
#pragma unroll
        for (uint32_t u = 0; u < PER; ++u) {
            const uint32_t k = b + u * kThreads + t;
            if (k < e && k >= rows_b && k < rows_e) __stcs(ro + k, lo[u]);
        }
        return;
    }
    __syncthreads();
    uint32_t v[PER], m = 0;
#pragma unroll
    for (uint32_t u = 0; u < PER; ++u) {
        m = max(m, mark[t * PER + u]);
        v[u] = m;
    }
    uint32_t s = m;  // inclusive maximum over the warp, then over the warps before
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= static_cast<uint32_t>(off)) s = max(s, o);
    }
    if (lane == 31) warp_max[warp] = s;
    uint32_t before = __shfl_up_sync(0xffffffffu, s, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    for (uint32_t w = 0; w < warp; ++w) before = max(before, warp_max[w]);
    before = max(before, r0);
#pragma unroll
    for (uint32_t u = 0; u < PER; ++u) mark[t * PER + u] = max(before, v[u]);
    __syncthreads();
    for (uint32_t i = t; i < e - b; i += kThreads)
        if (b + i >= rows_b && b + i < rows_e) __stcs(ro + b + i, mark[i]);
}

__global__ void fill_u32_kernel(uint32_t* p, uint64_t n, uint32_t v) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = v;
}

template <typename T>
__global__ void zero_dense_kernel(T* __restrict__ D, Dense dv, uint32_t rows, uint32_t cols) {
    const uint64_t total = static_cast<uint64_t>(rows) * cols;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint64_t major = dv.cm ? i / rows : i / cols, minor = dv.cm ? i % rows : i % cols;
        D[major * dv.ld + minor] = T(0);
    }
}

template <typename T>
__global__ void scatter_dense_kernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ cols,
                                     const T* __restrict__ vals, uint32_t nrows, T* __restrict__ D, Dense dv) {
    // one thread per row, entries in order: the last duplicate wins
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < nrows; r += stride)
        for (uint32_t k = rp[r]; k < rp[r + 1]; ++k) D[dv.at(r, cols[k])] = vals[k];
}

template <typename T>
__global__ void count_rows_kernel(const T* __restrict__ D, Dense dv, uint32_t rows, uint32_t cols,
                                  uint32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t r = warp; r < rows; r += nwarps) {
        uint32_t c = 0;
        for (uint32_t j0 = 0; j0 < cols; j0 += 32) {
            const uint32_t j = j0 + lane;
            const bool nz = j < cols && D[dv.at(r, j)] != T(0);
            c += __popc(__ballot_sync(0xffffffffu, nz));
        }
        if (lane == 0) cnt[r] = c;
    }
}

template <typename T>
__global__ void compact_rows_kernel(const T* __restrict__ D, Dense dv, uint32_t rows, uint32_t cols,
                                    const uint32_t* __restrict__ rp, uint32_t* __restrict__ ocols,
                                    T* __restrict__ ovals) {
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    for (uint64_t r = warp; r < rows; r += nwarps) {
        uint32_t pos = rp[r];
        for (uint32_t j0 = 0; j0 < cols; j0 += 32) {
            const uint32_t j = j0 + lane;
            const T v = j < cols ? D[dv.at(r, j)] : T(0);
            const unsigned ball = __ballot_sync(0xffffffffu, v != T(0));
            if (v != T(0)) {
                const uint32_t k = pos + __popc(ball & ((1u << lane) - 1u));
                ocols[k] = j;
                ovals[k] = v;
            }
            pos += __popc(ball);
        }
    }
}

// y = alpha * A * x + beta * y for a COO matrix sorted by row: G lanes per
// row find the row's entries [lower_bound(r), lower_bound(r + 1)) in the
// sorted row indices and reduce them (duplicates are summed); beta == 0
// overwrites y without reading it.
__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* __restrict__ a, uint32_t n, uint32_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (__ldg(a + mid) < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

template <typename T, int G>
__global__ void __launch_bounds__(kThreads)
    coomv_kernel(const uint32_t* __restrict__ ri, const uint32_t* __restrict__ ci, const T* __restrict__ vals,
                 uint32_t nnz, uint32_t nrows, const T* __restrict__ alpha_p, const T* __restrict__ x,
                 const T* __restrict__ beta_p, T* __restrict__ y) {
    const T alpha = *alpha_p, beta = *beta_p;
    const uint32_t lane = threadIdx.x & (G - 1);
    const uint64_t group = (static_cast<uint64_t>(blockIdx.x) * kThreads + threadIdx.x) / G;
    const uint64_t ngroups = static_cast<uint64_t>(gridDim.x) * kThreads / G;
    // every lane of the warp runs the same trips (the loop bound does not
    // depend on the group), so the full-warp shuffles below are uniform
    for (uint64_t base = 0; base < nrows; base += ngroups) {
        const uint64_t r = base + group;
        T acc = T(0);
        if (r < nrows) {
            const uint32_t lo = lower_bound_u32(ri, nnz, static_cast<uint32_t>(r));
            const uint32_t hi = lower_bound_u32(ri, nnz, static_cast<uint32_t>(r) + 1);
            for (uint32_t k = lo + lane; k < hi; k += G) acc = dev::fma_rn(alpha * vals[k], __ldg(x + ci[k]), acc);
        }
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off, G);
        if (r < nrows && lane == 0) y[r] = beta == T(0) ? acc : acc + beta * y[r];
    }
}

template <typename T>
clsparseStatus coomv(const clsparseScalar* alpha, const clsparseCooMatrix* A, const cldenseVector* x,
                     const clsparseScalar* beta, cldenseVector* y, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!alpha || !A || !x || !beta || !y) return clsparseInvalidValue;
    if (x->num_values < A->num_cols || y->num_values < A->num_rows) return clsparseInvalidSize;
    if (A->num_rows == 0) return clsparseSuccess;
    if (!alpha->value || !beta->value || !x->values || !y->values ||
        (A->num_nonzeros && (!A->values || !A->col_indices || !A->row_indices)))
        return clsparseInvalidMemObject;
    DeviceGuard g(control->device);
    constexpr int G = 8;
    // every lane of a warp runs the same number of rows: whole warps per CTA
    coomv_kernel<T, G><<<grid_for(static_cast<uint64_t>(A->num_rows) * G, control->sm_count), kThreads, 0,
                         control->stream>>>(
        dev_ptr<const uint32_t>(A->row_indices, A->off_row_indices),
        dev_ptr<const uint32_t>(A->col_indices, A->off_col_indices), dev_ptr<const T>(A->values, A->off_values),
        static_cast<uint32_t>(A->num_nonzeros), static_cast<uint32_t>(A->num_rows),
        dev_ptr<const T>(alpha->value, alpha->off_value), dev_ptr<const T>(x->values, x->off_values),
        dev_ptr<const T>(beta->value, beta->off_value), dev_ptr<T>(y->values, y->off_values));
    if (cudaGetLastError() != cudaSuccess) return clsparseInvalidKernelExecution;
    return finish_call(control);
}

bool check_ptrs(const void* a, const void* b, const void* c, size_t n) {
    return n == 0 || (a && b && c);
}

template <typename T>
clsparseStatus coo2csr(const clsparseCooMatrix* coo, clsparseCsrMatrix* csr, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!coo || !csr) return clsparseInvalidValue;
    if (!csr->row_pointer || !check_ptrs(coo->values, coo->col_indices, coo->row_indices, coo->num_nonzeros) ||
        !check_ptrs(csr->values, csr->col_indices, csr->row_pointer, coo->num_nonzeros))
        return clsparseInvalidMemObject;
    DeviceGuard g(control->device);
    csr->num_rows = coo->num_rows;
    csr->num_cols = coo->num_cols;
    csr->num_nonzeros = coo->num_nonzeros;
    cudaStream_t s = control->stream;
    const uint32_t nnz = static_cast<uint32_t>(coo->num_nonzeros), nrows = static_cast<uint32_t>(coo->num_rows);
    uint32_t* rp = dev_ptr<uint32_t>(csr->row_pointer, csr->off_row_pointer);
    if (nnz) {
        const uint32_t runs = (nnz - 1) / kChunk + 1, gap_ctas = nrows / kGapCta + 1;
        coo_to_csr_kernel<T><<<runs + gap_ctas, kThreads, 0, s>>>(
            dev_ptr<const uint32_t>(coo->row_indices, coo->off_row_indices),
            dev_ptr<const uint32_t>(coo->col_indices, coo->off_col_indices),
            dev_ptr<const T>(coo->values, coo->off_values), nnz, nrows, gap_ctas, rp,
            dev_ptr<uint32_t>(csr->col_indices, csr->off_col_indices), dev_ptr<T>(csr->values, csr->off_values));
    } else {
        fill_u32_kernel<<<grid_for(static_cast<uint64_t>(nrows) + 1, control->sm_count), kThreads, 0, s>>>(
            rp, static_cast<uint64_t>(nrows) + 1, 0u);
    }
    if (cudaGetLastError() != cudaSuccess) return clsparseInvalidKernelExecution;
    return finish_call(control);
}

template <typename T>
clsparseStatus csr2coo(const clsparseCsrMatrix* csr, clsparseCooMatrix* coo, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!coo || !csr) return clsparseInvalidValue;
    if (!csr->row_pointer || !check_ptrs(coo->values, coo->col_indices, coo->row_indices, csr->num_nonzeros) ||
        !check_ptrs(csr->values, csr->col_indices, csr->row_pointer, csr->num_nonzeros))
        return clsparseInvalidMemObject;
    DeviceGuard g(control->device);
    coo->num_rows = csr->num_rows;
    coo->num_cols = csr->num_cols;
    coo->num_nonzeros = csr->num_nonzeros;
    cudaStream_t s = control->stream;
    const uint32_t nnz = static_cast<uint32_t>(csr->num_nonzeros), nrows = static_cast<uint32_t>(csr->num_rows);
    if (nnz)
        csr_to_coo_kernel<T><<<(nnz - 1) / kChunk + 1, kThreads, 0, s>>>(
            dev_ptr<const uint32_t>(csr->row_pointer, csr->off_row_pointer),
            dev_ptr<const uint32_t>(csr->col_indices, csr->off_col_indices),
            dev_ptr<const T>(csr->values, csr->off_values), nnz, nrows,
            dev_ptr<uint32_t>(coo->row_indices, coo->off_row_indices),
            dev_ptr<uint32_t>(coo->col_indices, coo->off_col_indices), dev_ptr<T>(coo->values, coo->off_values));
    if (cudaGetLastError() != cudaSuccess) return clsparseInvalidKernelExecution;
    return finish_call(control);
}

template <typename T>
clsparseStatus csr2dense(const clsparseCsrMatrix* csr, cldenseMatrix* A, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!csr || !A) return clsparseInvalidValue;
    if (A->num_rows < csr->num_rows || A->num_cols < csr->num_cols || !dense_ok(A)) return clsparseInvalidSize;
    if (!A->values || !csr->row_pointer || (csr->num_nonzeros && (!csr->values || !csr->col_indices)))
        return clsparseInvalidMemObject;
    DeviceGuard g(control->device);
    cudaStream_t s = control->stream;
    const Dense dv = dense_view(A);
    T* D = dev_ptr<T>(A->values, A->off_values);
    const uint32_t rows = A->num_rows, cols = A->num_cols;
    zero_dense_kernel<T><<<grid_for(static_cast<uint64_t>(rows) * cols, control->sm_count), kThreads, 0, s>>>(
        D, dv, rows, cols);
    scatter_dense_kernel<T><<<grid_for(csr->num_rows, control->sm_count), kThreads, 0, s>>>(
        dev_ptr<const uint32_t>(csr->row_pointer, csr->off_row_pointer),
        dev_ptr<const uint32_t>(csr->col_indices, csr->off_col_indices), dev_ptr<const T>(csr->values, csr->off_values),
        static_cast<uint32_t>(csr->num_rows), D, dv);
    if (cudaGetLastError() != cudaSuccess) return clsparseInvalidKernelExecution;
    return finish_call(control);
}

template <typename T>
clsparseStatus dense2csr(const cldenseMatrix* A, clsparseCsrMatrix* csr, clsparseControl control) {
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (!csr || !A) return clsparseInvalidValue;
    if (!dense_ok(A)) return clsparseInvalidSize;
    if (!A->values || !csr->row_pointer || !csr->values || !csr->col_indices) return clsparseInvalidMemObject;
    const uint32_t rows = A->num_rows, cols = A->num_cols;
    const uint32_t nparts = (rows + 1023) / 1024;
    // the block totals use the partial-sum slots of the control's reduction
    // scratch (its tickets lie after them): at most 16.7 M rows
    if (static_cast<size_t>(nparts) * 4 > static_cast<size_t>(kMaxReduceCtas) * 4 * sizeof(double))
        return clsparseInvalidSize;
    DeviceGuard g(control->device);
    cudaStream_t s = control->stream;
    const Dense dv = dense_view(A);
    const T* D = dev_ptr<const T>(A->values, A->off_values);
    uint32_t* rp = dev_ptr<uint32_t>(csr->row_pointer, csr->off_row_pointer);
    // row counts into rp[1..rows], scanned in place (inclusive), rp[0] = 0
    uint32_t* part = static_cast<uint32_t*>(control->reduce_scratch.ptr);
    cudaMemsetAsync(rp, 0, 4, s);
    count_rows_kernel<T><<<grid_for(static_cast<uint64_t>(rows) * 32, control->sm_count), kThreads, 0, s>>>(
        D, dv, rows, cols, rp + 1);
    if (rows) {
        scan::inclusive_u32(rp + 1, rows, part, s);
    }
    uint32_t* hv = static_cast<uint32_t*>(control->pinned) + 512;
    cudaMemcpyAsync(hv, rp + rows, 4, cudaMemcpyDeviceToHost, s);
    compact_rows_kernel<T><<<grid_for(static_cast<uint64_t>(rows) * 32, control->sm_count), kThreads, 0, s>>>(
        D, dv, rows, cols, rp, dev_ptr<uint32_t>(csr->col_indices, csr->off_col_indices),
        dev_ptr<T>(csr->values, csr->off_values));
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
        return clsparseInvalidKernelExecution;
    csr->num_rows = rows;
    csr->num_cols = cols;
    csr->num_nonzeros = *hv;
    return finish_call(control);
}

}  // namespace
}  // namespace clsp

using namespace clsp;

extern "C" {

clsparseStatus clsparseScoomv(const clsparseScalar* alpha, const clsparseCooMatrix* matx, const cldenseVector* x,
                              const clsparseScalar* beta, cldenseVector* y, const clsparseControl control) {
    return coomv<float>(alpha, matx, x, beta, y, control);
}
clsparseStatus clsparseDcoomv(const clsparseScalar* alpha, const clsparseCooMatrix* matx, const cldenseVector* x,
                              const clsparseScalar* beta, cldenseVector* y, const clsparseControl control) {
    return coomv<double>(alpha, matx, x, beta, y, control);
}
clsparseStatus clsparseScoo2csr(const clsparseCooMatrix* coo, clsparseCsrMatrix* csr, const clsparseControl control) {
    return coo2csr<float>(coo, csr, control);
}
clsparseStatus clsparseDcoo2csr(const clsparseCooMatrix* coo, clsparseCsrMatrix* csr, const clsparseControl control) {
    return coo2csr<double>(coo, csr, control);
}
clsparseStatus clsparseScsr2coo(const clsparseCsrMatrix* csr, clsparseCooMatrix* coo, const clsparseControl control) {
    return csr2coo<float>(csr, coo, control);
}
clsparseStatus clsparseDcsr2coo(const clsparseCsrMatrix* csr, clsparseCooMatrix* coo, const clsparseControl control) {
    return csr2coo<double>(csr, coo, control);
}
clsparseStatus clsparseScsr2dense(const clsparseCsrMatrix* csr, cldenseMatrix* A, const clsparseControl control) {
    return csr2dense<float>(csr, A, control);
}
clsparseStatus clsparseDcsr2dense(const clsparseCsrMatrix* csr, cldenseMatrix* A, clsparseControl control) {
    return csr2dense<double>(csr, A, control);
}
clsparseStatus clsparseSdense2csr(const cldenseMatrix* A, clsparseCsrMatrix* csr, const clsparseControl control) {
    return dense2csr<float>(A, csr, control);
}
clsparseStatus clsparseDdense2csr(const cldenseMatrix* A, clsparseCsrMatrix* csr, const clsparseControl control) {
    return dense2csr<double>(A, csr, control);
}

}  // extern "C"
