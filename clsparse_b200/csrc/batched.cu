// Batched Jacobi-CG over many independent SPD systems in one persistent
// launch (clsparseScsrcgBatched), a project extension with no reference
// counterpart.
//
// The systems are stacked block-diagonally in one CSR matrix (rows and columns
// of system s are [off[s], off[s+1])). Each runs CG to completion on its own:
// FP32 vectors and FP32 matrix values, no grid synchronisation and no host
// round trip. When the recursive FP32 residual meets the tolerance, the true
// residual b - A x is recomputed in FP64; if that check fails, CG restarts
// from the current x with the FP64 residual (refinement) until the check
// passes or the iteration budget is spent.
//
// Banded systems (at most kBatchDiags column offsets, all inside their own
// rows; the offsets are found on the device at every call) that fit on chip
// are solved by the resident kernel (batched_resident.cuh), one launch per
// cluster size on streams of their own, the largest systems first.
//
// The others run in the persistent general kernel (a cliff: 52,900 rows take 6 us
// an iteration on eight SMs, 67,600 rows, which do not fit, 116 on one CTA here):
// one CTA per resident slot takes the next system from a device work queue
// (largest first). When all of them are banded (systems too large for a
// cluster's shared memory), their products come from a per-system
// diagonal-storage copy laid out at every call: one thread per row, the values
// and the vector entries independent loads instead of the row-pointer /
// column-index / vector chain of CSR, and rows whose whole stencil lies inside
// the system without clamps; otherwise, and when that copy cannot be had,
// each system's SpMV uses the lanes-per-row width the tuning table gives for
// its size class. The kernel is held to two CTAs per SM (64 registers): the
// diagonal loop would otherwise take 128 registers and halve the resident
// CTAs.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <vector>

#include "device_common.cuh"
#include "internal.h"

namespace clsp {
namespace {

constexpr int kThreads = 512;

// Diagonals a system may have to be solved from diagonal storage.
constexpr int kBatchDiags = 8;

}  // namespace
}  // namespace clsp

#include "batched_resident.cuh"

namespace clsp {
namespace {

struct BatchArgs {
    const float* vals;
    const uint32_t* cols;
    const uint32_t* rp;
    float* x;
    const float* b;
    float* r;
    float* p;
    float* q;
    float* invd;
    const uint32_t* off;      // num_systems + 1 row offsets
    const uint32_t* order;    // processing order of the systems
    const uint8_t* lanes;     // lanes per row for each system (1, 2, 4, 8, 16, 32)
    uint32_t* counter;        // work queue head
    int* iters;               // per system: CG iterations
    double* residual;         // per system: FP64 ||b - A x||_2 / ||b||_2 on exit
    int* converged;           // per system: 1 if residual <= tol
    uint32_t nsys;
    int max_iters;
    double tol;
    // Diagonal storage (nullptr: every system's products come from CSR):
    // system s's diagonal d at row r0 + i is dvals[dbase[s] + d * n_s + i],
    // its column offsets doffs[s * kBatchDiags + d] increasing, dnd[s] of them.
    const float* dvals;
    const uint64_t* dbase;
    const int32_t* doffs;
    const uint8_t* dnd;
};

__device__ __forceinline__ double cta_sum(double v, double* red) {
    return dev::block_sum(v, red);
}

// q = A v over the rows of one system, G lanes per row.
template <int G>
__device__ __forceinline__ void sys_spmv(const BatchArgs& a, uint32_t r0, uint32_t r1, const float* v,
                                         float* out) {
    const uint32_t grp = threadIdx.x / G, ln = threadIdx.x & (G - 1);
    const uint32_t groups = kThreads / G;
    for (uint32_t base = r0; base < r1; base += groups) {
        const uint32_t row = base + grp;
        float s = 0.f;
        if (row < r1) {
            const uint32_t nb = a.rp[row], ne = a.rp[row + 1];
            for (uint32_t j = nb + ln; j < ne; j += G) s = fmaf(a.vals[j], v[a.cols[j]], s);
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
        if (row < r1 && ln == 0) out[row] = s;
    }
}

__device__ __forceinline__ void spmv_dispatch(const BatchArgs& a, int g, uint32_t r0, uint32_t r1,
                                              const float* v, float* out) {
    switch (g) {
        case 1: sys_spmv<1>(a, r0, r1, v, out); break;
        case 2: sys_spmv<2>(a, r0, r1, v, out); break;
        case 4: sys_spmv<4>(a, r0, r1, v, out); break;
        case 8: sys_spmv<8>(a, r0, r1, v, out); break;
        case 16: sys_spmv<16>(a, r0, r1, v, out); break;
        default: sys_spmv<32>(a, r0, r1, v, out); break;
    }
}

// q = A v over the rows of one system from its diagonal storage: one thread
// per row, products in increasing column order, columns outside the system
// (the block diagonal) contribute nothing. The values and the v entries of
// a row are independent loads (no row-pointer / column-index chain).
__device__ __forceinline__ double sys_spmv_dia(const float* __restrict__ dv, uint32_t ns, uint32_t r0, uint32_t r1,
                                               const int32_t* soff, int nd, const float* v, float* out) {
    double dot = 0.0;
    const int32_t lo = nd > 0 ? soff[0] : 0, hi = nd > 0 ? soff[nd - 1] : 0;
    auto row_sum = [&](uint32_t row) {
        const uint32_t i = row - r0;
        float s = 0.f;
        if (static_cast<int64_t>(row) + lo >= r0 && static_cast<int64_t>(row) + hi < r1) {
            // every column of the row inside the system: no clamps
#pragma unroll
            for (int d = 0; d < kBatchDiags; ++d)
                if (d < nd)
                    s = fmaf(__ldg(dv + static_cast<size_t>(d) * ns + i), v[row + static_cast<uint32_t>(soff[d])], s);
        } else {
#pragma unroll
            for (int d = 0; d < kBatchDiags; ++d) {
                if (d < nd) {
                    const int64_t j = static_cast<int64_t>(row) + soff[d];
                    const bool in = j >= r0 && j < r1;
                    const float av = __ldg(dv + static_cast<size_t>(d) * ns + i);
                    const float xv = v[in ? static_cast<uint32_t>(j) : row];
                    s = fmaf(av, in ? xv : 0.f, s);
                }
            }
        }
        return s;
    };
    // two rows per pass, both rows' loads before the stores (see the update pass)
    for (uint32_t row = r0 + threadIdx.x; row < r1; row += 2 * kThreads) {
        const uint32_t row1 = row + kThreads;
        const bool has1 = row1 < r1;
        const uint32_t rb = has1 ? row1 : row;
        const float s0 = row_sum(row);
        const float s1 = row_sum(rb);
        const float v0 = v[row], v1 = v[rb];
        out[row] = s0;
        dot += static_cast<double>(v0) * s0;
        if (has1) {
            out[row1] = s1;
            dot += static_cast<double>(v1) * s1;
        }
    }
    return dot;  // this thread's part of <v, A v>
}

// r = b - A x in FP64 (the check), written back to r in FP32; returns
// sum r^2 and sum b^2 in every thread.
__device__ __forceinline__ void true_residual(const BatchArgs& a, uint32_t r0, uint32_t r1, double* red,
                                              double& rr, double& bb) {
    double acc_r = 0.0, acc_b = 0.0;
    for (uint32_t row = r0 + threadIdx.x; row < r1; row += kThreads) {
        double s = 0.0;
        for (uint32_t j = a.rp[row]; j < a.rp[row + 1]; ++j)
            s = fma(static_cast<double>(a.vals[j]), static_cast<double>(a.x[a.cols[j]]), s);
        const double bi = a.b[row];
        const double ri = bi - s;
        a.r[row] = static_cast<float>(ri);
        acc_r += ri * ri;
        acc_b += bi * bi;
    }
    rr = cta_sum(acc_r, red);
    bb = cta_sum(acc_b, red);
}

__global__ void __launch_bounds__(kThreads, 2) batched_cg_kernel(BatchArgs a) {
    __shared__ double red[32];
    __shared__ uint32_t slot;
    __shared__ int32_t soff[kBatchDiags];
    for (;;) {
        if (threadIdx.x == 0) slot = atomicAdd(a.counter, 1u);
        __syncthreads();
        const uint32_t k = slot;
        __syncthreads();
        if (k >= a.nsys) break;
        const uint32_t s = a.order[k];
        const uint32_t r0 = a.off[s], r1 = a.off[s + 1];
        const int g = a.lanes[s];
        const float* dv = a.dvals ? a.dvals + a.dbase[s] : nullptr;
        const int nd = a.dvals ? a.dnd[s] : 0;
        if (a.dvals && threadIdx.x < kBatchDiags) soff[threadIdx.x] = a.doffs[s * kBatchDiags + threadIdx.x];

        // Jacobi: inverse diagonal (first diagonal entry of each row; 1 if absent)
        for (uint32_t row = r0 + threadIdx.x; row < r1; row += kThreads) {
            float d = 0.f;
            for (uint32_t j = a.rp[row]; j < a.rp[row + 1]; ++j)
                if (a.cols[j] == row) {
                    d = a.vals[j];
                    break;
                }
            a.invd[row] = d != 0.f ? 1.f / d : 1.f;
        }
        __syncthreads();

        double rr, bb;
        true_residual(a, r0, r1, red, rr, bb);
        const double bnorm = sqrt(bb);
        int it = 0;
        bool ok = bnorm == 0.0 || sqrt(rr) <= a.tol * bnorm;
        double res64 = bnorm == 0.0 ? 0.0 : sqrt(rr) / bnorm;
        while (!ok && it < a.max_iters) {
            // (re)start: z = M r, p = z, rz = <r, z>
            double acc = 0.0;
            for (uint32_t row = r0 + threadIdx.x; row < r1; row += kThreads) {
                const float z = a.r[row] * a.invd[row];
                a.p[row] = z;
                acc += static_cast<double>(a.r[row]) * z;
            }
            double rz = cta_sum(acc, red);
            __syncthreads();
            bool inner_done = false;
            while (!inner_done && it < a.max_iters) {
                if (dv) {
                    // the row's thread also forms its part of <p, q>
                    acc = sys_spmv_dia(dv, r1 - r0, r0, r1, soff, nd, a.p, a.q);
                } else {
                    spmv_dispatch(a, g, r0, r1, a.p, a.q);
                    __syncthreads();
                    acc = 0.0;
                    for (uint32_t row = r0 + threadIdx.x; row < r1; row += kThreads)
                        acc += static_cast<double>(a.p[row]) * a.q[row];
                }
                const double pq = cta_sum(acc, red);  // its barriers also order q's stores
                const float alpha = static_cast<float>(rz / pq);
                double acc_rz = 0.0, acc_rr = 0.0;
                // two rows per pass, all their loads before any store (the
                // vectors are not __restrict__: a store holds back every later
                // load, so one row per pass would wait out each row's loads)
                for (uint32_t row = r0 + threadIdx.x; row < r1; row += 2 * kThreads) {
                    const uint32_t row1 = row + kThreads;
                    const bool has1 = row1 < r1;
                    const uint32_t rb = has1 ? row1 : row;
                    const float xi = fmaf(alpha, a.p[row], a.x[row]);
                    const float ri = fmaf(-alpha, a.q[row], a.r[row]);
                    const float z = ri * a.invd[row];
                    const float xj = fmaf(alpha, a.p[rb], a.x[rb]);
                    const float rj = fmaf(-alpha, a.q[rb], a.r[rb]);
                    const float zj = rj * a.invd[rb];
                    a.x[row] = xi;
                    a.r[row] = ri;
                    acc_rz += static_cast<double>(ri) * z;
                    acc_rr += static_cast<double>(ri) * ri;
                    if (has1) {
                        a.x[row1] = xj;
                        a.r[row1] = rj;
                        acc_rz += static_cast<double>(rj) * zj;
                        acc_rr += static_cast<double>(rj) * rj;
                    }
                }
                const double rz_new = cta_sum(acc_rz, red);
                const double rr_new = cta_sum(acc_rr, red);
                ++it;
                if (!(pq > 0.0) || !isfinite(rz_new)) {
                    inner_done = true;  // breakdown: fall through to the FP64 check
                    break;
                }
                if (sqrt(rr_new) <= a.tol * bnorm) {
                    inner_done = true;
                    break;
                }
                const float beta = static_cast<float>(rz_new / rz);
                rz = rz_new;
                for (uint32_t row = r0 + threadIdx.x; row < r1; row += 2 * kThreads) {
                    const uint32_t row1 = row + kThreads;
                    const bool has1 = row1 < r1;
                    const uint32_t rb = has1 ? row1 : row;
                    const float pi = fmaf(beta, a.p[row], a.r[row] * a.invd[row]);
                    const float pj = fmaf(beta, a.p[rb], a.r[rb] * a.invd[rb]);
                    a.p[row] = pi;
                    if (has1) a.p[row1] = pj;
                }
                __syncthreads();
            }
            __syncthreads();
            true_residual(a, r0, r1, red, rr, bb);
            res64 = sqrt(rr) / bnorm;
            ok = res64 <= a.tol;
            if (!isfinite(res64)) break;
        }
        if (threadIdx.x == 0) {
            a.iters[s] = it;
            a.residual[s] = res64;
            a.converged[s] = ok ? 1 : 0;
        }
        __syncthreads();
    }
}

// The distinct column offsets col - row of system blockIdx.x's rows
// [blockIdx.y * kDetectRows, ...) into its set (kBatchDiags slots preset to
// kNoOffset); over[s] = 1 when there are more, a column lies outside the
// system's rows, or columns are not strictly increasing in a row. A thread
// keeps the offsets it knows to be in the set in registers and goes to the
// shared set only for a new one (one CTA per system with every entry probing
// the set took 2.3 ms for 1024 systems of up to 50,000 rows).
constexpr int32_t kNoOffset = INT32_MIN;  // below any offset of a system of fewer than 2^31 rows
constexpr uint32_t kDetectRows = 4096;

__device__ __forceinline__ bool offset_insert(int32_t* set, int32_t o) {
    for (int t = 0; t < kBatchDiags; ++t) {
        const int32_t cur = *reinterpret_cast<volatile int32_t*>(&set[t]);
        if (cur == o) return true;
        if (cur == kNoOffset) {
            const int32_t old = atomicCAS(&set[t], kNoOffset, o);
            if (old == kNoOffset || old == o) return true;
        }
    }
    return false;
}

__global__ void __launch_bounds__(256)
    batch_dia_detect_kernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ cols,
                            const uint32_t* __restrict__ off, int32_t* sets, int* over) {
    __shared__ int32_t set[kBatchDiags];
    const uint32_t s = blockIdx.x;
    const uint32_t r0 = off[s], r1 = off[s + 1];
    const uint64_t begin = r0 + static_cast<uint64_t>(blockIdx.y) * kDetectRows;
    if (begin >= r1) return;
    const uint32_t end = static_cast<uint32_t>(min(static_cast<uint64_t>(r1), begin + kDetectRows));
    if (threadIdx.x < kBatchDiags) set[threadIdx.x] = kNoOffset;
    __syncthreads();
    bool bad = false;
    int32_t known[kBatchDiags];
#pragma unroll
    for (int t = 0; t < kBatchDiags; ++t) known[t] = kNoOffset;
    for (uint32_t row = static_cast<uint32_t>(begin) + threadIdx.x; row < end; row += blockDim.x) {
        const uint32_t kb = rp[row], ke = rp[row + 1];
        uint32_t prev = 0;
        for (uint32_t k = kb; k < ke; ++k) {
            const uint32_t c = cols[k];
            if (c < r0 || c >= r1 || (k > kb && c <= prev)) {
                bad = true;
            } else {
                const int32_t o = static_cast<int32_t>(static_cast<int64_t>(c) - static_cast<int64_t>(row));
                bool seen = false;
#pragma unroll
                for (int t = 0; t < kBatchDiags; ++t) seen |= known[t] == o;
                if (!seen) {
                    bad |= !offset_insert(set, o);
#pragma unroll
                    for (int t = 0; t < kBatchDiags; ++t) known[t] = *reinterpret_cast<volatile int32_t*>(&set[t]);
                }
            }
            prev = c;
        }
    }
    if (bad) atomicOr(over + s, 1);
    __syncthreads();
    if (threadIdx.x < kBatchDiags && set[threadIdx.x] != kNoOffset &&
        !offset_insert(sets + static_cast<size_t>(s) * kBatchDiags, set[threadIdx.x]))
        atomicOr(over + s, 1);
}

// The sets sorted: offsets of system s increasing at doffs[s * kBatchDiags],
// their number in dnd[s] (0: not banded, or no entries).
__global__ void batch_dia_sort_kernel(int32_t* doffs, const int* over, uint8_t* dnd, uint32_t nsys) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    int32_t v[kBatchDiags];
    int nd = 0;
    int32_t* o = doffs + static_cast<size_t>(s) * kBatchDiags;
    for (int t = 0; t < kBatchDiags; ++t)
        if (o[t] != kNoOffset) v[nd++] = o[t];
    if (over[s]) nd = 0;
    for (int t = 1; t < nd; ++t)  // insertion sort of at most kBatchDiags values
        for (int u = t; u > 0 && v[u - 1] > v[u]; --u) {
            const int32_t w = v[u];
            v[u] = v[u - 1];
            v[u - 1] = w;
        }
    for (int t = 0; t < kBatchDiags; ++t) o[t] = t < nd ? v[t] : 0;
    dnd[s] = static_cast<uint8_t>(nd);
}

__global__ void fill_i32_kernel(int32_t* p, size_t n, int32_t v) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// One CTA per system of `list`: its CSR values into diagonal storage (dv
// zeroed before).
__global__ void batch_dia_fill_kernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ cols,
                                      const float* __restrict__ vals, const uint32_t* __restrict__ off,
                                      const uint32_t* __restrict__ list, const int32_t* __restrict__ doffs, const uint8_t* __restrict__ dnd,
                                      const uint64_t* __restrict__ dbase, float* dv) {
    const uint32_t s = list[blockIdx.x];
    const uint32_t r0 = off[s], r1 = off[s + 1], ns = r1 - r0;
    const int nd = dnd[s];
    const int32_t* o = doffs + s * kBatchDiags;
    float* out = dv + dbase[s];
    for (uint32_t row = r0 + threadIdx.x; row < r1; row += blockDim.x) {
        int d = 0;
        for (uint32_t k = rp[row]; k < rp[row + 1]; ++k) {
            const int32_t c = static_cast<int32_t>(static_cast<int64_t>(cols[k]) - static_cast<int64_t>(row));
            while (d < nd && o[d] < c) ++d;  // columns increase, so d only moves forward
            if (d < nd && o[d] == c) out[static_cast<size_t>(d) * ns + (row - r0)] = vals[k];
        }
    }
}

__global__ void gather_bounds_kernel(const uint32_t* rp, const uint32_t* off, uint32_t nsys, uint32_t* bnd) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= nsys) bnd[i] = rp[off[i]];
}

int default_lanes(uint32_t n, uint32_t nnz) {
    const uint32_t per = n ? nnz / n : 0;
    if (per >= 24) return 8;
    if (per >= 12) return 4;
    return 2;
}

// ---- which systems the resident kernel takes, and how

constexpr int kResWide = 512;   // threads of a CTA, one CTA per SM
constexpr int kResSmall = 128;  // systems of up to 128 * kResRows rows: several CTAs per SM

// Shared memory a resident CTA may ask for: the 227 KB of an SM less the
// kernel's static part (the exchange's slots) and the CTA's reserve.
constexpr size_t kResSmem = 218 * 1024;

// One launch of the resident kernel: systems solved by clusters of the same size.
struct ResidentClass {
    int threads = 0, cluster = 0;
    size_t smem = 0;               // the largest of its systems
    std::vector<uint32_t> list;    // largest first
};

// Whether a system of n rows with nd sorted offsets runs on C CTAs of NT
// threads: its rows in the registers, its diagonals in shared memory, and its
// stencil reaching no further than the neighbouring CTA.
bool resident_fits(uint32_t n, const int32_t* off, int nd, uint32_t C, uint32_t NT, size_t& smem) {
    const uint64_t m = (static_cast<uint64_t>(n) + C - 1) / C;
    const uint64_t lo = off[0] < 0 ? static_cast<uint64_t>(-static_cast<int64_t>(off[0])) : 0;
    const uint64_t hi = off[nd - 1] > 0 ? static_cast<uint64_t>(off[nd - 1]) : 0;
    if (m > static_cast<uint64_t>(NT) * kResRows || (C > 1 && (lo > m || hi > m))) return false;
    smem = resident_smem(m, nd, lo, hi);
    return smem <= kResSmem;
}

template <int NT>
cudaError_t launch_resident(const ResidentArgs& a, const ResidentClass& k, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(batched_resident_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(kResSmem));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<uint32_t>(k.list.size()) * static_cast<uint32_t>(k.cluster));
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = k.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<uint32_t>(k.cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, batched_resident_kernel<NT>, a);
}

// Streams and events of the resident launches, made on first use.
bool ensure_streams(BatchWork& w, size_t count) {
    if (!w.begin && cudaEventCreateWithFlags(&w.begin, cudaEventDisableTiming) != cudaSuccess) return false;
    while (w.streams.size() < count) {
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return false;
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            cudaStreamDestroy(s);
            return false;
        }
        w.streams.push_back(s);
        w.ends.push_back(e);
    }
    return true;
}

}  // namespace
}  // namespace clsp

using namespace clsp;

extern "C" {

clsparseStatus clsparseScsrcgBatched(cldenseVector* x, const clsparseCsrMatrix* A, const cldenseVector* b,
                                     const clsparseIdx_t* systemOffsets, cl_int numSystems,
                                     const cl_int* lanesPerRow, clSParseSolverControl solverControl,
                                     clsparseB200BatchResult* result, clsparseControl control) {
    clsp::TraceRange trace_("clsparseScsrcgBatched");
    clsparseStatus st = check_entry(control);
    if (st != clsparseSuccess) return st;
    if (solverControl == nullptr) return clsparseInvalidSolverControlObject;
    if (!x || !A || !b || !systemOffsets || numSystems < 0) return clsparseInvalidValue;
    if (A->num_rows != A->num_cols || x->num_values != A->num_rows || b->num_values != A->num_rows)
        return clsparseInvalidSystemSize;
    const uint32_t nsys = static_cast<uint32_t>(numSystems);
    if (nsys == 0) return clsparseSuccess;
    if (systemOffsets[0] != 0 || systemOffsets[nsys] != A->num_rows) return clsparseInvalidSystemSize;
    for (uint32_t s = 0; s < nsys; ++s)
        if (systemOffsets[s + 1] < systemOffsets[s]) return clsparseInvalidSystemSize;
    DeviceGuard g(control->device);
    const size_t n = A->num_rows;
    if (!control->batch_work) control->batch_work = std::make_unique<BatchWork>();
    BatchWork& w = *control->batch_work;
    cudaStream_t s = control->stream;

    const size_t vb = ((n * 4 + 255) / 256) * 256;
    const size_t meta_bytes = 16 + (nsys + 1) * 4 * 2 + nsys * 4 * 2 + nsys + 256;
    const size_t out_bytes = nsys * (4 + 8 + 4) + 64;
    if (w.meta.ensure(meta_bytes) != cudaSuccess ||
        w.out.ensure(out_bytes) != cudaSuccess) {
        cudaGetLastError();
        return clsparseOutOfResources;
    }
    char* mb = static_cast<char*>(w.meta.ptr);
    uint32_t* d_counter = reinterpret_cast<uint32_t*>(mb);
    uint32_t* d_off = reinterpret_cast<uint32_t*>(mb + 16);
    uint32_t* d_bnd = d_off + (nsys + 1);
    uint32_t* d_order = d_bnd + (nsys + 1);
    uint32_t* d_rest = d_order + nsys;  // systems of the general kernel
    uint8_t* d_lanes = reinterpret_cast<uint8_t*>(d_rest + nsys);
    const uint32_t* rp = dev_ptr<const uint32_t>(A->row_pointer, A->off_row_pointer);

    // nonzeros per system from the row pointers at the system boundaries
    std::vector<uint32_t> off(systemOffsets, systemOffsets + nsys + 1), bnd(nsys + 1);
    cudaMemcpyAsync(d_off, off.data(), (nsys + 1) * 4, cudaMemcpyHostToDevice, s);
    gather_bounds_kernel<<<(nsys + 256) / 256, 256, 0, s>>>(rp, d_off, nsys, d_bnd);
    cudaMemcpyAsync(bnd.data(), d_bnd, (nsys + 1) * 4, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return clsparseInvalidMemObject;

    std::vector<uint32_t> order(nsys);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t p, uint32_t q) {
        return bnd[p + 1] - bnd[p] > bnd[q + 1] - bnd[q];
    });
    std::vector<uint8_t> lanes(nsys);
    for (uint32_t k = 0; k < nsys; ++k) {
        const uint32_t ns = off[k + 1] - off[k];
        const int l = lanesPerRow ? lanesPerRow[k] : default_lanes(ns, bnd[k + 1] - bnd[k]);
        if (l != 1 && l != 2 && l != 4 && l != 8 && l != 16 && l != 32) return clsparseInvalidValue;
        lanes[k] = static_cast<uint8_t>(l);
    }
    cudaMemcpyAsync(d_lanes, lanes.data(), nsys, cudaMemcpyHostToDevice, s);

    // Offsets of every system, found on the device at every call (so a matrix
    // changed in place is seen). CLSPARSE_B200_BATCH_DIA=0 keeps every system
    // on CSR.
    const char* dia_env = std::getenv("CLSPARSE_B200_BATCH_DIA");
    const bool dia = !(dia_env && std::atoi(dia_env) == 0);
    std::vector<uint8_t> hnd(nsys, 0);
    std::vector<int32_t> hoffs;
    int32_t* doffs = nullptr;
    uint64_t* dbase = nullptr;
    uint8_t* dnd = nullptr;
    const uint32_t* cols = dev_ptr<const uint32_t>(A->col_indices, A->off_col_indices);
    if (dia) {
        const size_t noff = static_cast<size_t>(nsys) * kBatchDiags;
        const size_t offs_b = ((noff * 4 + 255) / 256) * 256;
        const size_t base_b = ((static_cast<size_t>(nsys) * 8 + 255) / 256) * 256;
        const size_t over_b = ((static_cast<size_t>(nsys) * 4 + 255) / 256) * 256;
        if (w.dia_meta.ensure(offs_b + base_b + over_b + nsys + 256) != cudaSuccess) {
            cudaGetLastError();
            return clsparseOutOfResources;
        }
        char* dm = static_cast<char*>(w.dia_meta.ptr);
        doffs = reinterpret_cast<int32_t*>(dm);
        dbase = reinterpret_cast<uint64_t*>(dm + offs_b);
        int* over = reinterpret_cast<int*>(dm + offs_b + base_b);
        dnd = reinterpret_cast<uint8_t*>(dm + offs_b + base_b + over_b);
        uint32_t largest = 1;
        for (uint32_t k = 0; k < nsys; ++k) largest = std::max(largest, off[k + 1] - off[k]);
        const uint32_t chunks = std::min<uint32_t>((largest - 1) / kDetectRows + 1, 65535u);
        fill_i32_kernel<<<static_cast<uint32_t>((noff + 255) / 256), 256, 0, s>>>(doffs, noff, kNoOffset);
        cudaMemsetAsync(over, 0, static_cast<size_t>(nsys) * 4, s);
        if (static_cast<uint64_t>(chunks) * kDetectRows >= largest) {
            batch_dia_detect_kernel<<<dim3(nsys, chunks), 256, 0, s>>>(rp, cols, d_off, doffs, over);
            batch_dia_sort_kernel<<<(nsys + 255) / 256, 256, 0, s>>>(doffs, over, dnd, nsys);
            hoffs.resize(noff);
            cudaMemcpyAsync(hnd.data(), dnd, nsys, cudaMemcpyDeviceToHost, s);
            cudaMemcpyAsync(hoffs.data(), doffs, noff * 4, cudaMemcpyDeviceToHost, s);
            if (cudaStreamSynchronize(s) != cudaSuccess) return clsparseInvalidKernelExecution;
        }
    }

    // Systems of the resident kernel by CTA width and cluster size: the
    // smallest cluster that holds the system takes the least SM time (the
    // exchanges cost every CTA of a cluster alike); while the batch leaves
    // SMs idle, the clusters of systems with enough rows for it are doubled.
    // Measured, us an iteration of one system on 128 threads, 512, and 2, 4 and 8
    // CTAs of 512: 100 rows 2.5, 2.9, 3.5, 3.8, 4.0; 1024 rows 3.4, 3.2, 3.6,
    // 3.7, 3.9; 1764 rows 4.1, 3.5, 3.7, 3.8, 4.0; 3600 rows -, 4.1, 4.1, 3.9,
    // 4.0; 7056 rows -, 5.3, 4.7, 4.2, 4.2; 12,100 rows -, -, 5.5, 4.7, 4.5.
    constexpr uint64_t kWideRows = 896, kSplitRows = 1792;
    std::vector<ResidentClass> classes(5);
    const int sizes[5][2] = {{kResWide, 8}, {kResWide, 4}, {kResWide, 2}, {kResWide, 1}, {kResSmall, 1}};
    for (int k = 0; k < 5; ++k) {
        classes[k].threads = sizes[k][0];
        classes[k].cluster = sizes[k][1];
    }
    std::vector<int> at(nsys, -1);  // class of each system, -1: the general kernel
    auto place = [&](uint32_t k, int c) {
        size_t need = 0;
        return hnd[k] > 0 && resident_fits(off[k + 1] - off[k], &hoffs[static_cast<size_t>(k) * kBatchDiags], hnd[k],
                                           static_cast<uint32_t>(sizes[c][1]), static_cast<uint32_t>(sizes[c][0]), need)
                   ? need
                   : size_t(0);
    };
    uint64_t ctas = 0;
    for (uint32_t k = 0; k < nsys; ++k)
        for (int c = 4; c >= 0 && at[k] < 0; --c)
            if (place(k, c)) {
                at[k] = c;
                ctas += static_cast<uint64_t>(sizes[c][1]);
            }
    for (int step = 0; step < 4 && ctas > 0 && 2 * ctas <= static_cast<uint64_t>(control->sm_count); ++step) {
        ctas = 0;
        for (uint32_t k = 0; k < nsys; ++k) {
            const uint64_t rows = off[k + 1] - off[k];
            if (at[k] > 0 && rows > (at[k] == 4 ? kWideRows : kSplitRows * static_cast<uint64_t>(sizes[at[k]][1])) &&
                place(k, at[k] - 1))
                --at[k];
            if (at[k] >= 0) ctas += static_cast<uint64_t>(sizes[at[k]][1]);
        }
    }
    std::vector<uint32_t> lists, rest;  // the classes' systems one after another; the general kernel's
    for (uint32_t k : order) {
        if (at[k] < 0) {
            rest.push_back(k);
            continue;
        }
        classes[at[k]].list.push_back(k);
        classes[at[k]].smem = std::max(classes[at[k]].smem, place(k, at[k]));
    }
    for (const ResidentClass& c : classes) lists.insert(lists.end(), c.list.begin(), c.list.end());
    if (!lists.empty()) cudaMemcpyAsync(d_order, lists.data(), lists.size() * 4, cudaMemcpyHostToDevice, s);

    // The general kernel's vectors, and the diagonals of its systems when all
    // of them are banded; before anything is launched, so that x is untouched when
    // they cannot be had.
    std::vector<uint64_t> hbase;
    uint64_t total = 0;
    bool banded = false;
    auto general_memory = [&]() {
        banded = dia;
        for (uint32_t k : rest) banded = banded && hnd[k] > 0;
        total = 0;
        if (banded) {
            hbase.assign(nsys, 0);
            for (uint32_t k : rest) {
                hbase[k] = total;
                total += static_cast<uint64_t>(hnd[k]) * (off[k + 1] - off[k]);
            }
        }
        if (!test_fail("batched-alloc") && w.vecs.ensure(4 * vb + 256) == cudaSuccess) {
            if (banded && w.dia.ensure(total * sizeof(float) + 256) != cudaSuccess) {
                cudaGetLastError();
                banded = false;  // (their products from CSR then)
            }
            return true;
        }
        cudaGetLastError();
        return false;
    };
    if (!rest.empty() && !general_memory()) return clsparseOutOfResources;

    char* ob = static_cast<char*>(w.out.ptr);
    double* d_residual = reinterpret_cast<double*>(ob);
    int* d_iters = reinterpret_cast<int*>(ob + nsys * 8);
    int* d_converged = reinterpret_cast<int*>(ob + nsys * 12);
    const float* vals = dev_ptr<const float>(A->values, A->off_values);
    float* xp = dev_ptr<float>(x->values, x->off_values);
    const float* bp = dev_ptr<const float>(b->values, b->off_values);

    bool failed = false, no_memory = false;
    size_t forked = 0;
    if (!lists.empty()) {
        // each class on a stream of its own, after what the caller's stream holds
        size_t used = 0;
        for (const ResidentClass& c : classes) used += c.list.empty() ? 0 : 1;
        if (!ensure_streams(w, used) || cudaEventRecord(w.begin, s) != cudaSuccess) {
            cudaGetLastError();
            return clsparseOutOfResources;
        }
        ResidentArgs ra{vals, cols, rp,    xp,      bp,         d_off,       d_order,
                        doffs, dnd, d_iters, d_residual, d_converged, solverControl->maxIters,
                        solverControl->relativeTolerance};
        std::vector<uint32_t> refused;
        for (const ResidentClass& c : classes) {
            if (c.list.empty()) continue;
            cudaStream_t cs = w.streams[forked];
            failed |= cudaStreamWaitEvent(cs, w.begin, 0) != cudaSuccess;
            const cudaError_t e = failed || test_fail("batched-launch") ? cudaErrorLaunchOutOfResources
                                  : c.threads == kResWide               ? launch_resident<kResWide>(ra, c, cs)
                                                                        : launch_resident<kResSmall>(ra, c, cs);
            if (e != cudaSuccess) {
                cudaGetLastError();
                refused.insert(refused.end(), c.list.begin(), c.list.end());
            }
            failed |= cudaEventRecord(w.ends[forked], cs) != cudaSuccess;
            ++forked;
            ra.list += c.list.size();
            if (failed) break;
        }
        // systems whose launch was not taken: the general kernel's too
        if (!refused.empty() && !failed) {
            rest.insert(rest.begin(), refused.begin(), refused.end());
            no_memory = !general_memory();
        }
    }
    failed |= no_memory;
    if (!rest.empty() && !failed) {
        const uint32_t nrest = static_cast<uint32_t>(rest.size());
        cudaMemcpyAsync(d_rest, rest.data(), rest.size() * 4, cudaMemcpyHostToDevice, s);
        BatchArgs a;
        std::memset(&a, 0, sizeof(a));
        if (banded) {
            cudaMemcpyAsync(dbase, hbase.data(), nsys * 8, cudaMemcpyHostToDevice, s);
            cudaMemsetAsync(w.dia.ptr, 0, total * sizeof(float), s);
            batch_dia_fill_kernel<<<nrest, 256, 0, s>>>(rp, cols, vals, d_off, d_rest, doffs, dnd, dbase,
                                                        static_cast<float*>(w.dia.ptr));
            a.dvals = static_cast<const float*>(w.dia.ptr);
            a.dbase = dbase;
            a.doffs = doffs;
            a.dnd = dnd;
        }
        a.vals = vals;
        a.cols = cols;
        a.rp = rp;
        a.x = xp;
        a.b = bp;
        char* vbase = static_cast<char*>(w.vecs.ptr);
        a.r = reinterpret_cast<float*>(vbase);
        a.p = reinterpret_cast<float*>(vbase + vb);
        a.q = reinterpret_cast<float*>(vbase + 2 * vb);
        a.invd = reinterpret_cast<float*>(vbase + 3 * vb);
        a.off = d_off;
        a.order = d_rest;
        a.lanes = d_lanes;
        a.counter = d_counter;
        a.residual = d_residual;
        a.iters = d_iters;
        a.converged = d_converged;
        a.nsys = nrest;
        a.max_iters = solverControl->maxIters;
        a.tol = solverControl->relativeTolerance;
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_cg_kernel, kThreads, 0);
        const uint32_t grid = std::min(static_cast<uint32_t>(control->sm_count * std::max(per_sm, 1)), nrest);
        cudaMemsetAsync(d_counter, 0, 16, s);
        batched_cg_kernel<<<grid, kThreads, 0, s>>>(a);
        failed |= cudaGetLastError() != cudaSuccess;
    }
    for (size_t k = 0; k < forked; ++k) failed |= cudaStreamWaitEvent(s, w.ends[k], 0) != cudaSuccess;
    if (failed) {
        // nothing of this call stays in flight on the buffers
        cudaGetLastError();
        for (size_t k = 0; k < forked; ++k) cudaStreamSynchronize(w.streams[k]);
        cudaStreamSynchronize(s);
        return no_memory ? clsparseOutOfResources : clsparseInvalidKernelExecution;
    }

    std::vector<double> res(nsys);
    std::vector<int> its(nsys), conv(nsys);
    cudaMemcpyAsync(res.data(), d_residual, nsys * 8, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(its.data(), d_iters, nsys * 4, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(conv.data(), d_converged, nsys * 4, cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return clsparseInvalidKernelExecution;
    if (control->event) cudaEventRecord(control->event, s);
    int nconv = 0, maxit = 0;
    double worst = 0.0;
    for (uint32_t k = 0; k < nsys; ++k) {
        nconv += conv[k];
        maxit = std::max(maxit, its[k]);
        worst = std::max(worst, res[k]);
        if (result && result->iterations) result->iterations[k] = its[k];
        if (result && result->residuals) result->residuals[k] = res[k];
    }
    if (result) {
        result->systemsConverged = nconv;
        result->maxIterations = maxit;
        result->worstResidual = worst;
    }
    solverControl->nIters = maxit;
    solverControl->currentResidual = worst;
    return clsparseSuccess;
}

}  // extern "C"
