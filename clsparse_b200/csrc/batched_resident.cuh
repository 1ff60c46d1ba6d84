// Batched Jacobi-CG with a system held on chip: the kernel clsparseScsrcgBatched
// runs for every banded system that fits (batched.cu chooses).
//
// One system is solved by a cluster of C CTAs (C = 1, 2, 4 or 8), CTA c owning
// rows [c m, (c + 1) m), m = ceil(n / C). For the whole solve
//   x, r, q and D^-1 live in registers (row i of the CTA's rows in thread
//     i % NT, at index i / NT),
//   p and the values of the diagonals live in shared memory, p with the
//     neighbouring CTAs' rows its stencil reaches (the halo) beside it,
// so an iteration moves nothing through L2: two CTA- or cluster-wide
// exchanges of partial sums are left. The halo needs no exchange of its own:
// before the second exchange each CTA stores z = D^-1 r of its first and last
// rows into its neighbours' shared memory, and behind it every CTA updates its
// own copy of the neighbours' p from them (the same operations on the same
// values as in the owning CTA).
//
// Arithmetic as in the general kernel of batched.cu: FP32 vectors, products in
// increasing column order with FMAs, sums of products in FP64 (over threads,
// warps and CTAs in a fixed order), the true residual b - A x in FP64.
//
// What bounds it: shared-memory reads (about 18 words per row and iteration),
// then the two exchanges. 512 threads with 14 rows each: 7168 rows a CTA, what
// the diagonals of a seven-point stencil leave room for; systems of up to 1792
// rows run on 128 threads, three CTAs per SM.
//
// Measured (1024 stencil systems of 500 to 50,000 rows, 10.9 M rows, one
// call): 98.4 ms in the general kernel, bound by its largest systems (190 us
// an iteration for 50,000 rows on one CTA from L2); 25.0 ms here, the same
// iterates bit for bit.
#pragma once

#include <cooperative_groups.h>

#include "device_common.cuh"

namespace clsp {
namespace {

struct ResidentArgs {
    const float* vals;
    const uint32_t* cols;
    const uint32_t* rp;
    float* x;
    const float* b;
    const uint32_t* off;      // row offsets of the systems
    const uint32_t* list;     // systems of this launch, largest first
    const int32_t* doffs;     // column offsets of system s at s * kBatchDiags, increasing
    const uint8_t* dnd;       // their number
    int* iters;
    double* residual;
    int* converged;
    int max_iters;
    double tol;
};

constexpr int kMaxCluster = 8;
// Rows per thread: x, r, q and D^-1 take four registers each.
constexpr int kResRows = 14;

// Diagonals as the kernel stores them: the next size it is built for.
__host__ __device__ constexpr int resident_diags(int nd) { return nd <= 5 ? 5 : (nd <= 7 ? 7 : kBatchDiags); }

// Dynamic shared memory of a CTA with m rows, nd diagonals reaching `lo` rows
// down and `hi` up.
__host__ __device__ inline size_t resident_smem(size_t m, int nd, size_t lo, size_t hi) {
    return 4 * (m * (resident_diags(nd) + 1) + 2 * (lo + hi));
}

template <int NT>
struct ResidentCta {
    static constexpr int kWarps = NT / 32;
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    uint32_t C, rank;
    double (*red)[3][kMaxCluster * kWarps];  // [parity][value][CTA and warp]
    uint32_t epoch = 0;

    __device__ __forceinline__ void sync() {
        if (C == 1)
            __syncthreads();
        else
            cluster.sync();
    }
    // Sums K values over the cluster, the result in every thread and the same
    // bit for bit in every CTA; also a barrier of the cluster. Two buffers: a
    // slot is written again two exchanges later, when every warp has read it.
    template <int K>
    __device__ __forceinline__ void exchange(const double (&v)[K], double (&out)[K]) {
        const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        auto& buf = red[epoch & 1];
        ++epoch;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double w = dev::warp_sum(v[k]);
            if (lane < C) {
                double* slot = &buf[k][rank * kWarps + warp];
                if (C > 1) slot = cluster.map_shared_rank(slot, lane);
                *slot = w;
            }
        }
        sync();
        const uint32_t count = C * kWarps;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            double s = 0.0;
            for (uint32_t i = lane; i < count; i += 32) s += buf[k][i];
            out[k] = dev::warp_sum(s);
        }
    }
};

template <int NT, int ND>
__device__ __forceinline__ void resident_solve(const ResidentArgs& a, ResidentCta<NT>& cta, uint32_t s,
                                               const int32_t* soff, int nd) {
    constexpr int R = kResRows;
    extern __shared__ float smem[];
    const uint32_t r0 = a.off[s], n = a.off[s + 1] - r0;
    const uint32_t m = (n + cta.C - 1) / cta.C;                       // rows of a full CTA
    const uint32_t first = min(n, cta.rank * m);
    const uint32_t mine = min(m, n - first);                          // rows of this CTA
    const uint32_t base = r0 + first;                                 // its first row of A
    const uint32_t lo = soff[0] < 0 ? static_cast<uint32_t>(-soff[0]) : 0u;
    const uint32_t hi = soff[nd - 1] > 0 ? static_cast<uint32_t>(soff[nd - 1]) : 0u;
    float* P = smem;                // lo rows below, m own, hi above
    float* ZL = P + lo + m + hi;    // z of the lo rows below
    float* ZH = ZL + lo;            // z of the hi rows above
    float* DV = ZH + hi;            // diagonal d of own row i at d * m + i
    const uint32_t t = threadIdx.x;

    // ---- the system from CSR: diagonals, D^-1, x
    const uint32_t words = lo + m + hi + lo + hi + ND * m;
    for (uint32_t i = t; i < words; i += NT) smem[i] = 0.f;
    cta.sync();  // (of the cluster: the neighbours' stores come after every CTA's zeros)
    float x[R], r[R], q[R], inv[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const uint32_t i = t + k * NT;
        x[k] = r[k] = q[k] = inv[k] = 0.f;
        if (i < mine) {
            float diag = 0.f;
            int d = 0;
            const uint32_t ke = a.rp[base + i + 1];
            for (uint32_t e = a.rp[base + i]; e < ke; ++e) {
                const int32_t o = static_cast<int32_t>(static_cast<int64_t>(a.cols[e]) -
                                                       static_cast<int64_t>(base + i));
                const float v = a.vals[e];
                while (d < nd && soff[d] < o) ++d;  // columns increase, so d only moves forward
                if (d < nd && soff[d] == o) DV[d * m + i] = v;
                if (o == 0) diag = v;
            }
            inv[k] = diag != 0.f ? 1.f / diag : 1.f;
            x[k] = a.x[base + i];
        }
    }

    // This thread's first row in P, in P shifted by each diagonal's offset
    // (padding: offset 0, zero values) and in the diagonals; row k of the
    // thread is k * NT behind, a constant.
    // (Signed indices into shared memory: k * NT becomes an immediate.)
    const int own = static_cast<int>(lo + t);
    int pd[ND], dv[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        pd[d] = own + (d < nd ? soff[d] : 0);
        dv[d] = static_cast<int>(DV - smem) + d * static_cast<int>(m) + static_cast<int>(t);
    }
    const float* const bown = a.b + base + t;
    // Stores v, row i of this CTA, where the neighbours keep it: the last lo
    // rows below the next CTA's, the first hi above the previous one's.
    // (Pointers already moved by this thread's first row: row k is k * NT on.)
    float* next_lo = nullptr;
    float* prev_hi = nullptr;
    float* next_zl = nullptr;
    float* prev_zh = nullptr;
    const int to_next = static_cast<int>(lo + t) - static_cast<int>(m);
    if (cta.C > 1) {
        if (cta.rank + 1 < cta.C) {
            next_lo = cta.cluster.map_shared_rank(P, cta.rank + 1) + to_next;
            next_zl = cta.cluster.map_shared_rank(ZL, cta.rank + 1) + to_next;
        }
        if (cta.rank > 0) {
            prev_hi = cta.cluster.map_shared_rank(P + lo + m, cta.rank - 1) + t;
            prev_zh = cta.cluster.map_shared_rank(ZH, cta.rank - 1) + t;
        }
    }
    const int hi_t = static_cast<int>(hi) - static_cast<int>(t);
    auto push = [&](float* next, float* prev, int k, float v) {
        if (next && to_next + k * NT >= 0) next[k * NT] = v;  // (a next CTA with rows: this one is full)
        if (prev && k * NT < hi_t) prev[k * NT] = v;
    };
    // r = b - A x in FP64, kept in FP32; sums of r^2 and b^2.
    auto true_residual = [&](double (&tot)[2]) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint32_t i = t + k * NT;
            if (i < mine) {
                smem[own + k * NT] = x[k];
                push(next_lo, prev_hi, k, x[k]);
            }
        }
        cta.sync();
        double acc[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint32_t i = t + k * NT;
            if (i < mine) {
                double sum = 0.0;
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    sum = fma(static_cast<double>(smem[dv[d] + k * NT]), static_cast<double>(smem[pd[d] + k * NT]), sum);
                const double bi = bown[k * NT];
                const double ri = bi - sum;
                r[k] = static_cast<float>(ri);
                acc[0] += ri * ri;
                acc[1] += bi * bi;
            }
        }
        cta.template exchange<2>(acc, tot);
    };

    double tot[2];
    true_residual(tot);
    double rr = tot[0];
    const double bnorm = sqrt(tot[1]);
    int it = 0;
    bool ok = bnorm == 0.0 || sqrt(rr) <= a.tol * bnorm;
    double res64 = bnorm == 0.0 ? 0.0 : sqrt(rr) / bnorm;
    while (!ok && it < a.max_iters) {
        // (re)start: z = M r, p = z, rz = <r, z>
        double one[1] = {0.0}, sum1[1];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint32_t i = t + k * NT;
            if (i < mine) {
                const float z = r[k] * inv[k];
                smem[own + k * NT] = z;
                push(next_lo, prev_hi, k, z);
                one[0] += static_cast<double>(r[k]) * z;
            }
        }
        cta.template exchange<1>(one, sum1);
        double rz = sum1[0];
        for (;;) {
            // A: q = A p, <p, q>
            one[0] = 0.0;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const uint32_t i = t + k * NT;
                if (i < mine) {
                    float sum = 0.f;
#pragma unroll
                    for (int d = 0; d < ND; ++d) sum = fmaf(smem[dv[d] + k * NT], smem[pd[d] + k * NT], sum);
                    q[k] = sum;
                    one[0] += static_cast<double>(smem[own + k * NT]) * sum;
                }
            }
            cta.template exchange<1>(one, sum1);
            const double pq = sum1[0];
            const float alpha = static_cast<float>(rz / pq);
            // B: x, r, z of the edge rows to the neighbours; <r, z>, <r, r>
            double acc[2] = {0.0, 0.0}, sums[2];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const uint32_t i = t + k * NT;
                if (i < mine) {
                    x[k] = fmaf(alpha, smem[own + k * NT], x[k]);
                    r[k] = fmaf(-alpha, q[k], r[k]);
                    const float z = r[k] * inv[k];
                    push(next_zl, prev_zh, k, z);
                    acc[0] += static_cast<double>(r[k]) * z;
                    acc[1] += static_cast<double>(r[k]) * r[k];
                }
            }
            cta.template exchange<2>(acc, sums);
            ++it;
            if (!(pq > 0.0) || !isfinite(sums[0])) break;  // breakdown: fall through to the FP64 check
            if (sqrt(sums[1]) <= a.tol * bnorm) break;
            if (it >= a.max_iters) break;  // (here, not after C: the neighbours' halo is then still in use)
            const float beta = static_cast<float>(sums[0] / rz);
            rz = sums[0];
            // C: p = z + beta p, of the own rows and the halo
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const uint32_t i = t + k * NT;
                if (i < mine) smem[own + k * NT] = fmaf(beta, smem[own + k * NT], r[k] * inv[k]);
            }
            if (cta.C > 1) {
                for (uint32_t i = t; i < lo; i += NT) P[i] = fmaf(beta, P[i], ZL[i]);
                for (uint32_t i = t; i < hi; i += NT) P[lo + m + i] = fmaf(beta, P[lo + m + i], ZH[i]);
            }
            __syncthreads();
        }
        true_residual(tot);
        res64 = sqrt(tot[0]) / bnorm;
        ok = res64 <= a.tol;
        if (!isfinite(res64)) break;
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const uint32_t i = t + k * NT;
        if (i < mine) a.x[base + i] = x[k];
    }
    if (cta.rank == 0 && t == 0) {
        a.iters[s] = it;
        a.residual[s] = res64;
        a.converged[s] = ok ? 1 : 0;
    }
}

// Cluster g of the launch solves system list[g].
template <int NT>
__global__ void __launch_bounds__(NT, NT == 128 ? 3 : 1) batched_resident_kernel(ResidentArgs a) {
    __shared__ double red[2][3][kMaxCluster * (NT / 32)];
    __shared__ int32_t soff[kBatchDiags];
    ResidentCta<NT> cta;
    cta.C = cta.cluster.num_blocks();
    cta.rank = cta.cluster.block_rank();
    cta.red = red;
    const uint32_t s = a.list[blockIdx.x / cta.C];
    const int nd = a.dnd[s];
    if (threadIdx.x < kBatchDiags) soff[threadIdx.x] = a.doffs[s * kBatchDiags + threadIdx.x];
    __syncthreads();
    if (nd <= 5)
        resident_solve<NT, 5>(a, cta, s, soff, nd);
    else if (nd <= 7)
        resident_solve<NT, 7>(a, cta, s, soff, nd);
    else
        resident_solve<NT, kBatchDiags>(a, cta, s, soff, nd);
    cta.sync();  // no CTA leaves while another may still store into its shared memory
}

}  // namespace
}  // namespace clsp
