// The banded solves with the vectors held on chip.
//
// CTA c of the cooperative launch owns rows [c n / G, (c + 1) n / G) for the
// whole solve, row i of its rows in thread i % NT at index i / NT:
//   registers      x, r, q = A p (and D^-1 where they suffice)
//   shared memory  p of the own rows and of the rows its stencil reaches on
//                  either side (the halo); D^-1 and as many diagonals of A as
//                  fit, the others stay in L2
// Per iteration (CG): A) q = A p, <p,q>, exchange -> alpha; B) x, r, z = M r,
// <r,z>, ||r||, exchange -> beta; C) p = z + beta p. The halo's p needs no
// exchange of its own: in B a row another CTA reaches publishes its z (a tagged
// word, grid_words.cuh), and in C every CTA forms its own copy of the halo's
// p from it, the same operations on the same values as in the owning CTA.
// Where a CTA reaches further than its neighbours' words are worth (a halo of
// more rows than it owns), z goes out as a plain vector ordered by the exchange;
// wider still (halo_pays), the solve streams.
//
// What bounds it on small systems: latency, about half of it the two exchanges
// (1.0 us each bare at 148 CTAs, see kSlotWords) and the CTA-wide sums before
// them, the rest shared-memory reads and dependent FP64 operations with 16
// warps. On large ones the diagonals that stay in L2. Measured per iteration
// (streamed through L2 / here; FP64): 512^2 five-point 11.1 / 6.0 us, 1000^2
// 24.1 / 16.5, 64^3 seven-point 11.5 / 8.5, 100^3 33.6 / 29.2; FP32 512^2 10.2 /
// 5.3; BiCGStab on 300^2 18.3 / 8.8; the learned factor's inner iteration on
// 1024^2 19.6 / 13.
#include <algorithm>
#include <initializer_list>
#include <limits>

#include "device_common.cuh"
#include "dia.h"
#include "dia_resident.h"
#include "dia_rows.cuh"
#include "grid_words.cuh"
#include "internal.h"
#include "solver_state.cuh"

namespace clsp {
namespace {

// Threads of a CTA, one CTA per SM: 128 registers a thread. 14 rows of x, r and q
// take 84 of them in FP64, and those CG kernels (more than 2048 rows a CTA: from
// 303,105 rows on 148 SMs) store 200 to 340 bytes of others to the stack; FP64
// BiCGStab with four rows stores up to 184, FP32 kernels at most 64. (1024 threads
// of 64 registers measured slower in FP32: 6.6 us an iteration instead of 5.3 on
// 512^2, no change on 100^3.)
constexpr int kResThreads = 512;
constexpr int kFewRows = kResidentBicgRows / kResThreads;   // rows per thread the kernels are built for: 4,
constexpr int kManyRows = kResidentCgRows / kResThreads;    // 14

// Register arrays of R rows: D^-1 is the fourth when it fits beside x, r, q.
template <typename T, int R>
constexpr bool inv_in_regs() {
    return R * sizeof(T) <= 56;
}

// Rows of this CTA that a CSR-Adaptive block reduces over g > 1 lanes (a few,
// in the last block as a rule): which diagonals each holds, from CSR once, so
// that an iteration forms them from the diagonals and p at hand, without
// dependent global loads on the one CTA that has them.
constexpr uint32_t kLaneRows = 1024;
struct LaneTable {
    uint16_t mask[kLaneRows];
    uint32_t count;  // lane rows of the CTA
};

template <typename Args>
__device__ __forceinline__ void build_lane_table(const Args& a, uint32_t r0, uint32_t r1, LaneTable& tab) {
    uint32_t base = 0;
    for (int l = 0; l < a.nlanes; ++l) {
        const uint32_t b = max(r0, a.lanes[l].r0), e = min(r1, a.lanes[l].r1);
        if (b >= e) continue;
        for (uint32_t row = b + threadIdx.x; row < e; row += blockDim.x) {
            uint32_t m = 0;
            for (uint32_t k = a.rp[row]; k < a.rp[row + 1]; ++k) {
                const int32_t o = static_cast<int32_t>(static_cast<int64_t>(a.cols[k]) - static_cast<int64_t>(row));
                for (int d = 0; d < a.nd_real; ++d)
                    if (a.A.off[d] == o) m |= 1u << d;
            }
            if (base + row - b < kLaneRows) tab.mask[base + row - b] = static_cast<uint16_t>(m);
        }
        base += e - b;
    }
    if (threadIdx.x == 0) tab.count = base;
}

// Row `row` of the product in its block's lane order (csr_row_lanes) if it is a
// lane row: val(d) and vec(d) are its d-th diagonal's entry and the vector's.
template <typename T, int ND, typename Args, typename VF, typename XF, typename CF>
__device__ __forceinline__ bool lane_row(const Args& a, uint32_t r0, uint32_t r1, uint32_t row, const LaneTable& tab,
                                         VF val, XF vec, CF from_csr, T& out) {
    uint32_t base = 0;
    for (int l = 0; l < a.nlanes; ++l) {
        const uint32_t b = max(r0, a.lanes[l].r0), e = min(r1, a.lanes[l].r1);
        if (b >= e) continue;
        if (row >= b && row < e) {
            if (tab.count > kLaneRows) {
                out = from_csr(a.lanes[l].g);
                return true;
            }
            const uint32_t m = tab.mask[base + row - b];
            const uint32_t g = min(a.lanes[l].g, 16u);
            T v[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = T(0);
            uint32_t k = 0;
#pragma unroll
            for (int d = 0; d < ND; ++d)
                if (m >> d & 1u) {
                    const T prod = mul_rn(val(d), vec(d));
#pragma unroll
                    for (int w = 0; w < 16; ++w)
                        if ((k & (g - 1)) == static_cast<uint32_t>(w)) v[w] = add_rn(v[w], prod);
                    ++k;
                }
#pragma unroll
            for (int off = 8; off > 0; off >>= 1)
                if (static_cast<uint32_t>(off) < g) {
#pragma unroll
                    for (int w = 0; w < 8; ++w)
                        if (w < off) v[w] = add_rn(v[w], v[w + off]);
                }
            out = v[0];
            return true;
        }
        base += e - b;
    }
    return false;
}

// The kept diagonals into shared memory, and this thread's pointer to each
// diagonal's value at its first row (shared memory or L2).
template <int NT, int ND, typename V>
__device__ __forceinline__ void keep_diagonals(const DiaMat<V>& A, const ResidentPlan& pl, uint32_t n, uint32_t r0,
                                               uint32_t mine, V* kept, const V* (&dv)[ND]) {
    const uint32_t t = threadIdx.x;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const V* src = A.vals + static_cast<size_t>(d) * n + r0;
        dv[d] = src + t;
        if (pl.at[d] >= 0) {
            V* dst = kept + pl.at[d];
            const int first = -pl.lead[d];
            if (pl.lead[d] >= 0)
                for (int i = first + static_cast<int>(t); i < static_cast<int>(mine); i += NT)
                    dst[i] = i >= 0 || static_cast<uint32_t>(-i) <= r0 ? src[i] : V(0.f);
            dv[d] = dst + t;
        }
    }
}

// Words of diagonals a thread's rows may hold in registers, where its vectors
// leave room: the product then reads only the vector from shared memory, whose
// bandwidth bounds it. BiCGStab on 90,000 rows (two rows a thread, FP64, five
// diagonals: 20 words) 9.9 -> 8.8 us an iteration; with four rows a thread (40
// words) the CG spilled: 512^2 6.1 -> 6.9.
constexpr int kDiagRegs = 20;
template <typename T, int ND, int R>
constexpr bool diags_in_regs() {
    return ND * R * sizeof(T) / 4 <= kDiagRegs;
}

template <typename T>
struct DiaCgResidentArgs {
    DiaCgArgs<T> a;
    ResidentPlan plan;
    WordSync words;
};

// The drop-in CG (dia_cg_ref_kernel's arithmetic and bookkeeping) with its
// vectors on chip.
template <typename T, int ND, int R>
__global__ void __launch_bounds__(kResThreads, 1) dia_cg_resident_kernel(const __grid_constant__ DiaCgResidentArgs<T> args) {
    constexpr int NT = kResThreads;
    constexpr bool INV = inv_in_regs<T, R>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ WordSmem<NT> sm;
    __shared__ LaneTable tab;
    const DiaCgArgs<T>& a = args.a;
    const ResidentPlan& pl = args.plan;
    const WordSync& g = args.words;
    const uint32_t n = a.n, t = threadIdx.x;
    const uint32_t r0 = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x) * n / gridDim.x);
    const uint32_t r1 = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) + 1) * n / gridDim.x);
    const uint32_t mine = r1 - r0;
    const HaloRows halo{r0, r1, min(pl.lo, r0), min(pl.hi, n - r1)};
    const bool lead = blockIdx.x == 0 && t == 0;
    const bool jacobi = a.invD != nullptr;
    uint32_t epoch = 0;
    T* P = reinterpret_cast<T*>(smem_raw) + pl.lo;              // row i of the CTA at P[i], halo on both sides
    T* next = P + pl.mcap + pl.hi;                              // arrays kept in shared memory
    T* inv_s = next;
    if (pl.inv_smem) next += pl.mcap;
    const T* dv[ND];                                            // diagonal d of this thread's first row
    keep_diagonals<NT, ND>(a.A, pl, n, r0, mine, next, dv);
    constexpr bool DREG = diags_in_regs<T, ND, R>();
    const T* invp = (pl.inv_smem ? inv_s : a.invD + r0) + t;    // D^-1 where it is not in registers
    const T* pd[ND];                                            // P shifted by each offset
#pragma unroll
    for (int d = 0; d < ND; ++d) pd[d] = P + t + a.A.off[d];
    T* const own = P + t;
    const int hi_t = static_cast<int>(pl.hi) - static_cast<int>(t);                         // k NT < hi_t: an edge row
    const int lo_t = static_cast<int>(mine) - static_cast<int>(pl.lo) - static_cast<int>(t);  // k NT >= lo_t: too
    T* const zg = a.z + r0 + t;
    const uint32_t row_t = r0 + t;
    auto publish = [&](int k, T z) {
        if (pl.words) {
            if (k * NT < hi_t || k * NT >= lo_t) st_halo(g, row_t + k * NT, epoch + 1, z);
        } else if (k * NT < hi_t || k * NT >= lo_t) {
            zg[k * NT] = z;
        }
    };
    const DiaCgState in = *a.st;
    const int l2 = in.l2;
    auto term = [l2](T v) {
        const double d = static_cast<double>(v);
        return l2 ? mul_rn(d, d) : fabs(d);
    };
    auto finish_norm = [l2](double s) { return l2 ? sqrt(s) : s; };

    if (t == 0) sm.bad = 0;
    build_lane_table(a, r0, r1, tab);
    for (uint32_t i = t; i < pl.lo + pl.mcap + pl.hi; i += NT) (P - pl.lo)[i] = T(0);
    __syncthreads();

    // ---- prologue: r = b - A x, z = M r, p = z
    T av[DREG ? R : 1][ND];
    if constexpr (DREG) {
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int d = 0; d < ND; ++d)
                av[k][d] = t + k * NT < mine ? __ldg(a.A.vals + static_cast<size_t>(d) * n + row_t + k * NT) : T(0);
    }
    T x[R], r[R], q[R];
    T inv[INV ? R : 1];
    inv[0] = T(0);
    auto inv_of = [&](int k) {
        if constexpr (INV)
            return inv[k];
        else
            return invp[k * NT];
    };
    HaloTake<NT, T> take;
    auto prefetch = [&] {
        if (pl.words) take.begin(g, halo, epoch);
    };
    double tot0[4];
    {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
        for (uint32_t i = t; i < mine; i += NT) {
            const T y = cg_row<ND, false>(a, r0 + i, [&](uint32_t j) { return a.x[j]; });
            const T bi = __ldg(a.b + r0 + i);
            P[i] = add_rn(bi, -y);
            acc[0] = add_rn(acc[0], term(bi));
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint32_t i = t + k * NT;
            x[k] = r[k] = q[k] = T(0);
            if constexpr (INV) inv[k] = T(0);
            if (i < mine) {
                x[k] = a.x[r0 + i];
                r[k] = own[k * NT];
                T z = r[k];
                if (jacobi) {
                    const T d = __ldg(a.A.vals + static_cast<size_t>(a.d0) * n + r0 + i);
                    const T v = T(1) / d;
                    if constexpr (INV)
                        inv[k] = v;
                    else
                        const_cast<T*>(invp)[k * NT] = v;
                    z = mul_rn(r[k], v);
                    acc[3] += d == T(0) ? 1.0 : 0.0;
                }
                own[k * NT] = z;
                publish(k, z);
                acc[1] = add_rn(acc[1], term(r[k]));
                acc[2] = add_rn(acc[2], mul_rn(static_cast<double>(r[k]), static_cast<double>(z)));
            }
        }
        if (!words_exchange<4>(g, epoch, acc, tot0, sm, !pl.words, prefetch)) goto fail;
    }
    if (tot0[3] > 0.0) {
        if (lead) a.st->zero_diag = 1;
        return;
    }
    {
        // body(place in P, z) over the halo, z as published before the last exchange
        auto each_halo = [&](auto body) {
            if (pl.words) {
                take.end(g, halo, epoch, sm, [&](uint32_t j, T z) { body(halo.at(j), z); });
            } else {
                const uint32_t total = halo.count();
                for (uint32_t j0 = t; j0 < total; j0 += 4 * NT) {
                    T z[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j0 + u * NT < total) z[u] = __ldcg(a.z + halo.row(j0 + u * NT));
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j0 + u * NT < total) body(halo.at(j0 + u * NT), z[u]);
                }
            }
        };
        const T norm_b = static_cast<T>(finish_norm(tot0[0]));
        if (norm_b == T(0)) {
            for (uint32_t i = t; i < mine; i += NT) a.x[r0 + i] = __ldg(a.b + r0 + i);
            if (lead) {
                a.st->zero_b = 1;
                a.st->n_iters = 0;
            }
            return;
        }
        const T norm_r0 = static_cast<T>(finish_norm(tot0[1]));
        const double init_res = static_cast<double>(norm_r0 / norm_b);
        auto finished = [&](double res, int n_iters) {
            return res <= in.rel_tol || res <= in.abs_tol * init_res || n_iters >= in.max_iters ||
                   (in.stop_nonfinite && !isfinite(res));
        };
        T rz = static_cast<T>(tot0[2]);
        double cur_res = init_res;
        int n_iters = 0, status = 0;
        bool done = finished(init_res, in.n_iters_in);
        if (!done) {
            each_halo([&](int at, T z) { P[at] = z; });
            __syncthreads();
            if (sm.bad) goto fail;
        }
        for (int k = 0; !done; ++k) {
            // ---- A: q = A p, <q, p>
            double pq[1] = {0.0}, tq[1];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    T s = T(0);
#pragma unroll
                    for (int d = 0; d < ND; ++d)
                        s = add_rn(s, mul_rn(DREG ? av[DREG ? i : 0][d] : dv[d][i * NT], pd[d][i * NT]));
                    q[i] = s;
                }
            if (tab.count > 0) {
#pragma unroll 1
                for (int i = 0; i < R; ++i) {
                    const uint32_t row = row_t + i * NT;
                    T v = T(0);
                    if (row < r1 && lane_row<T, ND>(
                                        a, r0, r1, row, tab, [&](int d) { return dv[d][i * NT]; },
                                        [&](int d) { return pd[d][i * NT]; },
                                        [&](uint32_t lanes) {
                                            return csr_row_lanes(a.rp, a.cols, a.vals, row, lanes, [&](uint32_t j) {
                                                return P[static_cast<int>(j) - static_cast<int>(r0)];
                                            });
                                        },
                                        v)) {
#pragma unroll
                        for (int w = 0; w < R; ++w) q[w] = w == i ? v : q[w];
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine)
                    pq[0] = add_rn(pq[0], mul_rn(static_cast<double>(q[i]), static_cast<double>(own[i * NT])));
            if (!words_exchange<1>(g, epoch, pq, tq, sm, false)) goto fail;
            const T yp = static_cast<T>(tq[0]);
            const T alpha = rz / yp;
            if (!(yp > T(0))) status |= kStatusCurvature;
            // ---- B: x += alpha p, r -= alpha q, z = M r; <r,z>, ||r||
            double acc[2] = {0.0, 0.0}, tb[2];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    x[i] = add_rn(x[i], mul_rn(alpha, own[i * NT]));
                    r[i] = add_rn(r[i], -mul_rn(alpha, q[i]));
                    const T z = jacobi ? mul_rn(r[i], inv_of(i)) : r[i];
                    publish(i, z);
                    acc[0] = add_rn(acc[0], mul_rn(static_cast<double>(r[i]), static_cast<double>(z)));
                    acc[1] = add_rn(acc[1], term(r[i]));
                }
            if (!words_exchange<2>(g, epoch, acc, tb, sm, !pl.words, prefetch)) goto fail;
            const T rz_old = rz;
            rz = static_cast<T>(tb[0]);
            const T beta = rz / rz_old;
            const T res = static_cast<T>(finish_norm(tb[1])) / norm_b;
            n_iters = k;
            cur_res = static_cast<double>(res);
            if (!isfinite(cur_res)) status |= kStatusNonFinite;
            done = finished(cur_res, n_iters);
            if (done) break;
            // ---- C: p = z + beta p, own rows and halo
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    const T z = jacobi ? mul_rn(r[i], inv_of(i)) : r[i];
                    own[i * NT] = add_rn(z, mul_rn(beta, own[i * NT]));
                }
            each_halo([&](int at, T z) { P[at] = add_rn(z, mul_rn(beta, P[at])); });
            __syncthreads();
            if (sm.bad) goto fail;
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (t + i * NT < mine) a.x[r0 + t + i * NT] = x[i];
        if (lead) {
            a.st->n_iters = n_iters;
            a.st->init_res = init_res;
            a.st->cur_res = cur_res;
            atomicOr(&a.st->status, status);
        }
        return;
    }
fail:
    if (t == 0) atomicOr(&a.st->status, kStatusBarrierTimeout);
}

template <typename T>
struct DiaBicgResidentArgs {
    DiaBicgArgs<T> a;
    ResidentPlan plan;
    WordSync words;            // halo words of r
    unsigned long long* amp;   // halo words of A M p
};

// The drop-in BiCGStab (dia_bicg_ref_kernel's arithmetic and bookkeeping) with
// its vectors on chip: x, r, r*, p, A M p, A M s and D^-1 in registers, M p
// (then M s) in shared memory with its halo. The halo's M p and M s are formed
// from its r, p and A M p, of which every CTA keeps its own copies: A M p of
// the edge rows goes out with the first exchange of an iteration, r with the
// third, the second carries sums alone.
template <typename T, int ND, int R>
__global__ void __launch_bounds__(kResThreads, 1)
    dia_bicg_resident_kernel(const __grid_constant__ DiaBicgResidentArgs<T> args) {
    constexpr int NT = kResThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ WordSmem<NT> sm;
    __shared__ LaneTable tab;
    const DiaBicgArgs<T>& a = args.a;
    const ResidentPlan& pl = args.plan;
    const WordSync& g = args.words;
    WordSync ga = g;
    ga.halo = args.amp;
    const uint32_t n = a.n, t = threadIdx.x;
    const uint32_t r0 = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x) * n / gridDim.x);
    const uint32_t r1 = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) + 1) * n / gridDim.x);
    const uint32_t mine = r1 - r0;
    const HaloRows halo{r0, r1, min(pl.lo, r0), min(pl.hi, n - r1)};
    const bool lead = blockIdx.x == 0 && t == 0;
    const bool jacobi = a.invD != nullptr;
    uint32_t epoch = 0;
    T* const V = reinterpret_cast<T*>(smem_raw) + pl.lo;
    const uint32_t nh = pl.lo + pl.hi;
    T* const Rh = V + pl.mcap + pl.hi;   // the halo's r, p, A M p and D^-1
    T* const Ph = Rh + nh;
    T* const Ah = Ph + nh;
    T* const Ih = Ah + nh;
    T* const res_s = Ih + nh;            // diagonals kept in shared memory
    const T* dv[ND];
    keep_diagonals<NT, ND>(a.A, pl, n, r0, mine, res_s, dv);
    constexpr bool DREG = diags_in_regs<T, ND, R>();
    const T* pd[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) pd[d] = V + t + a.A.off[d];
    T* const own = V + t;
    const int hi_t = static_cast<int>(pl.hi) - static_cast<int>(t);
    const int lo_t = static_cast<int>(mine) - static_cast<int>(pl.lo) - static_cast<int>(t);
    const uint32_t row_t = r0 + t;
    auto publish = [&](const WordSync& w, int k, T v) {
        if (k * NT < hi_t || k * NT >= lo_t) st_halo(w, row_t + k * NT, epoch + 1, v);
    };
    const DiaCgState in = *a.st;
    const int l2 = in.l2;
    auto term = [l2](T v) {
        const double d = static_cast<double>(v);
        return l2 ? mul_rn(d, d) : fabs(d);
    };
    auto finish_norm = [l2](double v) { return l2 ? sqrt(v) : v; };
    auto dot = [](T u, T v) { return mul_rn(static_cast<double>(u), static_cast<double>(v)); };
    HaloTake<NT, T> take;
    T av[DREG ? R : 1][ND];
    if constexpr (DREG) {
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
            for (int d = 0; d < ND; ++d)
                av[k][d] = t + k * NT < mine ? __ldg(a.A.vals + static_cast<size_t>(d) * n + row_t + k * NT) : T(0);
    }
    T x[R], r[R], rs[R], p[R], amp[R], ams[R], inv[R];
#pragma unroll
    for (int k = 0; k < R; ++k) inv[k] = T(1);
    auto apply_m = [&](T v, int k) { return jacobi ? mul_rn(v, inv[k]) : v; };
    // out = A V for the own rows
    auto product = [&](T (&out)[R]) {
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (t + i * NT < mine) {
                T s = T(0);
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    s = add_rn(s, mul_rn(DREG ? av[DREG ? i : 0][d] : dv[d][i * NT], pd[d][i * NT]));
                out[i] = s;
            }
        if (tab.count > 0) {
#pragma unroll 1
            for (int i = 0; i < R; ++i) {
                const uint32_t row = row_t + i * NT;
                T v = T(0);
                if (row < r1 && lane_row<T, ND>(
                                    a, r0, r1, row, tab, [&](int d) { return dv[d][i * NT]; },
                                    [&](int d) { return pd[d][i * NT]; },
                                    [&](uint32_t lanes) {
                                        return csr_row_lanes(a.rp, a.cols, a.vals, row, lanes, [&](uint32_t j) {
                                            return V[static_cast<int>(j) - static_cast<int>(r0)];
                                        });
                                    },
                                    v)) {
#pragma unroll
                    for (int w = 0; w < R; ++w) out[w] = w == i ? v : out[w];
                }
            }
        }
    };
    if (t == 0) sm.bad = 0;
    build_lane_table(a, r0, r1, tab);
    for (uint32_t i = t; i < nh + pl.mcap; i += NT) (V - pl.lo)[i] = T(0);
    for (uint32_t j = t; j < halo.count(); j += NT) {
        Ih[j] = jacobi ? T(1) / __ldg(a.A.vals + static_cast<size_t>(a.d0) * n + halo.row(j)) : T(1);
        Ph[j] = Ah[j] = T(0);
    }
    __syncthreads();

    // ---- prologue: r = b - A x, r* = r, p = r
    double tot0[4];
    {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
        for (uint32_t i = t; i < mine; i += NT) {
            const T y = cg_row<ND, false>(a, r0 + i, [&](uint32_t j) { return a.x[j]; });
            const T bi = __ldg(a.b + r0 + i);
            V[i] = add_rn(bi, -y);
            acc[0] = add_rn(acc[0], term(bi));
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            x[k] = r[k] = rs[k] = p[k] = amp[k] = ams[k] = T(0);
            if (t + k * NT < mine) {
                x[k] = a.x[row_t + k * NT];
                r[k] = rs[k] = p[k] = own[k * NT];
                if (jacobi) {
                    const T d = __ldg(a.A.vals + static_cast<size_t>(a.d0) * n + row_t + k * NT);
                    inv[k] = T(1) / d;
                    acc[3] += d == T(0) ? 1.0 : 0.0;
                }
                publish(g, k, r[k]);
                acc[1] = add_rn(acc[1], term(r[k]));
                acc[2] = add_rn(acc[2], dot(r[k], r[k]));
            }
        }
        if (!words_exchange<4>(g, epoch, acc, tot0, sm, false, [&] { take.begin(g, halo, epoch); })) goto fail;
    }
    if (tot0[3] > 0.0) {
        if (lead) a.st->zero_diag = 1;
        return;
    }
    {
        const T norm_b = static_cast<T>(finish_norm(tot0[0]));
        if (norm_b <= std::numeric_limits<T>::min()) {
            for (uint32_t i = t; i < mine; i += NT) a.x[r0 + i] = __ldg(a.b + r0 + i);
            if (lead) {
                a.st->zero_b = 1;
                a.st->n_iters = 0;
            }
            return;
        }
        const double init_res = static_cast<double>(static_cast<T>(finish_norm(tot0[1])) / norm_b);
        auto finished = [&](double res, int n_iters) {
            return res <= in.rel_tol || res <= in.abs_tol * init_res || n_iters >= in.max_iters ||
                   (in.stop_nonfinite && !isfinite(res));
        };
        T rsr_old = static_cast<T>(tot0[2]);
        T beta = T(0), omega = T(0);
        double cur_res = init_res;
        int n_iters = in.n_iters_in, status = 0;
        bool done = finished(init_res, n_iters);
        if (done) n_iters = 0;
        for (int k = 0; !done; ++k) {
            // ---- 1: p_k, M p_k, AMp_k = A M p_k, <r*, AMp_k>
            const T bw = mul_rn(beta, omega);
            take.end(g, halo, epoch, sm, [&](uint32_t j, T v) {
                const T pj = k == 0 ? v : add_rn(add_rn(v, mul_rn(beta, Ph[j])), -mul_rn(bw, Ah[j]));
                Rh[j] = v;
                Ph[j] = pj;
                V[halo.at(j)] = jacobi ? mul_rn(pj, Ih[j]) : pj;
            });
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    if (k > 0) p[i] = add_rn(add_rn(r[i], mul_rn(beta, p[i])), -mul_rn(bw, amp[i]));
                    own[i * NT] = apply_m(p[i], i);
                }
            __syncthreads();
            if (sm.bad) goto fail;
            product(amp);
            double acc1[1] = {0.0}, t1[1];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    publish(ga, i, amp[i]);
                    acc1[0] = add_rn(acc1[0], dot(amp[i], rs[i]));
                }
            if (!words_exchange<1>(g, epoch, acc1, t1, sm, false, [&] { take.begin(ga, halo, epoch); })) goto fail;
            const T rs_amp = static_cast<T>(t1[0]);
            const T alpha = rsr_old / rs_amp;
            if (rs_amp == T(0)) status |= kStatusBicgBreakdown;
            // ---- 2: s, M s, AMs = A M s; ||s||, <AMs, s>, <AMs, AMs>
            auto s_of = [&](int i) { return add_rn(r[i], -mul_rn(alpha, amp[i])); };
            take.end(ga, halo, epoch, sm, [&](uint32_t j, T v) {
                Ah[j] = v;
                const T sj = add_rn(Rh[j], -mul_rn(alpha, v));
                V[halo.at(j)] = jacobi ? mul_rn(sj, Ih[j]) : sj;
            });
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) own[i * NT] = apply_m(s_of(i), i);
            __syncthreads();
            if (sm.bad) goto fail;
            product(ams);
            double acc2[3] = {0.0, 0.0, 0.0}, t2[3];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    const T si = s_of(i);
                    acc2[0] = add_rn(acc2[0], term(si));
                    acc2[1] = add_rn(acc2[1], dot(ams[i], si));
                    acc2[2] = add_rn(acc2[2], dot(ams[i], ams[i]));
                }
            if (!words_exchange<3>(g, epoch, acc2, t2, sm, false)) goto fail;
            {
                const T res_s = static_cast<T>(finish_norm(t2[0])) / norm_b;
                cur_res = static_cast<double>(res_s);
                if (!isfinite(cur_res)) status |= kStatusNonFinite;
                if (finished(cur_res, n_iters)) {
                    // biconjugate-gradients-stabilized.hpp:183-195: x += alpha M p
#pragma unroll
                    for (int i = 0; i < R; ++i) x[i] = add_rn(x[i], mul_rn(alpha, apply_m(p[i], i)));
                    n_iters = k;
                    break;
                }
            }
            const T amss = static_cast<T>(t2[1]);
            const T amsams = static_cast<T>(t2[2]);
            omega = amss / amsams;
            if (omega == T(0)) status |= kStatusBicgBreakdown;
            // ---- 3: x, r; ||r||, <r*, r>
            double acc3[2] = {0.0, 0.0}, t3[2];
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (t + i * NT < mine) {
                    const T si = s_of(i);
                    x[i] = add_rn(add_rn(x[i], mul_rn(alpha, apply_m(p[i], i))), mul_rn(omega, apply_m(si, i)));
                    r[i] = add_rn(si, -mul_rn(omega, ams[i]));
                    publish(g, i, r[i]);
                    acc3[0] = add_rn(acc3[0], term(r[i]));
                    acc3[1] = add_rn(acc3[1], dot(rs[i], r[i]));
                }
            if (!words_exchange<2>(g, epoch, acc3, t3, sm, false, [&] { take.begin(g, halo, epoch); })) goto fail;
            const T res = static_cast<T>(finish_norm(t3[0])) / norm_b;
            cur_res = static_cast<double>(res);
            if (!isfinite(cur_res)) status |= kStatusNonFinite;
            if (finished(cur_res, n_iters)) {
                n_iters = k;
                break;
            }
            const T rsr_new = static_cast<T>(t3[1]);
            beta = rsr_new / rsr_old;
            beta = beta * alpha;
            beta = beta / omega;
            rsr_old = rsr_new;
            n_iters = k + 1;
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (t + i * NT < mine) a.x[row_t + i * NT] = x[i];
        if (lead) {
            a.st->n_iters = n_iters;
            a.st->init_res = init_res;
            a.st->cur_res = cur_res;
            atomicOr(&a.st->status, status);
        }
        return;
    }
fail:
    if (t == 0) atomicOr(&a.st->status, kStatusBarrierTimeout);
}

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename VA, typename VG>
struct DiaPcgResidentArgs {
    DiaPcgArgs<VA, VG> a;
    ResidentPlan plan;
    WordSync words;            // halo words of z (or the plain vector a.z)
    unsigned long long* qw;    // halo words of q (learned factor)
};

// The refinement's inner PCG (dia_pcg_kernel's arithmetic: FP32 vectors and
// FMAs in column order, sums in FP64) with its vectors on chip. Jacobi / none:
// as the CG above. LEARNED (M^-1 = G^T G, G on offsets <= 0, G^T on >= 0): r
// in shared memory with its halo, updated there by every CTA from the halo's
// q, which goes out with the first exchange; t = G r of the own rows and the
// rows above that G^T reaches; z = G^T t in registers, its edge rows out with
// the second exchange.
template <typename VA, typename VG, int NDA, int NDG, int R, bool LEARNED>
__global__ void __launch_bounds__(kResThreads, 1)
    dia_pcg_resident_kernel(const __grid_constant__ DiaPcgResidentArgs<VA, VG> args) {
    constexpr int NT = kResThreads;
    constexpr bool INV = !LEARNED;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ WordSmem<NT> sm;
    const DiaPcgArgs<VA, VG>& a = args.a;
    const ResidentPlan& pl = args.plan;
    const WordSync& g = args.words;
    WordSync gq = g;
    gq.halo = args.qw;
    const uint32_t n = a.n, t = threadIdx.x;
    const uint32_t r0 = static_cast<uint32_t>(static_cast<uint64_t>(blockIdx.x) * n / gridDim.x);
    const uint32_t r1 = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) + 1) * n / gridDim.x);
    const uint32_t mine = r1 - r0;
    const HaloRows halo{r0, r1, min(pl.lo, r0), min(pl.hi, n - r1)};
    const HaloRows qhalo{r0, r1, min(pl.lo_g, r0), min(pl.hi_g, n - r1)};
    uint32_t epoch = 0;
    float* const P = reinterpret_cast<float*>(smem_raw) + pl.lo;
    float* next = P + pl.mcap + pl.hi;
    float* const Rs = next + (LEARNED ? pl.lo_g : 0);          // learned: r with its halo, t
    if (LEARNED) next = Rs + pl.mcap + pl.hi_g;
    float* const ts = next;
    if (LEARNED) next += pl.mcap + pl.hi_g;
    const float* invp = a.invD ? a.invD + r0 + t : nullptr;
    VA* res_s = reinterpret_cast<VA*>(next);
    const VA* dv[NDA];
    keep_diagonals<NT, NDA>(a.A, pl, n, r0, mine, res_s, dv);
    const float* pd[NDA];
#pragma unroll
    for (int d = 0; d < NDA; ++d) pd[d] = P + t + a.A.off[d];
    // learned: G and G^T at the CTA's first row
    const VG* gv[NDG];
    const VG* gtv[NDG];
    if constexpr (LEARNED) {
        VG* const g_s = reinterpret_cast<VG*>(res_s + pl.kept);
        const uint32_t span = pl.mcap + pl.hi_g;
#pragma unroll
        for (int d = 0; d < NDG; ++d) {
            gv[d] = a.G.vals + static_cast<size_t>(d) * n + r0;
            gtv[d] = a.GT.vals + static_cast<size_t>(d) * n + r0;
            if (pl.g_kept) {
                VG* dst = g_s + static_cast<size_t>(d) * span;
                for (uint32_t i = t; i < span; i += NT) dst[i] = i < mine + qhalo.above ? gv[d][i] : VG(0.f);
                gv[d] = dst;
                gtv[d] = g_s + static_cast<size_t>(pl.g_partner[d]) * span + a.GT.off[d];
            }
        }
    }
    const float* const diag32 = a.A.diag32 ? a.A.diag32 + r0 + t : nullptr;
    float* const own = P + t;
    const int hi_t = static_cast<int>(pl.hi) - static_cast<int>(t);
    const int lo_t = static_cast<int>(mine) - static_cast<int>(pl.lo) - static_cast<int>(t);
    const int hi_q = static_cast<int>(pl.hi_g) - static_cast<int>(t);
    const int lo_q = static_cast<int>(mine) - static_cast<int>(pl.lo_g) - static_cast<int>(t);
    const uint32_t row_t = r0 + t;
    float* const zg = a.z + r0 + t;
    auto publish_z = [&](int k, float z) {
        if (k * NT < hi_t || k * NT >= lo_t) {
            if (LEARNED || pl.words)
                st_halo(g, row_t + k * NT, epoch + 1, z);
            else
                zg[k * NT] = z;
        }
    };
    const DiaPcgState in = *a.st;
    const double tol2 = in.tol * in.tol;
    const float* const Po = a.p[in.pbuf & 1];
    double rz = 0.0, rr0 = 0.0, rr = 0.0;
    float beta = 0.f;
    int iters = 0, status = 0;
    float x[R], q[R];
    float r[LEARNED ? 1 : R], inv[INV ? R : 1], z[LEARNED ? R : 1];
    r[0] = inv[0] = z[0] = 0.f;
    HaloTake<NT, float> take;
    auto prefetch = [&] {
        if (LEARNED || pl.words) take.begin(g, halo, epoch);
    };
    auto each_halo = [&](auto body) {
        if (LEARNED || pl.words) {
            take.end(g, halo, epoch, sm, [&](uint32_t j, float v) { body(halo.at(j), j, v); });
        } else {
            const uint32_t total = halo.count();
            for (uint32_t j0 = t; j0 < total; j0 += 8 * NT) {
                float v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (j0 + u * NT < total) v[u] = __ldcg(a.z + halo.row(j0 + u * NT));
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (j0 + u * NT < total) body(halo.at(j0 + u * NT), j0 + u * NT, v[u]);
            }
        }
    };
    auto inv_of = [&](int k) { return inv[INV ? k : 0]; };
    // learned: t = G r of the own rows and the halo above, then z = G^T t; the
    // own rows' ||t||^2
    auto apply_factor = [&](double& tt) {
        if constexpr (LEARNED) {
            const uint32_t rows = mine + qhalo.above;
#pragma unroll 1
            for (uint32_t i0 = t; i0 < rows; i0 += 2 * NT) {
                float av[2][NDG], rv[2][NDG];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t i = min(i0 + u * NT, rows - 1);
#pragma unroll
                    for (int d = 0; d < NDG; ++d) {
                        av[u][d] = to_f(gv[d][i]);
                        rv[u][d] = Rs[static_cast<int>(i) + a.G.off[d]];
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const uint32_t i = i0 + u * NT;
                    float s = 0.f;
#pragma unroll
                    for (int d = 0; d < NDG; ++d) s = fmaf(av[u][d], rv[u][d], s);
                    if (i < rows) {
                        ts[i] = s;
                        if (i < mine) tt += static_cast<double>(s) * s;
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (t + k * NT < mine) {
                    float s = 0.f;
#pragma unroll
                    for (int d = 0; d < NDG; ++d)
                        s = fmaf(to_f(gtv[d][t + k * NT]), ts[static_cast<int>(t + k * NT) + a.GT.off[d]], s);
                    z[k] = s;
                    publish_z(k, s);
                }
        }
    };
    if (t == 0) sm.bad = 0;
    for (uint32_t i = t; i < pl.lo + pl.mcap + pl.hi; i += NT) (P - pl.lo)[i] = 0.f;
    if constexpr (LEARNED) {
        for (uint32_t i = t; i < pl.lo_g + pl.mcap + pl.hi_g; i += NT) (Rs - pl.lo_g)[i] = 0.f;
        for (uint32_t i = t; i < pl.mcap + pl.hi_g; i += NT) ts[i] = 0.f;
        __syncthreads();
        for (uint32_t i = t; i < mine; i += NT) Rs[i] = __ldg(a.b + r0 + i);
        for (uint32_t j = t; j < qhalo.count(); j += NT) Rs[qhalo.at(j)] = __ldg(a.b + qhalo.row(j));
    }
    __syncthreads();

    // ---- r = b, x = 0, z = M r, <r,z>, <r,r>
    {
        double acc[2] = {0.0, 0.0}, tot[2];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            x[k] = q[k] = 0.f;
            if constexpr (!LEARNED) r[k] = 0.f;
            if constexpr (INV) inv[k] = 0.f;
            if constexpr (LEARNED) z[k] = 0.f;
            if (t + k * NT < mine) {
                const float ri = __ldg(a.b + row_t + k * NT);
                acc[1] += static_cast<double>(ri) * ri;
                if constexpr (!LEARNED) {
                    if constexpr (INV) inv[k] = a.invD ? invp[k * NT] : 1.f;
                    r[k] = ri;
                    const float zi = a.invD ? ri * inv_of(k) : ri;
                    publish_z(k, zi);
                    acc[0] += static_cast<double>(ri) * zi;
                }
            }
        }
        apply_factor(acc[0]);
        if (!words_exchange<2>(g, epoch, acc, tot, sm, !LEARNED && !pl.words, prefetch)) goto fail;
        rz = tot[0];
        rr0 = rr = tot[1];
    }
    if (rr0 > 0.0 && in.max_iters > 0) {  // (b == 0: x = 0)
        // the first direction: z, or a previous solve's continued
        const bool warm = in.warm != 0;
        if (warm) beta = static_cast<float>(rz / in.rz_prev);
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (t + k * NT < mine) {
                float zi;
                if constexpr (LEARNED)
                    zi = z[k];
                else
                    zi = a.invD ? r[k] * inv_of(k) : r[k];
                own[k * NT] = warm ? fmaf(beta, __ldg(Po + row_t + k * NT), zi) : zi;
            }
        each_halo([&](int at, uint32_t j, float zi) { P[at] = warm ? fmaf(beta, __ldg(Po + halo.row(j)), zi) : zi; });
        __syncthreads();
        if (sm.bad) goto fail;
        for (;;) {
            // ---- A: q = A p, <p, q>
            double acc[1] = {0.0}, pq[1];
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (t + k * NT < mine) {
                    float s = 0.f;
#pragma unroll
                    for (int d = 0; d < NDA; ++d) s = fmaf(to_f(dv[d][k * NT]), pd[d][k * NT], s);
                    const float pi = own[k * NT];
                    if (diag32 != nullptr) s = fmaf(__ldg(diag32 + k * NT), pi, s);
                    q[k] = s;
                    if (LEARNED && (k * NT < hi_q || k * NT >= lo_q)) st_halo(gq, row_t + k * NT, epoch + 1, s);
                    acc[0] += static_cast<double>(pi) * s;
                }
            if (!words_exchange<1>(g, epoch, acc, pq, sm, false, [&] {
                    if (LEARNED) take.begin(gq, qhalo, epoch);
                }))
                goto fail;
            if (!(pq[0] > 0.0)) {  // lost positive curvature (or not finite): stop, the caller restarts
                status |= isfinite(pq[0]) ? kStatusCurvature : kStatusNonFinite;
                break;
            }
            const float alpha = static_cast<float>(rz / pq[0]);
            // ---- B: x, r, z = M r; <r, r>, <r, z>
            double acc2[2] = {0.0, 0.0}, tot[2];
            if constexpr (LEARNED) {
                take.end(gq, qhalo, epoch, sm, [&](uint32_t j, float qj) {
                    Rs[qhalo.at(j)] = fmaf(-alpha, qj, Rs[qhalo.at(j)]);
                });
#pragma unroll
                for (int k = 0; k < R; ++k)
                    if (t + k * NT < mine) {
                        x[k] = fmaf(alpha, own[k * NT], x[k]);
                        const float ri = fmaf(-alpha, q[k], Rs[t + k * NT]);
                        Rs[t + k * NT] = ri;
                        acc2[0] += static_cast<double>(ri) * ri;
                    }
                __syncthreads();
                if (sm.bad) goto fail;
                apply_factor(acc2[1]);
            } else {
#pragma unroll
                for (int k = 0; k < R; ++k)
                    if (t + k * NT < mine) {
                        x[k] = fmaf(alpha, own[k * NT], x[k]);
                        r[k] = fmaf(-alpha, q[k], r[k]);
                        const float zi = a.invD ? r[k] * inv_of(k) : r[k];
                        publish_z(k, zi);
                        acc2[0] += static_cast<double>(r[k]) * r[k];
                        acc2[1] += static_cast<double>(r[k]) * zi;
                    }
            }
            if (!words_exchange<2>(g, epoch, acc2, tot, sm, !LEARNED && !pl.words, prefetch)) goto fail;
            rr = tot[0];
            ++iters;
            if (!isfinite(rr)) {
                status |= kStatusNonFinite;
                break;
            }
            if (rr <= tol2 * rr0 || iters >= in.max_iters) break;
            beta = static_cast<float>(tot[1] / rz);
            rz = tot[1];
            // ---- C: p = z + beta p
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (t + k * NT < mine) {
                    float zi;
                    if constexpr (LEARNED)
                        zi = z[k];
                    else
                        zi = a.invD ? r[k] * inv_of(k) : r[k];
                    own[k * NT] = fmaf(beta, own[k * NT], zi);
                }
            each_halo([&](int at, uint32_t, float zi) { P[at] = fmaf(beta, P[at], zi); });
            __syncthreads();
            if (sm.bad) goto fail;
        }
    }
    // the solution, and the last direction for a continued solve (in the
    // buffer the previous one did not use: other CTAs' first directions)
    {
        float* const pn = a.p[(in.pbuf & 1) ^ 1];
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (t + k * NT < mine) {
                a.x[row_t + k * NT] = x[k];
                if (iters > 0) pn[row_t + k * NT] = own[k * NT];
            }
    }
    if (blockIdx.x == 0 && t == 0) {
        a.st->iters = iters;
        a.st->rr0 = rr0;
        a.st->rr = rr;
        a.st->rz_prev = rz;
        a.st->pbuf = iters > 0 ? (in.pbuf & 1) ^ 1 : in.pbuf & 1;
        a.st->xbuf = 0;
        atomicOr(&a.st->status, status);
    }
    return;
fail:
    if (t == 0) atomicOr(&a.st->status, kStatusBarrierTimeout);
}

// Dynamic shared memory a resident CTA may use: the 227 KB an SM gives one
// CTA, less the kernel's static part.
constexpr size_t kResidentSmem = 232448 - 4096;

// (The attribute belongs to the kernel, not to the launch: always the same
// value, so that another thread's smaller plan cannot come between.)
template <typename Args>
cudaError_t resident_launch(const void* k, Args& args, int threads, cudaStream_t s) {
    const cudaError_t e =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kResidentSmem));
    if (e != cudaSuccess) return e;
    void* p[] = {&args};
    return cudaLaunchCooperativeKernel(k, dim3(args.plan.grid), dim3(threads), p, args.plan.smem, s);
}

template <typename T, int ND>
cudaError_t cg_launch(DiaCgResidentArgs<T>& args, cudaStream_t s) {
    return resident_launch(args.plan.rows == 2 ? reinterpret_cast<const void*>(dia_cg_resident_kernel<T, ND, 2>)
                           : args.plan.rows == kFewRows
                               ? reinterpret_cast<const void*>(dia_cg_resident_kernel<T, ND, kFewRows>)
                               : reinterpret_cast<const void*>(dia_cg_resident_kernel<T, ND, kManyRows>),
                           args, kResThreads, s);
}
template <typename T, int ND>
cudaError_t bicg_launch(DiaBicgResidentArgs<T>& args, cudaStream_t s) {
    return resident_launch(args.plan.rows == 2 ? reinterpret_cast<const void*>(dia_bicg_resident_kernel<T, ND, 2>)
                                               : reinterpret_cast<const void*>(dia_bicg_resident_kernel<T, ND, kFewRows>),
                           args, kResThreads, s);
}
template <typename VA, typename VG, int NDA, int NDG, bool LEARNED>
cudaError_t pcg_launch(DiaPcgResidentArgs<VA, VG>& args, cudaStream_t s) {
    constexpr int few = kFewRows, many = kManyRows;
    return resident_launch(
        args.plan.rows == few ? reinterpret_cast<const void*>(dia_pcg_resident_kernel<VA, VG, NDA, NDG, few, LEARNED>)
                              : reinterpret_cast<const void*>(dia_pcg_resident_kernel<VA, VG, NDA, NDG, many, LEARNED>),
        args, kResThreads, s);
}

// Rows per CTA a solve aims at. An exchange costs more the more CTAs take part
// (each polls every other's words: 0.4 us bare with 2, 1.0 with 148), a CTA's own
// sums and products more the more rows it has. CG, FP64, us an iteration with
// 256, 512, 1024 and 2048 rows a CTA: 64^2 4.2, 3.7, 3.8, 4.4; 100^2 4.5, 4.5, 4.0,
// 4.4; 200^2 5.4, 4.3, 4.4, 5.1; 24^3 5.4, 5.7, 6.1, 6.5; 40^3 6.0, 5.9, 6.1, 7.3;
// BiCGStab 200^2 7.8, 7.5, 7.7, 9.5. (From 152,000 rows on every SM takes part
// either way.)
constexpr uint32_t kRowsPerCta = 1024;

// The part of a plan common to all methods: grid, rows, halo.
bool plan_rows(uint32_t n, const DiaOffsets& offs, int nd_pad, int sm_count, int threads,
               std::initializer_list<int> sizes, ResidentPlan& p) {
    p = ResidentPlan{};
    if (sm_count < 1 || sm_count > threads || n == 0 || nd_pad > kResidentDiags || offs.nd < 1) return false;
    p.grid = std::min<uint32_t>(static_cast<uint32_t>(sm_count), (n + kRowsPerCta - 1) / kRowsPerCta);
    p.mcap = (n + p.grid - 1) / p.grid;
    for (int r : sizes)
        if (p.rows == 0 && p.mcap <= static_cast<uint32_t>(r) * static_cast<uint32_t>(threads)) p.rows = r;
    const int32_t first = offs.off[0], last = offs.off[offs.nd - 1];
    p.lo = first < 0 ? static_cast<uint32_t>(-static_cast<int64_t>(first)) : 0u;
    p.hi = last > 0 ? static_cast<uint32_t>(last) : 0u;
    p.words = static_cast<uint64_t>(p.lo) + p.hi <= p.mcap ? 1 : 0;
    return p.rows != 0;
}

// Whether a halo is worth holding: every CTA reads all of it once an iteration,
// which a streaming kernel's L1 and L2 do for less when it is wide beside the
// CTA's own rows. At most `rows` rows, or twos / 2 times the CTA's own.
bool halo_pays(const ResidentPlan& p, uint64_t rows, uint64_t twos) {
    const uint64_t h = static_cast<uint64_t>(p.lo) + p.hi;
    return h <= rows || 2 * h <= twos * p.mcap;
}

// Hands out the shared memory of a plan.
struct SmemBudget {
    uint64_t left = kResidentSmem;
    bool take(uint64_t values, size_t size) {
        if (values * size > left) return false;
        left -= values * size;
        return true;
    }
    size_t used() const { return static_cast<size_t>(kResidentSmem - left); }
};

}  // namespace

namespace {

// Keeps as many diagonals as fit. With a symmetric A an upper diagonal is kept
// with the rows below the CTA that its lower partner needs, and serves both;
// they come before the main diagonal.
void keep_plan(const int32_t* off, int nd, bool sym, size_t size, SmemBudget& b, ResidentPlan& p) {
    for (int d = 0; d < kResidentDiags; ++d) p.at[d] = p.lead[d] = -1;
    auto keep = [&](int d, uint32_t lead) {
        if (p.at[d] >= 0 || !b.take(static_cast<uint64_t>(p.mcap) + lead, size)) return false;
        p.lead[d] = static_cast<int32_t>(lead);
        p.at[d] = static_cast<int32_t>(p.kept + lead);
        p.kept += p.mcap + lead;
        return true;
    };
    if (sym)
        for (int d = nd - 1; d >= 0 && off[d] > 0; --d)
            if (keep(d, static_cast<uint32_t>(off[d]))) p.at[nd - 1 - d] = p.at[d] - off[d];  // (lead stays -1)
    for (int d = 0; d < nd; ++d) keep(d, 0);
    if (p.kept % 2 && b.take(1, size)) ++p.kept;  // what follows starts on four bytes
}

}  // namespace

template <typename T>
bool resident_cg_plan(uint32_t n, const DiaOffsets& offs, int nd_pad, bool jacobi, bool sym, int sm_count,
                      ResidentPlan& p) {
    if (!plan_rows(n, offs, nd_pad, sm_count, kResThreads, {2, kFewRows, kManyRows}, p)) return false;
    // us an iteration on chip / streamed, halo rows and own rows: 8192 and 1024
    // 7.0 / 8.1 (FP64), 6.4 / 7.8 (FP32); 12,800 and 1024 8.5 / 9.4, 7.5 / 8.3;
    // 16,200 and 1013 9.2 / 8.8, 8.1 / 7.8; 20,000 and 3379 17.9 / 17.7, 13.1 / 15.4;
    // 28,800 and 6811 18.4 / 19.9 (FP32); 32,768 and 3543 16.8 / 14.7; 51,200
    // and 1384 16.8 / 9.8.
    if (!halo_pays(p, 14336, 12)) return false;
    SmemBudget b;
    if (!b.take(static_cast<uint64_t>(p.lo) + p.mcap + p.hi, sizeof(T))) return false;
    const bool regs = p.rows <= kFewRows ? inv_in_regs<T, kFewRows>() : inv_in_regs<T, kManyRows>();
    if (jacobi && !regs) {
        p.inv_smem = b.take(p.mcap, sizeof(T)) ? 1 : 0;  // (read twice an iteration)
        p.inv_global = 1 - p.inv_smem;
    }
    keep_plan(offs.off, nd_pad, sym, sizeof(T), b, p);
    p.smem = b.used();
    return true;
}

template <typename T>
bool resident_bicg_plan(uint32_t n, const DiaOffsets& offs, int nd_pad, int sm_count, ResidentPlan& p) {
    // (a neighbour's r and A M p only travel as words)
    if (!plan_rows(n, offs, nd_pad, sm_count, kResThreads, {2, kFewRows}, p)) return false;
    SmemBudget b;
    if (!b.take(5ull * (static_cast<uint64_t>(p.lo) + p.hi) + p.mcap, sizeof(T))) return false;
    keep_plan(offs.off, nd_pad, false, sizeof(T), b, p);
    p.smem = b.used();
    return true;
}

template <typename VA, typename VG>
bool resident_pcg_plan(const DiaPcgArgs<VA, VG>& a, bool learned, int sm_count, ResidentPlan& p) {
    DiaOffsets o;  // (padding diagonals, at offset 0, are in the list behind the real ones)
    int32_t lo = 0, hi = 0;
    for (int d = 0; d < a.A.nd; ++d) {
        lo = std::min(lo, a.A.off[d]);
        hi = std::max(hi, a.A.off[d]);
    }
    o.nd = 2;
    o.off[0] = lo;
    o.off[1] = hi;
    // (28 rows a thread, 2.1 M rows, measured slower than streaming: 58 us an
    // inner iteration on 128^3 instead of 38, the diagonals still from L2 with
    // too few loads in flight beside 84 registers of vectors)
    if (!plan_rows(a.n, o, a.A.nd, sm_count, kResThreads, {kFewRows, kManyRows}, p)) return false;
    // Jacobi, us an inner iteration on chip / streamed, halo rows and own rows:
    // 8192 and 1024 8.0 / 8.9; 12,800 and 1024 9.3 / 9.5, and 3460 12.6 / 12.8;
    // 13,122 and 3591 12.9 / 12.8; 16,200 and 1013 11.7 / 10.4, and 4926 14.5 / 15.5;
    // 20,000 and 4730 15.7 / 15.0, and 6757 17.7 / 18.1; 28,800 and 6811 20.3 / 18.5.
    // Learned (r's and q's halo beside p's): 4608 and 1024 10.1 / 11.2; 7200 and
    // 2432 14.9 / 15.4; 8192 and 1772 14.2 / 14.2; 9800 and 2318 17.8 / 16.6; 16,200
    // and 4926 30.2 / 23.4.
    if (!(learned ? halo_pays(p, 7680, 2) : halo_pays(p, 12800, 8))) return false;
    SmemBudget b;
    if (!b.take(static_cast<uint64_t>(p.lo) + p.mcap + p.hi, 4)) return false;
    if (learned) {
        if (a.G.nd > kResidentDiags || a.GT.nd != a.G.nd) return false;
        int real = 0;  // G's diagonals: offsets increasing to 0, then padding
        while (real < a.G.nd && a.G.off[real] < 0) ++real;
        if (real == a.G.nd || a.G.off[real] != 0) return false;
        ++real;
        bool mirrored = true;
        for (int d = 0; d < a.G.nd; ++d) {
            if (a.G.off[d] > 0 || a.GT.off[d] < 0) return false;
            p.lo_g = std::max(p.lo_g, static_cast<uint32_t>(-static_cast<int64_t>(a.G.off[d])));
            p.hi_g = std::max(p.hi_g, static_cast<uint32_t>(a.GT.off[d]));
            p.g_partner[d] = d < real ? real - 1 - d : d;
            mirrored = mirrored && a.GT.off[d] == -a.G.off[p.g_partner[d]];
        }
        if (!b.take(2ull * p.mcap + p.lo_g + 2ull * p.hi_g, 4)) return false;
        // G^T is the transpose of G value for value (the network exports it so)
        if (mirrored && b.take(static_cast<uint64_t>(a.G.nd) * (p.mcap + p.hi_g) + 2, sizeof(VG))) p.g_kept = 1;
    }
    keep_plan(a.A.off, a.A.nd, a.sym, sizeof(VA), b, p);
    p.smem = b.used();
    return true;
}

size_t word_sync_bytes(const ResidentPlan& p, uint32_t n, size_t value_bytes, int halos) {
    const size_t slots = 2 * static_cast<size_t>(p.grid) * kSlotWords;
    const size_t halo = static_cast<size_t>(n) * (value_bytes / 4) + 2;
    return 256 + (slots + halo * static_cast<size_t>(halos)) * sizeof(unsigned long long);
}

WordSync word_sync_at(void* base, const ResidentPlan& p, unsigned long long wait_ns, int never_release) {
    WordSync w;
    w.err = static_cast<int*>(base);
    w.slots = reinterpret_cast<unsigned long long*>(static_cast<char*>(base) + 256);
    w.halo = w.slots + 2 * static_cast<size_t>(p.grid) * kSlotWords;
    w.wait_ns = wait_ns;
    w.never_release = never_release;
    return w;
}

namespace {

// The second set of halo words behind the first (even: 16-byte aligned).
unsigned long long* second_halo(const WordSync& w, uint32_t n, size_t value_bytes) {
    return w.halo + ((static_cast<size_t>(n) * (value_bytes / 4) + 1) & ~size_t(1));
}

}  // namespace

template <typename T>
cudaError_t launch_cg_resident(const DiaCgArgs<T>& a, const ResidentPlan& plan, const WordSync& words, cudaStream_t s) {
    DiaCgResidentArgs<T> args{a, plan, words};
    switch (a.A.nd) {
        case 3: return cg_launch<T, 3>(args, s);
        case 5: return cg_launch<T, 5>(args, s);
        case 7: return cg_launch<T, 7>(args, s);
        case 9: return cg_launch<T, 9>(args, s);
        default: return cudaErrorInvalidConfiguration;
    }
}

template <typename T>
cudaError_t launch_bicg_resident(const DiaBicgArgs<T>& a, const ResidentPlan& plan, const WordSync& words,
                                 cudaStream_t s) {
    DiaBicgResidentArgs<T> args{a, plan, words, second_halo(words, a.n, sizeof(T))};
    switch (a.A.nd) {
        case 3: return bicg_launch<T, 3>(args, s);
        case 5: return bicg_launch<T, 5>(args, s);
        case 7: return bicg_launch<T, 7>(args, s);
        case 9: return bicg_launch<T, 9>(args, s);
        default: return cudaErrorInvalidConfiguration;
    }
}

template <typename VA, typename VG>
cudaError_t launch_pcg_resident(const DiaPcgArgs<VA, VG>& a, bool learned, const ResidentPlan& plan,
                                const WordSync& words, cudaStream_t s) {
    DiaPcgResidentArgs<VA, VG> args{a, plan, words, second_halo(words, a.n, sizeof(float))};
    if (learned) {
        if (a.A.nd == 5 && a.G.nd == 3) return pcg_launch<VA, VG, 5, 3, true>(args, s);
        if (a.A.nd == 7 && a.G.nd == 4) return pcg_launch<VA, VG, 7, 4, true>(args, s);
        if (a.A.nd == 9 && a.G.nd == 5) return pcg_launch<VA, VG, 9, 5, true>(args, s);
        return cudaErrorInvalidConfiguration;
    }
    switch (a.A.nd) {
        case 3: return pcg_launch<VA, VG, 3, 1, false>(args, s);
        case 5: return pcg_launch<VA, VG, 5, 1, false>(args, s);
        case 7: return pcg_launch<VA, VG, 7, 1, false>(args, s);
        case 9: return pcg_launch<VA, VG, 9, 1, false>(args, s);
        default: return cudaErrorInvalidConfiguration;
    }
}

#define CLSP_RES_INST(T)                                                                                           \
    template bool resident_cg_plan<T>(uint32_t, const DiaOffsets&, int, bool, bool, int, ResidentPlan&);           \
    template bool resident_bicg_plan<T>(uint32_t, const DiaOffsets&, int, int, ResidentPlan&);                     \
    template cudaError_t launch_cg_resident<T>(const DiaCgArgs<T>&, const ResidentPlan&, const WordSync&,          \
                                               cudaStream_t);                                                      \
    template cudaError_t launch_bicg_resident<T>(const DiaBicgArgs<T>&, const ResidentPlan&, const WordSync&,      \
                                                 cudaStream_t);
CLSP_RES_INST(float)
CLSP_RES_INST(double)
#undef CLSP_RES_INST
#define CLSP_RES_PCG(VA)                                                                                           \
    template bool resident_pcg_plan<VA, __nv_bfloat16>(const DiaPcgArgs<VA, __nv_bfloat16>&, bool, int,             \
                                                       ResidentPlan&);                                             \
    template cudaError_t launch_pcg_resident<VA, __nv_bfloat16>(const DiaPcgArgs<VA, __nv_bfloat16>&, bool,         \
                                                                const ResidentPlan&, const WordSync&, cudaStream_t);
CLSP_RES_PCG(float)
CLSP_RES_PCG(__nv_bfloat16)
#undef CLSP_RES_PCG

}  // namespace clsp
