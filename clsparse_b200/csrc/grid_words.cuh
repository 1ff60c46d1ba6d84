// Grid-wide exchanges of the on-chip solver kernels (one cooperative launch
// per solve, every CTA resident) through tagged words: a 32-bit half of a value and the
// 32-bit number of the exchange it belongs to are written as one 64-bit word,
// so a reader sees from the word itself that the value has arrived. No
// arrival counter, no fence and no second round trip: a sum costs one store
// and one polled load through L2 where the counter of grid_sync.cuh costs a
// release, an atomic, a polled load and a load of the partials.
//
// Every wait is bounded by the global timer; a wait that runs out sets the
// error flag, and every CTA leaves.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "dia_resident.h"

namespace clsp {

namespace {

__device__ __forceinline__ unsigned long long word_of(uint32_t half, uint32_t tag) {
    return static_cast<unsigned long long>(tag) << 32 | half;
}

// (No memory clobbers: a word carries its own tag, so nothing else has to keep
// its order beside it, and the loads of the rows around a published one may move
// past it.)
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}
__device__ __forceinline__ void st_words(unsigned long long* p, unsigned long long v0, unsigned long long v1) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v0), "l"(v1));
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void ld_words(const unsigned long long* p, unsigned long long& v0,
                                         unsigned long long& v1) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v0), "=l"(v1) : "l"(p));
}

// One bounded wait: expired() after every failed poll.
struct WordWait {
    uint64_t t0 = 0;
    uint32_t spins = 0;
    __device__ __forceinline__ bool expired(const WordSync& g) {
        if ((++spins & 63u) != 0u) return false;
        if (*reinterpret_cast<volatile int*>(g.err)) return true;
        uint64_t now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (t0 == 0) {
            t0 = now;
        } else if (now - t0 > g.wait_ns) {
            atomicExch(g.err, 1);
            return true;
        }
        return false;
    }
};

template <int NT>
struct WordSmem {
    double red[4][NT / 32];  // per-warp sums of the CTA's values
    double fin[4][NT / 32];  // per-warp sums of the grid's
    int bad;                 // a wait of this CTA ran out (zeroed by the kernel first)
};

// Sums K values per thread over the grid; the result in every thread, the
// same bit for bit in every CTA (warps, then CTAs, in a fixed order), and a
// barrier of the CTA. ++epoch numbers the exchange; a slot is rewritten two
// exchanges later, when every CTA has read it. With `publish`, plain global
// stores made before the call by any thread of any CTA are visible after it
// (fences on both sides). `meanwhile` runs in every thread between the CTA's
// own store and its polls (to start loads of its own). At most NT CTAs. False
// when the grid has to stop.
struct Nothing {
    __device__ __forceinline__ void operator()() const {}
};
template <int K, int NT, typename F = Nothing>
__device__ __forceinline__ bool words_exchange(const WordSync& g, uint32_t& epoch, const double (&v)[K],
                                               double (&out)[K], WordSmem<NT>& sm, bool publish, F meanwhile = {}) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t G = gridDim.x;
    ++epoch;
    unsigned long long* slots = g.slots + static_cast<size_t>(epoch & 1u) * G * kSlotWords;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const double w = dev::warp_sum(v[k]);
        if (lane == 0) sm.red[k][warp] = w;
    }
    __syncthreads();
    if (warp == 0) {
        // half a warp per value (at most 16 warps a CTA), two values at a time
        static_assert(NT <= 512, "a half-warp sums the warps' values");
        double mine = 0.0;
#pragma unroll
        for (int k0 = 0; k0 < K; k0 += 2) {
            const int k = k0 + static_cast<int>(lane >> 4);
            double w = k < K && (lane & 15) < NT / 32 ? sm.red[k < K ? k : 0][lane & 15] : 0.0;
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) w += __shfl_xor_sync(0xffffffffu, w, off);
            const double other = __shfl_xor_sync(0xffffffffu, w, 16);
            if (lane == static_cast<uint32_t>(k0)) mine = w;           // lanes 0..15 hold value k0
            if (lane == static_cast<uint32_t>(k0 + 1)) mine = other;   // and the other half k0 + 1
        }
        if (publish) __threadfence();
        if (lane < K && !(g.never_release && blockIdx.x == 0)) {
            const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(mine));
            st_words(slots + static_cast<size_t>(blockIdx.x) * kSlotWords + 2 * lane,
                     word_of(static_cast<uint32_t>(bits), epoch), word_of(static_cast<uint32_t>(bits >> 32), epoch));
        }
    }
    meanwhile();
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k] = 0.0;
    if (tid < G) {
        const unsigned long long* s = slots + static_cast<size_t>(tid) * kSlotWords;
        WordWait wait;
        for (;;) {
            unsigned long long w[2 * K];
            bool there = true;
#pragma unroll
            for (int k = 0; k < K; ++k) ld_words(s + 2 * k, w[2 * k], w[2 * k + 1]);
#pragma unroll
            for (int k = 0; k < 2 * K; ++k) there = there && static_cast<uint32_t>(w[k] >> 32) == epoch;
            if (there) {
#pragma unroll
                for (int k = 0; k < K; ++k)
                    acc[k] = __longlong_as_double(static_cast<long long>((w[2 * k + 1] << 32) | (w[2 * k] & 0xffffffffull)));
                break;
            }
            if (wait.expired(g)) {
                sm.bad = 1;
                break;
            }
        }
        if (publish) __threadfence();
    }
    const uint32_t warps = (G + 31) / 32;
    __syncwarp();
    if (warp < warps) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const double w = dev::warp_sum(acc[k]);
            if (lane == 0) sm.fin[k][warp] = w;
        }
    }
    __syncthreads();
    if (sm.bad) return false;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
        for (uint32_t w = 0; w < warps; ++w) s += sm.fin[k][w];
        out[k] = s;
    }
    return true;
}

// A halo value: row `row`'s words tagged `tag`.
__device__ __forceinline__ void st_halo(const WordSync& g, uint32_t row, uint32_t tag, float v) {
    st_word(g.halo + row, word_of(__float_as_uint(v), tag));
}
__device__ __forceinline__ void st_halo(const WordSync& g, uint32_t row, uint32_t tag, double v) {
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
    st_words(g.halo + 2 * static_cast<size_t>(row), word_of(static_cast<uint32_t>(bits), tag),
             word_of(static_cast<uint32_t>(bits >> 32), tag));
}
__device__ __forceinline__ bool try_halo(const WordSync& g, uint32_t row, uint32_t tag, float& v) {
    const unsigned long long w = ld_word(g.halo + row);
    v = __uint_as_float(static_cast<uint32_t>(w));
    return static_cast<uint32_t>(w >> 32) == tag;
}
__device__ __forceinline__ bool try_halo(const WordSync& g, uint32_t row, uint32_t tag, double& v) {
    unsigned long long w0, w1;
    ld_words(g.halo + 2 * static_cast<size_t>(row), w0, w1);
    v = __longlong_as_double(static_cast<long long>((w1 << 32) | (w0 & 0xffffffffull)));
    return static_cast<uint32_t>(w0 >> 32) == tag && static_cast<uint32_t>(w1 >> 32) == tag;
}

// The rows around a CTA's own [r0, r1) that its stencil reaches: `below` rows
// before and `above` rows after, clipped to the matrix.
struct HaloRows {
    uint32_t r0, r1, below, above;
    __device__ __forceinline__ uint32_t count() const { return below + above; }
    // row j of the halo; its place relative to the CTA's first row
    __device__ __forceinline__ uint32_t row(uint32_t j) const { return j < below ? r0 - below + j : r1 + (j - below); }
    __device__ __forceinline__ int at(uint32_t j) const { return static_cast<int>(row(j)) - static_cast<int>(r0); }
};

// The values of the halo rows from their tagged words: begin() starts a
// thread's first kHaloBatch loads (while an exchange is under way), end() polls
// for what was not there yet, loads the rest and calls body(j, value) for
// every halo row. A wait that runs out sets sm.bad, which the CTA sees behind
// its next barrier. (Polling to the end during the exchange, by the threads
// that poll no sums, measured slower: 6.4 instead of 6.0 us an iteration on
// 512^2 FP64, 31.3 instead of 28.8 on 100^3.)
constexpr int kHaloBatch = 4;
template <int NT, typename T>
struct HaloTake {
    T v[kHaloBatch];
    uint32_t missing;
    __device__ __forceinline__ void load(const WordSync& g, const HaloRows& h, uint32_t tag, uint32_t j0) {
        missing = 0;
#pragma unroll
        for (int u = 0; u < kHaloBatch; ++u) {
            const uint32_t j = j0 + u * NT;
            if (j < h.count() && !try_halo(g, h.row(j), tag, v[u])) missing |= 1u << u;
        }
    }
    __device__ __forceinline__ void begin(const WordSync& g, const HaloRows& h, uint32_t tag) {
        load(g, h, tag, threadIdx.x);
    }
    template <typename F>
    __device__ __forceinline__ void end(const WordSync& g, const HaloRows& h, uint32_t tag, WordSmem<NT>& sm, F body) {
        const uint32_t total = h.count();
        for (uint32_t j0 = threadIdx.x;;) {
            WordWait wait;
            while (missing) {
                if (wait.expired(g)) {
                    sm.bad = 1;
                    return;
                }
#pragma unroll
                for (int u = 0; u < kHaloBatch; ++u)
                    if ((missing >> u & 1u) && try_halo(g, h.row(j0 + u * NT), tag, v[u])) missing &= ~(1u << u);
            }
#pragma unroll
            for (int u = 0; u < kHaloBatch; ++u) {
                const uint32_t j = j0 + u * NT;
                if (j < total) body(j, v[u]);
            }
            j0 += NT * kHaloBatch;
            if (j0 >= total) return;
            load(g, h, tag, j0);
        }
    }
};

}  // namespace
}  // namespace clsp
