// Banded solves with their vectors held on chip (dia_resident.cu): what their
// callers (dia.cu) choose and allocate.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dia.h"
#include "dia_rows.cuh"

namespace clsp {

// Words of one launch, all zero when it starts (exchanges are numbered from
// 1): two buffers of a slot per CTA, and one word (FP32) or two (FP64) per
// matrix row for halo values. Slots lie 256 bytes apart: every CTA polls every
// slot, and slots that share a line or a pair of lines cost an exchange
// of 148 CTAs 2.2 us (32 bytes apart), 1.5 (64), 1.1 (128) instead of 1.0.
constexpr int kSlotWords = 32;
struct WordSync {
    unsigned long long* slots;
    unsigned long long* halo;
    int* err;
    unsigned long long wait_ns;
    int never_release;  // test switch: CTA 0 publishes nothing, so every wait runs out
};

constexpr int kResidentDiags = 9;  // padded diagonal counts the kernels are built for: 3, 5, 7, 9

// Layout of a resident CTA's shared memory, chosen on the host.
struct ResidentPlan {
    uint32_t lo = 0, hi = 0;   // rows the stencil reaches below / above
    uint32_t mcap = 0;         // rows of the largest CTA
    uint32_t grid = 0;         // CTAs, one per SM
    int rows = 0;              // rows per thread the kernel is built for
    int inv_smem = 0;          // D^-1 in shared memory
    int inv_global = 0;        // D^-1 in a vector of its own
    int words = 0;             // the halo's z as tagged words (else a plain vector)
    uint32_t lo_g = 0, hi_g = 0;  // learned factor: rows G reaches below, G^T above
    // Diagonal d kept in shared memory: row i of the CTA at value at[d] + i of
    // the kept ones (-1: it stays in L2), `lead` rows before the CTA's first kept
    // with it. A mirrored diagonal (lead -1) has no values of its own: A is
    // symmetric, and its row i is row i + off of its upper partner.
    int32_t at[kResidentDiags];
    int32_t lead[kResidentDiags];
    uint32_t kept = 0;         // values kept
    // Learned factor kept: diagonal d of G at value g_at + d (mcap + hi_g) of
    // the kept ones (its own type, behind A's), G^T's read from G's at the column's row.
    int g_kept = 0;
    int g_partner[kResidentDiags];
    size_t smem = 0;
};

// Rows a CTA of the drop-in CG / BiCGStab holds at most.
constexpr uint32_t kResidentCgRows = 7168, kResidentBicgRows = 2048;

// Whether a solve runs on chip, and its layout: the drop-in CG and BiCGStab on
// n rows, the refinement's inner PCG. `sym`: A is symmetric bit for bit, its
// offsets symmetric, no padding diagonals.
template <typename T>
bool resident_cg_plan(uint32_t n, const DiaOffsets& offs, int nd_pad, bool jacobi, bool sym, int sm_count,
                      ResidentPlan& p);
template <typename T>
bool resident_bicg_plan(uint32_t n, const DiaOffsets& offs, int nd_pad, int sm_count, ResidentPlan& p);
template <typename VA, typename VG>
bool resident_pcg_plan(const DiaPcgArgs<VA, VG>& a, bool learned, int sm_count, ResidentPlan& p);

// Whether a plan leaves diagonals in L2 (a symmetric A may then keep more).
inline bool resident_streams(const ResidentPlan& p, int nd) {
    for (int d = 0; d < nd; ++d)
        if (p.at[d] < 0) return true;
    return false;
}

// The exchange area of a launch with `halos` vectors whose edge rows travel as
// words: bytes to allocate and to zero before it, and its parts.
size_t word_sync_bytes(const ResidentPlan& p, uint32_t n, size_t value_bytes, int halos);
WordSync word_sync_at(void* base, const ResidentPlan& p, unsigned long long wait_ns, int never_release);

template <typename T>
cudaError_t launch_cg_resident(const DiaCgArgs<T>& a, const ResidentPlan& plan, const WordSync& words, cudaStream_t s);
template <typename T>
cudaError_t launch_bicg_resident(const DiaBicgArgs<T>& a, const ResidentPlan& plan, const WordSync& words,
                                 cudaStream_t s);
template <typename VA, typename VG>
cudaError_t launch_pcg_resident(const DiaPcgArgs<VA, VG>& a, bool learned, const ResidentPlan& plan,
                                const WordSync& words, cudaStream_t s);

}  // namespace clsp
