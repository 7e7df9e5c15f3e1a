// Shared by the segment kernels of both precisions: the collision candidates
// of a segment's steps.
#ifndef SPG_SEGMENT_CUH
#define SPG_SEGMENT_CUH

#include "philox.h"
#include "spg_internal.h"

namespace spg {

// Bit j: step c.step + j (j < L <= 64) of particle id is a collision candidate
// (its byte of the Philox block of its sixteen steps is zero).
__device__ __forceinline__ unsigned long long segment_candidates(const StepConst &c, uint32_t id, int L) {
    unsigned long long cand = 0ull;
    const int first = int(uint32_t(c.step) & 15u);
    for (int g = 0; 16 * g < first + L; ++g) {
        const unsigned long long m =
            candidate_mask(candidate_block(uint64_t(c.step) + 16ull * uint64_t(g), id, c.seed_lo, c.seed_hi));
        const int at = 16 * g - first;
        cand |= at >= 0 ? m << at : m >> -at;
    }
    return cand;
}

}  // namespace spg

#endif
