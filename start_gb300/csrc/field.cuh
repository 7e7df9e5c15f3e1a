// Stamp check of the lazily computed per-tet field (FieldArgs), shared by the
// FP64 and the mixed-form kernels. The stamp is read from L2, so a stamp that
// another SM swapped in this kernel is seen; the lane whose compare-and-swap
// succeeds computes the tet, every other lane skips it.
#ifndef SPG_FIELD_CUH
#define SPG_FIELD_CUH

#include <cstdint>

#include "spg_internal.h"

namespace spg {

// Sets or clears kRecEzero of a mixed-form record, whose other flags stay.
__device__ __forceinline__ void set_rec_ezero(TetRec32 &r, bool zero) {
    *reinterpret_cast<uint8_t *>(&r.ezero) = zero ? uint8_t(kRecEzero) : uint8_t(0);
}

// Whether a tet's field is of the current potential (stamp >= epoch) and was
// stored by a launch before the one that stamps with seq.
__device__ __forceinline__ bool stored_before(uint32_t stamp, uint32_t epoch, uint32_t seq) {
    return stamp >= epoch && stamp < seq;
}

template <class F>
__device__ __forceinline__ void refresh_tet(uint32_t *stamp, uint32_t epoch, int t, F compute) {
    const uint32_t old = __ldcg(stamp + t);
    if (old >= epoch) return;
    if (atomicCAS(stamp + t, old, epoch) == old) compute(t);
}

}  // namespace spg

#endif
