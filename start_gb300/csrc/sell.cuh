// SELL-32 sparse row times vector, shared by the PCG and AMG kernels.
#ifndef SPG_SELL_CUH
#define SPG_SELL_CUH

#include <cstdint>

#include "spg_internal.h"

namespace spg {

// Rows are grouped in slices of 32 (one warp), each slice padded to its
// longest row and stored column-major, so lane l of a warp reads entry j of its
// row at slice_ptr[s] + 32 j + l and a warp's 32 loads of one j are contiguous.
// Padding entries have value 0. The slice width is the same for the 32 lanes of
// a warp, so the loops branch uniformly.
//
// Band = true is for matrices most of whose slices are banded (band_sell32):
// entry j of lane l is in column sref[j] + l, as for the rows of a mesh numbered
// along lines, so the warp reads one column word per j instead of 32 and x at
// consecutive addresses. That is 4 of the 8 bytes (FP32) or 12 bytes (FP64) of
// an entry, and one memory latency: the values need not wait for the columns
// nor x for a gathered address. Jacobi step of the 1.03e6-node cube, FP32
// 11.6 -> 8.9 us, FP64 30.0 -> 24.5 us from L2. The few other slices of such a
// matrix (bit 0 of their word in stag is 0) take a plain loop; matrices with
// fewer banded slices than others take Band = false, eight entries of a row in
// flight at a time with their column and value loads issued before the
// gathers.
// xf(c) supplies x[c]: a plain gather, or a value formed from several vectors
// at the gathered column.
template <class T>
struct SellMat {
    const int64_t *slice_ptr;
    const int32_t *scol;
    const T *sval;
    const int64_t *stag;  // Band: slice_ptr with bit 0 marking the banded slices
    const int32_t *sref;  // Band: per slice and entry (slice_ptr / 32 + j), the column of lane 0
};

template <class T>
__device__ __forceinline__ SellMat<T> sell_of(const DevSellT<T> &M) {
    return {M.slice_ptr, M.scol, M.sval, M.stag, M.sref};
}

template <class T, class X>
__device__ __forceinline__ T sell_row_band(const SellMat<T> &M, X xf, int64_t i) {
    const int64_t s = i >> 5;
    const int lane = int(i & 31);
    const int64_t p0 = __ldg(M.stag + s), p1 = __ldg(M.stag + s + 1);
    const int w = int((p1 >> 5) - (p0 >> 5));
    const T *val = M.sval + (p0 & ~int64_t(31)) + lane;
    T a0 = T(0), a1 = T(0);
    if (p0 & 1) {
        const int32_t *ref = M.sref + (p0 >> 5);
#pragma unroll 1
        for (int j = 0; j < w; j += 8) {
            T v[8], xv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) {
                    v[u] = __ldg(val + 32 * (j + u));
                    xv[u] = xf(__ldg(ref + j + u) + lane);
                }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) {
                    if (u & 1)
                        a1 = fma(v[u], xv[u], a1);
                    else
                        a0 = fma(v[u], xv[u], a0);
                }
        }
    } else {
        const int32_t *col = M.scol + (p0 & ~int64_t(31)) + lane;
#pragma unroll 2
        for (int j = 0; j < w; ++j) a0 = fma(__ldg(val + 32 * j), xf(__ldg(col + 32 * j)), a0);
    }
    return a0 + a1;
}

template <class T, class X>
__device__ __forceinline__ T sell_row_plain(const SellMat<T> &M, X xf, int64_t i) {
    const int64_t s = i >> 5;
    const int64_t base = __ldg(M.slice_ptr + s) + (i & 31);
    const int w = int((__ldg(M.slice_ptr + s + 1) - __ldg(M.slice_ptr + s)) >> 5);
    T a0 = T(0), a1 = T(0);
    int j = 0;
    for (; j + 8 <= w; j += 8) {
        int32_t c[8];
        T v[8], xv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            c[u] = __ldg(M.scol + base + 32 * (j + u));
            v[u] = __ldg(M.sval + base + 32 * (j + u));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) xv[u] = xf(c[u]);
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            a0 = fma(v[u], xv[u], a0);
            a1 = fma(v[u + 1], xv[u + 1], a1);
        }
    }
    const int rem = w - j;  // 0..7, warp-uniform
    if (rem > 0) {
        int32_t c[7];
        T v[7], xv[7];
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (u < rem) {
                c[u] = __ldg(M.scol + base + 32 * (j + u));
                v[u] = __ldg(M.sval + base + 32 * (j + u));
            }
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (u < rem) xv[u] = xf(c[u]);
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (u < rem) {
                if (u & 1)
                    a1 = fma(v[u], xv[u], a1);
                else
                    a0 = fma(v[u], xv[u], a0);
            }
    }
    return a0 + a1;
}

template <bool Band, class T>
__device__ __forceinline__ T spmv_row_sell(const SellMat<T> &M, const T *__restrict__ x, int64_t i) {
    auto xf = [x](int32_t c) { return __ldg(x + c); };
    if constexpr (Band)
        return sell_row_band(M, xf, i);
    else
        return sell_row_plain(M, xf, i);
}

// A row read in two parts (FP32 kernels of a dependent chain): the head holds
// what does not depend on x, the extents and the first eight entries, and is
// loaded before the kernel waits for its predecessor. (In FP64 the head's 24
// registers cost more in resident warps than they hide: 29.0 against 26.8 us
// for the SpMV of the 1.03e6-node cube.)
template <class T, bool Band>
struct SellHead {
    int64_t base;  // of this lane
    int w;
    bool band;
    int32_t c[8];
    T v[8];

    __device__ __forceinline__ void fetch(const SellMat<T> &M, int lane, int j) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (j + u < w) v[u] = __ldg(M.sval + base + 32 * (j + u));
        if (Band && band) {
            const int32_t *ref = M.sref + ((base - lane) >> 5);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) c[u] = __ldg(ref + j + u) + lane;
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) c[u] = __ldg(M.scol + base + 32 * (j + u));
        }
    }
    __device__ __forceinline__ void load(const SellMat<T> &M, int64_t i) {
        const int64_t s = i >> 5;
        const int64_t *sp = Band ? M.stag : M.slice_ptr;
        const int64_t p0 = __ldg(sp + s), p1 = __ldg(sp + s + 1);
        band = p0 & 1;
        w = int((p1 >> 5) - (p0 >> 5));
        base = (p0 & ~int64_t(31)) + (i & 31);
        fetch(M, int(i & 31), 0);
    }
    template <class X>
    __device__ __forceinline__ T finish(const SellMat<T> &M, X xf, int64_t i) {
        T a0 = T(0), a1 = T(0);
        int j = 0;
        while (true) {
            T xv[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) xv[u] = xf(c[u]);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (j + u < w) {
                    if (u & 1)
                        a1 = fma(v[u], xv[u], a1);
                    else
                        a0 = fma(v[u], xv[u], a0);
                }
            j += 8;
            if (j >= w) return a0 + a1;
            fetch(M, int(i & 31), j);
        }
    }
};

}  // namespace spg

#endif
