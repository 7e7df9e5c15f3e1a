// V-cycle of the smoothed-aggregation AMG preconditioner (hierarchy from
// amg_setup.cpp). Per level: a damped Jacobi step from a zero guess, residual,
// restriction R = P^T, the coarser level, prolongation, and the same Jacobi
// step again; the coarsest level multiplies by its dense inverse. Pre- and
// post-smoother are the same, so the V-cycle is a symmetric positive definite
// operator and CG stays CG.
// Operators with short rows are stored SELL-32 with one thread per row (level
// 0 shares the solver's matrix); long rows (coarse operators, restriction)
// CSR with 4-32 lanes per row. No atomics, so z = M^-1 r is deterministic.
#include "pdl.cuh"
#include "sell.cuh"
#include "spg_internal.h"

namespace spg {

namespace {

constexpr int kT = 256;
constexpr int kBanded = kSellBanded;

// converged: 1 or 2 (plain PCG), or 3 (inner cap of the mixed form)
// (Every V-cycle kernel comes here before it reads a vector: pdl_wait orders it
// after its predecessor.)
__device__ __forceinline__ bool done(const PcgScalars *sc) {
    pdl_sync();
    return sc && *(volatile const int *)&sc->converged;
}

// Row `row` of M x, xf(c) = x[c], in two parts: RowHead holds what does not
// depend on x (the row's extents and its first entries) and is loaded before
// the kernel waits for its predecessor, so that a kernel whose grid is already
// on the chip spends its first two memory latencies while the predecessor
// ends. The small levels are bound by those latencies: one PCG iteration with
// the FP32 V-cycle took 41.4 us at 9,261 nodes, 75 at 132,651 and 235 at
// 1.03e6, and takes 32.7, 62.7 and 191 with the heads, the stored x0
// (k_restrict) and the banded level 0 (sell.cuh); with the FP64 V-cycle 50.6,
// 113 and 330 before, 40.5, 101 and 305 now (level 0 bound by FP64 issue: 8
// fused multiply-adds a row take 16.5 us at the measured rate).
// G = 0 or kBanded: SELL-32, the calling thread owns the row. G > 0: CSR, the
// G lanes of a group (lane = lane index within the group) stride over the
// row's entries, four per lane in flight, and a butterfly over the group leaves
// the sum in every lane of the group. Every lane of a warp joins the
// butterflies; rows past n read nothing.
template <class T, int G>
struct RowHead {
    int64_t k, k1;  // this lane's first entry, the row's end
    int32_t c[4];
    T v[4];
    __device__ __forceinline__ void fetch(const DevSellT<T> &M) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t kk = k + int64_t(u) * G;
            c[u] = kk < k1 ? __ldg(M.scol + kk) : -1;
            v[u] = kk < k1 ? __ldg(M.sval + kk) : T(0);
        }
    }
    __device__ __forceinline__ RowHead(const DevSellT<T> &M, int64_t row, int lane, int64_t n) {
        k = k1 = 0;
        if (row < n) {
            k = __ldg(M.slice_ptr + row) + lane;
            k1 = __ldg(M.slice_ptr + row + 1);
        }
        fetch(M);
    }
    template <class X>
    __device__ __forceinline__ T finish(const DevSellT<T> &M, X xf, int64_t, int64_t) {
        T a0 = T(0), a1 = T(0);
        while (true) {
            T x[4];
            const bool full = c[3] >= 0;  // four entries; else the lane's last ones
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = c[u] >= 0 ? xf(c[u]) : T(0);
            if (!full) {
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (c[u] >= 0) a0 = fma(v[u], x[u], a0);
                break;
            }
            a0 = fma(v[0], x[0], a0);
            a1 = fma(v[1], x[1], a1);
            a0 = fma(v[2], x[2], a0);
            a1 = fma(v[3], x[3], a1);
            k += 4 * G;
            fetch(M);
        }
        T s = a0 + a1;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off, G);
        return s;
    }
};

template <bool Band>
struct SellRow32 {
    SellHead<float, Band> h;
    __device__ __forceinline__ SellRow32(const DevSellT<float> &M, int64_t row, int, int64_t n) {
        if (row < n) h.load(sell_of(M), row);
    }
    template <class X>
    __device__ __forceinline__ float finish(const DevSellT<float> &M, X xf, int64_t row, int64_t n) {
        return row < n ? h.finish(sell_of(M), xf, row) : 0.0f;
    }
};
template <bool Band>
struct SellRow64 {
    __device__ __forceinline__ SellRow64(const DevSellT<double> &, int64_t, int, int64_t) {}
    template <class X>
    __device__ __forceinline__ double finish(const DevSellT<double> &M, X xf, int64_t row, int64_t n) {
        if (row >= n) return 0.0;
        if constexpr (Band)
            return sell_row_band(sell_of(M), xf, row);
        else
            return sell_row_plain(sell_of(M), xf, row);
    }
};
template <>
struct RowHead<float, 0> : SellRow32<false> {
    using SellRow32<false>::SellRow32;
};
template <>
struct RowHead<float, kBanded> : SellRow32<true> {
    using SellRow32<true>::SellRow32;
};
template <>
struct RowHead<double, 0> : SellRow64<false> {
    using SellRow64<false>::SellRow64;
};
template <>
struct RowHead<double, kBanded> : SellRow64<true> {
    using SellRow64<true>::SellRow64;
};

// Thread -> (row, lane within the row's group); `own`: this thread writes the row.
template <int G>
__device__ __forceinline__ void row_of(int64_t n, int64_t &row, int &lane, bool &own) {
    const int64_t t = int64_t(blockIdx.x) * kT + threadIdx.x;
    if constexpr (G <= 0) {
        row = t;
        lane = 0;
    } else {
        row = t / G;
        lane = int(t % G);
    }
    own = row < n && lane == 0;
}

template <class T>
__device__ __forceinline__ auto plain(const T *__restrict__ x) {
    return [x](int32_t c) { return __ldg(x + c); };
}

// r = b - A x_in
template <class T, int G>
__global__ void __launch_bounds__(kT) k_resid(const AmgLevelDevT<T> L, const T *__restrict__ b,
                                              const T *__restrict__ xin, const PcgScalars *sc) {
    int64_t i;
    int lane;
    bool own;
    row_of<G>(L.n, i, lane, own);
    pdl_trigger();
    RowHead<T, G> row(L.A, i, lane, L.n);
    if (done(sc)) return;
    const T ax = row.finish(L.A, plain(xin), i, L.n);
    if (own) L.r[i] = b[i] - ax;
}

// Degree 1 post-smoothing: x_out = x_in + D^-1 (b - A x_in) / theta
template <class T, int G>
__global__ void __launch_bounds__(kT) k_jacobi_step(const AmgLevelDevT<T> L, const T *__restrict__ b,
                                                    const T *__restrict__ xin, T *__restrict__ xout,
                                                    const PcgScalars *sc) {
    int64_t i;
    int lane;
    bool own;
    row_of<G>(L.n, i, lane, own);
    pdl_trigger();
    RowHead<T, G> row(L.A, i, lane, L.n);
    if (done(sc)) return;
    const T ax = row.finish(L.A, plain(xin), i, L.n);
    if (!own) return;
    const T r = b[i] - ax;
    xout[i] = xin[i] + T(L.inv_theta) * (L.dinv[i] * r);
}

// b_next = R r, and the next level's first smoothing step from x = 0 with it,
// x0 = D^-1 b / theta (x0 null: the next level is the coarsest, which has
// none). Level 0's x0 is written by the kernel that writes its b, the PCG's
// residual: so the residual and the prolongation of every level gather and
// read one stored vector, where forming x0 at each gathered column takes two
// (residual of 39,764 rows of 258 entries: 18.4 us so, 13.0 us from the stored
// vector), and no kernel is launched for it alone.
template <class T, int G>
__global__ void __launch_bounds__(kT) k_restrict(const DevSellT<T> R, const T *__restrict__ r, T *__restrict__ bnext,
                                                 const T *__restrict__ dinv, T inv_theta, T *__restrict__ x0,
                                                 const PcgScalars *sc) {
    int64_t i;
    int lane;
    bool own;
    row_of<G>(R.n, i, lane, own);
    pdl_trigger();
    RowHead<T, G> row(R, i, lane, R.n);
    const T di = own && x0 ? __ldg(dinv + i) : T(0);
    if (done(sc)) return;
    const T v = row.finish(R, plain(r), i, R.n);
    if (!own) return;
    bnext[i] = v;
    if (x0) x0[i] = inv_theta * (di * v);
}

// x_out = x_in + P x_coarse
template <class T, int G>
__global__ void __launch_bounds__(kT) k_prolong(const DevSellT<T> P, const T *__restrict__ xin,
                                                const T *__restrict__ xc, T *__restrict__ xout, const PcgScalars *sc) {
    int64_t i;
    int lane;
    bool own;
    row_of<G>(P.n, i, lane, own);
    pdl_trigger();
    RowHead<T, G> row(P, i, lane, P.n);
    if (done(sc)) return;
    const T v = row.finish(P, plain(xc), i, P.n);
    if (own) xout[i] = xin[i] + v;
}

// x = A_c^-1 b: one warp per row of the dense inverse, fixed-order lane sums.
template <class T>
__global__ void __launch_bounds__(kT) k_coarse(const T *__restrict__ inv, int64_t nc, const T *__restrict__ b,
                                               T *__restrict__ x, const PcgScalars *sc) {
    if (done(sc)) return;
    const int64_t row = (int64_t(blockIdx.x) * kT + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= nc) return;
    T s = T(0);
    for (int64_t k = lane; k < nc; k += 32) s += inv[row * nc + k] * b[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) x[row] = s;
}

inline unsigned blocks_for(int64_t n, int g = 0) {
    const int64_t threads = n * (g > 0 ? g : 1);
    return unsigned((threads + kT - 1) / kT);
}

#define SPG_AMG_DISPATCH(g, KERNEL, GRIDN, ...)                                             \
    switch (g) {                                                                            \
    case kBanded: launch_pdl(KERNEL<T, kBanded>, blocks_for(GRIDN, 0), kT, s, __VA_ARGS__); break; \
    case 4: launch_pdl(KERNEL<T, 4>, blocks_for(GRIDN, 4), kT, s, __VA_ARGS__); break;     \
    case 8: launch_pdl(KERNEL<T, 8>, blocks_for(GRIDN, 8), kT, s, __VA_ARGS__); break;     \
    case 16: launch_pdl(KERNEL<T, 16>, blocks_for(GRIDN, 16), kT, s, __VA_ARGS__); break;  \
    case 32: launch_pdl(KERNEL<T, 32>, blocks_for(GRIDN, 32), kT, s, __VA_ARGS__); break;  \
    default: launch_pdl(KERNEL<T, 0>, blocks_for(GRIDN, 0), kT, s, __VA_ARGS__); break;    \
    }

// xa holds x0 = D^-1 b / theta on entry (not on the coarsest level) and the
// result on return. skip_last: level 0's last Jacobi step (L.x[1] -> z) is
// left to the caller, which fuses it with the PCG's r.z.
template <class T>
void vcycle_level(const AmgDevT<T> &a, int l, const T *b, T *xa, const PcgScalars *sc, cudaStream_t s,
                  bool skip_last = false) {
    const AmgLevelDevT<T> &L = a.lev[l];
    if (l == a.levels - 1) {
        launch_pdl(k_coarse<T>, unsigned((a.nc * 32 + kT - 1) / kT), kT, s, a.coarse_inv, a.nc, b, xa, sc);
        return;
    }
    T *xb = L.x[1];
    const int ga = L.A.g;
    const AmgLevelDevT<T> &N = a.lev[l + 1];
    T *x0 = l + 2 < a.levels ? N.x[0] : nullptr;  // the coarsest level has no smoothing
    SPG_AMG_DISPATCH(ga, k_resid, L.n, L, b, xa, sc)
    SPG_AMG_DISPATCH(L.R.g, k_restrict, L.R.n, L.R, L.r, N.b, N.dinv, T(N.inv_theta), x0, sc)
    vcycle_level<T>(a, l + 1, N.b, N.x[0], sc, s);
    SPG_AMG_DISPATCH(L.P.g, k_prolong, L.P.n, L.P, xa, N.x[0], xb, sc)
    if (skip_last) return;
    SPG_AMG_DISPATCH(ga, k_jacobi_step, L.n, L, b, xb, xa, sc)
}

}  // namespace

void launch_amg_vcycle(const AmgDev &a, const double *r, double *z, const PcgScalars *sc, cudaStream_t s) {
    vcycle_level<double>(a, 0, r, z, sc, s, a.levels > 1);
}

void launch_amg_vcycle(const AmgDev32 &a, const float *r, float *z, const PcgScalars *sc, cudaStream_t s) {
    vcycle_level<float>(a, 0, r, z, sc, s, a.levels > 1);
}

}  // namespace spg
