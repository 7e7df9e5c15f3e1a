// Jacobi-preconditioned CG of a small or medium system as one kernel launch.
//
// The system lives on the chip for the whole solve: one thread per row holds
// x, r, p and the inverse diagonal in registers and its matrix row in shared
// memory, and what other rows need of a row, its record {z, p, u = D^-1 A p},
// lies in a pair of small arrays. An iteration has one exchange of sums:
//   p = z + beta p, q = A p (of a coupled row, z less alpha u and p plus beta
//   times the published p, so that no pass and no barrier is spent on the
//   updates), {z, p, u} stored into the other array of the pair;
//   the sums p.q, z.q, u.q, r.z and r.r over all rows;
//   alpha = r.z / p.q; x += alpha p, r -= alpha q, z = D^-1 r.
// The next r.z, which beta needs before the next sums, is predicted from this
// exchange, r.z - 2 alpha z.q + alpha^2 u.q, and formed from the vectors in the
// next one, so no rounding of a prediction is carried on ("predict and
// recompute", Chen and Carson, SIAM J. Sci. Comput. 42, 2020). The stop test
// sees r.r of an update one exchange later, before anything else is updated.
// With the values of k_spmv_dot, k_update and k_pupdate it differs by rounding
// alone (solves of up to 190 iterations: 1e-15 of x), and every sum has a fixed
// order, so a solve is deterministic.
//
// What bounds it is latency: the exchange (a tree over the block, a barrier over
// the blocks, a tree over their partial sums) and the FP64 chains around it. On
// GB300 an FP64 instruction holds its warp's scheduler for 63 cycles (about 1.7
// operations per clock and SM in all), a division takes 1,470.
// Two forms:
//   * cluster: up to 16 blocks in one cluster, the records in distributed shared
//     memory, the hardware barrier (400 to 600 cycles). Its 16 SMs issue few
//     FP64 operations, so it ends where the grid becomes faster, at 4,096 rows:
//     us an iteration, cluster / grid, 1,331 rows 4.1 / 5.1, 3,375 5.0 / 5.3,
//     4,096 5.4 / 5.3, 4,913 5.9 / 5.4 (3 % between cards).
//   * grid: up to one block per SM, cooperative launch, the records in L2, a counter
//     in global memory as the barrier (1.2 us). It ends at one row per thread,
//     155,648 rows on 152 SMs.
// Measured per iteration of the lattice Laplacian: three kernels per iteration in
// a graph; one launch with two exchanges per iteration ({z, p} published); one
// exchange: 1,331 rows 22, 4.4, 4.1 us; 5,832 rows -, 6.0, 5.2; 17,576 rows 22, 7.0,
// 5.6; 68,921 rows -, 9.1, 8.9; 132,651 rows 24, 12.4, 13.6 (there the FP64 pipe is
// full and the gathers' second multiply-add costs what the exchange saves).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "newton_div.h"
#include "pcg_resident.h"
#include "spg_internal.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSums = kResidentSums;
constexpr int kMaxCluster = 16;
// Polls of the grid barrier before a block gives up (each takes most of a
// microsecond): a few seconds. The cooperative launch makes every block
// resident, so the limit is never met in a healthy run.
constexpr int kMaxPolls = 1 << 22;

// Quotients on the critical path of every iteration (newton_div.h); operands
// beyond its range take the division, out of line so that it is not computed
// beside the fast form.
__device__ __noinline__ double divide(double a, double b) { return a / b; }
__device__ __forceinline__ double quotient(double a, double b, double y) {
    return newton_range(a) && newton_range(b) ? newton_quotient(a, b, y) : divide(a, b);
}

// Row access of the two matrix formats: entry k of the row is col[at(k)],
// val[at(k)], k < count.
struct RowRef {
    int64_t base;
    int stride, count;
    __device__ __forceinline__ int64_t at(int k) const { return base + int64_t(k) * stride; }
};

__device__ __forceinline__ RowRef row_ref(const ResidentArgs &a, int i) {
    if (a.slice_ptr) {
        const int s = i >> 5;
        const int64_t p0 = __ldg(a.slice_ptr + s), p1 = __ldg(a.slice_ptr + s + 1);
        return RowRef{p0 + (i & 31), 32, int((p1 - p0) >> 5)};
    }
    const int32_t k0 = __ldg(a.row_ptr + i), k1 = __ldg(a.row_ptr + i + 1);
    return RowRef{k0, 1, k1 - k0};
}

// What a row publishes for the rows coupled to it.
struct Zpu {
    double z, p, u;
};

__device__ __forceinline__ Zpu load_zpu(const ZpuRec *p) {
    Zpu r;  // not a read-only load: other blocks write the array between the barriers
    double unused;
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(r.z), "=d"(r.p), "=d"(r.u), "=d"(unused)
                 : "l"(p)
                 : "memory");
    return r;
}
__device__ __forceinline__ Zpu load_zpu_cluster(uint32_t addr) {
    Zpu r;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(r.z), "=d"(r.p) : "r"(addr) : "memory");
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(r.u) : "r"(addr + 16u) : "memory");
    return r;
}

__device__ __forceinline__ uint32_t shared_addr(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct Shared {
    double tot[kSums];                   // the totals of the last exchange
    double warp[4][kSums];               // the sums of the first four warps' columns
    double part[2][kSums][kMaxCluster];  // cluster form: every block's partial sums
    double alpha, beta;
    int stop, timed_out;
};

// v[k] summed over the warp; lane 16 (k & 1) + 8 (k >> 1) gets value k < 4, lane
// 4 value 4. Lanes hand over the value they do not keep, so the five sums take
// eight FP64 additions instead of 25.
__device__ __forceinline__ double warp_sums(const double (&v)[kSums]) {
    const int lane = threadIdx.x & 31;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    const double x01 = (b4 ? v[1] : v[0]) + __shfl_xor_sync(kFull, b4 ? v[0] : v[1], 16);
    const double x23 = (b4 ? v[3] : v[2]) + __shfl_xor_sync(kFull, b4 ? v[2] : v[3], 16);
    double x4 = v[4] + __shfl_xor_sync(kFull, v[4], 16);
    const double y = (b3 ? x23 : x01) + __shfl_xor_sync(kFull, b3 ? x01 : x23, 8);
    x4 += __shfl_xor_sync(kFull, x4, 8);
    double w = (b2 ? x4 : y) + __shfl_xor_sync(kFull, b2 ? y : x4, 4);
    w += __shfl_xor_sync(kFull, w, 2);
    w += __shfl_xor_sync(kFull, w, 1);
    return w;
}

// One exchange: the totals over all rows of the five values per thread in
// buf[k T + t], into s.tot[k] (read after the caller's barrier). Everything the
// block wrote before is visible to every block afterwards. An FP64 instruction
// holds its warp's scheduler for 63 cycles whatever its lanes and independence,
// so four warps, one per scheduler, add the columns of a large block and sum
// five values together, and half a warp each sums two values over the blocks.
// target: arrivals after which this exchange is complete (grid form). Out of
// line: one copy for every call.
template <bool CLUSTER>
__device__ __noinline__ void exchange(double *partials, unsigned int *arrived, Shared &s, double *buf, unsigned par,
                                      unsigned target) {
    const int T = blockDim.x, t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = T >> 5;
    const int G = int(gridDim.x);
    __syncthreads();
    if (t < 128) {
        double v[kSums];
#pragma unroll
        for (int k = 0; k < kSums; ++k) v[k] = buf[k * T + t];
        for (int j = t + 128; j < T; j += 128)
#pragma unroll
            for (int k = 0; k < kSums; ++k) v[k] += buf[k * T + j];
        const double w = warp_sums(v);
        if ((lane & 7) == 0) s.warp[wid][(lane >> 4) + 2 * ((lane >> 3) & 1)] = w;
        if (lane == 4) s.warp[wid][4] = w;
    }
    __syncthreads();
    if (wid == 0) {
        const int k = lane >> 2, w = lane & 3;
        double q = k < kSums && w < nw ? s.warp[w][k] : 0.0;
        q += __shfl_xor_sync(kFull, q, 1);
        q += __shfl_xor_sync(kFull, q, 2);
        if constexpr (CLUSTER) {
            for (int e0 = 0; e0 < kSums * G; e0 += 32) {  // value e % 5 to block e / 5
                const int e = e0 + lane, rank = e / kSums, v = e - rank * kSums;
                const double out = __shfl_sync(kFull, q, 4 * v);
                if (rank < G)
                    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(
                                     map_rank(shared_addr(&s.part[par][v][blockIdx.x]), unsigned(rank))),
                                 "d"(out)
                                 : "memory");
            }
        } else {
            if (k < kSums && w == 0) partials[(size_t(par) * kSums + k) * G + blockIdx.x] = q;
            __syncwarp();
            if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
        }
    }
    if constexpr (CLUSTER) cluster_barrier();
    const int hl = lane & 15;
    for (int k0 = 2 * wid; k0 < kSums; k0 += 2 * nw) {
        const int k = k0 + (lane >> 4);
        double w = 0.0;
        if constexpr (CLUSTER) {
            if (k < kSums && hl < G) w = s.part[par][k][hl];
        } else {
            unsigned got;
            int polls = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(arrived) : "memory");
            } while (got < target && ++polls < kMaxPolls);
            if (got < target) s.timed_out = 1;
            __syncwarp();
            // the blocks' partial sums, ten per lane in flight together
            const double *p = partials + (size_t(par) * kSums + (k < kSums ? k : 0)) * G;
            for (int b0 = 0; b0 < G; b0 += 160) {
                double u[10];
#pragma unroll
                for (int q = 0; q < 10; ++q) u[q] = b0 + 16 * q + hl < G ? __ldcg(p + b0 + 16 * q + hl) : 0.0;
#pragma unroll
                for (int q = 0; q < 10; ++q)
                    if (b0 + 16 * q < G) w += u[q];
            }
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) w += __shfl_xor_sync(kFull, w, off);
        if (hl == 0 && k < kSums) s.tot[k] = w;
        __syncwarp();
    }
}

// Positive and no NaN, by its bits.
__device__ __forceinline__ bool positive(double a) {
    const long long b = __double_as_longlong(a);
    return b > 0 && b <= 0x7ff0000000000000LL;
}

constexpr int kGathers = 6;  // gathers in flight per thread: the off-diagonal entries of a lattice row

template <bool CLUSTER, int TMAX>
__global__ void __launch_bounds__(TMAX, 1) k_pcg_resident(const __grid_constant__ ResidentArgs a) {
    extern __shared__ __align__(32) unsigned char dyn[];
    __shared__ Shared s;
    const int T = blockDim.x, t = threadIdx.x, wid = t >> 5;
    const int i = blockIdx.x * T + t;
    const bool act = i < a.n;
    // dynamic shared memory: cluster form's records [2][T], the exchange's
    // values [kSums][T], the staged matrix entries' values and places [staged][T]
    ZpuRec *zp_sh = reinterpret_cast<ZpuRec *>(dyn);
    double *buf = reinterpret_cast<double *>(zp_sh + (CLUSTER ? 2 * T : 0));
    double *mval = buf + kSums * T;
    int32_t *mcol = reinterpret_cast<int32_t *>(mval + size_t(a.staged) * T);
    unsigned par = 0, target = 0;
    auto sums = [&] {
        target += gridDim.x;
        exchange<CLUSTER>(a.partials, a.arrived, s, buf, par, target);
        par ^= 1u;
    };
    auto publish = [&](int half, double z, double p, double u) {
        if constexpr (CLUSTER)
            zp_sh[half * T + t] = ZpuRec{z, p, u, 0.0};
        else
            a.zpu[half][i] = ZpuRec{z, p, u, 0.0};
    };
    if (t == 0) s.timed_out = 0;

    const RowRef row = act ? row_ref(a, i) : RowRef{0, 1, 0};
    // place of column c's record: its index, or its shared address in the cluster
    auto place = [&](int32_t c) -> int32_t {
        if constexpr (CLUSTER) {
            const uint32_t rank = uint32_t(c) / uint32_t(T);
            return int32_t(map_rank(shared_addr(zp_sh + (uint32_t(c) - rank * uint32_t(T))), rank));
        } else {
            return c;
        }
    };

    // ---- r = b - A x, z = D^-1 r. The row's couplings to other rows go to
    // shared memory while they fit (entries from `next` on are read again in
    // every iteration); exact zeros are left out, the diagonal stays apart.
    double x = 0.0, r = 0.0, z = 0.0, p = 0.0, dinv = 1.0, diag = 0.0, last = 0.0;
    int staged = 0, next = row.count;
    double rz0 = 0.0, bb0 = 0.0, rr0 = 0.0, bad = 0.0;
    if (act) {
        double a0 = 0.0, a1 = 0.0;
        bool found = false;
        for (int k = 0; k < row.count; ++k) {
            const int32_t c = __ldg(a.col + row.at(k));
            const double m = __ldg(a.val + row.at(k));
            if (c == i) {
                diag += m;
                last = m;
                found = true;
            } else if (m != 0.0) {
                if (staged < a.staged) {
                    mval[staged * T + t] = m;
                    mcol[staged * T + t] = place(c);
                    ++staged;
                } else if (next == row.count) {
                    next = k;
                }
            }
            const double xc = a.x[c];
            if (k & 1)
                a1 = fma(m, xc, a1);
            else
                a0 = fma(m, xc, a0);
        }
        if (a.inv_diag) {
            dinv = __ldg(a.inv_diag + i);
        } else {
            // (of several entries on the diagonal, the last one, as in k_na_setup)
            if (!found || !(fabs(last) > 0.0) || !isfinite(last)) bad = 1.0;
            dinv = bad != 0.0 ? 1.0 : 1.0 / last;
        }
        x = a.x[i];
        const double b = a.b[i];
        r = b - (a0 + a1);
        z = r * dinv;
        rz0 = r * z;
        bb0 = b * b;
        rr0 = r * r;
        publish(0, z, 0.0, 0.0);
    }
    // the warp's rows filled up to one even count with zero couplings of a row
    // to itself (or, past the last row, of nothing to the last), so that the
    // gathers need no tests
    {
        int most = __reduce_max_sync(kFull, staged);
        most = min(most + (most & 1), a.staged);
        const int32_t self = place(act ? i : a.n - 1);
        for (; staged < most; ++staged) {
            mval[staged * T + t] = 0.0;
            mcol[staged * T + t] = self;
        }
    }
    buf[t] = rz0;
    buf[T + t] = bb0;
    buf[2 * T + t] = rr0;
    buf[3 * T + t] = bad;
    buf[4 * T + t] = 0.0;
    if constexpr (CLUSTER) cluster_barrier();  // every block runs before its shared memory is written
    sums();
    __syncthreads();
    double rz = s.tot[0], rr = s.tot[2], pq = 0.0, alpha = 0.0, beta = 0.0;
    const double bb = s.tot[1], tol2 = a.rtol2 * bb;
    int iters = 0;
    int stop = s.timed_out ? kPcgTimedOut : s.tot[3] > 0.0 ? kPcgBadDiagonal : (rr <= tol2 || bb == 0.0) ? 1 : 0;
    // a zero right-hand side of the allocation-free solve gives x = 0 whatever the start
    const bool zero_x = a.zero_on_zero_b && bb == 0.0 && !s.timed_out;

    int cur = 0;
    while (stop == 0) {
        // ---- p = z + beta p and q = A p: of another row c, z is the z it
        // published less alpha u, and p that plus beta times the p it published
        p = fma(beta, p, z);
        double q;
        {
            double a0 = diag * p, a1 = 0.0;
            const uint32_t half = CLUSTER ? uint32_t(cur) * uint32_t(T) * uint32_t(sizeof(ZpuRec)) : 0u;
            const ZpuRec *src = CLUSTER ? nullptr : a.zpu[cur];
            auto get = [&](int32_t at) -> Zpu {
                if constexpr (CLUSTER)
                    return load_zpu_cluster(uint32_t(at) + half);
                else
                    return load_zpu(src + at);
            };
            auto dir = [&](const Zpu &g) { return fma(beta, g.p, fma(-alpha, g.u, g.z)); };
            int k = 0;
            for (; k + kGathers <= staged; k += kGathers) {
                Zpu g[kGathers];
#pragma unroll
                for (int u = 0; u < kGathers; ++u) g[u] = get(mcol[(k + u) * T + t]);
#pragma unroll
                for (int u = 0; u < kGathers; u += 2) {
                    a0 = fma(mval[(k + u) * T + t], dir(g[u]), a0);
                    a1 = fma(mval[(k + u + 1) * T + t], dir(g[u + 1]), a1);
                }
            }
            for (; k + 2 <= staged; k += 2) {
                const Zpu g0 = get(mcol[k * T + t]), g1 = get(mcol[(k + 1) * T + t]);
                a0 = fma(mval[k * T + t], dir(g0), a0);
                a1 = fma(mval[(k + 1) * T + t], dir(g1), a1);
            }
            if (k < staged) a0 = fma(mval[k * T + t], dir(get(mcol[k * T + t])), a0);  // an odd capacity
            for (k = next; k < row.count; ++k) {
                const int32_t c = __ldg(a.col + row.at(k));
                const double m = __ldg(a.val + row.at(k));
                if (c == i || m == 0.0) continue;
                a0 = fma(m, dir(get(place(c))), a0);
            }
            q = a0 + a1;
        }
        const double u = q * dinv;
        cur ^= 1;
        if (act) publish(cur, z, p, u);
        buf[t] = act ? p * q : 0.0;
        buf[T + t] = act ? z * q : 0.0;
        buf[2 * T + t] = act ? u * q : 0.0;
        buf[3 * T + t] = act ? r * z : 0.0;
        buf[4 * T + t] = act ? r * r : 0.0;
        sums();
        __syncthreads();
        if (wid == 0) {
            pq = s.tot[0];
            rz = s.tot[3];
            // the stop test of the last update, then p.q: not positive if A is not SPD on
            // this subspace, or NaN
            const int why = s.timed_out               ? kPcgTimedOut
                            : s.tot[4] <= tol2        ? 1
                            : iters > 0 && iters >= a.max_iter ? 2
                            : positive(pq)            ? 0
                                                      : kPcgBreakdown;
            const double y = newton_reciprocal((t & 1) ? rz : pq);  // both at once
            const double y0 = __shfl_sync(kFull, y, 0), y1 = __shfl_sync(kFull, y, 1);
            alpha = why ? 0.0 : quotient(rz, pq, y0);
            const double next_rz = fma(alpha * alpha, s.tot[2], fma(-2.0 * alpha, s.tot[1], rz));
            beta = positive(next_rz) ? quotient(next_rz, rz, y1) : 0.0;
            if (t == 0) {
                s.stop = why;
                s.alpha = alpha;
                s.beta = beta;
            }
        }
        __syncthreads();
        stop = s.stop;
        rr = s.tot[4];
        pq = s.tot[0];
        rz = s.tot[3];
        if (stop) break;
        alpha = s.alpha;
        beta = s.beta;
        // ---- x, r, z of the row
        r = fma(-alpha, q, r);
        z = r * dinv;
        x = fma(alpha, p, x);
        ++iters;
    }
    // a refused system keeps the caller's x
    if (act && (iters > 0 || zero_x)) a.x[i] = zero_x ? 0.0 : x;
    if (blockIdx.x == 0 && t == 0) {
        PcgScalars o{};
        o.rz = rz;
        o.pq = pq;
        o.alpha = alpha;
        o.beta = beta;
        o.rr = rr;
        o.bb = bb;
        o.tol2 = tol2;
        o.iters = iters;
        o.converged = stop == kPcgBadDiagonal ? 0 : (stop == kPcgBreakdown ? a.breakdown : stop);
        o.max_iter = a.max_iter;
        o.flags = stop == kPcgBadDiagonal ? 1 : 0;
        *a.sc = o;
    }
    if constexpr (CLUSTER) cluster_barrier();  // no block leaves while its shared memory may be read
}

// Rows up to which one cluster of 16 blocks is used.
constexpr int64_t kClusterRows = 4096;

using Kernel = void (*)(ResidentArgs);
Kernel kernel_of(const ResidentPlan &p) {
    if (p.cluster) return k_pcg_resident<true, int(kClusterRows) / kMaxCluster>;
    return p.threads <= 512 ? k_pcg_resident<false, 512> : k_pcg_resident<false, 1024>;
}

size_t smem_of(int threads, int staged, bool cluster) {
    return size_t(threads) * ((cluster ? 2 * sizeof(ZpuRec) : 0) + 8 * kSums + 12 * size_t(staged));
}

cudaLaunchConfig_t config_of(const ResidentPlan &p, cudaLaunchAttribute *attr, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(p.blocks));
    cfg.blockDim = dim3(unsigned(p.threads));
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    if (p.cluster) {
        attr->id = cudaLaunchAttributeClusterDimension;
        attr->val.clusterDim.x = unsigned(p.blocks);
        attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    } else {
        attr->id = cudaLaunchAttributeCooperative;
        attr->val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether the device runs this plan (opt-in shared memory, cluster size, all
// blocks resident). A kernel's limit of dynamic shared memory is one value per
// device that all its plans share, and plans outlive this call: it is set to all
// that the kernel's own arrays leave of the opt-in size, whatever this plan needs.
bool fits(const ResidentPlan &p, int sms, int optin) {
    const Kernel k = kernel_of(p);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k) != cudaSuccess || p.smem + fa.sharedSizeBytes > size_t(optin) ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - int(fa.sharedSizeBytes)) !=
            cudaSuccess ||
        (p.cluster &&
         cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
        cudaGetLastError();
        return false;
    }
    int got = 0;
    if (p.cluster) {
        cudaLaunchAttribute attr;
        const cudaLaunchConfig_t cfg = config_of(p, &attr, nullptr);
        if (cudaOccupancyMaxActiveClusters(&got, k, &cfg) != cudaSuccess) got = 0;
    } else if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&got, k, p.threads, p.smem) != cudaSuccess) {
        got = 0;
    }
    cudaGetLastError();
    return p.cluster ? got >= 1 : int64_t(got) * sms >= p.blocks;
}

}  // namespace

ResidentPlan resident_plan(int64_t n) {
    ResidentPlan p;
    int dev = 0, sms = 0, optin = 0;
    if (n <= 0 || cudaGetDevice(&dev) != cudaSuccess) return p;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaGetLastError();
    auto shape = [&](int blocks, int threads, bool cluster) {
        p.blocks = blocks;
        p.threads = threads;
        p.cluster = cluster;
        const int64_t room = int64_t(optin) - 4096 - int64_t(smem_of(threads, 0, cluster));
        p.staged = int(std::min<int64_t>(32, std::max<int64_t>(0, room / (12 * int64_t(threads)))));
        p.smem = smem_of(threads, p.staged, cluster);
        return fits(p, sms, optin);
    };
    if (n <= kClusterRows) {
        const int threads = int(std::max<int64_t>(64, ((n + kMaxCluster - 1) / kMaxCluster + 31) / 32 * 32));
        if (shape(int((n + threads - 1) / threads), threads, true)) return p;
    }
    for (int threads = 128; threads <= 1024; threads *= 2) {
        if (n > int64_t(sms) * threads) continue;
        const int64_t blocks = (n + threads - 1) / threads;
        if (blocks <= 512 && shape(int(blocks), threads, false)) return p;
    }
    return ResidentPlan{};
}

cudaError_t launch_pcg_resident(const ResidentPlan &plan, ResidentArgs a, cudaStream_t s) {
    a.staged = plan.staged;
    if (!plan.cluster) {
        const cudaError_t e = cudaMemsetAsync(a.arrived, 0, sizeof(unsigned int), s);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = config_of(plan, &attr, s);
    return cudaLaunchKernelEx(&cfg, kernel_of(plan), a);
}

}  // namespace spg
