// Jacobi-preconditioned CG of a small or medium system as one kernel launch.
//
// The system lives on the chip for the whole solve: one thread per row holds
// x, r, p and the inverse diagonal in registers and its matrix row in shared
// memory, and the search direction's ingredients {z, p} of every row lie in a
// pair of small arrays. An iteration is
//   phase A  p_k = z + beta p (own row, and again at every gathered column, so
//            that no pass and no barrier is spent on the p update), q = A p_k,
//            reduction of p.q;
//   phase B  x += alpha p, r -= alpha q, z = D^-1 r, {z, p} of the row stored
//            into the other array of the pair, reduction of r.z and r.r.
// Every value is formed by the operations of the separate kernels (k_spmv_dot,
// k_update, k_pupdate); only the sums over the rows (and the place of the
// diagonal in a row's sum) are taken in another fixed order, so a solve is
// deterministic and differs from those kernels by rounding alone.
//
// What bounds it is latency: two exchanges of sums per iteration, each a tree
// over the block, a barrier over the blocks and a tree over their partial
// sums. On GB300 an FP64 instruction holds its warp's scheduler for 63 cycles
// (about 1.7 operations per clock and SM in all), a division takes 1,470.
// Two forms:
//   * cluster: up to 16 blocks in one cluster, {z, p} in distributed shared
//     memory, the hardware barrier (400 to 600 cycles). Its 16 SMs issue few
//     FP64 operations, so it ends where the grid becomes faster, about 6,000
//     rows: 5.5 us an iteration at 4,096 rows and 6.0 at 5,832 (cluster),
//     6.5 at 6,859 (grid), 6.8 at 4,913 in the grid form.
//   * grid: up to one block per SM, cooperative launch, {z, p} in L2, a counter
//     in global memory as the barrier (1.2 us). It ends at one row per thread,
//     155,648 rows on 152 SMs.
// Measured per iteration of the lattice Laplacian, three kernels per iteration
// in a graph before -> here: 1,331 rows 22 -> 4.4 us, 17,576 rows 22 -> 7.0,
// 132,651 rows 24 -> 12.4; of a caller's CSR system with 68,921 rows (three
// launches per iteration, the host asking every eight) 64 -> 9.1.
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "pcg_resident.h"
#include "spg_internal.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxSums = 4;
constexpr int kMaxCluster = 16;
// Polls of the grid barrier before a block gives up (each takes most of a
// microsecond): a few seconds. The cooperative launch makes every block
// resident, so the limit is never met in a healthy run.
constexpr int kMaxPolls = 1 << 22;

// Quotients on the critical path of every iteration, without the 1,470 cycles
// of the division sequence: reciprocal() is a seed and one third-order Newton
// step (y' = y + y (h + h^2), h = 1 - b y); quotient() corrects a y with its
// exact remainder. Operands whose steps could leave the normal range take the
// division, out of line so that it is not computed beside the fast form.
__device__ __forceinline__ double reciprocal(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double h = fma(-b, y, 1.0);
    return fma(y, fma(h, h, h), y);
}
__device__ __forceinline__ bool mid_range(double a) {
    const int e = (__double2hiint(a) >> 20) & 0x7ff;
    return e >= 300 && e <= 1700;
}
__device__ __noinline__ double divide(double a, double b) { return a / b; }
__device__ __forceinline__ double quotient(double a, double b, double y) {
    if (!(mid_range(a) && mid_range(b))) return divide(a, b);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
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

struct Zp {
    double z, p;
};

__device__ __forceinline__ Zp load_zp(const double2 *p) {
    Zp r;  // not a read-only load: other blocks write the array between the barriers
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(r.z), "=d"(r.p) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ Zp load_zp_cluster(uint32_t addr) {
    Zp r;
    asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(r.z), "=d"(r.p) : "r"(addr) : "memory");
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

// Sum over the first 2 * FROM lanes of a warp (result in lane 0).
template <int FROM>
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = FROM; off > 0; off >>= 1) v += __shfl_down_sync(kFull, v, off);
    return v;
}

struct Shared {
    double tot[kMaxSums];                   // the totals of the last exchange
    double part[2][kMaxSums][kMaxCluster];  // cluster form: every block's partial sums
    double alpha, beta, inv_rz;
    int stop, timed_out;
};

// One exchange: the totals over all rows of the n values per thread in
// buf[k T + t], into s.tot[k] by warp k modulo the block's warps (other warps
// read them after the caller's barrier). Everything the block wrote before is
// visible to every block afterwards. An FP64 instruction holds its warp's
// scheduler for 63 cycles whatever its lanes and independence, so at most four
// warps first add the columns of a large block, one per scheduler, and each
// value then has a warp of its own. target: arrivals after which this
// exchange is complete (grid form). Out of line: one copy for every phase.
template <bool CLUSTER>
__device__ __noinline__ void exchange(double *partials, unsigned int *arrived, Shared &s, double *buf, unsigned par,
                                      unsigned target, int n) {
    const int T = blockDim.x, t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = T >> 5;
    __syncthreads();
    if (T > 128) {
        if (t < 128)
            for (int k = 0; k < n; ++k) {
                double w = buf[k * T + t];
                for (int j = t + 128; j < T; j += 128) w += buf[k * T + j];
                buf[k * T + t] = w;
            }
        __syncthreads();
    }
    for (int k = wid; k < n; k += nw) {
        const double *b = buf + k * T + lane;
        double w = b[0] + b[32];
        if (T > 64) w += b[64];
        if (T > 96) w += b[96];
        w = warp_sum<16>(w);
        if constexpr (CLUSTER) {
            w = __shfl_sync(kFull, w, 0);
            if (unsigned(lane) < gridDim.x)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(
                                 map_rank(shared_addr(&s.part[par][k][blockIdx.x]), unsigned(lane))),
                             "d"(w)
                             : "memory");
        } else if (lane == 0) {
            partials[(size_t(par) * kMaxSums + k) * gridDim.x + blockIdx.x] = w;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
        }
    }
    if constexpr (CLUSTER) cluster_barrier();
    for (int k = wid; k < n; k += nw) {
        double w = 0.0;
        if constexpr (CLUSTER) {
            if (unsigned(lane) < gridDim.x) w = s.part[par][k][lane];
            w = warp_sum<8>(w);
        } else {
            unsigned got;
            int polls = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(arrived) : "memory");
            } while (got < target && ++polls < kMaxPolls);
            if (got < target) s.timed_out = 1;
            // the blocks' partial sums, five per lane in flight together
            const double *p = partials + (size_t(par) * kMaxSums + k) * gridDim.x;
            for (unsigned b = lane; b - lane < gridDim.x; b += 160) {
                double u[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) u[q] = b + 32 * q < gridDim.x ? __ldcg(p + b + 32 * q) : 0.0;
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (b - lane + 32 * q < gridDim.x) w += u[q];
            }
            w = warp_sum<16>(w);
        }
        if (lane == 0) s.tot[k] = w;
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
    extern __shared__ double2 dyn[];
    __shared__ Shared s;
    const int T = blockDim.x, t = threadIdx.x, wid = t >> 5;
    const int i = blockIdx.x * T + t;
    const bool act = i < a.n;
    // dynamic shared memory: cluster form's {z, p} pair [2][T], the exchange's
    // values [kMaxSums][T], the staged matrix entries' values and places [staged][T]
    double2 *zp_sh = dyn;
    double *buf = reinterpret_cast<double *>(dyn + (CLUSTER ? 2 * T : 0));
    double *mval = buf + kMaxSums * T;
    int32_t *mcol = reinterpret_cast<int32_t *>(mval + size_t(a.staged) * T);
    unsigned par = 0, target = 0;
    auto sums = [&](int n) {
        target += gridDim.x * unsigned(n);
        exchange<CLUSTER>(a.partials, a.arrived, s, buf, par, target, n);
        par ^= 1u;
    };
    if (t == 0) {
        s.timed_out = 0;
        s.inv_rz = 0.0;
    }

    const RowRef row = act ? row_ref(a, i) : RowRef{0, 1, 0};
    // place of column c's {z, p}: its index, or its shared address in the cluster
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
    double x = 0.0, r = 0.0, z = 0.0, p = 0.0, dinv = 1.0, diag = 0.0;
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
            if (!found || !(fabs(diag) > 0.0) || !isfinite(diag)) bad = 1.0;
            dinv = bad != 0.0 ? 1.0 : 1.0 / diag;
        }
        x = a.x[i];
        const double b = a.b[i];
        r = b - (a0 + a1);
        z = r * dinv;
        rz0 = r * z;
        bb0 = b * b;
        rr0 = r * r;
        if constexpr (CLUSTER)
            zp_sh[t] = make_double2(z, 0.0);
        else
            a.zp[0][i] = make_double2(z, 0.0);
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
    if constexpr (CLUSTER) cluster_barrier();  // every block runs before its shared memory is written
    sums(4);
    __syncthreads();
    double rz = s.tot[0], rr = s.tot[2], pq = 0.0, alpha = 0.0, beta = 0.0;
    const double bb = s.tot[1], tol2 = a.rtol2 * bb;
    int iters = 0;
    int stop = s.timed_out ? kPcgTimedOut : s.tot[3] > 0.0 ? kPcgBadDiagonal : (rr <= tol2 || bb == 0.0) ? 1 : 0;
    // a zero right-hand side of the allocation-free solve gives x = 0 whatever the start
    const bool zero_x = a.zero_on_zero_b && bb == 0.0 && !s.timed_out;

    int cur = 0;
    while (stop == 0) {
        // ---- phase A
        p = fma(beta, p, z);
        double q;
        {
            double a0 = diag * p, a1 = 0.0;
            const uint32_t half = CLUSTER ? uint32_t(cur) * uint32_t(T) * 16u : 0u;
            const double2 *src = CLUSTER ? nullptr : a.zp[cur];
            auto get = [&](int32_t at) -> Zp {
                if constexpr (CLUSTER)
                    return load_zp_cluster(uint32_t(at) + half);
                else
                    return load_zp(src + at);
            };
            int k = 0;
            for (; k + kGathers <= staged; k += kGathers) {
                Zp g[kGathers];
#pragma unroll
                for (int u = 0; u < kGathers; ++u) g[u] = get(mcol[(k + u) * T + t]);
#pragma unroll
                for (int u = 0; u < kGathers; u += 2) {
                    a0 = fma(mval[(k + u) * T + t], fma(beta, g[u].p, g[u].z), a0);
                    a1 = fma(mval[(k + u + 1) * T + t], fma(beta, g[u + 1].p, g[u + 1].z), a1);
                }
            }
            for (; k + 2 <= staged; k += 2) {
                const Zp g0 = get(mcol[k * T + t]), g1 = get(mcol[(k + 1) * T + t]);
                a0 = fma(mval[k * T + t], fma(beta, g0.p, g0.z), a0);
                a1 = fma(mval[(k + 1) * T + t], fma(beta, g1.p, g1.z), a1);
            }
            if (k < staged) {  // an odd capacity
                const Zp g = get(mcol[k * T + t]);
                a0 = fma(mval[k * T + t], fma(beta, g.p, g.z), a0);
            }
            for (k = next; k < row.count; ++k) {
                const int32_t c = __ldg(a.col + row.at(k));
                const double m = __ldg(a.val + row.at(k));
                if (c == i || m == 0.0) continue;
                const Zp g = get(place(c));
                a0 = fma(m, fma(beta, g.p, g.z), a0);
            }
            q = a0 + a1;
        }
        buf[t] = act ? p * q : 0.0;
        sums(1);
        if (wid == 0) {
            pq = s.tot[0];
            // not positive: A not SPD on this subspace, or NaN
            const int why = s.timed_out ? kPcgTimedOut : positive(pq) ? 0 : kPcgBreakdown;
            alpha = why ? 0.0 : quotient(rz, pq, reciprocal(pq));
            if (t == 0) {
                s.stop = why;
                s.alpha = alpha;
            }
        } else if (wid == 1) {
            const double y = reciprocal(rz);  // for beta, off its critical path
            if (t == 32) s.inv_rz = y;
        }
        __syncthreads();
        stop = s.stop;
        alpha = s.alpha;
        if (stop) break;
        // ---- phase B
        r = fma(-alpha, q, r);
        z = r * dinv;
        cur ^= 1;
        if (act) {
            if constexpr (CLUSTER)
                zp_sh[cur * T + t] = make_double2(z, p);
            else
                a.zp[cur][i] = make_double2(z, p);
        }
        buf[t] = act ? r * z : 0.0;
        buf[T + t] = act ? r * r : 0.0;
        x = fma(alpha, p, x);
        ++iters;
        sums(2);
        if (wid == 0) {
            beta = quotient(s.tot[0], rz, s.inv_rz);
            if (t == 0) s.beta = beta;
        } else if (wid == 1) {
            const int why = s.timed_out ? kPcgTimedOut : s.tot[1] <= tol2 ? 1 : iters >= a.max_iter ? 2 : 0;
            if (t == 32) s.stop = why;
        }
        __syncthreads();
        stop = s.stop;
        beta = s.beta;
        rz = s.tot[0];
        rr = s.tot[1];
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

using Kernel = void (*)(ResidentArgs);
Kernel kernel_of(const ResidentPlan &p) {
    if (p.cluster) return k_pcg_resident<true, 384>;
    return p.threads <= 512 ? k_pcg_resident<false, 512> : k_pcg_resident<false, 1024>;
}

// Rows up to which one cluster of 16 blocks is used.
constexpr int64_t kClusterRows = 6144;

size_t smem_of(int threads, int staged, bool cluster) {
    return size_t(threads) * ((cluster ? 32 : 0) + 8 * kMaxSums + 12 * size_t(staged));
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

// Whether the device runs this plan (opt-in shared memory, cluster size, all blocks resident).
bool fits(const ResidentPlan &p, int sms) {
    const Kernel k = kernel_of(p);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(p.smem)) != cudaSuccess ||
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
        return fits(p, sms);
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
