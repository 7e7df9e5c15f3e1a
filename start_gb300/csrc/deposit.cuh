// Persistent P1 charge deposit into the fixed-point node accumulators, shared
// by the FP64 and the mixed-form deposit kernels.
//
// Each block walks one contiguous range of 256-particle tiles (the grid is
// one wave of blocks), with the next tile's particle loads issued before the
// current tile is reduced. A warp whose tile lies in one tet (the common case
// in tet-sorted order: a beam puts thousands of particles in a tet) adds the
// weights to per-lane running sums and reduces them only when its tet
// changes. In other tiles (the ends of runs, and particles that moved to
// other tets since the last re-sort) every run of equal tets is summed by
// prefix sums. Either way the first lane adds the tet's four sums to the block's
// table of tets in shared memory: one probe, four adds. The table is flushed
// into the node accumulators at the end of the range (four global atomics per
// listed tet), and also every kDepCheckTiles tiles if it is more than half full,
// so a range whose particles are spread over many tets keeps aggregating. While
// the table is over half full a tet it does not hold goes to the node
// accumulators directly. Integer sums do not depend on order, so the result
// is the same as one atomic per particle.
//
// us per deposit, with a pass per key, 64-bit shared-memory adds (which are
// compare-and-swap loops) and, in FP64, unfused weights -> now: 6e6 ions of a
// Thompson source on 1.3e6 tets sorted 224 -> 147, ten and 19 steps after the
// sort 269 -> 153 and 309 -> 164 (FP64), 54 -> 59, 144 -> 102 and 200 -> 108 (mixed
// form); 3e6 all over 162,000 tets sorted 140 -> 90 and 65 -> 56, in random order
// 438 -> 242 and 370 -> 202. FP64 is bound by the issue of the weights' twelve
// instructions per particle (72 us for 3e6 at the measured rate).
#ifndef SPG_DEPOSIT_CUH
#define SPG_DEPOSIT_CUH

#include <algorithm>
#include <cstdint>

#include "spg_internal.h"

namespace spg {

constexpr int kDepThreads = 256;
constexpr int kDepSlots = 1024;          // tet slots of a block's table
constexpr int kDepOpen = kDepSlots / 2;  // new tets enter while the table holds fewer
constexpr int kDepCheckTiles = 16;       // tiles between checks of the table's fill

struct DepositTable {
    int tet[kDepSlots];  // -1: free; a slot's tet does not change until the table is cleared
    unsigned int lo[kDepSlots][4], hi[kDepSlots][4];  // the sums' halves
    unsigned int held;
};

// Sums of v[0..3] over the run of equal keys that begins at this lane (heads:
// the first lanes of the runs; other lanes' results are not used). Prefix sums
// over the warp (modulo 2^64, exact whenever the run's sum fits 64 bits) and
// their difference across the run: the same instructions for every warp,
// where reductions over the lanes of each key (match_any and the integer reduce
// unit) take a pass per key. v[0] = one - v[1] - v[2] - v[3] sums to count *
// one minus the others.
__device__ __forceinline__ void run_sums(unsigned heads, const long long v[4], long long one, long long sum[4]) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned after = heads & ~((2u << lane) - 1u);
    const int last = after ? __ffs(after) - 2 : 31;  // the run's last lane
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        unsigned long long p = (unsigned long long)v[q];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned long long t = __shfl_up_sync(kAll, p, off);
            if (lane >= off) p += t;
        }
        sum[q] = (long long)(__shfl_sync(kAll, p, last) - p + (unsigned long long)v[q]);
    }
    sum[0] = (long long)(last - lane + 1) * one - sum[1] - sum[2] - sum[3];
}

// Appends tet `key` to the list of occupied tets once per deposit (the
// generation stamp of the tet says whether it is listed already).
__device__ __forceinline__ void list_tet(const OccList &occ, int key) {
    if (occ.list && __ldcg(occ.gen_of + key) != occ.gen && atomicExch(occ.gen_of + key, occ.gen) != occ.gen)
        occ.list[atomicAdd(occ.n, 1u)] = key;
}

// A tet's four node sums into the node accumulators.
__device__ __forceinline__ void tet_to_nodes(int key, const unsigned long long sum[4],
                                             const int4 *__restrict__ tet_nodes,
                                             unsigned long long *__restrict__ node_fix, const OccList &occ) {
    list_tet(occ, key);
    const int4 tn = __ldg(tet_nodes + key);
    if (sum[0]) atomicAdd(node_fix + tn.x, sum[0]);
    if (sum[1]) atomicAdd(node_fix + tn.y, sum[1]);
    if (sum[2]) atomicAdd(node_fix + tn.z, sum[2]);
    if (sum[3]) atomicAdd(node_fix + tn.w, sum[3]);
}

// *(hi, lo) += v by 32-bit shared-memory atomics: the one on the low halves
// returns whether it carried. (A 64-bit add is a compare-and-swap loop there.)
__device__ __forceinline__ void add_halves(unsigned int *lo, unsigned int *hi, unsigned long long v) {
    const unsigned l = unsigned(v), h = unsigned(v >> 32);
    const unsigned old = atomicAdd(lo, l);
    const unsigned c = h + (old + l < l ? 1u : 0u);
    if (c) atomicAdd(hi, c);
}

// Adds a tet's four sums to its slot (open addressing, linear probing). A
// free slot is claimed by compare-and-swap only while the table is at most
// half full; otherwise a tet the table does not hold goes to the node
// accumulators. The probe run ends at the tet or a free slot: fewer than
// kDepOpen + kDepThreads slots are ever taken between clears.
__device__ __forceinline__ void table_add(DepositTable &s, int key, const long long sum[4],
                                          const int4 *__restrict__ tet_nodes,
                                          unsigned long long *__restrict__ node_fix, const OccList &occ) {
    int h = int((unsigned(key) * 2654435761u) >> 8) & (kDepSlots - 1);
    for (int probe = 0; probe < kDepSlots; ++probe) {
        int cur = s.tet[h];
        if (cur == -1) {
            if (*(volatile unsigned int *)&s.held >= unsigned(kDepOpen)) break;
            cur = atomicCAS(&s.tet[h], -1, key);
            if (cur == -1) {
                atomicAdd(&s.held, 1u);
                cur = key;
            }
        }
        if (cur == key) {
#pragma unroll
            for (int q = 0; q < 4; ++q) add_halves(&s.lo[h][q], &s.hi[h][q], (unsigned long long)sum[q]);
            return;
        }
        h = (h + 1) & (kDepSlots - 1);
    }
    const unsigned long long u[4] = {(unsigned long long)sum[0], (unsigned long long)sum[1],
                                     (unsigned long long)sum[2], (unsigned long long)sum[3]};
    tet_to_nodes(key, u, tet_nodes, node_fix, occ);
}

__device__ __forceinline__ void table_clear(DepositTable &s) {
    for (int k = threadIdx.x; k < kDepSlots; k += kDepThreads) {
        s.tet[k] = -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) s.lo[k][q] = s.hi[k][q] = 0u;
    }
    if (threadIdx.x == 0) s.held = 0u;
}

// Every held tet's sums into the node accumulators (after a barrier).
__device__ __forceinline__ void table_flush(const DepositTable &s, const int4 *__restrict__ tet_nodes,
                                            unsigned long long *__restrict__ node_fix, const OccList &occ) {
    for (int k = threadIdx.x; k < kDepSlots; k += kDepThreads)
        if (s.tet[k] >= 0) {
            unsigned long long sum[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) sum[q] = (unsigned long long)s.hi[k][q] << 32 | s.lo[k][q];
            tet_to_nodes(s.tet[k], sum, tet_nodes, node_fix, occ);
        }
}

// Warp sum of 64-bit values modulo 2^64 (three 21-bit pieces, the top one
// signed): exact whenever the true sum fits 64 bits.
__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned s0 = __reduce_add_sync(kAll, unsigned(v & 0x1FFFFFull));
    const unsigned s1 = __reduce_add_sync(kAll, unsigned((v >> 21) & 0x1FFFFFull));
    const int s2 = __reduce_add_sync(kAll, int((long long)v >> 42));
    return (unsigned long long)s0 + ((unsigned long long)s1 << 21) + ((unsigned long long)(long long)s2 << 42);
}

// The warp's running sums of tet key, reduced and added to the table by lane 0.
__device__ __forceinline__ void flush_running(DepositTable &s, int key, unsigned long long a1, unsigned long long a2,
                                              unsigned long long a3, int acnt, long long one,
                                              const int4 *__restrict__ tet_nodes,
                                              unsigned long long *__restrict__ node_fix, const OccList &occ) {
    long long sum[4];
    sum[1] = (long long)warp_sum64(a1);
    sum[2] = (long long)warp_sum64(a2);
    sum[3] = (long long)warp_sum64(a3);
    const unsigned long long cnt = __reduce_add_sync(0xffffffffu, unsigned(acnt));
    sum[0] = (long long)(cnt * (unsigned long long)one - (unsigned long long)sum[1] - (unsigned long long)sum[2] -
                         (unsigned long long)sum[3]);
    if ((threadIdx.x & 31) == 0) table_add(s, key, sum, tet_nodes, node_fix, occ);
}

// The deposit of particles [0, n) by one block of kDepThreads threads, its
// range of tiles given by blockIdx and gridDim. Src provides
//   Raw load(int64_t i, int64_t n): the particle's fields (a dead marker for i >= n);
//   int weights(const Raw &, long long v[4]): the tet (or -1: dead) and the
//     fixed-point weights v[0..3] summing to one (zeros for a dead particle);
//   long long one: the fixed-point one.
template <class Src>
__device__ __forceinline__ void deposit_tiles(const Src &src, int64_t n, const int4 *__restrict__ tet_nodes,
                                              unsigned long long *__restrict__ node_fix, const OccList &occ) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ DepositTable s;
    table_clear(s);
    __syncthreads();
    const int64_t tiles = (n + kDepThreads - 1) / kDepThreads;
    const int64_t per = (tiles + gridDim.x - 1) / gridDim.x;
    const int64_t t0 = int64_t(blockIdx.x) * per;
    const int64_t t1 = t0 + per < tiles ? t0 + per : tiles;
    const int lane = threadIdx.x & 31;
    int acc_key = -1;                           // warp-uniform: the tet of the running sums (-1: none)
    unsigned long long a1 = 0, a2 = 0, a3 = 0;  // modulo 2^64: the node totals fit 63 bits
    int acnt = 0;                               // this lane's alive particles in the running sums
    int64_t i = t0 * kDepThreads + threadIdx.x;
    typename Src::Raw nxt = src.load(i, t0 < t1 ? n : 0);
    for (int64_t t = t0; t < t1; ++t, i += kDepThreads) {
        if ((t - t0) % kDepCheckTiles == kDepCheckTiles - 1) {  // block-uniform
            __syncthreads();
            if (s.held >= unsigned(kDepOpen)) {
                table_flush(s, tet_nodes, node_fix, occ);
                __syncthreads();
                table_clear(s);
            }
            __syncthreads();
        }
        const typename Src::Raw cur = nxt;
        nxt = src.load(i + kDepThreads, t + 1 < t1 ? n : 0);
        long long v[4];
        const int key = src.weights(cur, v);
        const int kmax = __reduce_max_sync(kAll, key);
        if (__all_sync(kAll, key == kmax || key < 0)) {
            if (kmax != acc_key && kmax >= 0) {
                if (acc_key >= 0) flush_running(s, acc_key, a1, a2, a3, acnt, src.one, tet_nodes, node_fix, occ);
                acc_key = kmax;
                a1 = a2 = a3 = 0;
                acnt = 0;
            }
            a1 += (unsigned long long)v[1];
            a2 += (unsigned long long)v[2];
            a3 += (unsigned long long)v[3];
            acnt += key >= 0;
        } else {
            long long sum[4];
            const int prev = __shfl_up_sync(kAll, key, 1);
            const unsigned heads = __ballot_sync(kAll, lane == 0 || prev != key);
            run_sums(heads, v, src.one, sum);
            if (key >= 0 && ((heads >> lane) & 1u)) table_add(s, key, sum, tet_nodes, node_fix, occ);
        }
    }
    if (acc_key >= 0) flush_running(s, acc_key, a1, a2, a3, acnt, src.one, tet_nodes, node_fix, occ);
    __syncthreads();
    table_flush(s, tet_nodes, node_fix, occ);
}

// Blocks of `kernel` resident on the whole GPU at once (the deposit's one wave).
template <class K>
inline int resident_blocks(K kernel, int threads, size_t smem = 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    return std::max(1, sms * std::max(1, per_sm));
}

}  // namespace spg

#endif
