// Counting sort of particles by tet, by one of two routes.
//
// From an earlier sort (the particles are close to tet order): a histogram of
// the bins, a scan, and a scatter whose bins hand out their places by atomics.
// Consecutive warps hit the same bins, so warp groups of equal keys (match_any)
// are merged per block in a shared open-addressing table and a bin takes one
// global atomic per block. The destinations of a warp are a few runs.
//
// From no order (a new particle set): the destinations of a warp are 32 places
// in each of eight arrays, and writing 4 or 8 bytes of a 32-byte sector costs the
// sector eight times over. So the histogram pass keeps each particle's rank in
// its bin (its atomics return it; warps skip the table where the block's keys do
// not repeat), the particle goes as one record (32 or 64 bytes, whole sectors)
// to offset + rank of a scratch array, and a last kernel spreads the records over
// the arrays.
//
// us per sort from no order, histogram and scatter -> ranks and records, FP64 /
// mixed form: 1e7 ions of a Thompson source on 6.0e6 tets 1,116 -> 858 / 997 ->
// 543, 6e6 all over 1.3e6 tets 1,342 -> 386 / 1,193 -> 257, 1e6 on 7.5e5 143 -> 135
// / 144 -> 101, 6e6 in a beam on 6,000 tets 318 -> 347 / 300 -> 254. Twenty steps
// after a sort the ranks cost more than they save: 1e7 446 -> 566 / 404 -> 463.
#pragma once
#include <cstdint>

namespace spg {

constexpr int kSortBlock = 256;
constexpr int kSortSlots = 2 * kSortBlock;  // at most kSortBlock distinct keys per block
constexpr int kSortSpread = 192;            // warp groups in a block above which the table is skipped

struct SortTable {
    int key[kSortSlots];
    int count[kSortSlots];
    int base[kSortSlots];
};

__device__ __forceinline__ void sort_table_clear(SortTable &t) {
    for (int s = threadIdx.x; s < kSortSlots; s += blockDim.x) {
        t.key[s] = -1;
        t.count[s] = 0;
    }
}

// Slot of key (inserted if absent). The table has twice as many slots as the
// block has threads, so a free slot exists and the probe ends within
// kSortSlots steps.
__device__ __forceinline__ int sort_table_slot(SortTable &t, int key) {
    int h = int((unsigned(key) * 2654435761u) >> 23);  // 9 bits: kSortSlots = 512
    for (int probe = 0; probe < kSortSlots; ++probe) {
        const int old = atomicCAS(&t.key[h], -1, key);
        if (old == -1 || old == key) return h;
        h = (h + 1) & (kSortSlots - 1);
    }
    return -1;  // unreachable: at most kSortBlock keys are inserted
}

// Histogram of keys (key < 0: no particle) into cnt.
__device__ __forceinline__ void sort_hist_block(SortTable &t, int key, int32_t *cnt) {
    sort_table_clear(t);
    __syncthreads();
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31;
    if (key >= 0 && lane == __ffs(peers) - 1) {
        const int h = sort_table_slot(t, key);
        if (h >= 0) atomicAdd(&t.count[h], __popc(peers));
    }
    __syncthreads();
    for (int s = threadIdx.x; s < kSortSlots; s += blockDim.x)
        if (t.key[s] >= 0) atomicAdd(cnt + t.key[s], t.count[s]);
}

// Destination index of this thread's particle (key < 0: none, returns -1):
// offs[key] is the next free index of bin key.
__device__ __forceinline__ int64_t sort_dest_block(SortTable &t, int key, int32_t *offs) {
    sort_table_clear(t);
    __syncthreads();
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int h = -1, local = 0;
    if (key >= 0 && lane == leader) {
        h = sort_table_slot(t, key);
        if (h >= 0) local = atomicAdd(&t.count[h], __popc(peers));
    }
    __syncthreads();
    for (int s = threadIdx.x; s < kSortSlots; s += blockDim.x)
        if (t.key[s] >= 0) t.base[s] = atomicAdd(offs + t.key[s], t.count[s]);
    __syncthreads();
    int64_t first = 0;
    if (key >= 0 && lane == leader && h >= 0) first = int64_t(t.base[h]) + local;
    first = __shfl_sync(0xffffffffu, first, leader);
    if (key < 0) return -1;
    return first + __popc(peers & ((1u << lane) - 1u));
}

// Rank of this thread's particle in bin key (key < 0: none), counted into cnt.
// shared_bin: a bin that any warp may use (the dead), always merged per block.
__device__ __forceinline__ int sort_rank_block(SortTable &t, int key, int shared_bin, int32_t *cnt) {
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    const bool lead = key >= 0 && lane == leader;
    // (a shared bin in the block counts as too few groups)
    const int groups = __syncthreads_count(lead) - 2 * kSortBlock * __syncthreads_or(key == shared_bin);
    int first = 0;
    if (groups > kSortSpread) {
        if (lead) first = atomicAdd(cnt + key, __popc(peers));
    } else {
        sort_table_clear(t);
        __syncthreads();
        int h = -1, local = 0;
        if (lead) {
            h = sort_table_slot(t, key);
            if (h >= 0) local = atomicAdd(&t.count[h], __popc(peers));
        }
        __syncthreads();
        for (int s = threadIdx.x; s < kSortSlots; s += blockDim.x)
            if (t.key[s] >= 0) t.base[s] = atomicAdd(cnt + t.key[s], t.count[s]);
        __syncthreads();
        if (h >= 0) first = t.base[h] + local;
    }
    first = __shfl_sync(0xffffffffu, first, leader);
    return first + __popc(peers & ((1u << lane) - 1u));
}

// One particle as whole 32-byte sectors.
struct alignas(32) SortRec32 {
    float x, y, z, vx, vy, vz;
    int32_t tet;
    uint32_t idf;
};
struct alignas(32) SortRec64 {
    double x, y, z, vx, vy, vz;
    int32_t tet;
    uint32_t idf;
    double unused;
};

__device__ __forceinline__ void store_sector(void *p, const uint32_t (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// Counting-sort scatter of one particle array set (DevParticles or
// DevParticles32): the eight fields are loaded before the bin offsets are
// taken, so the loads overlap the atomics.
template <class P>
__device__ __forceinline__ void sort_scatter_block(SortTable &t, const P &src, P &dst, int64_t n, int n_tets,
                                                   uint32_t dead_mask, int32_t *offs) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool have = i < n;
    const int64_t k = have ? i : 0;
    const auto x = src.x[k], y = src.y[k], z = src.z[k];
    const auto vx = src.vx[k], vy = src.vy[k], vz = src.vz[k];
    const int32_t tet = src.tet[k];
    const uint32_t idf = src.idf[k];
    const int key = have ? ((idf & dead_mask) ? n_tets : tet) : -1;
    const int64_t j = sort_dest_block(t, key, offs);
    if (j < 0) return;
    dst.x[j] = x;
    dst.y[j] = y;
    dst.z[j] = z;
    dst.vx[j] = vx;
    dst.vy[j] = vy;
    dst.vz[j] = vz;
    dst.tet[j] = tet;
    dst.idf[j] = idf;
}

// Particle i of src to record offs[bin] + rank[i].
__device__ __forceinline__ void put_record(SortRec32 *rec, float x, float y, float z, float vx, float vy, float vz,
                                           int32_t tet, uint32_t idf) {
    const uint32_t w[8] = {__float_as_uint(x),  __float_as_uint(y),  __float_as_uint(z), __float_as_uint(vx),
                           __float_as_uint(vy), __float_as_uint(vz), uint32_t(tet),      idf};
    store_sector(rec, w);
}
__device__ __forceinline__ void put_record(SortRec64 *rec, double x, double y, double z, double vx, double vy, double vz,
                                           int32_t tet, uint32_t idf) {
    const double a[6] = {x, y, z, vx, vy, vz};
    uint32_t w[16];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        w[2 * k] = uint32_t(__double2loint(a[k]));
        w[2 * k + 1] = uint32_t(__double2hiint(a[k]));
    }
    w[12] = uint32_t(tet);
    w[13] = idf;
    w[14] = w[15] = 0u;
    store_sector(rec, reinterpret_cast<const uint32_t(&)[8]>(w[0]));
    store_sector(reinterpret_cast<uint32_t *>(rec) + 8, reinterpret_cast<const uint32_t(&)[8]>(w[8]));
}

template <class P, class R>
__device__ __forceinline__ void sort_to_records(const P &src, R *__restrict__ rec, int64_t n, int n_tets,
                                                uint32_t dead_mask, const int32_t *__restrict__ offs,
                                                const int32_t *__restrict__ rank) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t tet = src.tet[i];
    const uint32_t idf = src.idf[i];
    const int64_t j = int64_t(__ldg(offs + ((idf & dead_mask) ? n_tets : tet))) + rank[i];
    put_record(rec + j, src.x[i], src.y[i], src.z[i], src.vx[i], src.vy[i], src.vz[i], tet, idf);
}

// Records in order to the arrays.
template <class R, class P>
__device__ __forceinline__ void sort_unpack(const R *__restrict__ rec, const P &dst, int64_t n) {
    const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const R r = rec[j];
    dst.x[j] = r.x;
    dst.y[j] = r.y;
    dst.z[j] = r.z;
    dst.vx[j] = r.vx;
    dst.vy[j] = r.vy;
    dst.vz[j] = r.vz;
    dst.tet[j] = r.tet;
    dst.idf[j] = r.idf;
}

}  // namespace spg
