// One-launch Jacobi PCG of a system that fits on the chip (kernels_pcg_resident.cu).
#ifndef SPG_PCG_RESIDENT_H
#define SPG_PCG_RESIDENT_H

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace spg {

struct PcgScalars;

// PcgScalars::converged beyond 1 (converged) and 2 (max_iter): CG breakdown
// (written as ResidentArgs::breakdown), a barrier that gave up; and a row
// without a usable diagonal (flags = 1, converged = 0).
constexpr int kPcgBreakdown = 3;
constexpr int kPcgTimedOut = 4;
constexpr int kPcgBadDiagonal = 5;

// Launch shape chosen from the row count: `blocks` blocks of `threads` threads
// with one row per thread (0 blocks: the system does not fit), as one cluster
// or as a cooperative grid; `staged` matrix entries per row in shared memory.
struct ResidentPlan {
    int blocks = 0, threads = 0, staged = 0;
    bool cluster = false;
    size_t smem = 0;
};

// The system and its working memory. SELL-32 (slice_ptr) or CSR (row_ptr);
// inv_diag nullptr: taken from the matrix, and a row without a finite nonzero
// diagonal entry is refused. zpu: two arrays of n records (grid form only);
// partials: kResidentPartials doubles; arrived: zeroed by the launch.
struct alignas(32) ZpuRec {
    double z, p, u, unused;  // D^-1 r, the search direction, D^-1 A p
};
constexpr int kResidentSums = 5;
struct ResidentArgs {
    int n = 0;
    const int64_t *slice_ptr = nullptr;
    const int32_t *row_ptr = nullptr;
    const int32_t *col = nullptr;
    const double *val = nullptr, *inv_diag = nullptr, *b = nullptr;
    double *x = nullptr;
    ZpuRec *zpu[2] = {nullptr, nullptr};
    double *partials = nullptr;
    unsigned int *arrived = nullptr;
    PcgScalars *sc = nullptr;
    double rtol2 = 0.0;
    int max_iter = 0, breakdown = 2, staged = 0;
    bool zero_on_zero_b = false;
};

constexpr size_t kResidentPartials = 2 * kResidentSums * 512;  // two parities, at most 512 blocks

ResidentPlan resident_plan(int64_t n);
cudaError_t launch_pcg_resident(const ResidentPlan &plan, ResidentArgs a, cudaStream_t s);

}  // namespace spg

#endif
