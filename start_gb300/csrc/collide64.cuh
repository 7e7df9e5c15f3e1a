// Gas collision decision of the FP64 form, shared by the step kernel and the
// adjoint (both built with --fmad=false): decided mostly in FP32, equal to the
// FP64 test in every case.
#ifndef SPG_COLLIDE64_CUH
#define SPG_COLLIDE64_CUH

#include "philox.h"
#include "screen.h"
#include "spg_internal.h"

namespace spg {

namespace {

constexpr double kPi = 3.14159265358979323846;

// Collision probability exactly as the reference evaluates it:
// HSModel.cpp:12-15, VHSModel.cpp:14-25 (and VSSModel.cpp, same formula).
__device__ __noinline__ double probability64(const StepConst &c, double vx, double vy, double vz) {
    const double vmod = sqrt(vx * vx + vy * vy + vz * vz);
    double sigma;
    if (c.model == SPG_COLL_HS) {
        sigma = c.sigma_hs;
    } else {
        const double base = c.two_kT / ((c.mr * vmod) * vmod);
        const double d2 = c.vhs_c1 * pow(base, c.expo);
        sigma = kPi * d2;
    }
    return ((sigma * vmod) * c.gas_n) * c.dt;
}

// Gas collision decision (the candidate-byte test of philox.h), equal to the
// FP64 test and taken mostly in FP32:
//  * a step that is no candidate (255 of 256) with v^2 at most c.v2_cand_f,
//    computed from the 20-bit components (below the true v^2), has P below
//    q: no collision, no FP64 instruction;
//  * otherwise P_f = kp (v^2)^pexp from the 20-bit components (relative
//    error below 2e-5) decides P against q outside the band q (1 -+ 1e-4),
//    a candidate's u_acc against 256 P outside 256 P_f (1 -+ 1e-4), and
//    u_f against (P - q) / (1 - q) outside a band of 3e-5 P_f + 2e-7;
//  * P is computed in FP64 only inside a band.
// The test where the common case cannot decide it: a candidate, or P that
// may exceed q (out of line, so the step loop carries none of it).
__device__ __noinline__ bool collision_test64(const StepConst &c, uint32_t id, uint64_t step, uint32_t byte, float v2,
                                              double vx, double vy, double vz) {
    constexpr float qf = float(kCandQ);
    const float pf = c.kp_f * exp2f(c.pexp_f * log2f(v2));
    if (byte == 0u) {
        // a candidate: P > q collides; P <= q collides iff u_acc < 256 P
        if (pf > qf * (1.0f + 1e-4f)) return true;
        const Philox4 r = collision_draw(step, 3u, id, c.seed_lo, c.seed_hi);
        if (pf < qf * (1.0f - 1e-4f)) {
            const float ulo = float(r.v[0] >> 8) * 5.9604644775390625e-8f;  // 2^-24
            const float uhi = ulo + 5.9604644775390625e-8f;
            const float a = pf * 256.0f;
            if (uhi < a * (1.0f - 1e-4f)) return true;
            if (ulo > a * (1.0f + 1e-4f)) return false;
        }
        const double P = probability64(c, vx, vy, vz);
        return P > kCandQ || u01_from(r.v[0], r.v[1]) < P * 256.0;
    }
    if (pf < qf * (1.0f - 1e-4f)) return false;
    const Philox4 r = collision_draw(step, 4u, id, c.seed_lo, c.seed_hi);
    const float ulo = float(r.v[0] >> 8) * 5.9604644775390625e-8f;  // 2^-24
    const float uhi = ulo + 5.9604644775390625e-8f;
    const float tf = (pf - qf) / (1.0f - qf), band = 3e-5f * pf + 2e-7f;
    if (pf > qf * (1.0f + 1e-4f) && uhi < tf - band) return true;
    if (pf > qf * (1.0f + 1e-4f) && ulo > tf + band) return false;
    const double P = probability64(c, vx, vy, vz);
    return P > kCandQ && u01_from(r.v[0], r.v[1]) < (P - kCandQ) / (1.0 - kCandQ);
}

// The FP32 screens of collision_test64 that rule a collision out: for a
// candidate (P certainly below q) u_acc certainly beyond 256 P; else P
// certainly below q, or u_f certainly beyond its threshold (fast particles in
// a dense gas, where P exceeds q in every step). False: not certain.
__device__ __forceinline__ bool no_collision_sure(const StepConst &c, uint32_t id, uint64_t step, bool cand, float v2) {
    constexpr float qf = float(kCandQ);
    const float pf = c.kp_f * exp2f(c.pexp_f * log2f(v2));
    const bool below = pf < qf * (1.0f - 1e-4f);
    if (!cand && below) return true;
    if (cand && !below) return false;
    const uint32_t u = collision_draw(step, cand ? 3u : 4u, id, c.seed_lo, c.seed_hi).v[0] >> 8;
    const float ulo = float(u) * 5.9604644775390625e-8f;  // 2^-24
    if (cand) return ulo > pf * 256.0f * (1.0f + 1e-4f);
    const float tf = (pf - qf) / (1.0f - qf), band = 3e-5f * pf + 2e-7f;
    return pf > qf * (1.0f + 1e-4f) && ulo > tf + band;
}

}  // namespace

}  // namespace spg

#endif
