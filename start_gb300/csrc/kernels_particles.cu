// Particle kernels of the FP64 form: fused push + move + gas collision +
// tet walk + surface settle, P1 deposit, per-tet E, point location, re-sort.
//
// Compiled with --fmad=false: every a*b+c stays a separate multiply and add,
// matching the CPU oracle (built with -ffp-contract=off) bit for bit on the
// collisionless path. Division and sqrt are IEEE (CUDA defaults for double).
//
// FP64 on GB300 issues at about 2 instructions per clock per SM (FP32: ~128),
// and double<->float conversions share that pipe. The step kernel therefore
// keeps FP64 semantics exactly while spending FP64 instructions only where the
// result is stored: push, move and the offset from the tet origin. Every
// yes/no decision of the reference algorithm (slow particle, inside the
// modelling box, degenerate segment, inside the tet, collision) is taken by an
// integer or FP32 screen with a proven error bound; when a screen cannot
// decide, the exact FP64 expression (the oracle's) decides. The state written
// is therefore identical to an all-FP64 evaluation.
#include <cmath>
#include <cstdio>

#include "philox.h"
#include "collide64.cuh"
#include "deposit.cuh"
#include "field.cuh"
#include "exact_div.h"
#include "screen.h"
#include "segment.cuh"
#include "sort_block.cuh"
#include "spg_internal.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;

enum WalkStatus { W_INSIDE = 0, W_SURFACE = 1, W_EXIT = 2, W_CAP = 3 };

struct TetGeo {
    double M[9];
    double x0[3];
};

__device__ __forceinline__ void load_geo(const TetRec *__restrict__ rec, int t, TetGeo &g) {
    const double2 *rp = reinterpret_cast<const double2 *>(rec + t);
    double2 a = __ldg(rp + 0), b = __ldg(rp + 1), c = __ldg(rp + 2), d = __ldg(rp + 3);
    double2 e = __ldg(rp + 4), f = __ldg(rp + 5);
    g.M[0] = a.x; g.M[1] = a.y; g.M[2] = b.x; g.M[3] = b.y; g.M[4] = c.x; g.M[5] = c.y;
    g.M[6] = d.x; g.M[7] = d.y; g.M[8] = e.x;
    g.x0[0] = e.y; g.x0[1] = f.x; g.x0[2] = f.y;
}

// Barycentric coordinates from the tet's record in memory (L1-resident
// during a walk), so a walk holds no FP64 map in registers; same values as
// the oracle's evaluation order.
__device__ __forceinline__ void bary_rec(const TetRec *__restrict__ r, double px, double py, double pz,
                                         double l[4]) {
    const double2 *rp = reinterpret_cast<const double2 *>(r);
    const double2 e = __ldg(rp + 4), f = __ldg(rp + 5);
    const double d0 = px - e.y, d1 = py - f.x, d2 = pz - f.y;
    const double2 a = __ldg(rp + 0), b = __ldg(rp + 1);
    l[1] = a.x * d0 + a.y * d1 + b.x * d2;
    const double2 c = __ldg(rp + 2), d = __ldg(rp + 3);
    l[2] = b.y * d0 + c.x * d1 + c.y * d2;
    l[3] = d.x * d0 + d.y * d1 + e.x * d2;
    l[0] = 1.0 - l[1] - l[2] - l[3];
}

__device__ __forceinline__ int comp(const int4 &v, int f) {
    return f == 0 ? v.x : (f == 1 ? v.y : (f == 2 ? v.z : v.w));
}

// ---------------------------------------------------------------- screens
// Order-preserving integer key of a double (see order_key_host).
__device__ __forceinline__ long long order_key(double x) {
    long long b = __double_as_longlong(x);
    if (b == (long long)0x8000000000000000ULL) b = 0;
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}

// IEEE equality of two finite doubles from their bit patterns.
__device__ __forceinline__ bool same_value(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return x == y || ((x | y) << 1) == 0;
}

// Screened inside test from the tet's TetScreen record: true = lambda(p) >= 0
// in all four coordinates for certain; false = undecided (the caller
// evaluates the exact FP64 walk). No FP64 instruction runs: M is truncated to
// 20 mantissa bits (hi_float, once per tet on the host) and
// d = p - x0 is formed in FP32 from p and x0 truncated the same way (integer
// ops). With S_i = sum_j |M_ij d_j|, the truncation of M and the FP32
// products put lambda_i within 2.2e-6 S_i of its value for the exact d; the
// margin takes 4e-6 S_i + 1e-30 (for terms flushed to zero).
// |p - pf| < 2^-20 |p| <= 9.6e-7 |pf| (pf truncates toward zero) and the FP32
// difference rounds by at most 2^-24 |d_f|, so each d_k is within
// delta_k = 9.6e-7 (|pf_k| + |x0f_k|) + 6e-8 |d_fk| + 1e-30 of p_k - x0_k.
// That adds sum_k |M_ik| delta_k (times 1.01 for the truncation of M) to the
// margin of lambda_i; lambda_0 = 1 - sum gets the sum of the three margins
// plus 1e-6 for its own FP32 rounding.
struct ScreenRegs {
    float4 q0, q1, q2;
};

__device__ __forceinline__ ScreenRegs load_screen(const TetScreen *__restrict__ scr) {
    const float4 *sp = reinterpret_cast<const float4 *>(scr);
    return ScreenRegs{__ldg(sp), __ldg(sp + 1), __ldg(sp + 2)};
}

__device__ __forceinline__ bool inside_sure(const ScreenRegs &scr, double px, double py, double pz) {
    const float4 q0 = scr.q0, q1 = scr.q1, q2 = scr.q2;
    const float M[9] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x};
    const float X0[3] = {q2.y, q2.z, q2.w};
    const float pf[3] = {hi_float(px), hi_float(py), hi_float(pz)};
    float e[3], dl[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float x0 = X0[k];
        e[k] = pf[k] - x0;
        dl[k] = fmaf(9.6e-7f, fabsf(pf[k]) + fabsf(x0), fmaf(6e-8f, fabsf(e[k]), 1e-30f));
    }
    float l[3], b[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float m0 = M[3 * r], m1 = M[3 * r + 1], m2 = M[3 * r + 2];
        l[r] = fmaf(m2, e[2], fmaf(m1, e[1], m0 * e[0]));
        const float s = fmaf(fabsf(m2), fabsf(e[2]), fmaf(fabsf(m1), fabsf(e[1]), fabsf(m0) * fabsf(e[0])));
        const float pd = fmaf(fabsf(m2), dl[2], fmaf(fabsf(m1), dl[1], fabsf(m0) * dl[0]));
        b[r] = fmaf(4e-6f, s, fmaf(1.01f, pd, 1e-30f));
    }
    const float l0 = 1.0f - l[0] - l[1] - l[2];
    const float b0 = b[0] + b[1] + b[2] + 1e-6f;
    return l[0] > b[0] && l[1] > b[1] && l[2] > b[2] && l0 > b0;
}

struct WalkOut {
    int tet, status, tri, crossings, face;
    double s;
};

// The walk's decision in one tet from the FP64 barycentrics (the oracle's):
// kScreenInside, or the exit face.
__device__ __noinline__ int exact_exit(const TetRec *__restrict__ rt, double p0x, double p0y, double p0z, double p1x,
                                       double p1y, double p1z, int enter) {
    double l1[4];
    bary_rec(rt, p1x, p1y, p1z, l1);
    int ncand = 0, best = -1;
#pragma unroll
    for (int f = 0; f < 4; ++f)
        if (f != enter && l1[f] < 0.0) {
            ++ncand;
            best = f;
        }
    if (ncand == 0) return kScreenInside;
    if (ncand > 1) {
        double l0[4], sb = 0.0;
        bary_rec(rt, p0x, p0y, p0z, l0);
        best = -1;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            if (f == enter || !(l1[f] < 0.0)) continue;
            const double s = l0[f] / (l0[f] - l1[f]);
            if (best < 0 || s < sb) {
                best = f;
                sb = s;
            }
        }
    }
    return best;
}

// Crossing parameter of face f along p0 -> p1.
__device__ __noinline__ double exit_parameter(const TetRec *__restrict__ rt, double p0x, double p0y, double p0z,
                                              double p1x, double p1y, double p1z, int f) {
    double l0[4], l1[4];
    bary_rec(rt, p0x, p0y, p0z, l0);
    bary_rec(rt, p1x, p1y, p1z, l1);
    const double a = f == 0 ? l0[0] : f == 1 ? l0[1] : f == 2 ? l0[2] : l0[3];
    const double b = f == 0 ? l1[0] : f == 1 ? l1[1] : f == 2 ? l1[2] : l1[3];
    return a / (a - b);
}

// Straight walk of the segment p0 -> p1 starting in tet t.
// In each tet: if p1 is inside (no lambda < 0 but of the entry face) stop.
// Otherwise leave through the face, other than the entry face, with
// lambda(p1) < 0 whose crossing parameter s = l0/(l0 - l1) along the segment is
// smallest (lowest local face index on ties). A face carrying a surface
// triangle stops the walk there (when stop_surface); a boundary face without
// one is an exit.
// The decisions come from FP32 with bounds (screen_exit); the FP64 evaluation
// runs where the bounds leave one open (about one decision in a thousand) and
// for the crossing parameter that is returned. Deciding in FP64 the walks took
// a third of the step's FP64 instructions: a lane that needs the second set of
// barycentrics or a division (a dozen instructions and 1,470 cycles) costs its
// whole warp.
__device__ __forceinline__ WalkOut walk64(const MeshDev &m, int t, double p0x, double p0y, double p0z, double p1x,
                                       double p1y, double p1z, int max_cross, bool stop_surface) {
    WalkOut o;
    o.crossings = 0;
    o.tri = -1;
    o.face = -1;
    o.s = 1.0;
    int enter = -1;
    const double p0[3] = {p0x, p0y, p0z}, p1[3] = {p1x, p1y, p1z};
    for (;;) {
        const TetRec *rt = m.rec + t;
        int best;
        {
            const ScreenRegs scr = load_screen(m.screen + t);
            const float4 q0 = scr.q0, q1 = scr.q1, q2 = scr.q2;
            const float M[9] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x};
            const double2 e = __ldg(reinterpret_cast<const double2 *>(rt) + 4);
            const double2 f = __ldg(reinterpret_cast<const double2 *>(rt) + 5);
            const double x0[3] = {e.y, f.x, f.y};
            best = screen_exit(M, x0, p0, p1, enter);
        }
        if (best == kScreenUndecided) best = exact_exit(rt, p0x, p0y, p0z, p1x, p1y, p1z, enter);
        o.tet = t;
        if (best == kScreenInside) {
            o.status = W_INSIDE;
            return o;
        }
        const int tri = comp(__ldg(m.ftri + t), best);
        const int nb = comp(__ldg(m.nbr + t), best);
        if (stop_surface && tri >= 0) {
            o.status = W_SURFACE;
            o.tri = tri;
            o.face = best;
            o.s = exit_parameter(rt, p0x, p0y, p0z, p1x, p1y, p1z, best);
            return o;
        }
        if (nb < 0) {
            o.status = W_EXIT;
            return o;
        }
        if (o.crossings == max_cross) {
            o.status = W_CAP;
            return o;
        }
        o.crossings++;
        t = nb >> 2;
        enter = nb & 3;
    }
}

// Post-collision velocity (HSModel.cpp:24-39, VHSModel.cpp:31-46,
// VSSModel.cpp:32-48): stationary target; v' = m_p/(m_p+m_t) v + |m_t/(m_p+m_t) v| n.
// The azimuth phi = 2 pi u2 enters as cospi(2 u2), sinpi(2 u2) (no argument
// reduction), and the VSS frame angles beta = acos(pz/|p|), gamma =
// atan2(py, px) as their cosines and sines formed algebraically: the same
// quantities, rounded differently, at a fraction of the FP64 instructions
// (collisional runs are compared with the reference statistically).
__device__ __noinline__ void scatter64(const StepConst &c, double u1, double u2, double &vx, double &vy, double &vz) {
    double xi_cos;
    if (c.model == SPG_COLL_HS)
        xi_cos = -1.0 + 2.0 * u1;
    else if (c.model == SPG_COLL_VHS)
        xi_cos = u1;
    else
        xi_cos = 2.0 * pow(u1, c.inv_alpha) - 1.0;
    const double xi_sin = sqrt(1.0 - xi_cos * xi_cos);
    double sphi, cphi;
    sincospi(2.0 * u2, &sphi, &cphi);
    const double nx = xi_sin * cphi, ny = xi_sin * sphi, nz = xi_cos;
    const double cmx = vx * c.mass_cp, cmy = vy * c.mass_cp, cmz = vz * c.mass_cp;
    const double pvx = c.mass_ct * vx, pvy = c.mass_ct * vy, pvz = c.mass_ct * vz;
    const double mp = sqrt(pvx * pvx + pvy * pvy + pvz * pvz);
    double ex = nx * mp, ey = ny * mp, ez = nz * mp;
    if (c.model == SPG_COLL_VSS) {
        // GeometryVector::calcBetaGamma + rotation (GeometryVector.hpp:448-471, 66-90)
        const double cb = fmin(1.0, fmax(-1.0, pvz / mp)), sb = sqrt(1.0 - cb * cb);
        const double tx = cb * ex + sb * ez, tz = -sb * ex + cb * ez;
        ex = tx;
        ez = tz;
        const double rxy = sqrt(pvx * pvx + pvy * pvy);
        const double cg = rxy > 0.0 ? pvx / rxy : 1.0, sg = rxy > 0.0 ? pvy / rxy : 0.0;
        const double ux = cg * ex - sg * ey, uy = sg * ex + cg * ey;
        ex = ux;
        ey = uy;
    }
    vx = ex + cmx;
    vy = ey + cmy;
    vz = ez + cmz;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned v) { return __reduce_add_sync(kFull, v); }

// Finite test from the exponent bits (no FP64 compare).
__device__ __forceinline__ bool finite_bits(double x) {
    return ((__double2hiint(x) >> 20) & 0x7ff) != 0x7ff;
}

// E per tet: E = -sum_i phi_i grad(lambda_i) = -sum_r (phi_{r+1} - phi_0) M_r
// (VolumetricMesh::computeElectricFields, VolumetricMesh.cpp:382-411, with the
// sign and scale of E = -grad(phi)), plus the push increment
// H = ((q E / m) dt) / 2, the operations of Particle::electroMagneticPush.
struct Field64 {
    double E[3], H[3];
    uint32_t ezero;
};

__device__ __forceinline__ Field64 field_values64(const FieldArgs &f, int64_t t) {
    const int4 tn = __ldg(f.tet_nodes + t);
    const double f0 = f.phi[tn.x], f1 = f.phi[tn.y], f2 = f.phi[tn.z], f3 = f.phi[tn.w];
    const double d1 = f1 - f0, d2 = f2 - f0, d3 = f3 - f0;
    TetGeo r;
    load_geo(f.rec, int(t), r);
    Field64 o;
#pragma unroll
    for (int k = 0; k < 3; ++k) o.E[k] = -((d1 * r.M[k] + d2 * r.M[3 + k]) + d3 * r.M[6 + k]);
    const double half_dt = 0.5 * f.dt;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double a = div_by_known(f.charge * o.E[k], f.mass, f.inv_mass);  // (q E) / m
        o.H[k] = a * half_dt;  // (a dt) / 2: halving is exact
    }
    o.ezero = (((__double_as_longlong(o.E[0]) | __double_as_longlong(o.E[1]) | __double_as_longlong(o.E[2])) << 1) == 0)
                  ? 1u : 0u;  // all three +-0
    return o;
}

__device__ __forceinline__ void store_field64(const FieldArgs &f, int64_t t, const Field64 &v) {
    TetRec &r = f.rec[t];
#pragma unroll
    for (int k = 0; k < 3; ++k) f.efield[3 * t + k] = v.E[k];
    *reinterpret_cast<double2 *>(r.H) = make_double2(v.H[0], v.H[1]);
    r.H[2] = v.H[2];
    r.ezero = v.ezero;
}

__device__ __forceinline__ void field_of_tet64(const FieldArgs &f, int64_t t) {
    store_field64(f, t, field_values64(f, t));
}

// ---------------------------------------------------------------- steps
// Steps c.step .. c.step + L - 1 of every particle in one launch, in the order
// of ParticleDynamicsProcessor.cpp:161-200: settled? -> |v| < vmin? -> outside
// bbox? -> E push (Boris, B = 0) -> move -> gas collision -> surface crossing
// along the move segment.
//
// A lane keeps its particle and the tet's push increment in registers and steps
// it until a step needs what few lanes need: the exact walk (the end point is
// not certainly inside the tet) or a collision that FP32 cannot rule out. An FP64
// instruction costs its warp the pipe whatever its active lanes (1.7
// thread-operations per clock and SM), so every warp schedules its lanes: such
// a particle's state goes to the warp's pool in shared memory and the lane takes
// a ready one from there. What is the same for all of them runs in full warps:
// loading 32 new particles with their push increments and the Philox blocks of
// the segment (prepare64), and the walks, or the scatterings, of 32 waiting
// particles (run_pool64). Only the end of a warp's range runs with idle lanes.
//
// Against one launch per step with a second one for the walks, the state moves
// once per segment instead of once per step and a scattering no longer costs
// 32 lanes (at 4.6e-4 collisions per particle-step every 70th warp-step paid
// one). The FP64 pipe bounds it, with the twelve operations of push and move:
// 76 % active (pure FP64 additions reach 81 %), 158 FP64 instructions per warp
// and ten steps against 171 with blocks that step in lockstep and 190 with the
// walks decided in FP64. Per step and 1e7 ions on 6.0e6 tets 415 -> 328 us;
// 1e6 ions on 7.5e5 tets 59 -> 36 us, 3e5 on 94,000 33 -> 14 us, 1e4 on 6,000
// 21 -> 3.8 us (there the launches and one warp's serial FP64 latency).
// The values are those of single steps in the same order for every particle,
// so the segment length changes no result.
//
// A walk may enter a tet whose field is of an older potential. Stamps count up
// with every launch that can write fields: a field that an earlier launch computed
// (stored_before) is read; otherwise the lane forms it in registers, and the lane
// whose compare-and-swap sets the stamp to seq also stores it for later launches.
// Nothing orders these stores with a read in the same launch, and no lane makes
// one: a new particle's tet was entered in an earlier launch, and an item that
// leaves the pool looks at the stamp, whether its walk entered a tet or not.

// Items of a warp's pool: those waiting for their walk at [0, np), those ready
// to step at [kPool - nr, kPool), those with a collision to decide at
// [kPool, kPool + ns) (while there is room; a scattering is over a hundred FP64
// instructions, so they wait for a batch of their own instead of costing the
// walks' batches theirs).
// Words: position (waiting: at the step's start); waiting: end position, ready:
// push increment; velocity; tet and id word; index, step and flags; bit j: step
// j of the segment is a collision candidate.
// np + nr <= 64 + idle lanes always holds: a step adds what it idles, taking a
// ready item keeps it, and what adds up to 32 ready items (new particles, a
// collision batch) runs only while np + nr <= 32 + idle lanes. So a step's
// 32 - idle items fit kPool = 96.
constexpr int kPool = 96, kSide = 24, kPoolWords = 12;
constexpr int kRefill = 2;   // idle lanes that make a warp look for work (8: 343 us per step of 1e7, 4: 331, 2: 328)
constexpr int kDrain = 16;   // idle lanes that make it run a part-filled batch when nothing else is left
template <int ITEMS>
struct PoolOf {
    double w[kPoolWords][ITEMS];
    unsigned int cross, settled, lost, capped, coll;
};
using WarpPool = PoolOf<kPool + kSide>;
using StepPool = PoolOf<64>;  // single steps: waiting items only
// Waiting items: the walk; the collision test; a position that is no number.
constexpr int kNeedWalk = 1, kNeedTest = 2, kNeedLost = 4;
// Ready items: the field is not zero; the tet lies inside the modelling box; a
// new particle (its place in its tet not yet shown, its arrays unchanged).
constexpr int kPush = 1, kInterior = 2, kNew = 4;
constexpr int kFlagBits = 3;

struct Seg64 {
    MeshDev m;
    DevParticles p;
    int64_t n;
    unsigned int *tri_count;
    DevCounters *ctr;
    LandRec *land;     // nullable: landing records (adjoint)
    HistRec *hist;     // nullable: tet and velocity at the start of every alive step
    int64_t hist_n;    // particles of a history plane
    int L;
    uint32_t seq;
};

// Push increment and flags of a tet whose field an earlier launch wrote.
struct Push64 {
    double hx, hy, hz;
    int flags;
};

__device__ __forceinline__ Push64 load_push(const TetRec *__restrict__ rec, int t) {
    // the record's last 32 bytes, from L2: an L1 line may be older
    const double2 *hp = reinterpret_cast<const double2 *>(rec + t) + 6;
    const double2 a = __ldcg(hp), b = __ldcg(hp + 1);
    const unsigned long long w = (unsigned long long)__double_as_longlong(b.y);
    return Push64{a.x, a.y, b.x, ((w & 0xffffffffull) == 0ull ? kPush : 0) | ((w >> 32) != 0ull ? kInterior : 0)};
}

template <class Pool>
__device__ __forceinline__ void put_ready(Pool &P, int k, double x, double y, double z, const Push64 &h, double vx,
                                          double vy, double vz, int tet, uint32_t idf, int i, int word, double cand) {
    P.w[0][k] = x;
    P.w[1][k] = y;
    P.w[2][k] = z;
    P.w[3][k] = h.hx;
    P.w[4][k] = h.hy;
    P.w[5][k] = h.hz;
    P.w[6][k] = vx;
    P.w[7][k] = vy;
    P.w[8][k] = vz;
    P.w[9][k] = __hiloint2double(int(idf), tet);
    P.w[10][k] = __hiloint2double(word | h.flags, i);
    P.w[11][k] = cand;
}

// New particles [base, base + 32) of the warp: the alive ones become ready
// items. Returns the new count of ready items.
__device__ __noinline__ int prepare64(const Seg64 &a, const StepConst &c, WarpPool &P, int64_t base, int nr) {
    const int lane = threadIdx.x & 31;
    const int64_t i = base + lane;
    uint32_t idf = kDead;
    if (i < a.n) idf = a.p.idf[i];
    const bool alive = !(idf & kDead);
    const unsigned go = __ballot_sync(kFull, alive);
    if (alive) {
        const int tet = a.p.tet[i];
        const double x = a.p.x[i], y = a.p.y[i], z = a.p.z[i];
        const double vx = a.p.vx[i], vy = a.p.vy[i], vz = a.p.vz[i];
        const Push64 h = load_push(a.m.rec, tet);
        unsigned long long cand = 0ull;
        if (c.model != SPG_COLL_NONE) cand = segment_candidates(c, idf & kIdMask, a.L);
        put_ready(P, kPool - 1 - nr - __popc(go & ((1u << lane) - 1u)), x, y, z, h, vx, vy, vz, tet, idf, int(i), kNew,
                  __longlong_as_double((long long)cand));
    }
    __syncwarp();
    return nr + __popc(go);
}

// The waiting items [first, first + take) of the warp's pool, one per lane:
// collision, walk, landing. An item that goes on becomes a ready one, the
// others are written to the particle arrays. Returns the new count of ready items.
template <class Pool>
__device__ __noinline__ int run_pool64(const Seg64 &a, const StepConst &c, const FieldArgs &f, Pool &P, int first,
                                       int take, int nr) {
    const int lane = threadIdx.x & 31;
    const bool mine = lane < take;
    double x = 0.0, y = 0.0, z = 0.0, vx = 0.0, vy = 0.0, vz = 0.0, cand = 0.0;
    int tet = 0, i = 0, j = 0;
    uint32_t idf = 0;
    bool on = false;
    unsigned cross = 0;
    int status = W_INSIDE;
    bool hit = false;
    Push64 h{};
    if (mine) {
        const int k = first + lane;
        x = P.w[0][k];
        y = P.w[1][k];
        z = P.w[2][k];
        double nx = P.w[3][k], ny = P.w[4][k], nz = P.w[5][k];
        vx = P.w[6][k];
        vy = P.w[7][k];
        vz = P.w[8][k];
        const double ti = P.w[9][k], ij = P.w[10][k];
        cand = P.w[11][k];
        tet = __double2loint(ti);
        idf = uint32_t(__double2hiint(ti));
        i = __double2loint(ij);
        const int need = __double2hiint(ij);
        j = need >> kFlagBits;
        if (need & kNeedTest) {
            const uint64_t step = uint64_t(c.step) + uint64_t(j);
            const uint32_t id = idf & kIdMask;
            const float fx = hi_float(vx), fy = hi_float(vy), fz = hi_float(vz);
            const uint32_t is_cand = uint32_t((unsigned long long)__double_as_longlong(cand) >> j) & 1u;
            hit = collision_test64(c, id, step, is_cand ^ 1u, fmaf(fz, fz, fmaf(fy, fy, fx * fx)), vx, vy, vz);
            if (hit) {
                const Philox4 r = collision_draw(step, 1u, id, c.seed_lo, c.seed_hi);
                scatter64(c, u01_from(r.v[0], r.v[1]), u01_from(r.v[2], r.v[3]), vx, vy, vz);
            }
        }
        bool entered = false;
        if (need & kNeedLost) {
            idf |= kLost;
            status = W_EXIT;
            a.p.idf[i] = idf;
            nx = x;
            ny = y;
            nz = z;
        } else if (need & kNeedWalk) {
            const WalkOut w = walk64(a.m, tet, x, y, z, nx, ny, nz, c.max_cross, true);
            cross = unsigned(w.crossings);
            status = w.status;
            if (w.status == W_SURFACE) {
                nx = x + w.s * (nx - x);
                ny = y + w.s * (ny - y);
                nz = z + w.s * (nz - z);
                atomicAdd(a.tri_count + w.tri, 1u);
                idf |= kSettled;
                if (a.land) {
                    a.land[i].step = int32_t(c.step + j);
                    a.land[i].face = w.face;
                    a.land[i].tet = w.tet;
                    a.land[i].s = w.s;
                }
            } else if (w.status != W_INSIDE) {
                idf |= kLost;
            }
            if (w.status != W_INSIDE) {
                a.p.idf[i] = idf;
            } else {
                entered = w.tet != tet;
            }
            tet = w.tet;
        }
        x = nx;
        y = ny;
        z = nz;
        on = status == W_INSIDE && j + 1 < a.L;
        if (on || entered) {
            // Also where the tet stays the same: the particle may have entered it earlier
            // in this launch, and then its field is being stored by another lane.
            const uint32_t st = __ldcg(f.stamp + tet);
            if (!stored_before(st, f.epoch, a.seq)) {
                const Field64 v = field_values64(f, tet);
                h.hx = v.H[0];
                h.hy = v.H[1];
                h.hz = v.H[2];
                h.flags = (v.ezero == 0u ? kPush : 0) | (__ldcg(&a.m.rec[tet].interior) != 0u ? kInterior : 0);
                if (st < f.epoch && atomicCAS(f.stamp + tet, st, a.seq) == st) store_field64(f, tet, v);
            } else if (on) {
                h = load_push(a.m.rec, tet);
            }
        }
        if (!on) {
            a.p.x[i] = x;
            a.p.y[i] = y;
            a.p.z[i] = z;
            a.p.vx[i] = vx;
            a.p.vy[i] = vy;
            a.p.vz[i] = vz;
            a.p.tet[i] = tet;
        }
    }
    __syncwarp();
    const unsigned go = __ballot_sync(kFull, on);
    if (on)
        put_ready(P, kPool - 1 - nr - __popc(go & ((1u << lane) - 1u)), x, y, z, h, vx, vy, vz, tet, idf, i,
                  (j + 1) << kFlagBits, cand);
    const unsigned n0 = __reduce_add_sync(kFull, cross), n4 = __popc(__ballot_sync(kFull, hit));
    const unsigned n1 = __popc(__ballot_sync(kFull, status == W_SURFACE));
    const unsigned n2 = __popc(__ballot_sync(kFull, status == W_EXIT || status == W_CAP));
    const unsigned n3 = __popc(__ballot_sync(kFull, status == W_CAP));
    if (lane == 0) {
        P.cross += n0;
        P.settled += n1;
        P.lost += n2;
        P.capped += n3;
        P.coll += n4;
    }
    __syncwarp();
    return nr + __popc(go);
}

template <bool HIST>
__global__ void __launch_bounds__(128, 4) k_seg64(const __grid_constant__ Seg64 a, const __grid_constant__ StepConst c,
                                                  const __grid_constant__ FieldArgs f) {
    extern __shared__ __align__(16) unsigned char pool_bytes[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    WarpPool &P = reinterpret_cast<WarpPool *>(pool_bytes)[wid];
    if (lane == 0) P.cross = P.settled = P.lost = P.capped = P.coll = 0u;
    __syncwarp();
    unsigned processed = 0;
    int np = 0, nr = 0, ns = 0;
    // new particles: 32 at a time, the warps of the grid in turn
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    int64_t base = int64_t(blockIdx.x) * blockDim.x + 32 * wid;
    bool have = false;
    double x = 0.0, y = 0.0, z = 0.0, vx = 0.0, vy = 0.0, vz = 0.0, hx = 0.0, hy = 0.0, hz = 0.0;
    int tet = 0, i = 0, j = 0, flags = 0;
    uint32_t idf = 0;
    unsigned long long cand = 0ull;
    bool dirty = false;
    for (;;) {
        unsigned idle = __ballot_sync(kFull, !have);
        if (__popc(idle) >= kRefill) {
            if (nr < __popc(idle) && base < a.n && np + nr <= 32 + __popc(idle)) {
                nr = prepare64(a, c, P, base, nr);
                base += stride;
            }
            if (nr > 0) {
                const int take = min(nr, __popc(idle));
                const int k = kPool - nr + __popc(idle & below);
                if (!have && __popc(idle & below) < take) {
                    x = P.w[0][k];
                    y = P.w[1][k];
                    z = P.w[2][k];
                    hx = P.w[3][k];
                    hy = P.w[4][k];
                    hz = P.w[5][k];
                    vx = P.w[6][k];
                    vy = P.w[7][k];
                    vz = P.w[8][k];
                    const double ti = P.w[9][k], ij = P.w[10][k];
                    cand = (unsigned long long)__double_as_longlong(P.w[11][k]);
                    tet = __double2loint(ti);
                    idf = uint32_t(__double2hiint(ti));
                    i = __double2loint(ij);
                    flags = __double2hiint(ij);
                    j = flags >> kFlagBits;
                    dirty = !(flags & kNew);
                    have = true;
                }
                nr -= take;
                __syncwarp();
                idle = __ballot_sync(kFull, !have);
            }
        }
        const bool drain = base >= a.n && __popc(idle) >= kDrain;
        if (np >= 32 || (np > 0 && drain)) {
            const int take = min(np, 32);
            np -= take;
            nr = run_pool64(a, c, f, P, np, take, nr);
            continue;
        }
        if ((ns == kSide || (ns > 0 && drain)) && np + nr <= 32 + __popc(idle)) {
            nr = run_pool64(a, c, f, P, kPool, ns, nr);
            ns = 0;
            continue;
        }
        if (idle == kFull) {
            if (nr > 0 || base < a.n) continue;
            break;  // nothing waits and no new particle is left
        }
        // ---- one step of every lane that has a particle
        int need = 0;
        double nx = 0.0, ny = 0.0, nz = 0.0;
        bool done = false;
        if (have) {
            if constexpr (HIST) {
                double2 *o = reinterpret_cast<double2 *>(a.hist + int64_t(j) * a.hist_n + i);
                o[0] = make_double2(vx, vy);
                o[1] = make_double2(vz, __hiloint2double(0, tet));
            }
            ++processed;
            // |v| < vmin: certainly false when some |v_k| >= 2 vmin (bit compare of
            // non-negative doubles); otherwise the exact FP64 test.
            const long long ax = __double_as_longlong(vx) & 0x7fffffffffffffffLL;
            const long long ay = __double_as_longlong(vy) & 0x7fffffffffffffffLL;
            const long long az = __double_as_longlong(vz) & 0x7fffffffffffffffLL;
            bool stays = false;
            if (ax < c.two_vmin_bits && ay < c.two_vmin_bits && az < c.two_vmin_bits)
                stays = sqrt(vx * vx + vy * vy + vz * vz) < c.vmin;
            if ((flags & (kNew | kInterior)) != kInterior) {
                // outside the modelling box; skipped where this launch has shown the
                // particle to lie in its tet and the tet lies inside the box
                const long long kx = order_key(x), ky = order_key(y), kz = order_key(z);
                stays = stays || !(kx >= c.lo_key[0] && kx <= c.hi_key[0] && ky >= c.lo_key[1] && ky <= c.hi_key[1] &&
                                   kz >= c.lo_key[2] && kz <= c.hi_key[2]);
            }
            if (stays) {  // nothing moves it any more
                if constexpr (!HIST) {
                    processed += unsigned(a.L - 1 - j);
                    j = a.L - 1;
                }
            } else {
                if (flags & kPush) {
                    // Particle::electroMagneticPush (Particle.cpp:196-234) with B = 0:
                    // v- = v + a dt/2, the rotation is the identity, v = v- + a dt/2.
                    vx = (vx + hx) + hx;
                    vy = (vy + hy) + hy;
                    vz = (vz + hz) + hz;
                }
                dirty = true;
                // Particle::updatePosition (Particle.cpp:157-165)
                nx = x + vx * c.dt;
                ny = y + vy * c.dt;
                nz = z + vz * c.dt;
                if (!(same_value(nx, x) && same_value(ny, y) && same_value(nz, z))) {
                    if (c.model != SPG_COLL_NONE) {
                        // no candidate and v^2 at most v2_cand_f (from the 20-bit components): no collision
                        const bool is_cand = (cand >> j) & 1ull;
                        const float fx = hi_float(vx), fy = hi_float(vy), fz = hi_float(vz);
                        const float v2 = fmaf(fz, fz, fmaf(fy, fy, fx * fx));
                        if ((is_cand || !(v2 <= c.v2_cand_f)) &&
                            !no_collision_sure(c, idf & kIdMask, uint64_t(c.step) + uint64_t(j), is_cand, v2))
                            need = kNeedTest;
                    }
                    if (!(finite_bits(nx) && finite_bits(ny) && finite_bits(nz))) {
                        need |= kNeedLost;
                    } else {
                        if (!inside_sure(load_screen(a.m.screen + tet), nx, ny, nz)) need |= kNeedWalk;
                        flags &= ~kNew;  // of the next step's position, walked or not
                        if (!need) {
                            x = nx;
                            y = ny;
                            z = nz;
                        }
                    }
                }
            }
            if (!need) done = ++j == a.L;
        }
        const unsigned out = __ballot_sync(kFull, need != 0);
        if (out) {
            // collisions to the side while it has room, the rest to the waiting items
            const unsigned test = __ballot_sync(kFull, (need & kNeedTest) != 0);
            const int room = kSide - ns;
            const bool side = (need & kNeedTest) && __popc(test & below) < room;
            const unsigned main_out = __ballot_sync(kFull, need != 0 && !side);
            if (need) {
                const int k = side ? kPool + ns + __popc(test & below) : np + __popc(main_out & below);
                P.w[0][k] = x;
                P.w[1][k] = y;
                P.w[2][k] = z;
                P.w[3][k] = nx;
                P.w[4][k] = ny;
                P.w[5][k] = nz;
                P.w[6][k] = vx;
                P.w[7][k] = vy;
                P.w[8][k] = vz;
                P.w[9][k] = __hiloint2double(int(idf), tet);
                P.w[10][k] = __hiloint2double((j << kFlagBits) | need, i);
                P.w[11][k] = __longlong_as_double((long long)cand);
                have = false;
            }
            np += __popc(main_out);
            ns += min(__popc(test), room);
            __syncwarp();
        }
        if (done) {
            if (dirty) {
                a.p.x[i] = x;
                a.p.y[i] = y;
                a.p.z[i] = z;
                a.p.vx[i] = vx;
                a.p.vy[i] = vy;
                a.p.vz[i] = vz;
                a.p.tet[i] = tet;
            }
            have = false;
        }
    }
    // one atomic per counter and warp
    const unsigned long long n0 = warp_sum(processed);
    if (lane == 0) {
        const unsigned long long n1 = P.coll, n3 = P.cross, n4 = P.settled, n5 = P.capped, n6 = P.lost;
        if (n0) atomicAdd(&a.ctr->processed, n0);
        if (n1) atomicAdd(&a.ctr->collisions, n1);
        if (n3) atomicAdd(&a.ctr->crossings, n3);
        if (n4) atomicAdd(&a.ctr->settled, n4);
        if (n5) atomicAdd(&a.ctr->capped, n5);
        if (n6) atomicAdd(&a.ctr->lost, n6);
    }
}

// A single step (a call of one step, or steps between which the trajectories are
// sampled). Nothing is gained there by a lane that takes another particle at
// once: a warp steps 32 particles straight from the arrays, writes those that stay
// in their tet, and pools the others; 32 of these are walked and decided in a
// full warp and written. No state lives across the pool, so the kernel holds 80
// registers and 24 warps per SM instead of 128 and 16, which hides the loads that
// a step of its own needs. The operations are those of k_seg64's step. us per
// step, a step and a walk kernel with a queue in memory / k_seg64 with L = 1 /
// here: 1e7 ions on 6.0e6 tets 417, 523, 390; 1e6 of a Thompson source 58, 62, 48,
// all over the mesh 71, 78, 60; 1e5 27, 20, 17. (Blocks per SM 5 / 6 / 8: 408, 390,
// 495 at 1e7.)
__global__ void __launch_bounds__(128, 6) k_step64(const __grid_constant__ Seg64 a, const __grid_constant__ StepConst c,
                                                   const __grid_constant__ FieldArgs f) {
    extern __shared__ __align__(16) unsigned char pool_bytes[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    StepPool &P = reinterpret_cast<StepPool *>(pool_bytes)[wid];
    if (lane == 0) P.cross = P.settled = P.lost = P.capped = P.coll = 0u;
    __syncwarp();
    unsigned processed = 0;
    int np = 0;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t base = int64_t(blockIdx.x) * blockDim.x + 32 * wid; base < a.n; base += stride) {
        const int64_t i = base + lane;
        uint32_t idf = kDead;
        if (i < a.n) idf = a.p.idf[i];
        int need = 0, tet = 0;
        double x = 0.0, y = 0.0, z = 0.0, vx = 0.0, vy = 0.0, vz = 0.0, nx = 0.0, ny = 0.0, nz = 0.0;
        uint32_t is_cand = 0u;
        if (!(idf & kDead)) {
            ++processed;
            tet = a.p.tet[i];
            x = a.p.x[i];
            y = a.p.y[i];
            z = a.p.z[i];
            vx = a.p.vx[i];
            vy = a.p.vy[i];
            vz = a.p.vz[i];
            const ScreenRegs scr = load_screen(a.m.screen + tet);
            const Push64 h = load_push(a.m.rec, tet);
            // the tests of k_seg64's step, in its order
            const long long ax = __double_as_longlong(vx) & 0x7fffffffffffffffLL;
            const long long ay = __double_as_longlong(vy) & 0x7fffffffffffffffLL;
            const long long az = __double_as_longlong(vz) & 0x7fffffffffffffffLL;
            bool stays = false;
            if (ax < c.two_vmin_bits && ay < c.two_vmin_bits && az < c.two_vmin_bits)
                stays = sqrt(vx * vx + vy * vy + vz * vz) < c.vmin;
            const long long kx = order_key(x), ky = order_key(y), kz = order_key(z);
            stays = stays || !(kx >= c.lo_key[0] && kx <= c.hi_key[0] && ky >= c.lo_key[1] && ky <= c.hi_key[1] &&
                               kz >= c.lo_key[2] && kz <= c.hi_key[2]);
            if (!stays) {
                if (h.flags & kPush) {
                    vx = (vx + h.hx) + h.hx;
                    vy = (vy + h.hy) + h.hy;
                    vz = (vz + h.hz) + h.hz;
                }
                nx = x + vx * c.dt;
                ny = y + vy * c.dt;
                nz = z + vz * c.dt;
                if (!(same_value(nx, x) && same_value(ny, y) && same_value(nz, z))) {
                    if (c.model != SPG_COLL_NONE) {
                        const uint32_t id = idf & kIdMask;
                        is_cand = candidate_byte(candidate_block(uint64_t(c.step), id, c.seed_lo, c.seed_hi),
                                                 uint64_t(c.step)) == 0u;
                        const float fx = hi_float(vx), fy = hi_float(vy), fz = hi_float(vz);
                        const float v2 = fmaf(fz, fz, fmaf(fy, fy, fx * fx));
                        if ((is_cand || !(v2 <= c.v2_cand_f)) &&
                            !no_collision_sure(c, id, uint64_t(c.step), is_cand, v2))
                            need = kNeedTest;
                    }
                    if (!(finite_bits(nx) && finite_bits(ny) && finite_bits(nz)))
                        need |= kNeedLost;
                    else if (!inside_sure(scr, nx, ny, nz))
                        need |= kNeedWalk;
                }
                if (!need) {
                    a.p.x[i] = nx;
                    a.p.y[i] = ny;
                    a.p.z[i] = nz;
                    a.p.vx[i] = vx;
                    a.p.vy[i] = vy;
                    a.p.vz[i] = vz;
                }
            }
        }
        const unsigned out = __ballot_sync(kFull, need != 0);
        if (need) {
            const int k = np + __popc(out & below);
            P.w[0][k] = x;
            P.w[1][k] = y;
            P.w[2][k] = z;
            P.w[3][k] = nx;
            P.w[4][k] = ny;
            P.w[5][k] = nz;
            P.w[6][k] = vx;
            P.w[7][k] = vy;
            P.w[8][k] = vz;
            P.w[9][k] = __hiloint2double(int(idf), tet);
            P.w[10][k] = __hiloint2double(need, int(i));
            P.w[11][k] = __longlong_as_double((long long)is_cand);
        }
        np += __popc(out);  // at most 31 + 32
        __syncwarp();
        if (np >= 32) {
            np -= 32;
            run_pool64(a, c, f, P, np, 32, 0);
        }
    }
    if (np > 0) run_pool64(a, c, f, P, 0, np, 0);
    const unsigned long long n0 = warp_sum(processed);
    if (lane == 0) {
        const unsigned long long n1 = P.coll, n3 = P.cross, n4 = P.settled, n5 = P.capped, n6 = P.lost;
        if (n0) atomicAdd(&a.ctr->processed, n0);
        if (n1) atomicAdd(&a.ctr->collisions, n1);
        if (n3) atomicAdd(&a.ctr->crossings, n3);
        if (n4) atomicAdd(&a.ctr->settled, n4);
        if (n5) atomicAdd(&a.ctr->capped, n5);
        if (n6) atomicAdd(&a.ctr->lost, n6);
    }
}

// round(x * 2^k) for k <= 52 with integer ops only (round half away from zero
// on the magnitude). |x| < 2^(52 - k), as every barycentric of a particle inside
// its tet, takes no branch: the shift is at least 1, and a zero, a subnormal
// or any |x| 2^k < 1/2 shifts out.
__device__ __forceinline__ long long fix_round(double x, int k) {
    const long long b = __double_as_longlong(x);
    const int e = int((b >> 52) & 0x7ff);
    const long long mant = (b & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
    const int sh = 1075 - e - k;
    const int s1 = min(max(sh, 1), 63);
    long long r = (mant + (1LL << (s1 - 1))) >> s1;
    if (sh < 1) r = mant << (-sh);
    return b < 0 ? -r : r;
}

// P1 deposit in fixed point: each alive particle adds round(lambda_i 2^k) for
// i = 1..3 and 2^k minus their sum for lambda_0, so its four node shares are
// exactly 2^k and charge is conserved exactly. Integer sums do not depend on
// summation order, so the result is the same for any particle order, grid
// or atomic interleaving. Lanes of a warp hold consecutive (tet-sorted)
// particles; runs of equal tet are summed per warp and merged in the
// block's node table over its range of tiles (deposit.cuh).
struct DepSrc64 {
    struct Raw {
        uint32_t idf;
        int32_t tet;
        double x, y, z;
    };
    DevParticles p;
    const TetRec *rec;
    int k;
    long long one;
    __device__ __forceinline__ Raw load(int64_t i, int64_t n) const {
        Raw r{kDead, -1, 0.0, 0.0, 0.0};
        if (i < n) {
            r.idf = __ldg(p.idf + i);
            r.tet = __ldg(p.tet + i);
            r.x = __ldg(p.x + i);
            r.y = __ldg(p.y + i);
            r.z = __ldg(p.z + i);
        }
        return r;
    }
    __device__ __forceinline__ int weights(const Raw &r, long long v[4]) const {
        v[0] = v[1] = v[2] = v[3] = 0;
        if (r.idf & kDead) return -1;
        TetGeo g;
        load_geo(rec, r.tet, g);
        const double d0 = r.x - g.x0[0], d1 = r.y - g.x0[1], d2 = r.z - g.x0[2];
        // fused: nothing compares a weight bit by bit, and 12 FP64 instructions
        // instead of 18 issue
        const double l1 = __fma_rn(g.M[2], d2, __fma_rn(g.M[1], d1, g.M[0] * d0));
        const double l2 = __fma_rn(g.M[5], d2, __fma_rn(g.M[4], d1, g.M[3] * d0));
        const double l3 = __fma_rn(g.M[8], d2, __fma_rn(g.M[7], d1, g.M[6] * d0));
        v[1] = fix_round(l1, k);
        v[2] = fix_round(l2, k);
        v[3] = fix_round(l3, k);
        v[0] = one - v[1] - v[2] - v[3];
        return r.tet;
    }
};

__global__ void __launch_bounds__(kDepThreads)
    k_deposit64(const DepSrc64 src, int64_t n, const int4 *__restrict__ tet_nodes,
                unsigned long long *__restrict__ node_fix, const OccList occ) {
    deposit_tiles(src, n, tet_nodes, node_fix, occ);
}

__global__ void k_fix_to_charge(const unsigned long long *__restrict__ node_fix, double scale,
                                double *__restrict__ node_q, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    node_q[i] = double((long long)node_fix[i]) * scale;
}

// The field of the tets listed by the deposit (each once).
__global__ void k_field64_list(const __grid_constant__ FieldArgs f, const int32_t *__restrict__ list,
                               const unsigned int *__restrict__ list_n) {
    const unsigned nl = *list_n;
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < nl; j += gridDim.x * blockDim.x) {
        const int t = list[j];
        field_of_tet64(f, t);
        f.stamp[t] = f.epoch;
    }
}

// Every tet's field. Bound by the FP64 pipe (33 instructions per tet: 0.40 ms for
// 6.0e6 tets at the measured rate). 829 us before, with scalar loads of the map
// and a division wherever a component was zero, which a potential that is flat
// over most of the mesh has in every warp: 576 us for a charged potential, 441
// for the electrodes' start values now.
__global__ void k_field64_full(const __grid_constant__ FieldArgs f, int64_t n) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    field_of_tet64(f, t);
    f.stamp[t] = f.epoch;
}

// The field of every tet holding an alive particle. Particles are tet-sorted
// (up to the drift since the last re-sort), so only the first lane of each
// run of equal tets in a warp checks the stamp.
__global__ void k_refresh64(DevParticles p, int64_t n, const __grid_constant__ FieldArgs f) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int key = (i < n && !(p.idf[i] & kDead)) ? p.tet[i] : -1;
    const int prev = __shfl_up_sync(kFull, key, 1);
    if (key >= 0 && ((threadIdx.x & 31) == 0 || prev != key))
        refresh_tet(f.stamp, f.epoch, key, [&f](int t) { field_of_tet64(f, t); });
}

__global__ void k_interior_flags(TetRec *__restrict__ rec, const int4 *__restrict__ tet_nodes,
                                 const double *__restrict__ xyz, int64_t n, double lx, double ly, double lz, double hx,
                                 double hy, double hz) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int4 tn = tet_nodes[t];
    const int nd[4] = {tn.x, tn.y, tn.z, tn.w};
    bool in = true;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double x = xyz[3 * int64_t(nd[k])], y = xyz[3 * int64_t(nd[k]) + 1], z = xyz[3 * int64_t(nd[k]) + 2];
        in = in && x >= lx && x <= hx && y >= ly && y <= hy && z >= lz && z <= hz;
    }
    rec[t].interior = in ? 1u : 0u;
}

// E = 0 and H = 0 in tets [t0, t1), stamped, by the `threads` threads of which
// this is number `thread` (before the first solve). Of a record only the words
// of its form are written and none is read (a read of the strided sectors costs
// more than all stores: 529 us in the mixed form), E and the stamps in the order
// of memory. 6.0e6 tets: mixed form 664 -> 127 us, FP64 227 -> 215 us (32 of each
// 128 bytes).
__device__ __forceinline__ void zero_field_range(const FieldArgs &f, int64_t t0, int64_t t1, int thread, int threads) {
    for (int64_t t = t0 + thread; t < t1; t += threads) {
        if (f.rec32) {
            TetRec32 &rt = f.rec32[t];
            rt.H[0] = 0.0f;
            *reinterpret_cast<float2 *>(rt.H + 1) = make_float2(0.0f, 0.0f);
            set_rec_ezero(rt, true);
        } else {
            TetRec &rt = f.rec[t];
            *reinterpret_cast<double2 *>(rt.H) = make_double2(0.0, 0.0);
            rt.H[2] = 0.0;
            rt.ezero = 1u;
        }
        f.stamp[t] = f.epoch;
    }
    for (int64_t k = 3 * t0 + thread; k < 3 * t1; k += threads) f.efield[k] = 0.0;
}

__global__ void __launch_bounds__(256) k_zero_field(const __grid_constant__ FieldArgs f, int64_t n) {
    const int64_t t0 = int64_t(blockIdx.x) * 256;
    zero_field_range(f, t0, t0 + 256 < n ? t0 + 256 : n, threadIdx.x, 256);
}

__global__ void k_count_lost(const int32_t *__restrict__ tet, int64_t n, unsigned long long *out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const unsigned v = (i < n && tet[i] < 0) ? 1u : 0u;
    const unsigned s = __reduce_add_sync(kFull, v);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, (unsigned long long)s);
}

// Point location: walk from the centroid of the voxel's seed tet to p.
__global__ void k_locate(const double *__restrict__ pos, int64_t n, const __grid_constant__ MeshDev m, const int32_t *__restrict__ vox_seed,
                         double ox, double oy, double oz, double ix, double iy, double iz, int dx, int dy, int dz,
                         int max_cross, int32_t *__restrict__ tet_out) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
    if (!(finite_bits(px) && finite_bits(py) && finite_bits(pz))) {
        tet_out[i] = -1;
        return;
    }
    const int vx = min(dx - 1, max(0, int(floor((px - ox) * ix))));
    const int vy = min(dy - 1, max(0, int(floor((py - oy) * iy))));
    const int vz = min(dz - 1, max(0, int(floor((pz - oz) * iz))));
    const int seed = vox_seed[vx + int64_t(dx) * (vy + int64_t(dy) * vz)];
    const int4 tn = __ldg(m.tet_nodes + seed);
    double c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        c[k] = 0.25 * (((m.node_xyz[3 * tn.x + k] + m.node_xyz[3 * tn.y + k]) + m.node_xyz[3 * tn.z + k]) +
                       m.node_xyz[3 * tn.w + k]);
    const WalkOut w = walk64(m, seed, c[0], c[1], c[2], px, py, pz, max_cross, false);
    tet_out[i] = w.status == W_INSIDE ? w.tet : -1;
}

// Upload and location in one pass, reading the caller's position and
// velocity arrays where they lie (host memory the GPU reaches over the C2C
// link), so the copy overlaps the location walks: the same tet and state as
// k_locate followed by k_init_particles (FP64 form) or k_to_local (mixed form,
// cen != nullptr: FP32 position about the tet's centroid, FP32 velocity).
__global__ void __launch_bounds__(128) k_upload(const double *__restrict__ pos, const double *__restrict__ vel, int64_t n,
                         const __grid_constant__ MeshDev m, const int32_t *__restrict__ vox_seed, double ox, double oy, double oz, double ix, double iy,
                         double iz, int dx, int dy, int dz, int max_cross, DevParticles p, DevParticles32 q,
                         const double *__restrict__ cen, unsigned long long *lost, const __grid_constant__ FieldArgs f,
                         int64_t zero_tets, int zero_per_block) {
    // the block's share of the tets whose field is set to zero: its stores go to
    // HBM while the link brings the particles
    if (zero_per_block > 0) {
        const int64_t t0 = int64_t(blockIdx.x) * zero_per_block;
        const int64_t t1 = t0 + zero_per_block;
        zero_field_range(f, t0 < zero_tets ? t0 : zero_tets, t1 < zero_tets ? t1 : zero_tets, threadIdx.x, 128);
    }
    // the block's xyz triples come in as one contiguous run per array (whole
    // lines per warp load), then each thread takes its particle's
    __shared__ double sp[3 * 128], sv[3 * 128];
    const int64_t i0 = int64_t(blockIdx.x) * 128;
    const int64_t i = i0 + threadIdx.x;
    const int cnt = n - i0 < 128 ? int(n - i0) : 128;
    for (int k = threadIdx.x; k < 3 * cnt; k += 128) {
        sp[k] = pos[3 * i0 + k];
        sv[k] = vel[3 * i0 + k];
    }
    __syncthreads();
    unsigned is_lost = 0;
    if (i < n) {
        const double px = sp[3 * threadIdx.x], py = sp[3 * threadIdx.x + 1], pz = sp[3 * threadIdx.x + 2];
        const double vx = sv[3 * threadIdx.x], vy = sv[3 * threadIdx.x + 1], vz = sv[3 * threadIdx.x + 2];
        int32_t t = -1;
        if (finite_bits(px) && finite_bits(py) && finite_bits(pz)) {
            const int cx = min(dx - 1, max(0, int(floor((px - ox) * ix))));
            const int cy = min(dy - 1, max(0, int(floor((py - oy) * iy))));
            const int cz = min(dz - 1, max(0, int(floor((pz - oz) * iz))));
            const int seed = vox_seed[cx + int64_t(dx) * (cy + int64_t(dy) * cz)];
            const int4 tn = __ldg(m.tet_nodes + seed);
            double c[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
                c[k] = 0.25 * (((m.node_xyz[3 * tn.x + k] + m.node_xyz[3 * tn.y + k]) + m.node_xyz[3 * tn.z + k]) +
                               m.node_xyz[3 * tn.w + k]);
            const WalkOut w = walk64(m, seed, c[0], c[1], c[2], px, py, pz, max_cross, false);
            t = w.status == W_INSIDE ? w.tet : -1;
        }
        is_lost = t < 0 ? 1u : 0u;
        const uint32_t idf = uint32_t(i) | (t < 0 ? kLost : 0u);
        if (cen) {
            const int64_t tc = t < 0 ? 0 : t;
            q.x[i] = float(px - (t < 0 ? 0.0 : cen[3 * tc]));
            q.y[i] = float(py - (t < 0 ? 0.0 : cen[3 * tc + 1]));
            q.z[i] = float(pz - (t < 0 ? 0.0 : cen[3 * tc + 2]));
            q.vx[i] = float(vx);
            q.vy[i] = float(vy);
            q.vz[i] = float(vz);
            q.tet[i] = t;
            q.idf[i] = idf;
        } else {
            p.x[i] = px;
            p.y[i] = py;
            p.z[i] = pz;
            p.vx[i] = vx;
            p.vy[i] = vy;
            p.vz[i] = vz;
            p.tet[i] = t;
            p.idf[i] = idf;
        }
    }
    const unsigned s = __reduce_add_sync(kFull, is_lost);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(lost, (unsigned long long)s);
}

__global__ void k_init_particles(const double *__restrict__ pos, const double *__restrict__ vel,
                                 const int32_t *__restrict__ tet, int64_t n, DevParticles p, int64_t id_base) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t j = id_base + i;
    p.x[j] = pos[3 * i];
    p.y[j] = pos[3 * i + 1];
    p.z[j] = pos[3 * i + 2];
    p.vx[j] = vel[3 * i];
    p.vy[j] = vel[3 * i + 1];
    p.vz[j] = vel[3 * i + 2];
    const int32_t t = tet[i];
    p.tet[j] = t;
    p.idf[j] = uint32_t(j) | (t < 0 ? kLost : 0u);
}

// Slot of each particle id. The ids are a permutation of 0..n-1 (set, inject
// and restore keep it so); an id out of range is not written.
__global__ void k_slot_of_id(const uint32_t *__restrict__ idf, int64_t n, int32_t *__restrict__ slot) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = idf[i] & kIdMask;
    if (int64_t(id) < n) slot[id] = int32_t(i);
}

// One thread per id: scattered reads of its slot, writes in id order. The
// block's xyz triples go through shared memory and out as one contiguous run
// per array, so each warp store covers whole lines (the arrays may be the
// caller's pinned host memory, written over the C2C link).
__global__ void __launch_bounds__(256) k_gather_by_id(DevParticles p, int64_t n, const int32_t *__restrict__ slot,
                                                      double *pos, double *vel, int32_t *tet, uint32_t *flags) {
    __shared__ double sp[3 * 256], sv[3 * 256];
    const int64_t id0 = int64_t(blockIdx.x) * 256;
    const int64_t id = id0 + threadIdx.x;
    const int m = n - id0 < 256 ? int(n - id0) : 256;
    if (id < n) {
        const int64_t i = slot[id];
        const uint32_t idf = p.idf[i];
        if (pos) {
            sp[3 * threadIdx.x] = p.x[i];
            sp[3 * threadIdx.x + 1] = p.y[i];
            sp[3 * threadIdx.x + 2] = p.z[i];
        }
        if (vel) {
            sv[3 * threadIdx.x] = p.vx[i];
            sv[3 * threadIdx.x + 1] = p.vy[i];
            sv[3 * threadIdx.x + 2] = p.vz[i];
        }
        if (tet) tet[id] = p.tet[i];
        if (flags) flags[id] = ((idf & kSettled) ? SPG_FLAG_SETTLED : 0u) | ((idf & kLost) ? SPG_FLAG_LOST : 0u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 3 * m; k += 256) {
        if (pos) pos[3 * id0 + k] = sp[k];
        if (vel) vel[3 * id0 + k] = sv[k];
    }
}

// ------------------------------------------------------------------ re-sort
// Counting sort by tet (dead particles get key n_tets and go last).

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kSortBlock) k_sort_hist(const int32_t *__restrict__ tet,
                                                          const uint32_t *__restrict__ idf, int64_t n, int n_tets,
                                                          int32_t *__restrict__ cnt) {
    __shared__ SortTable t;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int key = i < n ? ((idf[i] & kDead) ? n_tets : tet[i]) : -1;
    sort_hist_block(t, key, cnt);
}

__global__ void __launch_bounds__(kSortBlock) k_sort_rank(const int32_t *__restrict__ tet,
                                                          const uint32_t *__restrict__ idf, int64_t n, int n_tets,
                                                          int32_t *__restrict__ cnt, int32_t *__restrict__ rank) {
    __shared__ SortTable t;
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int key = i < n ? ((idf[i] & kDead) ? n_tets : tet[i]) : -1;
    const int r = sort_rank_block(t, key, n_tets, cnt);
    if (i < n) rank[i] = r;
}

// Block-local exclusive scan of one tile; tile total to sums[blockIdx.x].
// Also counts non-empty tet bins (occupied tets).
__global__ void __launch_bounds__(kScanThreads) k_scan_tile(int32_t *__restrict__ a, int64_t len, int n_tets,
                                                            int32_t *__restrict__ sums,
                                                            unsigned long long *__restrict__ occupied) {
    __shared__ int32_t ws[kScanThreads / 32];
    const int64_t base = int64_t(blockIdx.x) * kScanTile + int64_t(threadIdx.x) * kScanItems;
    int32_t v[kScanItems];
    int32_t run = 0;
    unsigned occ = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t j = base + k;
        const int32_t x = j < len ? a[j] : 0;
        if (j < n_tets && x > 0) occ++;
        v[k] = run;
        run += x;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t incl = run;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int32_t up = __shfl_up_sync(kFull, incl, off);
        if (lane >= off) incl += up;
    }
    if (lane == 31) ws[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int32_t w = lane < kScanThreads / 32 ? ws[lane] : 0;
        int32_t wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t up = __shfl_up_sync(kFull, wi, off);
            if (lane >= off) wi += up;
        }
        if (lane < kScanThreads / 32) ws[lane] = wi - w;
    }
    __syncthreads();
    const int32_t offset = ws[wid] + (incl - run);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const int64_t j = base + k;
        if (j < len) a[j] = v[k] + offset;
    }
    if (threadIdx.x == kScanThreads - 1) sums[blockIdx.x] = offset + run;
    const unsigned long long occw = __reduce_add_sync(kFull, occ);
    if (lane == 0 && occw) atomicAdd(occupied, occw);
}

// Exclusive scan of the tile sums by one block, carrying across chunks.
__global__ void __launch_bounds__(1024) k_scan_sums(int32_t *__restrict__ sums, int64_t nb) {
    __shared__ int32_t ws[32];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t c0 = 0; c0 < nb; c0 += 1024) {
        const int64_t j = c0 + threadIdx.x;
        const int32_t x = j < nb ? sums[j] : 0;
        int32_t incl = x;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int32_t up = __shfl_up_sync(kFull, incl, off);
            if (lane >= off) incl += up;
        }
        if (lane == 31) ws[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int32_t w = ws[lane];
            int32_t wi = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int32_t up = __shfl_up_sync(kFull, wi, off);
                if (lane >= off) wi += up;
            }
            ws[lane] = wi - w;
        }
        __syncthreads();
        const int32_t excl = carry + ws[wid] + incl - x;
        if (j < nb) sums[j] = excl;
        __syncthreads();
        if (threadIdx.x == 1023) carry = excl + x;
        __syncthreads();
    }
}

__global__ void k_scan_add(int32_t *__restrict__ a, int64_t len, const int32_t *__restrict__ sums, int n_tets,
                           int64_t *__restrict__ n_alive) {
    const int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= len) return;
    const int32_t v = a[j] + sums[j / kScanTile];
    a[j] = v;
    if (j == n_tets) *n_alive = v;
}

__global__ void __launch_bounds__(kSortBlock) k_sort_scatter(DevParticles src, DevParticles dst, int64_t n, int n_tets,
                                                             int32_t *__restrict__ offs) {
    __shared__ SortTable t;
    sort_scatter_block(t, src, dst, n, n_tets, kDead, offs);
}

__global__ void __launch_bounds__(kSortBlock) k_sort_records(DevParticles src, SortRec64 *rec, int64_t n, int n_tets,
                                                             const int32_t *__restrict__ offs,
                                                             const int32_t *__restrict__ rank) {
    sort_to_records(src, rec, n, n_tets, kDead, offs, rank);
}
__global__ void __launch_bounds__(kSortBlock) k_sort_unpack(const SortRec64 *__restrict__ rec, DevParticles dst,
                                                            int64_t n) {
    sort_unpack(rec, dst, n);
}

inline unsigned grid_for(int64_t n, int block) { return unsigned((n + block - 1) / block); }

}  // namespace

void launch_segment64(const DevParticles &p, int64_t n, const MeshDev &m, const StepConst &c, int L,
                      unsigned int *tri_count, DevCounters *ctr, const FieldArgs &f, uint32_t seq, cudaStream_t s,
                      LandRec *land, HistRec *hist, int64_t hist_n) {
    if (n <= 0 || L <= 0) return;
    Seg64 a{};
    a.m = m;
    a.p = p;
    a.n = n;
    a.tri_count = tri_count;
    a.ctr = ctr;
    a.land = land;
    a.hist = hist;
    a.hist_n = hist_n;
    a.L = L;
    a.seq = seq;
    if (L == 1 && !hist) {
        static int blocks = 0;
        constexpr size_t bytes = sizeof(StepPool) * 4;
        if (blocks == 0) blocks = resident_blocks(k_step64, 128, bytes);
        const int T = n >= int64_t(blocks) * 128 ? 128 : 32;
        const unsigned grid = unsigned(std::min<int64_t>(grid_for(n, T), int64_t(blocks) * (128 / T)));
        k_step64<<<grid, T, bytes * T / 128, s>>>(a, c, f);
        return;
    }
    // one wave: SMs x resident blocks (same on every device of this build);
    // few particles spread over smaller blocks so that every SM has some
    static int resident[2] = {0, 0};
    int &r = resident[hist ? 1 : 0];
    constexpr int kT = 128;
    constexpr size_t smem = sizeof(WarpPool) * kT / 32;
    static_assert(smem <= 48 * 1024, "a block's pools fit the default limit of dynamic shared memory");
    if (r == 0) r = hist ? resident_blocks(k_seg64<true>, kT, smem) : resident_blocks(k_seg64<false>, kT, smem);
    const int T = n >= int64_t(r) * kT ? kT : 32;
    const unsigned grid = unsigned(std::min<int64_t>(grid_for(n, T), int64_t(r) * (kT / T)));
    if (hist)
        k_seg64<true><<<grid, T, smem * T / kT, s>>>(a, c, f);
    else
        k_seg64<false><<<grid, T, smem * T / kT, s>>>(a, c, f);
}

void launch_deposit64(const DevParticles &p, int64_t n, const MeshDev &m, int k, unsigned long long *node_fix,
                      const OccList &occ, cudaStream_t s) {
    if (n <= 0) return;
    static int blocks = 0;  // one wave
    if (blocks == 0) blocks = resident_blocks(k_deposit64, kDepThreads);
    const DepSrc64 src{p, m.rec, k, 1LL << k};
    const unsigned grid = unsigned(std::min<int64_t>(grid_for(n, kDepThreads), blocks));
    k_deposit64<<<grid, kDepThreads, 0, s>>>(src, n, m.tet_nodes, node_fix, occ);
}

void launch_fix_to_charge(const unsigned long long *node_fix, double scale, double *node_q, int64_t n,
                          cudaStream_t s) {
    k_fix_to_charge<<<grid_for(n, 256), 256, 0, s>>>(node_fix, scale, node_q, n);
}

void launch_field64_full(const FieldArgs &f, int64_t n_tets, cudaStream_t s) {
    if (n_tets > 0) k_field64_full<<<grid_for(n_tets, 256), 256, 0, s>>>(f, n_tets);
}

void launch_field64_list(const FieldArgs &f, const int32_t *list, const unsigned int *list_n, cudaStream_t s) {
    k_field64_list<<<152 * 4, 256, 0, s>>>(f, list, list_n);
}

void launch_refresh64(const DevParticles &p, int64_t n, const FieldArgs &f, cudaStream_t s) {
    if (n > 0) k_refresh64<<<grid_for(n, 256), 256, 0, s>>>(p, n, f);
}

void launch_zero_field(const FieldArgs &f, int64_t n_tets, cudaStream_t s) {
    if (n_tets > 0) k_zero_field<<<grid_for(n_tets, 256), 256, 0, s>>>(f, n_tets);
}

void launch_interior_flags(TetRec *rec, const int4 *tet_nodes, const double *node_xyz, int64_t n_tets,
                           const double *lo, const double *hi, double margin, cudaStream_t s) {
    if (n_tets > 0)
        k_interior_flags<<<grid_for(n_tets, 256), 256, 0, s>>>(rec, tet_nodes, node_xyz, n_tets, lo[0] + margin,
                                                              lo[1] + margin, lo[2] + margin, hi[0] - margin,
                                                              hi[1] - margin, hi[2] - margin);
}

void launch_count_lost(const int32_t *tet, int64_t n, unsigned long long *out, cudaStream_t s) {
    if (n <= 0) return;
    k_count_lost<<<grid_for(n, 256), 256, 0, s>>>(tet, n, out);
}

void launch_locate(const double *pos, int64_t n, const MeshDev &m, const int32_t *vox_seed,
                   const double *oi, const int32_t *dims, int max_cross, int32_t *tet_out, cudaStream_t s) {
    if (n <= 0) return;
    k_locate<<<grid_for(n, 128), 128, 0, s>>>(pos, n, m, vox_seed, oi[0], oi[1], oi[2], oi[3], oi[4], oi[5],
                                               dims[0], dims[1], dims[2], max_cross, tet_out);
}

void launch_init_particles(const double *pos, const double *vel, const int32_t *tet, int64_t n, DevParticles p,
                           cudaStream_t s, int64_t id_base) {
    if (n <= 0) return;
    k_init_particles<<<grid_for(n, 256), 256, 0, s>>>(pos, vel, tet, n, p, id_base);
}

void launch_upload(const double *pos, const double *vel, int64_t n, const MeshDev &m, const int32_t *vox_seed,
                   const double *oi, const int32_t *dims, int max_cross, const DevParticles &p,
                   const DevParticles32 &q, const double *cen, unsigned long long *lost, const FieldArgs &f,
                   int64_t zero_tets, cudaStream_t s) {
    if (n <= 0) return;
    const unsigned grid = grid_for(n, 128);  // 128: staging
    const int per_block = int((zero_tets + grid - 1) / grid);
    k_upload<<<grid, 128, 0, s>>>(pos, vel, n, m, vox_seed, oi[0], oi[1], oi[2], oi[3], oi[4], oi[5], dims[0], dims[1],
                                  dims[2], max_cross, p, q, cen, lost, f, zero_tets, per_block);
}

void launch_slot_of_id(const uint32_t *idf, int64_t n, int32_t *slot, cudaStream_t s) {
    if (n > 0) k_slot_of_id<<<grid_for(n, 256), 256, 0, s>>>(idf, n, slot);
}

void launch_gather_by_id(const DevParticles &p, int64_t n, int32_t *slot, double *pos, double *vel,
                         int32_t *tet, uint32_t *flags, cudaStream_t s) {
    if (n <= 0) return;
    launch_slot_of_id(p.idf, n, slot, s);
    k_gather_by_id<<<grid_for(n, 256), 256, 0, s>>>(p, n, slot, pos, vel, tet, flags);  // 256: the staging size
}

int64_t sort_scratch_words(int64_t n_tets) {
    const int64_t len = n_tets + 1;
    const int64_t nb = (len + kScanTile - 1) / kScanTile;
    // 64-bit occupied-tet counter (2 words), counts/offsets, tile sums
    return 2 + len + nb;
}

unsigned long long *sort_occupied_counter(int32_t *scratch) {
    return reinterpret_cast<unsigned long long *>(scratch);
}

int32_t *sort_offsets(int32_t *scratch) { return scratch + 2; }

void launch_sort_prepare(const int32_t *tet, const uint32_t *idf, int64_t n, int64_t n_tets, int32_t *scratch,
                         int32_t *rank, int64_t *n_alive_dev, cudaStream_t s) {
    const int64_t len = n_tets + 1;
    const int64_t nb = (len + kScanTile - 1) / kScanTile;
    unsigned long long *occupied = sort_occupied_counter(scratch);
    int32_t *cnt = sort_offsets(scratch);
    int32_t *sums = cnt + len;
    cudaMemsetAsync(cnt, 0, sizeof(int32_t) * len, s);
    cudaMemsetAsync(occupied, 0, sizeof(unsigned long long), s);
    if (n > 0 && rank)
        k_sort_rank<<<grid_for(n, kSortBlock), kSortBlock, 0, s>>>(tet, idf, n, int(n_tets), cnt, rank);
    else if (n > 0)
        k_sort_hist<<<grid_for(n, kSortBlock), kSortBlock, 0, s>>>(tet, idf, n, int(n_tets), cnt);
    k_scan_tile<<<unsigned(nb), kScanThreads, 0, s>>>(cnt, len, int(n_tets), sums, occupied);
    k_scan_sums<<<1, 1024, 0, s>>>(sums, nb);
    k_scan_add<<<grid_for(len, 256), 256, 0, s>>>(cnt, len, sums, int(n_tets), n_alive_dev);
}

void launch_resort(const DevParticles &src, DevParticles dst, int64_t n, int64_t n_tets, int32_t *scratch,
                   int32_t *rank, void *records, int64_t *n_alive_dev, cudaStream_t s) {
    launch_sort_prepare(src.tet, src.idf, n, n_tets, scratch, records ? rank : nullptr, n_alive_dev, s);
    if (n <= 0) return;
    const unsigned grid = grid_for(n, kSortBlock);
    if (records) {
        SortRec64 *rec = static_cast<SortRec64 *>(records);
        k_sort_records<<<grid, kSortBlock, 0, s>>>(src, rec, n, int(n_tets), sort_offsets(scratch), rank);
        k_sort_unpack<<<grid, kSortBlock, 0, s>>>(rec, dst, n);
    } else {
        k_sort_scatter<<<grid, kSortBlock, 0, s>>>(src, dst, n, int(n_tets), sort_offsets(scratch));
    }
}

}  // namespace spg
