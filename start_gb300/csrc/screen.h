// FP32 screens of the FP64 step: the truncated-float view of a double, the
// per-tet record of the inside screen and the screened decision of the walk.
// Shared by the kernels, the host code that builds the records and a host-side
// check against the FP64 decisions, so all truncate with the same integer ops.
#ifndef SPG_SCREEN_H
#define SPG_SCREEN_H

#include "exact_div.h"

namespace spg {

// Float from the high word of a double (sign, exponent, top 20 mantissa
// bits), integer ops only: |f - x| <= 2^-20 |x| for 2^-126 <= |x| < 2^128;
// 0 below that range, +-inf above.
SPG_XHD inline float hi_float(double x) {
    const int hi = int(as_bits(x) >> 32);
    const int a = hi & 0x7fffffff;
    const int r = a < (897 << 20) ? 0 : (a >= (1151 << 20) ? 0x7f800000 : ((a - (896 << 20)) << 3));
    const int bits = r | (hi & int(0x80000000));
#ifdef __CUDA_ARCH__
    return __int_as_float(bits);
#else
    float f;
    std::memcpy(&f, &bits, 4);
    return f;
#endif
}

// hi_float of a tet's barycentric map (M row-major, origin x0): what the
// inside screen reads, 48 bytes instead of the 96 of the FP64 map.
struct alignas(16) TetScreen {
    float M[9];
    float x0[3];
};
static_assert(sizeof(TetScreen) == 48, "TetScreen is three 16-byte words");

// Float of the mantissa bits that hi_float(x) leaves out: x = hi_float(x) +
// lo_float(x) to 2^-44 |x|, integer ops and one 32-bit conversion (no FP64
// instruction). 0 below 2^-74, where those bits are under 2^-94, and from 2^180 on.
SPG_XHD inline float lo_float(double x) {
    const long long b = as_bits(x);
    const int hi = int(b >> 32);
    const int e = (hi >> 20) & 0x7ff;
    const uint32_t lo = uint32_t(b);
    const int bits = (e < 949 || e > 1202) ? 0 : (((e - 948) << 23) | (hi & int(0x80000000)));  // +-2^(e - 1075)
#ifdef __CUDA_ARCH__
    return __uint2float_rn(lo) * __int_as_float(bits);
#else
    float f;
    std::memcpy(&f, &bits, 4);
    return float(lo) * f;
#endif
}

// The four barycentric coordinates of a point in FP32, each with a bound of
// its distance from the exact value. M: the map truncated to 20 bits (TetScreen),
// x0 and p in full. d = p - x0 from the float pairs of both: the two
// subtractions and the sum round by at most 2^-24 of their results, the pairs
// leave out 2^-44 of |p| and |x0|, so d is within
// delta = 1.2e-7 (|hi difference| + |d|) + 1e-12 (|p| + |x0|) + 1e-27. With
// S = sum_j |M_j d_j| the truncation of M and the products put lambda_i within
// 2.2e-6 S (4e-6 S is taken), and delta adds 1.01 sum_j |M_j| delta_j;
// lambda_0 gets the three bounds and 1e-6 for its own sum.
struct Lam4 {
    float l[4], b[4];
};

SPG_XHD inline Lam4 screen_lambda(const float M[9], const double x0[3], const double p[3]) {
    float d[3], dl[3];
    for (int k = 0; k < 3; ++k) {
        const float ph = hi_float(p[k]), xh = hi_float(x0[k]);
        const float hd = ph - xh;
        d[k] = hd + (lo_float(p[k]) - lo_float(x0[k]));
        dl[k] = fmaf(1.2e-7f, fabsf(hd) + fabsf(d[k]), fmaf(1e-12f, fabsf(ph) + fabsf(xh), 1e-27f));
    }
    Lam4 o;
    float sl = 0.0f, sb = 0.0f;
    for (int r = 0; r < 3; ++r) {
        const float m0 = M[3 * r], m1 = M[3 * r + 1], m2 = M[3 * r + 2];
        const float l = fmaf(m2, d[2], fmaf(m1, d[1], m0 * d[0]));
        const float s = fmaf(fabsf(m2), fabsf(d[2]), fmaf(fabsf(m1), fabsf(d[1]), fabsf(m0) * fabsf(d[0])));
        const float q = fmaf(fabsf(m2), dl[2], fmaf(fabsf(m1), dl[1], fabsf(m0) * dl[0]));
        o.l[r + 1] = l;
        o.b[r + 1] = fmaf(4e-6f, s, fmaf(1.01f, q, 1e-30f));
        sl += l;
        sb += o.b[r + 1];
    }
    o.l[0] = 1.0f - sl;
    o.b[0] = sb + 1e-6f;
    return o;
}

// One decision of the segment walk p0 -> p1 in a tet entered through face
// `enter` (-1: the first tet): kScreenInside when no face but the entry has
// lambda(p1) < 0, else the face with lambda(p1) < 0 whose crossing parameter
// lambda(p0) / (lambda(p0) - lambda(p1)) is smallest. Decided only where the
// bounds leave no other answer; kScreenUndecided otherwise (the caller
// evaluates the FP64 expressions). A crossing parameter is compared as a
// product, with both denominators certainly positive.
constexpr int kScreenInside = 4, kScreenUndecided = -1;

SPG_XHD inline int screen_exit(const float M[9], const double x0[3], const double p0[3], const double p1[3],
                               int enter) {
    const Lam4 e = screen_lambda(M, x0, p1);
    int neg = 0;
    bool sure = true;
    for (int f = 0; f < 4; ++f) {
        const bool in = e.l[f] > e.b[f], out = e.l[f] < -e.b[f];
        if (f != enter) {
            sure = sure && (in || out);
            neg |= out ? 1 << f : 0;
        }
    }
    if (!sure) return kScreenUndecided;
    if (neg == 0) return kScreenInside;
    if ((neg & (neg - 1)) == 0) return (neg & 1) ? 0 : (neg & 2) ? 1 : (neg & 4) ? 2 : 3;
    const Lam4 s = screen_lambda(M, x0, p0);
    int best = -1;
    float lb = 0.0f, bb = 0.0f, db = 0.0f, eb = 0.0f;  // lambda(p0), its bound; denominator, its bound
    for (int f = 0; f < 4; ++f) {
        if (!(neg & (1 << f))) continue;
        const float l = s.l[f], b = s.b[f], d = l - e.l[f];
        const float ed = fmaf(1e-6f, fabsf(l) + fabsf(e.l[f]), b + e.b[f]);
        sure = sure && d > ed;
        if (best < 0) {
            best = f;
            lb = l;
            bb = b;
            db = d;
            eb = ed;
            continue;
        }
        // s_f < s_best <=> l db < lb d
        const float x = l * db, y = lb * d;
        const float err = (b * (db + eb) + fabsf(l) * eb) + (bb * (d + ed) + fabsf(lb) * ed) +
                          1e-6f * (fabsf(x) + fabsf(y)) + 1e-30f;
        if (x < y - err) {
            best = f;
            lb = l;
            bb = b;
            db = d;
            eb = ed;
        } else {
            sure = sure && x > y + err;
        }
    }
    return sure ? best : kScreenUndecided;
}

}  // namespace spg

#endif
