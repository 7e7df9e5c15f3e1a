// FP64 quotients by Newton's iteration, for code in which a division stands on
// the critical path (1,470 cycles on GB300, an FP64 fused multiply-add 63).
//
// The reciprocal is one Newton-Raphson step y' = y + y (1 - b y), which squares the
// relative error, from an FP32 reciprocal of b's leading 24 bits: 2^-23 from
// leaving out the other bits and 2^-24 from rounding it make 1.8e-7, then 3.3e-14.
// The quotient is corrected once by its remainder with a fused multiply-add, q' =
// q + y (a - b q) (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), which squares the error
// again, to 1.1e-27: before its rounding q' is within 2^-36 ulp of a/b, so it is
// the rounded quotient or, next to a midpoint between two doubles, its neighbour.
// Nothing overflows or leaves the normal range for operands between 2^-423 and 2^424;
// others take the division. The same bits on the host, where they are checked
// against the division.
#ifndef SPG_NEWTON_DIV_H
#define SPG_NEWTON_DIV_H

#include "exact_div.h"

namespace spg {

SPG_XHD inline bool newton_range(double a) {
    const int e = int((as_bits(a) >> 52) & 0x7ff);
    return e >= 600 && e <= 1446;
}

// 1 / b to 3.3e-14 for newton_range(b); any number otherwise.
SPG_XHD inline double newton_reciprocal(double b) {
    const long long bb = as_bits(b);
    const int e = int((bb >> 52) & 0x7ff);
    // m in [1, 2): b's leading 24 bits, without an FP64 conversion; r in (1/2, 1]
    const int mb = 0x3f800000 | int((bb >> 29) & 0x7fffff);
#ifdef __CUDA_ARCH__
    const int rb = __float_as_int(1.0f / __int_as_float(mb));
#else
    float m;
    std::memcpy(&m, &mb, 4);
    const float r = 1.0f / m;
    int rb;
    std::memcpy(&rb, &r, 4);
#endif
    // r 2^(1023 - e) with b's sign, from the exponents
    const long long eb = (rb >> 23) - 127 + 2046 - e;
    const double y = from_bits((bb & (-0x7fffffffffffffffLL - 1)) | (eb << 52) | ((long long)(rb & 0x7fffff) << 29));
    return std::fma(y, std::fma(-b, y, 1.0), y);
}

// a / b with y = newton_reciprocal(b), for newton_range(a) and newton_range(b).
SPG_XHD inline double newton_quotient(double a, double b, double y) {
    const double q = a * y;
    return std::fma(std::fma(-b, q, a), y, q);
}

}  // namespace spg

#endif
