// Checks newton_reciprocal and newton_quotient (start_gb300/csrc/newton_div.h)
// against the division: random operands of both signs over the whole accepted
// range, quotients next to midpoints between doubles, powers of two and their
// neighbours, both ends of the range, and values that must be turned away.
// Prints the largest relative error of the reciprocal, the largest difference of
// the quotient in ulp, and of those that are not the rounded quotient the largest
// distance, in ulp, of a / b from the midpoint between the two.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include <limits>
#include <random>

#include "newton_div.h"

using spg::as_bits;

static long long ulps(double a, double b) {
    const long long d = as_bits(a) - as_bits(b);
    return d < 0 ? -d : d;
}

int main(int argc, char **argv) {
    const long long n = argc > 1 ? std::atoll(argv[1]) : 4000000;
    std::mt19937_64 g(2025);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    const double lo = std::ldexp(1.0, -423), hi = std::nextafter(std::ldexp(1.0, 424), 0.0);
    double worst_r = 0.0;
    double from_mid = 0.0;
    long long worst_q = 0, tested = 0, wrong_range = 0;
    auto check = [&](double a, double b) {
        const double y = spg::newton_reciprocal(b), q = spg::newton_quotient(a, b, y);
        const double dr = std::fabs(std::fma(-b, y, 1.0));
        const long long dq = ulps(q, a / b);
        worst_r = dr > worst_r ? dr : worst_r;
        worst_q = dq > worst_q ? dq : worst_q;
        if (dq == 1) {
            // a/b lies next to the midpoint of q and c: the nearer to zero plus half an ulp.
            // The remainder and its difference from b ulp / 2 are exact.
            const double c = a / b, lo2 = std::fabs(q) < std::fabs(c) ? q : c;
            const double ulp = (std::fabs(q) < std::fabs(c) ? c : q) - lo2;
            const double d = std::fabs((std::fma(-b, lo2, a) - 0.5 * ulp * b) / (ulp * b));
            from_mid = d > from_mid ? d : from_mid;
        }
        ++tested;
        wrong_range += !spg::newton_range(a) || !spg::newton_range(b);
    };
    auto draw = [&] {
        double v = 1.0 + u(g);
        if (u(g) < 0.2) v = 1.0 + std::ldexp(double(int(u(g) * 5.0)), -52);          // just above a power of two
        if (u(g) < 0.2) v = 2.0 - std::ldexp(1.0 + double(int(u(g) * 4.0)), -52);  // just below
        v = std::ldexp(v, int(u(g) * 847.0) - 423);
        v = v > hi ? hi : v;
        return u(g) < 0.5 ? -v : v;
    };
    for (long long i = 0; i < n; ++i) {
        const double b = draw();
        double a = draw();
        if (i % 3 == 0) {  // a quotient next to a midpoint
            const double q = std::ldexp(1.0 + u(g), int(u(g) * 60.0) - 30);
            a = (q + 0.5 * (std::nextafter(q, 2.0 * q) - q)) * b;
            if (!spg::newton_range(a)) a = b;
        }
        check(a, b);
    }
    for (double a : {lo, hi, 1.0, -lo, -hi, std::nextafter(lo, hi), std::nextafter(hi, 0.0)})
        for (double b : {lo, hi, 1.0, -lo, -hi, std::nextafter(lo, hi), std::nextafter(hi, 0.0)}) check(a, b);
    const double inf = std::numeric_limits<double>::infinity();
    for (double v : {0.0, -0.0, inf, -inf, std::numeric_limits<double>::quiet_NaN(), std::nextafter(lo, 0.0),
                     std::nextafter(hi, inf), 5e-324, 2.2e-308, 1.7e308, -1.7e308})
        wrong_range += spg::newton_range(v);
    std::printf("%lld %.3e %lld %.3e %lld\n", tested, worst_r, worst_q, from_mid, wrong_range);
    return 0;
}
