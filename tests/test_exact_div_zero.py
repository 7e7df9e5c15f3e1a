"""div_by_known of a zero (exact_div.h): the bits of the division, for divisors of both
signs, at the ends of the normal range, subnormal, zero, infinite and NaN."""
import subprocess

from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

SRC = r"""
#include <cstdio>
#include <initializer_list>
#include <limits>
#include "exact_div.h"
int main() {
    const double inf = std::numeric_limits<double>::infinity();
    const double ms[] = {1.0, 7.95e-26, -3.0, 1e300, -1e-300, 2.2250738585072014e-308, 1.7976931348623157e308,
                         5e-324, -1e-310, 0.0, inf, -inf, std::numeric_limits<double>::quiet_NaN()};
    int wrong = 0;
    for (double m : ms)
        for (double x : {0.0, -0.0}) {
            const double a = spg::div_by_known(x, m, 1.0 / m), b = x / m;
            wrong += !(spg::as_bits(a) == spg::as_bits(b) || (a != a && b != b));
        }
    std::printf("%d\n", wrong);
}
"""


def test_zero_over_every_kind_of_divisor(tmp_path):
    src, exe = tmp_path / "z.cpp", tmp_path / "z"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'start_gb300' / 'csrc'}", "-o", str(exe),
                    str(src)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"
