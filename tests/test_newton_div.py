"""newton_reciprocal and newton_quotient (newton_div.h) against the division.

IEEE operations alone, so the host's bits are the device's. Bounds as derived
in the header: the reciprocal to 3.3e-14, the quotient the rounded one or its
neighbour, and the neighbour only where a / b lies within 2^-36 ulp of the
midpoint between the two (many of the operands are made to sit there).
"""
import subprocess

from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_quotients_over_the_accepted_range(tmp_path):
    exe = tmp_path / "nd"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'start_gb300' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "newton_div_check.cpp")], check=True)
    out = subprocess.run([str(exe), "4000000"], check=True, capture_output=True, text=True).stdout.split()
    tested, worst_r, worst_q, from_mid, wrong_range = int(out[0]), float(out[1]), int(out[2]), float(out[3]), int(out[4])
    assert tested >= 4_000_000 and wrong_range == 0
    assert worst_r <= 3.3e-14 and worst_q <= 1 and from_mid <= 2.0**-36
