"""newton_reciprocal and newton_quotient (newton_div.h) against the division.

IEEE operations alone, so the host's bits are the device's. Bounds as derived
in the header: the reciprocal within 2 ulp, the quotient the rounded one or its
neighbour, with the neighbour only next to midpoints (the operands here are made
to sit there, a third of them; 1 in 100 is far above what they can give).
"""
import subprocess

from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_quotients_over_the_accepted_range(tmp_path):
    exe = tmp_path / "nd"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'start_gb300' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "newton_div_check.cpp")], check=True)
    out = subprocess.run([str(exe), "4000000"], check=True, capture_output=True, text=True).stdout.split()
    tested, worst_r, worst_q, off, wrong_range = int(out[0]), int(out[1]), int(out[2]), float(out[3]), int(out[4])
    assert tested >= 4_000_000 and wrong_range == 0
    assert worst_r <= 2 and worst_q <= 1 and off < 0.01
