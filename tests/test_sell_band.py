"""Banded SELL-32 slices (sell_build.h) against the CSR rows they stand for.

A host build checks lattices of 7 and 15 couplings per node (with exact zeros
and identity rows, one to 6,000 nodes, lines shorter and longer than a slice)
in line, reversed and random node order: every row read through the plain
columns and through the band references holds the row's entries, and every
column of every lane, padding included, lies inside the matrix.
"""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_banded_slices_hold_their_rows(tmp_path):
    exe = tmp_path / "sell_band_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), str(HERE / "native" / "sell_band_check.cpp"),
                    str(HERE.parent / "start_gb300" / "csrc" / "sell_build.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(int(v) for v in line.split()) for line in out.splitlines()]
    assert len(rows) == 48
    assert all(wrong == 0 for _, _, wrong in rows), rows
    # the 101-node lines in their own order: most slices band
    slices, banded, _ = rows[30]
    assert slices == 111 and banded > slices // 2, rows[30]
