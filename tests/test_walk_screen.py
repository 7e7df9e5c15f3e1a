"""The walk's FP32-screened decisions (screen.h) against the FP64 evaluation.

A host build of the header runs 4e5 random decisions for each kind of tet and
step (sizes, distances from the origin, slivers, start points on faces and
edges, ends on vertices and beyond edges, entered tets): a decision may be left
open, never wrong, and with the tets and steps of the workloads nearly all of
the generic ones are taken.
"""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_no_decision_differs(tmp_path):
    exe = tmp_path / "walk_screen_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(exe),
                    str(HERE / "native" / "walk_screen_check.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(int(v) for v in line.split()) for line in out.splitlines()]
    assert len(rows) == 11
    assert all(wrong == 0 for _, _, wrong in rows), rows
    # of the six ways to place the segment two start on a face or an edge or end
    # on a vertex for certain, and one aims at a vertex: at least half are generic
    decided, undecided, _ = rows[0]
    assert decided >= 0.5 * (decided + undecided), rows[0]
