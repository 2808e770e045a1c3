"""The importon histogram's octant rule (octant_of) against the angle it stands
for, compiled for the host."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_octant_by_comparison_equals_the_arc_tangent(tmp_path):
    exe = str(tmp_path / "octant_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "octant_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
