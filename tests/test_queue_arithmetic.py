"""Queues of up to 2^31 - 1 rays: launch sizes and the end of the queue."""

import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sizes_up_to_the_largest_int(tmp_path):
    exe = str(tmp_path / "queue_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "queue_check.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_traces_use_them():
    """No sum of a ray count and a group size (it overflows) in the traces."""
    for f in ("trace.cu", "traverse.cuh"):
        src = open(os.path.join(ROOT, "xyz_b200", "csrc", f)).read()
        assert not re.search(r"\(n \+ \w+ - 1\) /", src), f
