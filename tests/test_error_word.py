"""An error that a guide's kernels report is not left for the next call."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_error_word_is_cleared_by_its_own_call(tmp_path):
    exe = str(tmp_path / "error_word_check")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", "error_word_check.cpp"), "-o", exe],
                   check=True)
    assert subprocess.run([exe]).returncode == 0


def test_every_guide_call_holds_the_error_word():
    """Each entry point that checks the word took hold of it before its first launch."""
    src = open(os.path.join(ROOT, "xyz_b200", "csrc", "guide.cu")).read()
    checks = src.count("return check_err(word,")
    assert checks == 4
    for part in src.split("return check_err(word,")[:-1]:
        body = part[part.rindex("extern \"C\"") if "extern \"C\"" in part else 0:]
        last = body[body.rindex("\nint xyzgpu_"):]
        assert last.index("error_word(g, st)") < min(last.index(k) for k in ("_launch(", "render_launch(") if k in last)
