"""The statistics' lines per block against an SM's shared memory, on the CPU
(tests/native/spline_check.cpp)."""

import os
import subprocess

from conftest import PKG, ROOT


def test_two_blocks_of_spline_lines_fit_an_sm(tmp_path):
    exe = str(tmp_path / "spline_check")
    subprocess.run(["g++", "-O1", "-std=c++17", f"-I{PKG}/csrc", os.path.join(ROOT, "tests", "native", "spline_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
