"""The FP64 path's reciprocal and reciprocal square root against the exact
values (tests/native/recip_check.cu)."""

import os
import subprocess

import pytest

from conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_reciprocals_within_one_unit_in_the_last_place(tmp_path):
    """One hardware approximation and one third-order step each.  Bounds: the
    step leaves e^3 of the approximation's error e (below 2^-19) and rounds once,
    half a unit; the reciprocal square root's e carries the rounding of x y, at
    most another half unit."""
    exe = str(tmp_path / "recip_check")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-fmad=false", "-gencode", "arch=compute_100a,code=sm_100a",
                    f"-I{PKG}/csrc", os.path.join(ROOT, "tests", "native", "recip_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
