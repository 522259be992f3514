"""The reciprocals and roots of the cell kernels (rds_math.cuh) on a million numbers, in a program
that fails when its kernel did not run and counts the numbers it evaluated."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_reciprocals_and_roots(tmp_path):
    """rcp_fast within 1 unit in the last place (its last operation's rounding), rsqrt_fast within 2
    of the library's, itself off by one; the FP32 root correctly rounded. The FP64 root x y, with y
    off by up to 1.5 2^-52 relative, by that and 2^-53 of its own: 4 units of at least 2^-53. Its
    inverse y differs from the reciprocal of the rounded root by 2 1.5 2^-52 + 2^-52: 8 units."""
    exe = tmp_path / "roots_test"
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I" + os.path.join(ROOT, "pdekit_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "roots_test.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    points, rcp, rsqrt, root32, root64, inverse = map(int, out.split())
    assert points == 4096 * 256
    assert rcp <= 1 and rsqrt <= 2
    assert root32 == 0
    assert root64 <= 4 and inverse <= 8
