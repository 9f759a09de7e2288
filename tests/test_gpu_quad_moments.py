"""The moments of a quad mesh's cells, from which its smoothness indicators are
formed (tests/cpp/quad_moments_check.cu). Bound: a coordinate in the cell's
frame carries the rounding of the centre and the corner, 2^-53 / h each, and a
moment sums products of at most four such coordinates of order one over its
points: 64 such roundings."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_moments_equal_extended_precision(cuda_lib, tmp_path):
    from mantlepar_b200 import build as B
    exe, obj = str(tmp_path / "moments"), str(tmp_path / "tables.o")
    subprocess.run([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "--fmad=false", "-c",
                    os.path.join(B.CSRC, "quad_table_kernels.cu"), "-o", obj], check=True)
    subprocess.run([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "-I", B.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "quad_moments_check.cu"), os.path.join(B.CSRC, "quad_tables.cpp"),
                    obj, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert float(r.stdout) <= 64.0
