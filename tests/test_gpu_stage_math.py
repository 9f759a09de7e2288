"""The rule that flags a cell plain (tests/cpp/stage_math_check.cu)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def results(tmp_path_factory):
    from mantlepar_b200 import build as B
    exe = str(tmp_path_factory.mktemp("math") / "stage_math_check")
    subprocess.run([B.nvcc()] + B.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I", B.CSRC, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "stage_math_check.cu"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return {line.split()[0]: [float(v) for v in line.split()[1:]] for line in r.stdout.splitlines()}


def test_plain_cells_keep_a_margin(results):
    flagged, close = results["plain"]
    assert flagged > 100 and close == 0
