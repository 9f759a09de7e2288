"""The short reciprocal, quotient and square root of the stage kernels, and
the rule that flags a cell plain (tests/cpp/stage_math_check.cu).

Bounds, with u = 2^-53. The seeds are approximations of relative error below
2^-19. One third-order step leaves the cube of that, 2^-57, plus one rounding:
a reciprocal off by at most one representable double. The quotient's remainder
step on top of it: one. Two Newton steps leave 1.5 delta^3 < 2^-56 of the
square root's seed, plus one rounding: one. The inverse square root carries
the root's error (1.2 u), its own 2^-57 and a rounding: 2.3 u against the
exact value, so at most two from the rounded one."""
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


@pytest.mark.parametrize("name,worst", [("rcp", 1), ("div", 1), ("sqrt", 1), ("rsqrt", 2)])
def test_short_arithmetic(results, name, worst):
    count, other, far, seed = results[name]
    assert count > 2e6
    assert far <= worst
    assert seed <= -19.0


def test_plain_cells_keep_a_margin(results):
    flagged, close = results["plain"]
    assert flagged > 100 and close == 0
