"""The fixed-point quadrature points of the FP64-grade assembly on the host: the
functions the kernel calls (csrc/bie_fix64.cuh), compiled with g++ and compared
with long double over random regular pairs (the complex-wavenumber damping is
covered by tests/test_gpu_fix64.py)."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

GXX = shutil.which("g++")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if GXX is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("fix64") / "fix64_points"
    subprocess.run([GXX, "-O2", "-std=gnu++17", "-I", str(PKG / "csrc"), str(ROOT / "tests" / "fix64_points.cpp"),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("seed", [1, 2])
def test_points_against_long_double(driver, seed):
    out = subprocess.run([driver, str(seed)], check=True, capture_output=True, text=True).stdout.split()
    assert out[0] == "1"            # every table index inside its table
    assert float(out[1]) <= 1.0     # largest error as a multiple of its bound


@pytest.mark.parametrize("seed", [1, 2])
def test_functions_against_long_double(tmp_path, seed):
    """Roots: their fixed-point value is good to 2^-59, so 0.52 units after
    rounding; the exponential adds 2^-56 of its series and 2^-63 |x| of log2(e)
    (|x| below 700): 0.9; sine and cosine 2^-59 + 2^-61 |x| besides the rounding."""
    if GXX is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "fix64_math"
    subprocess.run([GXX, "-O2", "-std=gnu++17", "-I", str(PKG / "csrc"), str(ROOT / "tests" / "fix64_math.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(seed)], check=True, capture_output=True, text=True).stdout.split()
    assert float(out[0]) <= 0.52 and float(out[1]) <= 0.52
    assert float(out[2]) <= 0.9
    assert float(out[3]) <= 1.0
    assert out[4] == "1"


@pytest.mark.parametrize("seed", [1, 2])
def test_division_and_roots_are_ieee(tmp_path, seed):
    if GXX is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "fix64_divide"
    subprocess.run([GXX, "-O2", "-std=gnu++17", "-ffp-contract=off", "-I", str(PKG / "csrc"),
                    str(ROOT / "tests" / "fix64_divide.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), str(seed)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0", "0", "1"]
