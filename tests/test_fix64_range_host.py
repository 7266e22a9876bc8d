"""Index arithmetic and scales of the fixed-point assembly on the host: the
functions of csrc/bie_fix64.cuh at sizes and values no quick GPU test reaches."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

GXX = shutil.which("g++")


@pytest.fixture(scope="module")
def build(tmp_path_factory):
    if GXX is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("fix64_range")

    def make(name):
        exe = out / name
        subprocess.run([GXX, "-O2", "-std=gnu++17", "-I", str(PKG / "csrc"), str(ROOT / "tests" / f"{name}.cpp"),
                        "-o", str(exe)], check=True)

        def run(*args):
            return subprocess.run([str(exe), *map(str, args)], check=True, capture_output=True, text=True).stdout.split()
        return run
    return make


@pytest.mark.parametrize("capacity,percent", [(0, 100), (7, 100), (500, 100), (500, 30), (100000, 100), (100000, 5)])
def test_deferred_pairs_are_counted_once_per_row_and_slice(build, capacity, percent):
    """Every deferred pair is integrated once, and the counter of list places stays
    within the list's length and one per (row, slice) however many there are."""
    out = build("fix64_defer")(1, 40, 5, 60, capacity, percent)
    assert out[0] == "1" and out[1] == "1"


def test_columns_of_many_rows(build):
    # 2^28 rows and more: a column is 4 GB
    assert build("fix64_columns")() == ["1"]


@pytest.mark.parametrize("seed", [1, 2])
def test_element_factors_of_any_magnitude(build, seed):
    """Value times factor, in the value's unit (2^-59 of its range): the final
    shift rounds to half a unit, the two products of low limbs that are left out
    are below 2^62 2^-62 = 1 each, and the factor's own rounding 2^-62 of a
    component counts an eighth: 2.7 units.  The factor's exponent is its own, so
    this holds whatever other elements carry."""
    out = build("fix64_factor")(seed)
    assert float(out[0]) <= 2.7 and out[1] == "1"


@pytest.mark.parametrize("exponent", [-6, -3, 0, 3, 6, 8, 9, 12, 15, 17, 19, 24, 31, 40, 48])
def test_sine_and_cosine_over_their_range(build, exponent):
    """Besides the final rounding 2^-59 for every argument that is taken: the series
    2^-60, the truncated turn 2 pi 2^-64, and below 2^9 1 / 2 pi in one word
    (2^-69.4 |x|)."""
    assert float(build("fix64_sine")(1, exponent)[0]) <= 1.0


@pytest.mark.parametrize("exponent", [-1022, -300, -60, -31, -30, -29, -20, -15, -12, -10, -9])
def test_sine_of_small_arguments(build, exponent):
    """Below 2^-8 the sine is relative to its argument: half a unit of rounding, and
    2^-58 of the value from x^2 (Q72), the two series terms (the next one is
    x^6 / 5040 < 2^-60) and the product: 0.52 units."""
    out = build("fix64_sine")(1, exponent)
    assert float(out[0]) <= 1.0 and float(out[1]) <= 0.52


@pytest.mark.parametrize("cplx", [0, 1])
@pytest.mark.parametrize("turns", [-8, 0, 9, 15, 25])
def test_points_of_many_turns_and_complex_wavenumbers(build, turns, cplx):
    """As the real points of few turns: 2^-50 for the roundings and 2^-53 of the phase
    (r to 2^-55, the turn's fraction with 58 + 32 bits), and for complex k 2^-53 of
    the damping's exponent, relative to the element's near end."""
    out = build("fix64_complex")(1, turns, cplx)
    assert out[0] == "1" and float(out[1]) <= 1.0
