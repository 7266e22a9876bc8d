"""Warp code of the GMRES kernels (csrc/bie_krylov.cuh) on the host, one thread per
lane: nothing may depend on lanes running in step between warp operations."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

GXX = shutil.which("g++")


@pytest.fixture(scope="module")
def rotate(tmp_path_factory):
    if GXX is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("krylov") / "krylov_rotate"
    subprocess.run([GXX, "-O1", "-std=gnu++20", "-fno-strict-aliasing", "-pthread", "-I",
                    str(ROOT / "tests" / "host_cuda"), "-I", str(PKG / "csrc"),
                    str(ROOT / "tests" / "krylov_rotate.cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("late", [0, 3, 12, 1, 8])
@pytest.mark.parametrize("rotations", [0, 1, 2, 19])
def test_rotations_with_late_lanes(rotate, late, rotations):
    """Each of up to 19 rotations rounds its sums of three products: 1e-14."""
    out = subprocess.run([rotate, str(late), str(rotations)], check=True, capture_output=True, text=True, timeout=60)
    assert float(out.stdout) <= 1e-14
