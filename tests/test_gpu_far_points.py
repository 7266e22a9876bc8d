"""FP64 assembly at field points up to a hundred million wavelengths away."""
from __future__ import annotations

import numpy as np
import pytest

import biegpu
import oracle
from biegpu import mesh as bm

from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [3e2, 3e3, 1e5, 1e7, 3e8])
@pytest.mark.parametrize("M", [40, 700])
@pytest.mark.parametrize("geometry", ["linear", "quadratic"])
def test_far_field_points(geometry, M, radius):
    """The oracle rounds r and k r, and the distance takes two roundings of the point:
    2^-53 k r each, a few of them beside the 1e-12 of near points."""
    k = 10.0
    t = np.random.default_rng(5).normal(size=(3, M))
    t *= radius / np.linalg.norm(t, axis=0)
    mesh = bm.icosphere(4, geometry=geometry)
    ctx = biegpu.get_context(mesh, n=2, m=2)
    F, G, _ = ctx.assemble(k, targets=t)
    want = oracle.assemble(mesh, k, targets=t, n=2, m=2)
    for a, b in ((F, want[0]), (G, want[1])):
        assert np.all(np.isfinite(a))
        assert rel_fro(a, b) <= 1e-12 + 4 * 2.0**-53 * k * radius


@pytest.mark.parametrize("radius", [3e3, 1e5, 1e6, 1e7])
@pytest.mark.parametrize("k", [10.0, 10.0 + 1e-5j])
@pytest.mark.parametrize("M", [40, 3000])
def test_far_field_points_without_ties(M, k, radius):
    """One physics node per element: the nearest node is never a tie, so such points
    stay in fixed point to 2^25 turns."""
    t = np.random.default_rng(5).normal(size=(3, M))
    t *= radius / np.linalg.norm(t, axis=0)
    mesh = bm.icosphere(4, physics="disctriconstant")
    ctx = biegpu.get_context(mesh, n=2, m=2)
    F, G, _ = ctx.assemble(k, targets=t)
    want = oracle.assemble(mesh, k, targets=t, n=2, m=2)
    for a, b in ((F, want[0]), (G, want[1])):
        assert np.all(np.isfinite(a))
        assert rel_fro(a, b) <= 1e-12 + 4 * 2.0**-53 * abs(k) * radius
