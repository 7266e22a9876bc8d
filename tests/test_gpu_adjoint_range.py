"""Adjoint gradients where the arithmetic's ranges matter: admittances of very
different size in one mesh."""
from __future__ import annotations

import numpy as np
import pytest

import biegpu
import oracle

from test_gpu_adjoint import RHO_C, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "df64"])
@pytest.mark.parametrize("ratio", [1e3, 1e6, 1e10])
def test_soft_patch_beside_hard_elements(ratio, precision):
    """A patch of small impedance makes rho c k |Y| of its elements large beside
    the double layer, so every other element's factor has to keep its own bits.
    The solve stops at a relative residual of 1e-13; a decade for the system's
    condition: 1e-12."""
    mesh, Z, X = setup(3, nfield=8)
    Z[:mesh.n_elements // 20] /= ratio
    _, pf, _, _, info = biegpu.farfield_objective(mesh, 3.0, Z, X, rho_c=RHO_C, precision=precision)
    _, want = oracle.farfield_objective(mesh, 3.0, Z, X, rho_c=RHO_C)
    assert info["forward_converged"]
    assert np.linalg.norm(pf - want) <= 1e-12 * np.linalg.norm(want)
