"""Adjoint gradients where the arithmetic's ranges matter: admittances of very
different size in one mesh, meshes away from the origin."""
from __future__ import annotations

import numpy as np
import pytest

import biegpu
import oracle
from biegpu import mesh as bm

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


def moved(mesh, shift, scale=1.0):
    P = mesh.coordinates * scale + np.asarray(shift, dtype=np.float64)[:, None]
    return bm._finish(P, mesh.topology, "linear", "geometry")


def against_forward_mode(mesh, k, Z, X, precision, tol):
    from oracle import forward_mode as fm
    _, _, dX, dZ, info = biegpu.farfield_objective(mesh, k, Z, X, rho_c=RHO_C, precision=precision)
    assert info["forward_converged"] and info["adjoint_converged"]
    rng = np.random.default_rng(11)
    for _ in range(3):
        V = rng.normal(size=mesh.coordinates.shape)
        _, dJ = fm.farfield_directional_derivative(mesh, k, Z, X, Vdir=V, rho_c=RHO_C)
        assert abs(float(np.sum(dX * V)) - dJ) <= tol * np.linalg.norm(dX) * np.linalg.norm(V)
        dz = rng.normal(size=mesh.n_elements) + 1j * rng.normal(size=mesh.n_elements)
        _, dJz = fm.farfield_directional_derivative(mesh, k, Z, X, dZ=dz, rho_c=RHO_C)
        gz = float(np.sum(dZ.real * dz.real + dZ.imag * dz.imag))
        assert abs(gz - dJz) <= tol * np.linalg.norm(dZ) * np.linalg.norm(dz)


@pytest.mark.parametrize("shift", [(0.0, 0.0, 0.0), (300.0, -200.0, 150.0)])
@pytest.mark.parametrize("precision", ["fp64"])
def test_gradient_to_the_precision_asked_for(precision, shift):
    """Gradients against the exact derivative of the CPU restatement.  A point's
    coordinate carries 2^-53 |x| (|x| about 400 on the moved mesh: 4.4e-14), the
    nearest pairs are some 0.03 away and the derivative goes with the third power
    of the distance: 4.4e-12 at most, and 1e-12 from the solves (1e-13 each, a
    decade for the system's condition).  Double-float coordinates (2^-48) would
    be 32 times as far off."""
    mesh, Z, X = setup(3, nfield=8)
    tol = 5.4e-12 if shift[0] else 1e-12
    against_forward_mode(moved(mesh, shift), 3.0, Z, X + np.asarray(shift)[:, None], precision, tol)


@pytest.mark.parametrize("shift,scale", [((0.0, 0.0, 0.0), 1.0), ((0.0, 0.0, 0.0), 1e-3), ((0.0, 0.0, 0.0), 3e4),
                                         ((300.0, -200.0, 160.0), 1.0)])
def test_double_float_gradient_beside_fp64(shift, scale):
    """Regular pairs in 48 bits stay within 1e-13 of FP64 where the mesh is near the
    origin (1e-12 with the solves).  Moved by 400 both precisions carry the
    coordinates' 2^-53 |x| = 4.4e-14, over the nearest distance of 0.03 1.5e-12; a
    distance taken between coordinates that were rounded to float pairs (2^-48)
    would put 32 times that into the nearer pairs."""
    mesh, Z, X = setup(6, nfield=8)
    mesh = moved(mesh, shift, scale)
    X = X * scale + np.asarray(shift)[:, None]
    a, b = (biegpu.farfield_objective(mesh, 3.0 / scale, Z, X, rho_c=RHO_C, precision=p) for p in ("fp64", "df64"))
    for i in (2, 3):
        assert np.linalg.norm(b[i] - a[i]) <= (1.5e-12 if shift[0] else 1e-12) * np.linalg.norm(a[i])


@pytest.mark.parametrize("scale,radius", [(1.0, 1e10), (1e9, 1e6), (1e15, 10.0), (1e-15, 10.0)])
def test_double_float_gradient_at_the_ends_of_its_range(scale, radius):
    """Lengths and distances whose products leave FP32's range (the adjoint pressure
    falls with the field points' distance): such calls take the FP64 reverse pass."""
    mesh, Z, X = setup(5, nfield=8)
    mesh = moved(mesh, (0.0, 0.0, 0.0), scale)
    k = (3.0 if radius == 10.0 else 1e-3) / scale
    X = X * (radius / 10.0 * scale)
    a, b = (biegpu.farfield_objective(mesh, k, Z, X, rho_c=RHO_C, precision=p) for p in ("fp64", "df64"))
    for i in (2, 3):
        size = np.max(np.abs(a[i]))
        assert np.linalg.norm((b[i] - a[i]) / size) <= 1e-12 * np.linalg.norm(a[i] / size)


@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_few_and_many_field_points(precision):
    """Few field points take slices down to single elements with every node shared,
    many the flagged slices; with admittances over six decades both sum the same
    integers, so the pressures agree to the FP64 additions (1e-13 of the largest)."""
    mesh, Z, X = setup(9, nfield=2000)
    Z = Z * 10.0 ** np.random.default_rng(8).uniform(-3, 3, mesh.n_elements)
    many = biegpu.farfield_objective(mesh, 3.0, Z, X, rho_c=RHO_C, precision=precision, gradient=False)[1]
    for M in (1, 8, 200):
        few = biegpu.farfield_objective(mesh, 3.0, Z, X[:, :M], rho_c=RHO_C, precision=precision, gradient=False)[1]
        assert np.max(np.abs(few - many[:M])) <= 1e-13 * np.max(np.abs(many))
