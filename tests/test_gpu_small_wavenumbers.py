"""Imaginary parts at small wavenumbers.  With k r small e^{ikr} is nearly real: the
imaginary part of G is about k times its real part, that of F about k^3, and each is
a result of its own (it carries the radiated power).  FP64 calls keep each part to
FP64, not only the modulus."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest
import torch

import biegpu
import oracle
from biegpu import mesh as bm

from conftest import rel_fro

pytestmark = pytest.mark.gpu


def check_parts(F, G, wantF, wantG, k):
    """G: sin(k r) to a few units, summed over some ten points: 1e-14.  F: the
    difference k r cos(k r) - sin(k r) of terms that round at 2^-53 k r (r at most 2
    here), a few dozen points of either sign: 2^-48 k of the modulus."""
    assert rel_fro(G.imag, wantG.imag) <= 1e-14
    assert np.linalg.norm(F.imag - wantF.imag) <= 2.0**-48 * k * np.linalg.norm(wantF.real)
    assert rel_fro(F, wantF) <= 1e-12 and rel_fro(G, wantG) <= 1e-12


@pytest.mark.parametrize("k", [1e-8, 1e-5, 1e-2, 0.3])
def test_near_field(k):
    mesh = bm.icosphere(3, geometry="quadratic")
    F, G = biegpu.assemble_parallel(mesh, k, sparse=True, depth=1, offset=0.2)
    o = oracle.nearfield(mesh, k, depth=1, offset=0.2)
    check_parts(F.data, G.data, *o[2:4], k)


@pytest.mark.parametrize("geometry", ["linear", "quadratic"])
@pytest.mark.parametrize("k", [1e-8, 1e-5, 1e-2, 0.3])
def test_matrix_free_product(geometry, k):
    mesh = bm.icosphere(4, geometry=geometry)
    want = oracle.assemble(mesh, k, n=2, m=2)
    x = np.random.default_rng(2).uniform(0.5, 1.5, mesh.n_sources).astype(np.complex128)
    F, G = ((op(mesh, k, n=2, m=2, precision="fp64") @ torch.from_numpy(x).cuda()).cpu().numpy()
            for op in (biegpu.GPUFOperator, biegpu.GPUGOperator))
    check_parts(F, G, want[0] @ x, want[1] @ x, k)


@pytest.mark.parametrize("geometry", ["linear", "quadratic"])
@pytest.mark.parametrize("targets", [0, 40])
@pytest.mark.parametrize("k", [0.0, 1e-8, 1e-5, 1e-2, 0.3])
def test_assembly(geometry, targets, k):
    mesh = bm.icosphere(4, geometry=geometry)
    t = None
    if targets:
        t = np.random.default_rng(3).normal(size=(3, targets))
        t *= 1.8 / np.linalg.norm(t, axis=0)
    ctx = biegpu.get_context(mesh, n=2, m=2)
    F, G, _ = ctx.assemble(k, targets=t)
    want = oracle.assemble(mesh, k, targets=t, n=2, m=2)
    if k == 0.0:
        assert not np.any(F.imag) and not np.any(G.imag)
        assert rel_fro(F, want[0]) <= 1e-12 and rel_fro(G, want[1]) <= 1e-12
    else:
        check_parts(F, G, want[0], want[1], k)


def test_sweep_over_both_kernels():
    """A sweep whose wavenumbers lie on both sides of the line records the FP64 kernel;
    solutions as with one wavenumber at a time."""
    mesh = bm.icosphere(5)
    ks = np.array([1e-3, 0.2, 0.8, 2.0, 3.0])
    w = np.random.default_rng(4).normal(size=mesh.n_sources) + 0j
    p, _ = biegpu.sweep([mesh], ks, [w], precision="fp64", n=2, m=2)
    for j, k in enumerate(ks):
        q, _ = biegpu.sweep([mesh], ks[j:j + 1], [w], precision="fp64", n=2, m=2)
        a, b = np.asarray(p[0])[:, j], np.asarray(q[0])[:, 0]
        assert np.linalg.norm(a - b) <= 1e-7 * np.linalg.norm(b)


@pytest.mark.parametrize("order", [[0, 1, 2, 3, 4, 5], [5, 4, 3, 2, 1, 0], [3, 0, 4, 1, 5, 2]])
@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_sweep_in_any_order(order, precision):
    """Wavenumbers on both sides of the line, in three orders, on two meshes of which
    the smaller one puts the line elsewhere."""
    small = bm.icosphere(4)
    meshes = [bm.icosphere(5), dataclasses.replace(small, sources=0.2 * small.sources, coordinates=0.2 * small.coordinates)]
    ks = np.array([0.1, 0.3, 0.6, 1.5, 2.5, 3.5])
    rng = np.random.default_rng(4)
    w = [rng.normal(size=m.n_sources) + 0j for m in meshes]
    p, _ = biegpu.sweep(meshes, ks[order], w, precision=precision, n=2, m=2)
    for i, mesh in enumerate(meshes):
        for j, k in enumerate(ks[order]):
            q, _ = biegpu.sweep([mesh], [k], [w[i]], precision=precision, n=2, m=2)
            a, b = np.asarray(p[i])[:, j], np.asarray(q[0])[:, 0]
            assert np.linalg.norm(a - b) <= 1e-7 * np.linalg.norm(b)
