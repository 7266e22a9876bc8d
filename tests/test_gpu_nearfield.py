"""GPU near-field (sparse) assembly against the oracle restatement of
sparse_assemble_parallel! and partial_assemble_parallel!; FP64, relative
2-norm error of the CSR values <= 1e-12."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import biegpu
import oracle
from biegpu import mesh as bm
from biegpu.assembly import nearfield_values

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("geo,phys,f", [("linear", "geometry", 4), ("quadratic", "geometry", 3),
                                        ("quadratic", "linear", 3)])
@pytest.mark.parametrize("depth", [1, 2])
def test_nearfield_accurate(geo, phys, f, depth):
    mesh = bm.icosphere(f, geometry=geo, physics=phys)
    ctx = biegpu.get_context(mesh)
    k = 2.0 + 0.1j if depth == 2 else 3.0
    rp, cols, F, G = nearfield_values(ctx, k, depth=depth)
    rpo, colso, Fo, Go = oracle.nearfield(mesh, k, depth=depth)
    assert np.array_equal(rp, rpo) and np.array_equal(cols, colso)
    assert rel(F, Fo) <= 1e-12 and rel(G, Go) <= 1e-12


@pytest.mark.parametrize("offset", [0.2])
def test_nearfield_offset_and_coarse(offset):
    mesh = bm.icosphere(4)
    ctx = biegpu.get_context(mesh)
    _, _, F, G = nearfield_values(ctx, 1.5, offset=offset)
    _, _, Fo, Go = oracle.nearfield(mesh, 1.5, offset=offset)
    assert rel(F, Fo) <= 1e-12 and rel(G, Go) <= 1e-12
    _, _, F, G = nearfield_values(ctx, 1.5, coarse=True, n_gauss=3)
    _, _, Fo, Go = oracle.nearfield(mesh, 1.5, coarse=True, n_gauss=3)
    assert rel(F, Fo) <= 1e-12 and rel(G, Go) <= 1e-12


def test_sparse_assemble_parallel_api():
    mesh = bm.icosphere(3, geometry="quadratic")
    # the dispatcher's default depth is 2 (src/3d/assembly_collocation.jl:259-260)
    F, G = biegpu.assemble_parallel(mesh, 2.0, mesh.sources, sparse=True)
    assert F.shape == (mesh.n_sources, mesh.n_sources)
    rp, cols, Fo, Go = oracle.nearfield(mesh, 2.0, depth=2)
    assert rel(F.data, Fo) <= 1e-12
    # the diagonal (self) entries of G are the largest single-layer values
    assert np.all(np.abs(G.diagonal()) > 0)


def test_nearfield_flat_six_node_elements():
    """Flat 6-node elements: F of connected pairs is the rounding of n . (x - t), so
    it agrees with the oracle only if interpolation, cross product, hypot and
    divisions round as there."""
    mesh = bm.icosphere(3, geometry="quadratic")
    X = np.array(mesh.coordinates)
    T = np.asarray(mesh.topology) - np.min(mesh.topology)
    T = T if T.shape[0] == 6 else T.T
    for m, (a, b) in zip((3, 4, 5), ((0, 1), (1, 2), (2, 0))):
        X[:, T[m]] = 0.5 * (X[:, T[a]] + X[:, T[b]])
    mesh = dataclasses.replace(mesh, coordinates=X, sources=X.copy())
    ctx = biegpu.get_context(mesh)
    _, _, F, G = nearfield_values(ctx, 2.0, depth=1)
    _, _, Fo, Go = oracle.nearfield(mesh, 2.0, depth=1)
    assert rel(F, Fo) <= 1e-12 and rel(G, Go) <= 1e-12
