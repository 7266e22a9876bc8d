"""Fixed-point assembly (K10) at the edges of its ranges, against the oracle.

Tolerance 1e-12 (relative Frobenius), the bound every FP64 assembly test uses:
the fixed-point values carry 2^-54 or better, so what differs is FP64 rounding
in the oracle and in the near pairs."""
from __future__ import annotations

import dataclasses

import numpy as np
import pytest

import biegpu
import oracle
from biegpu import mesh as bm

from conftest import rel_fro

pytestmark = pytest.mark.gpu

TOL = 1e-12


def moved(mesh, scale, shift):
    s = np.asarray(shift, dtype=np.float64)[:, None]
    return dataclasses.replace(mesh, sources=mesh.sources * scale + s, coordinates=mesh.coordinates * scale + s)


def check(mesh, k, n, m, targets=None, precision="fp64"):
    ctx = biegpu.Context(mesh, n=n, m=m)
    got = ctx.assemble(k, targets=targets, precision=precision)
    want = oracle.assemble(mesh, k, targets=targets, n=n, m=m)
    for a, b in zip(got[:2], want[:2]):
        assert np.all(np.isfinite(a))
        assert rel_fro(a, b) <= TOL
    if targets is None:
        assert rel_fro(got[2], want[2]) <= TOL
    ctx.close()


@pytest.mark.parametrize("scale,shift", [(1e-9, (0, 0, 0)), (3e7, (0, 0, 0)), (1.0, (40.0, -25.0, 3.0)),
                                         (0.01, (0.0, 0.5, 0.0))])
@pytest.mark.parametrize("geometry", ["linear", "quadratic"])
def test_scaled_and_moved_meshes(geometry, scale, shift):
    mesh = moved(bm.icosphere(3, geometry=geometry), scale, shift)
    check(mesh, 2.5 / scale, 2, 2)


@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (3, 2), (5, 5)])
@pytest.mark.parametrize("k", [0.0, 3.0, -2.0, 2.0 + 1.5j, 1.0 - 0.5j])
def test_rules_and_wavenumbers(n, m, k):
    check(bm.icosphere(2, geometry="quadratic"), k, n, m)


@pytest.mark.parametrize("M", [1, 31, 129])
@pytest.mark.parametrize("radius", [1.05, 9.0, 4000.0])
def test_field_points(M, radius):
    rng = np.random.default_rng(M)
    t = rng.normal(size=(3, M))
    t *= radius / np.linalg.norm(t, axis=0)
    mesh = bm.icosphere(3)
    k = 0.3 if radius > 100 else 4.0 + 0.5j
    check(mesh, k, 2, 2, targets=t)


def test_more_fp64_pairs_than_the_list_holds():
    # targets beyond the fixed coordinates: every pair goes to FP64, 6 times more than
    # the list of deferred pairs takes
    rng = np.random.default_rng(7)
    t = rng.normal(size=(3, 150))
    t *= 3e13 / np.linalg.norm(t, axis=0)
    mesh = bm.icosphere(6)
    assert 150 * mesh.n_elements > 6 * (150 * 64 + 4096)
    check(mesh, 0.0, 2, 2, targets=t)


@pytest.mark.parametrize("level", range(8))
def test_every_slicing(level):
    mesh = bm.icosphere(4, geometry="quadratic")
    ctx = biegpu.Context(mesh, n=2, m=2)
    ctx.force_shape("df64_assembly", level)
    F, G, C = ctx.assemble(3.0, precision="df64")
    ctx.force_shape("df64_assembly", -1)
    for a, b in zip((F, G, C), oracle.assemble(mesh, 3.0, n=2, m=2)):
        assert rel_fro(a, b) <= TOL
    only = ctx.assemble(3.0, fOn=True, gOn=False, cOn=False)[0], ctx.assemble(3.0, fOn=False, gOn=True, cOn=False)[1]
    assert rel_fro(only[0], F) <= TOL and rel_fro(only[1], G) <= TOL
    ctx.close()


def test_graded_mesh():
    # element sizes over a factor of 1000 (pairs too close for the fixed range go to FP64)
    mesh = bm.icosphere(4)
    z = mesh.coordinates[2]
    s = 1e-3 + (1 - 1e-3) * ((1 + z) / 2) ** 4
    c = mesh.coordinates * s
    check(dataclasses.replace(mesh, coordinates=c, sources=c.copy()), 2.0, 2, 2)



@pytest.mark.parametrize("geo,phys", [("linear", "geometry"), ("quadratic", "geometry"),
                                      ("quadratic", "disctrilinear")])
@pytest.mark.parametrize("k", [3.0, 2.0 + 0.4j])
def test_few_rows_match_many(geo, phys, k):
    """Few targets take slices down to single elements with every node shared, many
    the flagged slices.  Every entry is a sum of the same integers, so rows agree
    but for the FP64 additions of near pairs: some 30 at 2^-53 of the entries they
    add to, below 1e-14 of the row."""
    mesh = bm.icosphere(9, geometry=geo, physics=phys)
    ctx = biegpu.get_context(mesh, n=2, m=2)
    r = np.random.default_rng(4)
    t = r.normal(size=(3, 2600))
    t *= r.uniform(1.05, 4.0, 2600) / np.linalg.norm(t, axis=0)
    F, G, _ = biegpu.assemble_parallel(mesh, k, t, n=2, m=2)
    for M in (1, 40, 129, 300, 1792):
        f, g, _ = biegpu.assemble_parallel(mesh, k, t[:, :M], n=2, m=2)
        for a, b in ((f, F[:M]), (g, G[:M])):
            assert np.max(np.abs(a - b) / np.max(np.abs(b), axis=1, keepdims=True)) <= 1e-14


@pytest.mark.parametrize("power", [1, 4, 12])
@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_graded_meshes_in_both_precisions(power, precision):
    # few, half and most of the elements small against the mesh
    mesh = bm.icosphere(6)
    s = 1e-3 + (1 - 1e-3) * ((1 + mesh.coordinates[2]) / 2) ** power
    c = mesh.coordinates * s
    check(dataclasses.replace(mesh, coordinates=c, sources=c.copy()), 2.0, 2, 2, precision=precision)
