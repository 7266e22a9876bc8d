"""The work a user of this framework has it do, as cases that can be timed and compared.

A case names an entry point ("kind"), the mesh and the options; sizes come
from the repository's own configurations, tests and benchmark (geodesic spheres
and 3:2:1 ellipsoids with 3- and 6-node triangles, 162 to 40962 nodes).  Every
preparation turns the mesh by a random rotation and draws the wavenumber and
the data, so inputs of another seed are another problem of the same size.

``exact`` restates the collocation integrals with plain torch in 64 bits.
"""
from __future__ import annotations

import dataclasses
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
for _p in (str(ROOT / "boundaryintegralequations.jl_gb300"), str(ROOT)):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import biegpu  # noqa: E402
from biegpu import mesh as bm  # noqa: E402

DEVICE = "cuda:0"
RHO_C = 1.21 * 343.0


def listed():
    return [
        # a small first study with the defaults of assemble_parallel (n = m = 4, FP64):
        # latency and launches
        {"name": "assemble_fp64_small", "kind": "assemble", "f": 6, "geometry": "linear", "physics": "geometry",
         "precision": "fp64", "n": 4, "m": 4, "targets": 0, "complex_k": False},
        # pulsating sphere, plain FP64, 4-point rules, 20480 linear triangles
        {"name": "assemble_fp64_pulsating", "kind": "assemble", "f": 32, "geometry": "linear", "physics": "geometry",
         "precision": "fp64", "n": 2, "m": 2, "targets": 0, "complex_k": False},
        # rigid sphere, 6-node triangles, mixed precision: the headline assembly
        {"name": "assemble_mixed_rigid_p2", "kind": "assemble", "f": 17, "geometry": "quadratic",
         "physics": "geometry", "precision": "mixed", "n": 2, "m": 2, "targets": 0, "complex_k": False},
        # the same kind of mesh at FP64 grade with double-float arithmetic
        {"name": "assemble_df64_p2", "kind": "assemble", "f": 12, "geometry": "quadratic", "physics": "geometry",
         "precision": "df64", "n": 2, "m": 2, "targets": 0, "complex_k": False},
        # F and G at field points (a ragged number of them) for a complex wavenumber,
        # discontinuous quadratic physics
        {"name": "field_points_fp64", "kind": "assemble", "f": 8, "geometry": "quadratic",
         "physics": "disctriquadratic", "precision": "fp64", "n": 3, "m": 3, "targets": 1333, "complex_k": True},
        # one matrix-free product of GMRES on the 40962-node sphere
        {"name": "product_mixed_p2", "kind": "product", "f": 32, "geometry": "quadratic", "physics": "geometry",
         "precision": "mixed", "which": "F", "n": 2, "m": 2, "targets": 0, "complex_k": False},
        # products with a block of right-hand sides on the tensor cores
        {"name": "products_multi_rhs", "kind": "multi", "f": 16, "geometry": "quadratic", "physics": "geometry",
         "precision": "fp16_split", "which": "G", "n": 2, "m": 2, "rhs": 96, "complex_k": False},
        # frequency sweep of the 2562-node sphere, assembly and solve of every wavenumber
        {"name": "sweep_mixed", "kind": "sweep", "f": 16, "geometry": "linear", "physics": "geometry",
         "precision": "mixed", "n": 2, "m": 2, "nk": 8},
        # GMRES on an assembled dense system, default precision
        {"name": "gmres_dense", "kind": "gmres", "f": 22, "geometry": "linear", "physics": "geometry",
         "precision": "fp64", "n": 2, "m": 2},
        # shape and impedance gradient of the far field, ellipsoid, ka = 3
        {"name": "adjoint_gradient", "kind": "adjoint", "f": 22, "geometry": "linear", "physics": "geometry",
         "precision": "fp64", "n": 2, "m": 2, "points": 32},
        # near-field (sparse) F and G with the adaptive singular rules
        {"name": "near_field_sparse", "kind": "nearfield", "f": 16, "geometry": "linear", "physics": "geometry",
         "depth": 1, "offset": 0.2, "complex_k": False},
        # product with the visco-thermal system at 100 Hz (nested solves)
        {"name": "lossy_product", "kind": "lossy", "f": 16, "geometry": "linear", "physics": "geometry",
         "freq": 100.0},
    ]


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "product", "product", "multi", "sweep", "gmres",
                       "adjoint", "nearfield", "lossy"])

    def between(lo, hi):   # whole numbers spread over their logarithm
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = {"kind": kind, "geometry": rng.choice(["linear", "quadratic"]), "physics": "geometry"}
    if kind in ("assemble", "product"):
        c["precision"] = rng.choice(["fp64", "mixed", "df64"])
        c["n"] = c["m"] = rng.choice([2, 2, 3, 4])
        c["complex_k"] = rng.random() < 0.3
        most = 8e8 if c["precision"] == "fp64" else 8e8 * 2      # quadrature evaluations at most
        per = c["n"] * c["m"] * (1.6 if c["geometry"] == "quadratic" else 1.0)
        if kind == "assemble":
            c["physics"] = rng.choice(["geometry", "geometry", "geometry", "linear", "disctriconstant",
                                       "disctrilinear", "disctriquadratic"])
            c["targets"] = rng.choice([0, 0, between(33, 4000)])
        else:
            c["targets"] = 0
            c["which"] = rng.choice(["F", "G"])
            c["physics"] = "geometry"
        top = 32
        if c["complex_k"]:
            most /= 2
        while True:
            c["f"] = between(4, top)
            el = 20 * c["f"] ** 2
            nodes = _nodes(c)
            rows = c["targets"] or nodes
            if rows * el * per <= most and rows * nodes <= 1.4e8:
                break
    elif kind == "multi":
        c.update(f=between(4, 16), precision=rng.choice(["fp16", "bf16", "fp16_split", "bf16_split"]),
                 which=rng.choice(["F", "G"]), n=2, m=2, rhs=between(8, 256), complex_k=rng.random() < 0.3)
    elif kind == "sweep":
        c.update(geometry="linear", f=between(5, 16), precision="mixed", n=2, m=2, nk=between(3, 12))
    elif kind == "gmres":
        c.update(geometry="linear", f=between(5, 26), precision="fp64", n=2, m=2)
    elif kind == "adjoint":
        c.update(geometry="linear", f=between(5, 22), precision=rng.choice(["fp64", "df64"]), n=2, m=2,
                 points=between(5, 65))
    elif kind == "nearfield":
        c.update(f=between(4, 14), depth=1, offset=rng.choice([0.15, 0.2, 0.3]), complex_k=rng.random() < 0.5)
    else:
        c.update(geometry="linear", f=between(5, 16), freq=float(rng.choice([50.0, 100.0, 200.0])))
    return c


def _nodes(c):
    f = c["f"]
    v = 10 * f * f + 2
    per = {"disctriconstant": 1, "disctrilinear": 3, "disctriquadratic": 6}.get(c["physics"])
    if per:
        return 20 * f * f * per
    return 40 * f * f + 2 if c["geometry"] == "quadratic" and c["physics"] == "geometry" else v


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _base_mesh(f, geometry, physics, ellipsoid):
    axes = (1.0, 2.0 / 3.0, 1.0 / 3.0) if ellipsoid else None
    return bm.icosphere(f, geometry=geometry, physics=physics, axes=axes)


def _rotation(rng):
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    return q if np.linalg.det(q) > 0 else -q


def _mesh(case, rng):
    b = _base_mesh(case["f"], case["geometry"], case["physics"], case["kind"] == "adjoint")
    R = _rotation(rng)
    # collocation points that are mesh vertices stay bit-identical to them
    return dataclasses.replace(b, **{a: R @ getattr(b, a) for a in ("sources", "coordinates", "normals", "tangents",
                                                                    "sangents")})


def _crandn(rng, *shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def _inputs(case, seed):
    """Mesh, wavenumber and data of a case: numpy, from the seed alone."""
    rng = np.random.default_rng([int(seed), 20])
    mesh = _mesh(case, rng)
    N = mesh.n_sources
    k = float(rng.uniform(1.0, 10.0)) if case["f"] >= 12 else float(rng.uniform(0.5, 4.0))
    d = {"mesh": mesh, "k": complex(k, 0.4 * k) if case.get("complex_k") else k}
    if case.get("targets"):
        t = rng.normal(size=(3, case["targets"]))
        d["targets"] = t / np.linalg.norm(t, axis=0) * rng.uniform(1.5, 6.0, size=case["targets"])
    kind = case["kind"]
    if kind == "product":
        d["x"] = _crandn(rng, N)
    elif kind == "multi":
        d["X"] = _crandn(rng, case["rhs"], N)
    elif kind == "sweep":
        d["ks"] = np.sort(rng.uniform(0.1, 4.0, size=case["nk"]))
        d["w"] = _crandn(rng, N)
    elif kind == "gmres":
        d["k"] = float(rng.uniform(0.5, 4.0))
        dirn = rng.normal(size=3)
        d["b"] = np.exp(-1j * d["k"] * ((dirn / np.linalg.norm(dirn)) @ mesh.sources))
    elif kind == "adjoint":
        d["k"] = float(rng.uniform(2.5, 3.5))
        d["Z"] = RHO_C * (1.0 + 0.3 * rng.normal(size=mesh.n_elements) + 0.3j * rng.normal(size=mesh.n_elements))
        v = rng.normal(size=(3, case["points"]))
        d["points"] = 10.0 * v / np.linalg.norm(v, axis=0)
    elif kind == "lossy":
        d["x"] = _crandn(rng, N)
    return d


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    mesh, kind = s["mesh"], case["kind"]
    N = mesh.n_sources
    if kind == "assemble":
        s["ctx"] = biegpu.get_context(mesh, n=case["n"], m=case["m"])
        M = case["targets"] or N
        s["out"] = [torch.empty((N, M), dtype=torch.complex128, device=DEVICE),
                    torch.empty((N, M), dtype=torch.complex128, device=DEVICE),
                    torch.empty(M, dtype=torch.complex128, device=DEVICE)]
        s["t"] = torch.from_numpy(np.ascontiguousarray(s["targets"].T)).to(DEVICE) if case["targets"] else None
    elif kind == "product":
        op = biegpu.GPUFOperator if case["which"] == "F" else biegpu.GPUGOperator
        s["op"] = op(mesh, s["k"], n=case["n"], m=case["m"], precision=case["precision"])
        s["xd"] = torch.from_numpy(s["x"]).to(DEVICE)
    elif kind == "multi":
        op = biegpu.GPUFOperator if case["which"] == "F" else biegpu.GPUGOperator
        s["op"] = op(mesh, s["k"], n=case["n"], m=case["m"], multi_precision=case["precision"])
        s["Xd"] = torch.from_numpy(s["X"]).to(DEVICE).T
    elif kind == "gmres":
        s["ctx"] = biegpu.get_context(mesh, n=case["n"], m=case["m"])
        A = torch.empty((N, N), dtype=torch.complex128, device=DEVICE)
        C = torch.empty(N, dtype=torch.complex128, device=DEVICE)
        s["ctx"].assemble_device(s["k"], F=A, Cv=C, precision="fp64")
        A.diagonal().add_(1.0 - C)
        s["A"], s["bd"] = A, torch.from_numpy(s["b"]).to(DEVICE)
    elif kind == "lossy":
        s["L"] = biegpu.LossyGlobalOuter(mesh, case["freq"], depth=1, n=3)
    elif kind in ("sweep", "adjoint"):
        biegpu.get_context(mesh, n=case["n"], m=case["m"])
    else:
        s["ctx"] = biegpu.get_context(mesh)
        biegpu.assembly.nearfield_pattern(s["ctx"], case["depth"])   # the sparsity pattern a program keeps
    return s


def run(s):
    case, mesh = s["case"], s["mesh"]
    kind = case["kind"]
    if kind == "assemble":
        F, G, C = s["out"]
        s["ctx"].assemble_device(s["k"], F=F, G=G, Cv=C, targets=s["t"], precision=case["precision"])
        return {"F": F, "G": G, "C": C}
    if kind == "product":
        return s["op"] @ s["xd"]
    if kind == "multi":
        return s["op"] @ s["Xd"]
    if kind == "sweep":
        p, _ = biegpu.sweep([mesh], s["ks"], [s["w"]], precision=case["precision"], n=case["n"], m=case["m"])
        return p[0]
    if kind == "gmres":
        return biegpu.gmres(s["A"], s["bd"], precision=case["precision"], ctx=s["ctx"])
    if kind == "adjoint":
        J, pf, dX, dZ, _ = biegpu.farfield_objective(mesh, s["k"], s["Z"], s["points"], rho_c=RHO_C, n=case["n"],
                                                     m=case["m"], precision=case["precision"])
        return {"J": J, "pf": pf, "dX": dX, "dZ": dZ}
    if kind == "lossy":
        return s["L"] @ s["x"]
    F, G = biegpu.assemble_parallel(mesh, s["k"], sparse=True, depth=case["depth"], offset=case["offset"])
    return {"F": F.data, "G": G.data}


def work(case):
    f, kind = case["f"], case["kind"]
    E, N = 20 * f * f, _nodes(case)
    NP = {"linear": 3, "disctriconstant": 1, "disctrilinear": 3, "disctriquadratic": 6}.get(
        case["physics"], 6 if case["geometry"] == "quadratic" else 3)
    mesh_bytes = 24 * N + E * 8 * (3 + NP)
    q = case.get("n", 2) * case.get("m", 2)
    if case["geometry"] == "quadratic" and NP == 6:
        q *= 1.4                         # half of the nearest nodes are midpoints with the larger rule
    quad = 32 + 8 * NP                   # per quadrature evaluation
    if kind == "assemble":
        M = case["targets"] or N
        return {"bytes": mesh_bytes + 24 * M + 32.0 * M * N + 16 * M, "flops": float(M) * E * q * quad}
    if kind == "product":
        return {"bytes": mesh_bytes + 32.0 * N, "flops": float(N) * E * q * (quad - 8 * NP + 8)}
    if kind == "multi":
        return {"bytes": mesh_bytes + 32.0 * N * case["rhs"],
                "flops": float(N) * E * q * quad + 8.0 * N * N * case["rhs"]}
    if kind == "sweep":                  # assembly of F, G and C and about 25 products per wavenumber
        return {"bytes": mesh_bytes + 16.0 * N * case["nk"],
                "flops": case["nk"] * (float(N) * E * q * quad + 25 * 8.0 * N * N)}
    if kind == "gmres":
        return {"bytes": 16.0 * N * N + 32.0 * N, "flops": 10 * 8.0 * N * N}
    if kind == "adjoint":                # forward assembly, two solves, reverse pass of about twice the work
        return {"bytes": mesh_bytes + 32.0 * E + 24 * N,
                "flops": float(N + case["points"]) * E * q * 3 * quad + 50 * 8.0 * N * N}
    if kind == "lossy":
        return {"bytes": 2 * 16.0 * N * N + 32.0 * N, "flops": 2 * 8.0 * N * N}
    pairs = (6 if case["geometry"] == "linear" else 18) * (E / 2.0)
    return {"bytes": mesh_bytes + 32.0 * 7 * N, "flops": pairs * 800 * quad}


# ---------------------------------------------------------------------------
# the same integrals in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _gauss01(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _rules(n, m, count):
    """Quadrature rules clustered at the corners (Duffy) and at the edge midpoints (two half-Duffy triangles)."""
    def grid(a, b):
        (x, wx), (y, wy) = _gauss01(a), _gauss01(b)
        return np.tile(x, b), np.repeat(y, a), np.tile(wx, b) * np.repeat(wy, a)

    u, v, w = grid(n, m)
    out = [(u * v, (1 - u) * v, w * v), (u, v * (1 - u), w * (1 - u)), (v * (1 - u), u, w * (1 - u))]
    if count > 3:
        u, v, w = grid(n, 2 * ((m + 1) // 2))
        X = np.concatenate([0.5 * u, (u - 0.5) * v + 0.5])
        Y = np.concatenate([v * (1 - u), v * (1 - u)])
        W = np.concatenate([w * 0.5 * (1 - u), w * 0.5 * v])
        out += [(X, Y, W), (1 - X - Y, X, W), (Y, 1 - X - Y, W)]
    return out[:count]


def _shape(kind, u, v, beta=0.0):
    """Values and u-, v-derivatives (nodes x points)."""
    l = 1.0 - u - v
    z, o = np.zeros_like(u), np.ones_like(u)
    if kind == "disctriconstant":
        return np.stack([o]), None, None
    if kind.startswith("disc"):
        l, u, v = ((s - beta) / (1 - 3 * beta) for s in (l, u, v))
    if kind in ("linear", "disctrilinear"):
        return np.stack([l, u, v]), np.stack([-o, o, z]), np.stack([-o, z, o])
    val = np.stack([l * (2 * l - 1), u * (2 * u - 1), v * (2 * v - 1), 4 * u * l, 4 * u * v, 4 * v * l])
    du = np.stack([1 - 4 * l, 4 * u - 1, z, 4 * (l - u), 4 * v, -4 * v])
    dv = np.stack([1 - 4 * l, z, 4 * v - 1, -4 * u, 4 * u, 4 * (l - v)])
    return val, du, dv


class _Dense:
    """Rows of F, G, C of a mesh on the GPU in 64 bits."""

    def __init__(self, mesh, n, m):
        T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)   # noqa: E731
        self.X = T(mesh.coordinates.T)
        self.S = T(mesh.sources.T)
        self.topo, self.ptopo = T(mesh.topology.T - 1), T(mesh.physics_topology.T - 1)
        self.N, self.E, self.NP = self.S.shape[0], self.topo.shape[0], self.ptopo.shape[1]
        corners = mesh.shape_function == "linear"
        tables = _rules(n, m, min(self.NP, 3) if corners else self.NP)
        tables = [tables[min(r, len(tables) - 1)] for r in range(self.NP)]
        qmax = max(len(t[2]) for t in tables)
        pad = lambda a: np.concatenate([a, np.repeat(a[..., -1:], qmax - a.shape[-1], axis=-1)], axis=-1)  # noqa
        val, du, dv, phi, w = [], [], [], [], []
        for u, v, wt in tables:
            a, b, c = _shape(mesh.shape_function, u, v)
            val.append(pad(a)), du.append(pad(b)), dv.append(pad(c))
            phi.append(pad(_shape(mesh.physics_function, u, v, mesh.physics_beta)[0]))
            w.append(np.concatenate([wt, np.zeros(qmax - len(wt))]))
        self.val, self.du, self.dv, self.phi = (T(np.stack(x)) for x in (val, du, dv, phi))   # R x nodes x Q
        self.w = T(np.stack(w))
        self.Q = qmax
        self.geometry(self.X)

    def geometry(self, X):
        V = X[self.topo]                                          # E x nodes x 3
        self.x = torch.einsum("eak,raq->erqk", V, self.val)
        a, b = torch.einsum("eak,raq->erqk", V, self.du), torch.einsum("eak,raq->erqk", V, self.dv)
        nn = torch.linalg.cross(a, b)
        jac = torch.linalg.vector_norm(nn, dim=-1)
        self.nrm = -nn / jac[..., None]
        self.jw = jac * self.w

    def chunk(self):
        return max(1, int(2.5e7 / (self.E * self.Q)))

    def nearest(self, t):
        """First nearest physics node of every (row, element): largest component scaled out, each step rounded."""
        best, c = None, None
        for a in range(self.NP):
            P = self.S[self.ptopo[:, a]]
            x, y, z = ((P[None, :, i] - t[:, None, i]).abs() for i in range(3))
            mx = torch.maximum(torch.maximum(x, y), z)
            one = torch.where(mx == 0, torch.ones_like(mx), mx)
            x, y, z = x / one, y / one, z / one
            h = mx * torch.sqrt((x * x + y * y) + z * z)
            if a == 0:
                best, c = h, torch.zeros_like(h, dtype=torch.int64)
            else:
                c = torch.where(h < best, torch.full_like(c, a), c)
                best = torch.minimum(h, best)
        return c

    def kernels(self, t, k, c=None):
        """F, G, C integrands (rows x E x Q) with the rule of every pair, and that rule."""
        with torch.no_grad():
            c = self.nearest(t) if c is None else c
        e = torch.arange(self.E, device=DEVICE)[None]
        d = self.x[e, c] - t[:, None, None]
        r = torch.sqrt((d * d).sum(-1))
        jw = self.jw[e, c] / (4 * math.pi)
        dn = (d * self.nrm[e, c]).sum(-1) * jw / r**3
        k = complex(k)
        ph = torch.polar(torch.exp(-k.imag * r), k.real * r) if k.imag else torch.complex(torch.cos(k.real * r),
                                                                                        torch.sin(k.real * r))
        return ph * torch.complex(-1 - k.imag * r, k.real * r) * dn, ph * (jw / r), -dn, c

    def rows(self, t, k):
        """F, G (rows x N) and C (rows)."""
        f, g, cc, c = self.kernels(t, k)
        P = self.phi.transpose(1, 2).to(f.dtype)                  # R x Q x NP
        out = []
        for v in (f, g):
            pair = torch.zeros(v.shape[:2] + (self.NP,), dtype=f.dtype, device=DEVICE)
            for r in range(self.NP):
                sel = c == r
                pair[sel] = v[sel] @ P[r]
            A = torch.zeros((t.shape[0], self.N), dtype=f.dtype, device=DEVICE)
            out.append(A.index_add_(1, self.ptopo.reshape(-1), pair.reshape(t.shape[0], -1)))
        return out[0], out[1], cc.sum((1, 2)).to(f.dtype)

    def matrices(self, t, k, take):
        """take(first row, F rows, G rows, C rows) over all rows of t."""
        step = self.chunk()
        for i in range(0, t.shape[0], step):
            take(i, *self.rows(t[i:i + step], k))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("nearfield", "lossy"):      # adaptive rules; nested iterative solves
        return None
    d = _inputs(case, seed)
    mesh, k = d["mesh"], d.get("k")
    D = _Dense(mesh, case["n"], case["m"])
    t = torch.from_numpy(np.ascontiguousarray(d["targets"].T)).to(DEVICE) if case.get("targets") else D.S
    M, N = t.shape[0], D.N
    z = functools.partial(torch.zeros, dtype=torch.complex128, device=DEVICE)
    if kind == "assemble":
        F, G, C = z((N, M)), z((N, M)), z(M)

        def take(i, f, g, c):
            F[:, i:i + len(c)], G[:, i:i + len(c)], C[i:i + len(c)] = f.T, g.T, c
        D.matrices(t, k, take)
        return {"F": F, "G": G, "C": C}
    if kind in ("product", "multi"):
        X = torch.from_numpy(d["x"] if kind == "product" else d["X"].T.copy()).to(DEVICE)
        y = z((M,) + tuple(X.shape[1:]))

        def take(i, f, g, c):
            y[i:i + len(c)] = (f if case["which"] == "F" else g) @ X
        D.matrices(t, k, take)
        return y
    if kind in ("sweep", "gmres"):
        ks = d["ks"] if kind == "sweep" else [k]
        p = z((N, len(ks)))
        for j, kj in enumerate(ks):
            A, rhs = z((N, N)), z(N)
            w = torch.from_numpy(d["w"]).to(DEVICE) if kind == "sweep" else None

            def take(i, f, g, c):
                A[i:i + len(c)] = f
                A[i:i + len(c), i:i + len(c)].diagonal().add_(1 - c)
                if w is not None:
                    rhs[i:i + len(c)] = g @ w
            D.matrices(D.S, float(kj), take)
            p[:, j] = torch.linalg.solve(A, rhs if w is not None else torch.from_numpy(d["b"]).to(DEVICE))
        return p if kind == "sweep" else p[:, 0]
    return _exact_adjoint(case, d, D)


def _exact_adjoint(case, d, D):
    """J, pressures and gradients by torch's autograd, row block by row block, with the adjoint solution held."""
    k = d["k"]
    z = functools.partial(torch.zeros, dtype=torch.complex128, device=DEVICE)
    Y = 1.0 / torch.from_numpy(d["Z"]).to(DEVICE)
    xf = torch.from_numpy(np.ascontiguousarray(d["points"].T)).to(DEVICE)
    e3 = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=DEVICE)
    N, M, step = D.N, xf.shape[0], max(1, D.chunk() // 8)
    P = D.phi.transpose(1, 2).to(torch.complex128)

    def incident(t):
        s = -k * (t @ e3)
        return torch.complex(torch.cos(s), torch.sin(s))

    def both(t, Yv, c=None):
        """Element contributions rows x E x 3 of F and of G with element factors, and C."""
        f, g, cc, c = D.kernels(t, k, c)
        pick = P[c]                                              # rows x E x Q x 3
        return torch.einsum("meq,meqa->mea", f, pick), torch.einsum("meq,meqa->mea", g * Yv[None, :, None], pick), cc.sum((1, 2))

    def matrix(t, a_f, a_g):
        A = z((t.shape[0], N))
        cs = z(t.shape[0])
        for i in range(0, t.shape[0], step):
            f, g, c = both(t[i:i + step], Y)
            A[i:i + step].index_add_(1, D.ptopo.reshape(-1), (a_f * f + a_g * g).reshape(f.shape[0], -1))
            cs[i:i + step] = c
        return A, cs

    with torch.no_grad():
        A, cs = matrix(D.S, 1.0, -1j * RHO_C * k)
        A.diagonal().add_(1 - cs)
        B, _ = matrix(xf, -1.0, 1j * RHO_C * k)
        p = torch.linalg.solve(A, incident(D.S))
        pf = incident(xf) + B @ p
        g = pf.conj()
        lam = torch.linalg.solve(A.T, B.T @ g)
    X = D.X.clone().requires_grad_()
    Yl = Y.clone().requires_grad_()
    gX, gY = torch.zeros_like(X), torch.zeros_like(Yl)
    pe = p[D.ptopo]                                              # E x 3
    for at, wt, a_f, a_g in ((None, -lam, 1.0, -1j * RHO_C * k), (xf, g, -1.0, 1j * RHO_C * k)):
        total = N if at is None else M
        for i in range(0, total, step):
            D.geometry(X)
            rows = X[i:i + step] if at is None else at[i:i + step]
            wi = wt[i:i + step]
            f, gg, c = both(rows, Yl)
            val = ((a_f * f + a_g * gg) * pe[None]).sum((1, 2))
            L = wi * val
            if at is None:
                L = L - wi * c * p[i:i + step] - wi * incident(rows)
            a, b = torch.autograd.grad(2 * L.sum().real, (X, Yl), allow_unused=True)
            gX += a
            gY += b
    # torch's gradient of a real function with respect to Y is dL/dRe Y + i dL/dIm Y; Z = 1 / Y
    dZ = gY * (-(Y * Y)).conj()
    return {"J": float((pf.abs() ** 2).sum()), "pf": pf, "dX": gX.T.contiguous(), "dZ": dZ}
