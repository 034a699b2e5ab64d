"""The calls whose speed counts: assembly, loads, gradients, solves, energies and batches through the public API.

Seven kinds of call, each over the range of sizes, element types, integrands and value types that the tests, the
benchmark and the shipped configurations use:

  assemble   ``ElementAssembler`` on given points and a per-element coefficient -> the CSR values
  load       ``NodeAssembler`` of a source function -> the load vector
  gradient   an assembly and the gradients of <G, values> in the points and the coefficient (shape and
             coefficient optimisation)
  solve      ``K.solve`` of a condensed Poisson system
  poisson    the whole calculation: assembly, load, condensation, solve, recovery
  energy     the Neo-Hookean energy and its displacement gradient (one evaluation of a Newton or descent step)
  batched    many independent Poisson problems of uneven size in one call

A case is a dict: ``kind``, ``element``, ``n`` (cells per side of the unit square or cube), ``dtype`` and what the kind
needs besides.  ``exact`` restates every result in float64 with plain torch.
"""
import math

import numpy as np
import torch

import tensormesh_gb300 as tg
from tensormesh_gb300.batched import BatchedPoisson
from tensormesh_gb300.forms import elasticity_block, reference_lame

DEV = "cuda"
DTYPES = {"f64": torch.float64, "f32": torch.float32}
DIM = {"triangle": 2, "triangle6": 2, "tetra": 3, "tetra10": 3}
NU = 0.3
RTOL = 1e-10        # of the FP64 solves, as the adjoint configuration and the smoke run use it
BATCH_RTOL = 1e-5   # of the float32 batch


def listed():
    return [
        # the smallest call: a coarse 2D mesh inside an optimisation or time loop; launches and host work count
        {"name": "laplace tri small", "kind": "assemble", "element": "triangle", "form": "laplace", "n": 16,
         "dtype": "f64", "order": 2, "jitter": True, "numbering": "grid"},
        # the 64 x 64 Poisson problem as a tutorial user runs it, from the coefficient to the solution
        {"name": "poisson 2d whole", "kind": "poisson", "element": "triangle", "n": 64, "dtype": "f64", "order": 2},
        # the largest assembly configuration: 12.6 M tetrahedra of a structured cube, per-element coefficient
        {"name": "laplace tet 128", "kind": "assemble", "element": "tetra", "form": "laplace", "n": 128,
         "dtype": "f64", "order": 1, "jitter": False, "numbering": "grid"},
        # an unstructured float32 mesh of odd size, numbered as a Delaunay generator leaves it
        {"name": "laplace tet f32 odd", "kind": "assemble", "element": "tetra", "form": "laplace", "n": 75,
         "dtype": "f32", "order": 2, "jitter": True, "numbering": "random"},
        # linear elasticity with a modulus per element, the 64^3 configuration
        {"name": "elasticity tet 64", "kind": "assemble", "element": "tetra", "form": "elasticity", "n": 64,
         "dtype": "f64", "order": 1, "jitter": False, "numbering": "grid"},
        # quadratic tetrahedra, curved by moving every node: the general geometry at each quadrature point
        {"name": "laplace tet10 27", "kind": "assemble", "element": "tetra10", "form": "laplace", "n": 27,
         "dtype": "f64", "order": 2, "jitter": True, "numbering": "grid"},
        # the load of a source function f(x) on a large mesh
        {"name": "load tet 64", "kind": "load", "element": "tetra", "n": 64, "dtype": "f64", "order": 2,
         "jitter": True},
        # forward and backward assembly: the gradient step of a 3D shape and coefficient optimisation
        {"name": "gradient tet 48", "kind": "gradient", "element": "tetra", "form": "laplace", "n": 48,
         "dtype": "f64", "order": 2},
        # a large 3D system with jumping coefficients (bandwidth-bound iterations)
        {"name": "solve 3d 96", "kind": "solve", "element": "tetra", "n": 96, "dtype": "f64"},
        # the 256 x 256 system of the adjoint configuration (latency-bound iterations)
        {"name": "solve 2d 256", "kind": "solve", "element": "triangle", "n": 256, "dtype": "f64"},
        # hyperelastic energy and internal forces on a large mesh
        {"name": "energy tet 64", "kind": "energy", "element": "tetra", "n": 64, "dtype": "f64", "order": 2},
        # a data-generation batch: 64 uneven 2D problems assembled and solved in one launch
        {"name": "batched 64", "kind": "batched", "element": "triangle", "count": 64, "lo": 32, "hi": 161,
         "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "assemble", "load", "gradient", "gradient", "solve",
                       "poisson", "energy", "batched"])
    element = rng.choice(["triangle", "triangle6", "tetra", "tetra", "tetra10"])
    dtype = rng.choice(["f64", "f64", "f32"])
    order = rng.choice([1, 2])
    if kind == "assemble":
        form = rng.choice(["laplace", "laplace", "mass", "elasticity"])
        top = {"laplace": {"triangle": 1000, "triangle6": 300, "tetra": 112, "tetra10": 27},
               "mass": {"triangle": 1000, "triangle6": 300, "tetra": 96, "tetra10": 24},
               "elasticity": {"triangle": 400, "triangle6": 100, "tetra": 56, "tetra10": 12}}[form][element]
        return {"kind": kind, "element": element, "form": form, "n": _log_int(rng, 4, top), "dtype": dtype,
                "order": order, "jitter": rng.random() < 0.5, "numbering": rng.choice(["grid", "grid", "random"])}
    if kind == "load":
        top = {"triangle": 700, "triangle6": 250, "tetra": 80, "tetra10": 27}[element]
        return {"kind": kind, "element": element, "n": _log_int(rng, 4, top), "dtype": dtype, "order": 2,
                "jitter": rng.random() < 0.5}
    if kind == "gradient":
        element = rng.choice(["triangle", "tetra"])
        return {"kind": kind, "element": element, "form": rng.choice(["laplace", "laplace", "elasticity"]),
                "n": _log_int(rng, 4, 300 if element == "triangle" else 30), "dtype": dtype, "order": order}
    if kind in ("solve", "poisson"):
        element = rng.choice(["triangle", "tetra"])
        return {"kind": kind, "element": element, "n": _log_int(rng, 8, 250 if element == "triangle" else 80),
                "dtype": "f64", **({"order": 2} if kind == "poisson" else {})}
    if kind == "energy":
        element = rng.choice(["triangle", "tetra", "tetra"])
        return {"kind": kind, "element": element, "n": _log_int(rng, 4, 400 if element == "triangle" else 60),
                "dtype": dtype, "order": order}
    return {"kind": kind, "element": "triangle", "count": rng.randint(8, 56), "lo": rng.randint(16, 48),
            "hi": rng.randint(64, 150), "dtype": "f32"}


# -- inputs ------------------------------------------------------------------------------------------------------------
def _grid(dim, n):
    """(points [N, dim], cells [E, dim + 1], boundary mask [N]) of the split unit square or the Kuhn cube."""
    m = n + 1
    xs = torch.linspace(0.0, 1.0, m, dtype=torch.float64, device=DEV)
    ax = torch.meshgrid(*([xs] * dim), indexing="ij")
    pts = torch.stack([a.reshape(-1) for a in reversed(ax)], 1)
    ix = torch.meshgrid(*([torch.arange(n, device=DEV)] * dim), indexing="ij")
    step = [m ** d for d in range(dim)]
    base = sum(i * s for i, s in zip(reversed(ix), step)).reshape(-1)
    perms = [(0, 1), (1, 0)] if dim == 2 else [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
    cells = []
    for p in perms:
        v = [base]
        for d in p:
            v.append(v[-1] + step[d])
        if dim == 2 and p == (1, 0):
            v = [v[0], v[2], v[1]]   # counter-clockwise
        cells.append(torch.stack(v, 1))
    cells = torch.stack(cells, 1).reshape(-1, dim + 1)
    return pts, cells, ((pts == 0.0) | (pts == 1.0)).any(1)


EDGES = {2: ((1, 2), (0, 2), (0, 1)), 3: ((2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1))}


def _quadratic(pts, cells):
    dim, N = pts.shape[1], pts.shape[0]
    pairs = torch.stack([torch.sort(cells[:, list(e)], 1).values for e in EDGES[dim]], 1)
    uniq, inv = torch.unique(pairs[..., 0] * N + pairs[..., 1], return_inverse=True)
    mid = 0.5 * (pts[uniq // N] + pts[uniq % N])
    return torch.cat([pts, mid]), torch.cat([cells, N + inv], 1)


def _geometry(case, gen):
    """(points float64, cells, boundary mask) of a case."""
    element, n = case["element"], case["n"]
    dim = DIM[element]
    pts, cells, bd = _grid(dim, n)
    if element in ("triangle6", "tetra10"):
        pts, cells = _quadratic(pts, cells)
        bd = ((pts == 0.0) | (pts == 1.0)).any(1)
    if case.get("jitter"):
        move = 0.05 if element in ("triangle6", "tetra10") else 0.2
        pts = pts + move / n * (2.0 * torch.rand(pts.shape, generator=gen, dtype=torch.float64, device=DEV) - 1.0)
    if case.get("numbering") == "random":
        new = torch.randperm(pts.shape[0], generator=gen, device=DEV)
        moved = torch.empty_like(pts)
        moved[new] = pts
        mask = torch.empty_like(bd)
        mask[new] = bd
        pts, bd, cells = moved, mask, new[cells]
        cells = cells[torch.randperm(cells.shape[0], generator=gen, device=DEV)]
    return pts, cells.contiguous(), bd


def _source(x, phase=0.0):
    return torch.sin(3.0 * x[..., 0] + phase) * torch.cos(2.0 * x[..., 1]) + 2.0


def _inputs(case, seed):
    """Every tensor a case's call is given, made from the seed alone."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    dt = DTYPES[case["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, dtype=torch.float64, device=DEV)

    if case["kind"] == "batched":
        rng = np.random.default_rng(case["count"] * 1000003 + case["lo"] * 1009 + case["hi"])
        geo = [_grid(2, int(k)) for k in rng.integers(case["lo"], case["hi"], size=case["count"])]
        return {"geo": geo, "kappa": torch.exp(normal(sum(g[1].shape[0] for g in geo))).to(dt)}
    pts, cells, bd = _geometry(case, gen)
    out = {"points": pts.to(dt), "cells": cells, "boundary": bd}
    E, N, dim = cells.shape[0], pts.shape[0], pts.shape[1]
    if case["kind"] in ("assemble", "gradient", "poisson"):
        out["kappa"] = torch.exp(normal(E)).to(dt)
    if case["kind"] == "solve":
        # log kappa ~ N(0, 1) on blocks of cells (a layered medium), as the benchmark's generator draws it
        blocks = 4
        centre = pts[cells].mean(1)
        at = (centre.clamp(0, 1 - 1e-9) * blocks).long()
        field = torch.exp(normal(blocks ** dim))
        out["kappa"] = field[(at * torch.tensor([blocks ** d for d in range(dim)], device=DEV)).sum(1)]
        out["rhs"] = _source(pts) / case["n"] ** dim * (1.0 + 0.1 * normal(N))
    if case["kind"] == "gradient":
        out["seed_values"] = int(seed) + 77
    if case["kind"] == "load":
        out["phase"] = 3.0 * float(torch.rand(1, generator=gen, dtype=torch.float64, device=DEV))
    if case["kind"] == "energy":
        wave = torch.sin(3.0 * pts + normal(dim)) * 0.02
        out["u"] = (wave + 0.1 / case["n"] * 0.2 * normal(N, dim).clamp(-2, 2)).to(dt)
    return out


class _KappaLaplace(tg.ElementAssembler):
    def forward(self, gradu, gradv, kappa):
        return kappa * (gradu @ gradv)


class _KappaMass(tg.ElementAssembler):
    def forward(self, u, v, kappa):
        return kappa * u * v


class _KappaElasticity(tg.ElementAssembler):
    def forward(self, gradu, gradv, kappa):
        lam, mu = reference_lame(1.0, NU)
        return kappa * elasticity_block(gradu, gradv, lam, mu)


_FORMS = {"laplace": _KappaLaplace, "mass": _KappaMass, "elasticity": _KappaElasticity}


class _Source(tg.NodeAssembler):
    def __post_init__(self, phase):
        self.phase = phase

    def forward(self, x, v):
        return _source(x, self.phase) * v


def prepare(case, seed):
    """What the caller's program holds before the call: mesh, data, assemblers and, for a solve, the system."""
    i = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batched":
        meshes = [tg.Mesh(points=p, cells={"triangle": c}, point_data={"is_boundary": b}) for p, c, b in i["geo"]]
        return {"kind": kind, "batch": BatchedPoisson(meshes), "kappa": i["kappa"]}
    mesh = tg.Mesh(points=i["points"], cells={case["element"]: i["cells"]}, point_data={"is_boundary": i["boundary"]})
    s = {"kind": kind, "points": mesh.points}
    order = case.get("order", 1)
    if kind == "assemble":
        s["asm"], s["data"] = _FORMS[case["form"]].from_mesh(mesh, order), {"kappa": i["kappa"]}
    elif kind == "load":
        s["asm"] = _Source.from_mesh(mesh, order, phase=i["phase"])
    elif kind == "gradient":
        s["asm"] = _FORMS[case["form"]].from_mesh(mesh, order)
        s["points"] = mesh.points.clone().requires_grad_(True)
        s["kappa"] = i["kappa"].clone().requires_grad_(True)
        H = DIM[case["element"]] if case["form"] == "elasticity" else 1
        gen = torch.Generator(device=DEV).manual_seed(i["seed_values"])
        s["G"] = torch.randn(s["asm"].topology.pattern.nnz * H * H, generator=gen, dtype=torch.float64,
                             device=DEV).to(mesh.points.dtype)
    elif kind == "energy":
        s["asm"] = tg.NeoHookeanModel.from_mesh(mesh, order)
        s["u"] = i["u"].clone().requires_grad_(True)
    else:
        s["asm"], s["data"] = _KappaLaplace.from_mesh(mesh, order), {"kappa": i["kappa"]}
        s["condenser"] = tg.Condenser(mesh.boundary_mask)
        if kind == "poisson":
            s["load"] = tg.const_node_assembler(1.0).from_mesh(mesh, order)
        else:
            s["K"], s["f"] = s["condenser"](s["asm"](mesh.points, element_data=s["data"]), i["rhs"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "assemble":
        return s["asm"](s["points"], element_data=s["data"]).values
    if kind == "load":
        return s["asm"](s["points"])
    if kind == "gradient":
        K = s["asm"](s["points"], element_data={"kappa": s["kappa"]})
        dx, dk = torch.autograd.grad(K.values, (s["points"], s["kappa"]), s["G"])
        return {"values": K.values, "points": dx, "kappa": dk}
    if kind == "energy":
        e = s["asm"].energy(s["u"], s["points"])
        (force,) = torch.autograd.grad(e, (s["u"],))
        return {"energy": e, "force": force}
    if kind == "solve":
        return s["K"].solve(s["f"], rtol=RTOL)
    if kind == "poisson":
        K = s["asm"](s["points"], element_data=s["data"])
        K_ii, f_i = s["condenser"](K, s["load"](s["points"]))
        return {"u": s["condenser"].recover(K_ii.solve(f_i, rtol=RTOL)), "values": K.values}
    u, info = s["batch"](s["kappa"], rtol=BATCH_RTOL)
    return {"u": u, "status": info.status}


# -- the work of a pass ------------------------------------------------------------------------------------------------
# nodes and CSR entries per cell of a large mesh
_NODES = {"triangle": 1, "triangle6": 4, "tetra": 1, "tetra10": 8}
_DEGREE = {"triangle": 7, "triangle6": 11.5, "tetra": 15, "tetra10": 28.5}


def work(case):
    if case["kind"] == "batched":
        cells = case["count"] * (case["lo"] + case["hi"]) ** 2 / 4.0 * 1.05
        return {"bytes": cells * (2 * 12 + 2 * 4 + 2 * 4 + 7 * 8 + 8), "flops": cells * 200 * 2 * 7}
    el, n, size = case["element"], case["n"], DTYPES[case["dtype"]].itemsize
    dim = DIM[el]
    E = (2 if dim == 2 else 6) * n ** dim
    N = _NODES[el] * (n + 0.5) ** dim
    B = {"triangle": 3, "triangle6": 6, "tetra": 4, "tetra10": 10}[el]
    H = dim if case.get("form") == "elasticity" else 1
    nnz = N * _DEGREE[el] * H * H
    mesh = 4 * B * E + size * dim * N                 # connectivity and coordinates
    pair = {"laplace": 2 * dim + 2, "mass": 3, "elasticity": 5 * dim * dim}
    if case["kind"] == "assemble":
        return {"bytes": mesh + size * (E + nnz), "flops": E * (B * B * pair[case["form"]] + 60)}
    if case["kind"] == "load":
        return {"bytes": mesh + size * N, "flops": E * (B * 8 * case["order"] + 60)}
    if case["kind"] == "gradient":
        return {"bytes": 2 * mesh + size * (2 * E + 2 * nnz + dim * N), "flops": 3 * E * (B * B * pair[case["form"]] + 60)}
    if case["kind"] == "energy":
        return {"bytes": mesh + 2 * size * dim * N, "flops": E * (B * 6 * dim + 250)}
    system = nnz * 12 + 24 * N                        # values, columns, right-hand side, solution
    if case["kind"] == "solve":
        return {"bytes": system, "flops": 2 * nnz + 10 * N}
    return {"bytes": mesh + size * (E + nnz) + system, "flops": E * (B * B * pair["laplace"] + 60) + 2 * nnz}


# -- the same results in float64, plain torch --------------------------------------------------------------------------
_A, _B = 0.5854101966249685, 0.1381966011250105
_RULE = {
    (2, 1): ([0.5], [[1 / 3, 1 / 3]]),
    (2, 2): ([1 / 6] * 3, [[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]]),
    (3, 1): ([1 / 6], [[0.25] * 3]),
    (3, 2): ([1 / 24] * 4, [[_A, _B, _B], [_B, _B, _B], [_B, _B, _A], [_B, _A, _B]]),
}


def _shape(element, xi):
    """Shape functions [B] and their reference gradients [B, D] at one point."""
    dim = DIM[element]
    lam = torch.cat([1.0 - xi.sum().reshape(1), xi])
    dlam = torch.cat([-torch.ones(1, dim, dtype=torch.float64, device=DEV),
                      torch.eye(dim, dtype=torch.float64, device=DEV)])
    if element in ("triangle", "tetra"):
        return lam, dlam
    N = [l * (2 * l - 1) for l in lam] + [4 * lam[a] * lam[b] for a, b in EDGES[dim]]
    dN = [(4 * l - 1) * d for l, d in zip(lam, dlam)]
    dN += [4 * (lam[a] * dlam[b] + lam[b] * dlam[a]) for a, b in EDGES[dim]]
    return torch.stack(N), torch.stack(dN)


def _points_of(element, order, X):
    """(shape functions, weight, physical gradients [E, B, D], |det J| [E]) at each quadrature point."""
    w, xi = _RULE[(DIM[element], order)]
    for wq, x in zip(w, xi):
        N, dN = _shape(element, torch.tensor(x, dtype=torch.float64, device=DEV))
        J = torch.einsum("ebj,bi->eji", X, dN)                    # dx_j / dxi_i
        yield N, wq, torch.einsum("bi,eij->ebj", dN, torch.linalg.inv(J)), torch.linalg.det(J).abs()


def _element_matrices(element, form, order, X, kappa):
    """[E, B, B] or, for elasticity, [E, B, D, B, D]."""
    total = 0
    for N, wq, g, det in _points_of(element, order, X):
        cw = kappa * wq * det
        if form == "mass":
            total = total + cw[:, None, None] * (N[:, None] * N[None, :])
        elif form == "laplace":
            total = total + cw[:, None, None] * (g @ g.transpose(1, 2))
        else:
            mu = float(np.float32(1.0 / (2.0 * (1.0 + NU))))
            lam = float(np.float32(NU / ((1.0 + NU) * (1.0 - 2.0 * NU))))
            c = cw[:, None, None, None, None]
            eye = torch.eye(g.shape[2], dtype=torch.float64, device=DEV)
            blk = lam * torch.einsum("eai,ebj->eaibj", g, g) + mu * torch.einsum("eaj,ebi->eaibj", g, g)
            total = total + c * (blk + mu * torch.einsum("eab,ij->eaibj", g @ g.transpose(1, 2), eye))
    return total


def _csr(cells, Ke, N):
    """(row, column, values) of the global matrix, rows then columns ascending; differentiable in Ke."""
    if Ke.dim() == 5:
        H = Ke.shape[2]
        cells = (cells[:, :, None] * H + torch.arange(H, device=DEV)).reshape(cells.shape[0], -1)
        N, Ke = N * H, Ke.reshape(Ke.shape[0], cells.shape[1], cells.shape[1])
    key = (cells[:, :, None] * N + cells[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(key, return_inverse=True)
    vals = torch.zeros(uniq.shape[0], dtype=torch.float64, device=DEV).index_add(0, inv, Ke.reshape(-1))
    return uniq // N, uniq % N, vals


def _source_vector(element, order, X, cells, N, f):
    out = torch.zeros(N, dtype=torch.float64, device=DEV)
    for Nq, wq, _, det in _points_of(element, order, X):
        x = torch.einsum("ebj,b->ej", X, Nq)
        out.index_add_(0, cells.reshape(-1), ((f(x) * wq * det)[:, None] * Nq).reshape(-1))
    return out


def _conjugate_gradients(row, col, val, N, keep, b):
    """K x = b on the dofs of ``keep`` (zero elsewhere), to about 1e-15, Jacobi-preconditioned."""
    inside = keep[row] & keep[col]
    at = torch.cumsum(keep.long(), 0) - 1
    r, c, v = at[row[inside]], at[col[inside]], val[inside]
    n = int(keep.sum())
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    A = torch.sparse_csr_tensor(ptr, c, v, size=(n, n))
    d = torch.zeros(n, dtype=torch.float64, device=DEV)
    d[r[r == c]] = v[r == c]
    rhs = b[keep]
    x = torch.zeros_like(rhs)
    for _ in range(2):                      # the second pass refines the first
        res = rhs - A @ x
        z = res / d
        p, rz = z.clone(), torch.dot(res, z)
        dx = torch.zeros_like(x)
        stop = max(1e-15 * float(rhs.norm()), 1e-9 * float(res.norm()))
        for k in range(20000):
            q = A @ p
            a = rz / torch.dot(p, q)
            dx += a * p
            res = res - a * q
            if k % 25 == 24 and float(res.norm()) <= stop:
                break
            z = res / d
            rz, old = torch.dot(res, z), rz
            p = z + (rz / old) * p
        x = x + dx
    out = torch.zeros(N, dtype=torch.float64, device=DEV)
    out[keep] = x
    return out


def exact(case, seed):
    i = _inputs(case, seed)
    kind, element = case["kind"], case["element"]
    if kind == "batched":
        shift, pts, cells, keep = 0, [], [], []
        for p, c, b in i["geo"]:
            pts.append(p.float().double())
            cells.append(c + shift)
            keep.append(~b)
            shift += p.shape[0]
        pts, cells, keep = torch.cat(pts), torch.cat(cells), torch.cat(keep)
        row, col, val = _csr(cells, _element_matrices(element, "laplace", 1, pts[cells], i["kappa"].double()), shift)
        b = _source_vector(element, 1, pts[cells], cells, shift, lambda x: torch.ones_like(x[..., 0]))
        return {"u": _conjugate_gradients(row, col, val, shift, keep, b), "status": None}
    pts, cells = i["points"].double(), i["cells"]
    N, order = pts.shape[0], case.get("order", 1)
    if kind == "load":
        return _source_vector(element, order, pts[cells], cells, N, lambda x: _source(x, i["phase"]))
    if kind == "energy":
        mu, lam = 1.0 / (2 * (1 + NU)), NU / ((1 + NU) * (1 - 2 * NU))
        u = i["u"].double().requires_grad_(True)
        total = 0.0
        dim = pts.shape[1]
        for _, wq, g, det in _points_of(element, order, pts[cells]):
            F = torch.eye(dim, dtype=torch.float64, device=DEV) + torch.einsum("ebi,ebj->eij", u[cells], g)
            lnJ = torch.log(torch.linalg.det(F))
            psi = 0.5 * mu * ((F * F).sum((1, 2)) - dim) - mu * lnJ + 0.5 * lam * lnJ ** 2
            total = total + (wq * det * psi).sum()
        (force,) = torch.autograd.grad(total, (u,))
        return {"energy": total.detach(), "force": force}
    kappa = i["kappa"].double()
    if kind == "gradient":
        pts, kappa = pts.requires_grad_(True), kappa.requires_grad_(True)
        _, _, val = _csr(cells, _element_matrices(element, case["form"], order, pts[cells], kappa), N)
        gen = torch.Generator(device=DEV).manual_seed(i["seed_values"])
        G = torch.randn(val.shape[0], generator=gen, dtype=torch.float64, device=DEV).to(DTYPES[case["dtype"]]).double()
        dx, dk = torch.autograd.grad(val, (pts, kappa), G)
        return {"values": val.detach(), "points": dx, "kappa": dk}
    row, col, val = _csr(cells, _element_matrices(element, case.get("form", "laplace"), order, pts[cells], kappa), N)
    if kind == "assemble":
        return val
    keep = ~i["boundary"]
    if kind == "solve":
        return _conjugate_gradients(row, col, val, N, keep, i["rhs"])[keep]
    b = _source_vector(element, order, pts[cells], cells, N, lambda x: torch.ones_like(x[..., 0]))
    return {"u": _conjugate_gradients(row, col, val, N, keep, b), "values": val}
