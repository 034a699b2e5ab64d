"""Element-once assembly of P1 meshes (tm_assemble_gather): sizes around the
32-row groups, random numbering, every coefficient kind, high-valence nodes,
and the group lists themselves.

Bars: float64 values within 1e-12 of max|K| of the oracle (the bar of every
float64 assembly), float32 within 1e-5, CSR values symmetric and bitwise
repeatable."""
import numpy as np
import pytest
import torch

import tensormesh_gb300 as tg
from oracle import fem

pytestmark = pytest.mark.gpu
DEV = "cuda"


class KappaLaplace(tg.ElementAssembler):
    def forward(self, gradu, gradv, kappa):
        return kappa * (gradu @ gradv)


class EElasticity(tg.ElementAssembler):
    def forward(self, gradu, gradv, kappa):
        lam, mu = tg.forms.reference_lame(1.0, 0.3)
        return kappa * tg.forms.elasticity_block(gradu, gradv, lam, mu)


@pytest.fixture(autouse=True)
def every_size(monkeypatch):
    """The element-once path at any size (its dispatch keeps small meshes on
    the one-launch patch kernels)."""
    monkeypatch.setattr("tensormesh_gb300.assemble._GATHER_MIN_ELEMENTS", dict.fromkeys(tg.element.ELEMENT_TYPES, 0))


FORMS = {"laplace": KappaLaplace, "elasticity": EElasticity}


def ragged(etype, n, seed):
    base = tg.Mesh.gen_unit_square(n) if etype == "triangle" else tg.Mesh.gen_unit_cube(n)
    rng = np.random.default_rng(seed)
    pts = base.points.numpy() + rng.uniform(-0.2, 0.2, size=tuple(base.points.shape)) / n
    new = rng.permutation(pts.shape[0])
    moved = np.empty_like(pts)
    moved[new] = pts
    el = new[base.cells[etype].numpy()]
    return moved, el[rng.permutation(el.shape[0])]


def check(pts, el, etype, form, coef, dtype=torch.float64, q=2, data="element_data"):
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV, dtype=dtype), cells={etype: torch.tensor(el, device=DEV)})
    asm = FORMS[form].from_mesh(mesh, quadrature_order=q)
    c = torch.tensor(coef, device=DEV, dtype=dtype)
    call = lambda: asm(mesh.points, **{data: {"kappa": c}})  # noqa: E731
    K = call()
    assert asm.topology.gather.struct(1) is not None
    p64, c64 = mesh.points.double().cpu().numpy(), c.double().cpu().numpy()
    oc = {"coef": c64} if data == "element_data" else {"coef": element_mean(c64, el)}
    ip, ix, dv = fem.assemble_csr(p64, el, etype, form, q, **oc)
    assert np.array_equal(K.indptr.cpu().numpy(), ip) and np.array_equal(K.indices.cpu().numpy(), ix)
    err = np.max(np.abs(K.values.double().cpu().numpy() - dv)) / np.max(np.abs(dv))
    assert err <= (1e-12 if dtype == torch.float64 else 1e-5), err
    assert torch.equal(call().values, K.values)


def element_mean(c, el):
    # an order-2 rule integrates a linear coefficient against constant gradients exactly
    return c[el].mean(1)


@pytest.mark.parametrize("etype,n", [("triangle", 1), ("triangle", 5), ("triangle", 11), ("tetra", 1), ("tetra", 3),
                                     ("tetra", 6)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_ragged_groups_match_oracle(etype, n, form, dtype):
    pts, el = ragged(etype, n, 3 * n)
    check(pts, el, etype, form, np.exp(np.random.default_rng(n).normal(size=el.shape[0])), dtype)


@pytest.mark.parametrize("form", ["laplace", "elasticity"])
def test_point_coefficients(form):
    pts, el = ragged("tetra", 4, 9)
    check(pts, el, "tetra", form, np.exp(np.random.default_rng(1).normal(size=pts.shape[0])), data="point_data")


@pytest.mark.parametrize("ring", [90, 200])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
def test_high_valence_nodes(ring, form):
    """Two apexes with `ring` + 1 neighbours each: lists and rows far longer
    than a regular mesh's."""
    t = np.arange(ring) * 2 * np.pi / ring
    pts = np.concatenate([[[0.0, 0.0, -0.3], [0.0, 0.0, 0.3]], np.stack([np.cos(t), np.sin(t), 0 * t], 1)])
    el = np.array([[0, 2 + k, 2 + (k + 1) % ring, 1] for k in range(ring)], dtype=np.int64)
    check(pts, el, "tetra", form, np.exp(np.random.default_rng(ring).normal(size=ring)))


def test_zero_and_far_coefficients():
    """Zero coefficients, and coefficients far outside the common exponent's
    window on either side of element 0's, in one call: every entry keeps its
    own relative accuracy where a single element makes it."""
    pts, el = ragged("tetra", 3, 5)
    g = np.exp(np.random.default_rng(6).normal(size=el.shape[0]))
    for scale in (0.0, 1e-40, 1e40):
        check(pts, el, "tetra", "laplace", g * np.where(np.arange(el.shape[0]) % 3 == 1, scale, 1.0))
        check(pts, el, "tetra", "elasticity", g * np.where(np.arange(el.shape[0]) % 3 == 0, scale, 1.0))


def test_an_element_that_repeats_a_node_keeps_the_patch_kernels():
    pts, el = ragged("tetra", 2, 8)
    bad = np.concatenate([el, el[:1]])
    bad[-1, 3] = bad[-1, 0]
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV), cells={"tetra": torch.tensor(bad, device=DEV)})
    assert KappaLaplace.from_mesh(mesh).topology.gather.struct(1) is None


@pytest.mark.parametrize("etype,n", [("triangle", 7), ("tetra", 4)])
@pytest.mark.parametrize("H", [1, 0])
def test_group_lists_cover_every_entry(etype, n, H):
    """The lists decoded on the host name, for every CSR position off the
    diagonal, the elements that hold its node pair, ascending."""
    pts, el = ragged(etype, n, 2)
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV), cells={etype: torch.tensor(el, device=DEV)})
    topo = KappaLaplace.from_mesh(mesh).topology
    H = H or topo.dim
    topo.gather.struct(H)
    s, keep = topo.gather._structs[H]
    B = el.shape[1]
    P = B * (B - 1) // 2
    pairs = [(a, b) for a in range(B) for b in range(a + 1, B)]
    k = {name: t.cpu().numpy() for name, t in keep.items()}
    ent, rec = k["gent"].view(np.uint32), k["grec"].view(np.uint16)
    ip, ix = topo.pattern.indptr.cpu().numpy(), topo.pattern.indices.cpu().numpy()
    holds = {}
    for e, nodes in enumerate(el):
        for i in nodes:
            for j in nodes:
                if i != j:
                    holds.setdefault((i, j), []).append(e)
    assert sorted(k["order"].tolist()) == list(range(pts.shape[0]))
    for g in range(k["base"].shape[0] - 1):
        e0, t, r0 = k["base"][g]
        elems = k["gelem"][e0:k["base"][g + 1][0]]
        assert np.all(np.diff(elems) > 0)
        for lr, r in enumerate(k["order"][g * s.rows_per_cta:(g + 1) * s.rows_per_cta]):
            for c in ix[ip[r]:ip[r + 1]]:
                w = int(ent[t])
                t += 1
                if c == r:
                    assert w == 0xffffffff
                    continue
                assert (w >> 16) & 63 == lr
                at, got = r0 + (w & 0xffff) * (4 if H == 1 else 1), []
                while True:
                    v = int(rec[at])
                    if H == 1:
                        if (v & 0x7fff) // P < len(elems):
                            e = int(elems[(v & 0x7fff) // P])
                            assert set(el[e][list(pairs[(v & 0x7fff) % P])]) == {r, c}
                            got.append(e)
                        at += 1
                        if (at - r0) % 4 == 0 and v & 0x8000:
                            break
                    else:
                        e = int(elems[(v & 0x7fff) >> 4])
                        assert (el[e][(v >> 2) & 3], el[e][v & 3]) == (r, c)
                        got.append(e)
                        at += 1
                        if v & 0x8000:
                            break
                assert got == holds[(r, c)]


# -- quadrature kernels: P2 elements, mass matrices, loads ------------------------------
class KappaMass(tg.ElementAssembler):
    def forward(self, u, v, kappa):
        return kappa * u * v


FORMS["mass"] = KappaMass


def curved(etype, n, seed):
    """A P2 mesh with every node moved and renumbered."""
    base = (tg.Mesh.gen_unit_square(n) if etype == "triangle6" else tg.Mesh.gen_unit_cube(n)).to_p2()
    rng = np.random.default_rng(seed)
    pts = base.points.numpy() + rng.uniform(-0.04, 0.04, size=tuple(base.points.shape)) / n
    new = rng.permutation(pts.shape[0])
    moved = np.empty_like(pts)
    moved[new] = pts
    return moved, new[base.cells[etype].numpy()]


MESHES = [("triangle6", 1), ("triangle6", 5), ("tetra10", 1), ("tetra10", 3)]


@pytest.mark.parametrize("etype,n", MESHES)
@pytest.mark.parametrize("form", ["laplace", "mass", "elasticity"])
@pytest.mark.parametrize("q", [1, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_p2_forms_match_oracle(etype, n, form, q, dtype):
    pts, el = curved(etype, n, n)
    check(pts, el, etype, form, np.exp(np.random.default_rng(n).normal(size=el.shape[0])), dtype, q=q)


@pytest.mark.parametrize("etype,n", [("triangle", 6), ("tetra", 4)])
@pytest.mark.parametrize("q", [1, 2, 4])
def test_p1_mass_matches_oracle(etype, n, q):
    pts, el = ragged(etype, n, n)
    check(pts, el, etype, "mass", np.exp(np.random.default_rng(n).normal(size=el.shape[0])), q=q)


@pytest.mark.parametrize("etype,n", [("triangle", 6), ("tetra", 4)] + MESHES[1::2])
@pytest.mark.parametrize("scale", [1e-9, 1e9])
def test_units_and_far_coefficients_with_quadrature(etype, n, scale):
    """Mass matrices (length^D) in extreme units, with elements whose
    coefficient is zero or far outside the common exponent's window."""
    pts, el = ragged(etype, n, 1) if n >= 4 and etype in ("triangle", "tetra") else curved(etype, n, 1)
    g = np.exp(np.random.default_rng(2).normal(size=el.shape[0]))
    for far in (0.0, 1e-40, 1e40):
        check(pts * scale, el, etype, "mass", g * np.where(np.arange(el.shape[0]) % 3 == 1, far, 1.0))
        if etype in ("triangle6", "tetra10"):
            check(pts * scale, el, etype, "elasticity", g * np.where(np.arange(el.shape[0]) % 3 == 1, far, 1.0))


def test_slivers_with_quadrature():
    """Needle elements (conditioning 1e7) take the native pass of their CTA."""
    ring, height = 30, 200.0
    t = np.arange(ring) * 2 * np.pi / ring
    pts = np.concatenate([[[0.0, 0.0, -height], [0.0, 0.0, height]], np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(3 * t)], 1)])
    el = np.array([[0, 2 + k, 2 + (k + 1) % ring, 1] for k in range(ring)], dtype=np.int64)
    kappa = np.exp(np.random.default_rng(ring).normal(size=ring))
    check(pts, el, "tetra", "mass", kappa)
    p2 = tg.Mesh(points=torch.tensor(pts), cells={"tetra": torch.tensor(el)}).to_p2()
    check(p2.points.numpy(), p2.cells["tetra10"].numpy(), "tetra10", "laplace", kappa)


@pytest.mark.parametrize("etype,n", [("triangle", 6), ("tetra", 4)] + MESHES)
@pytest.mark.parametrize("q", [1, 2, 4])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_loads_match_oracle(etype, n, q, dtype):
    pts, el = (ragged if etype in ("triangle", "tetra") else curved)(etype, n, 4)
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV, dtype=dtype), cells={etype: torch.tensor(el, device=DEV)})
    p64 = mesh.points.double().cpu().numpy()

    class PointLoad(tg.NodeAssembler):
        def forward(self, v, f):
            return v * f

    f = torch.tensor(np.random.default_rng(3).normal(size=(pts.shape[0], 3)), device=DEV, dtype=dtype)
    cases = [
        (tg.const_node_assembler(torch.tensor([2.0, -1.0], device=DEV, dtype=dtype)).from_mesh(mesh, quadrature_order=q)(mesh.points),
         fem.assemble_load(p64, el, etype, q, "const", [2.0, -1.0])),
        # a source that decays by 40 orders of magnitude over the mesh, and one with zeros
        (tg.func_node_assembler(lambda x: torch.exp(-90.0 * x[..., 0])).from_mesh(mesh, quadrature_order=q)(mesh.points),
         fem.assemble_load(p64, el, etype, q, "func", lambda x: np.exp(-90.0 * x[..., 0]))),
        (tg.func_node_assembler(lambda x: torch.relu(x[..., 0] - 0.5)).from_mesh(mesh, quadrature_order=q)(mesh.points),
         fem.assemble_load(p64, el, etype, q, "func", lambda x: np.maximum(x[..., 0] - 0.5, 0.0))),
        (PointLoad.from_mesh(mesh, quadrature_order=q)(mesh.points, point_data={"f": f}),
         fem.assemble_load(p64, el, etype, q, "point", f.double().cpu().numpy())),
    ]
    for got, ref in cases:
        err = np.max(np.abs(got.double().cpu().numpy() - ref)) / np.max(np.abs(ref))
        assert err <= (1e-12 if dtype == torch.float64 else 1e-5), err


@pytest.mark.parametrize("etype", ["triangle", "tetra"])
@pytest.mark.parametrize("q", [1, 2, 4])
@pytest.mark.parametrize("far", [1.0, 1e-150, 1e150, 1e-285])
def test_p1_loads_of_slivers_far_units_and_far_sources(etype, q, far):
    """Needle elements (native FP64), meshes in extreme units, and sources that
    are tiny, huge, or zero at some points, one to three components: 1e-12 of
    the largest entry (order 4 has more points than a thread keeps)."""
    ring = 33
    t = np.arange(ring) * 2 * np.pi / ring
    if etype == "tetra":
        pts = np.concatenate([[[0.0, 0.0, -200.0], [0.0, 0.0, 200.0]],
                              np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(3 * t)], 1)])
        el = np.array([[0, 2 + k, 2 + (k + 1) % ring, 1] for k in range(ring)], dtype=np.int64)
    else:
        pts = np.concatenate([[[0.0, 3e5]], np.stack([np.cos(t), np.sin(t)], 1)])
        el = np.array([[0, 1 + k, 1 + (k + 1) % ring] for k in range(ring)], dtype=np.int64)
    ragged_pts, ragged_el = ragged(etype, 6 if etype == "triangle" else 4, 7)
    for p, e, scale in ((pts, el, 1.0), (ragged_pts, ragged_el, 1e-9), (ragged_pts, ragged_el, 1e9)):
        if far == 1e-285 and scale < 1.0:
            continue   # subnormal results
        p = p * scale
        mesh = tg.Mesh(points=torch.tensor(p, device=DEV), cells={etype: torch.tensor(e, device=DEV)})
        for H in (1, 2, 3):
            class PointLoad(tg.NodeAssembler):
                def forward(self, v, f):
                    return v * f

            f = far * np.random.default_rng(H).normal(size=(p.shape[0], H))
            f[::3] = 0.0
            got = PointLoad.from_mesh(mesh, quadrature_order=q)(
                mesh.points, point_data={"f": torch.tensor(f[:, 0] if H == 1 else f, device=DEV)}).cpu().numpy()
            ref = fem.assemble_load(p, e, etype, q, "point", f)
            assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref)), (scale, H)


# -- backward ----------------------------------------------------------------------
def torch_values(pts, el, kappa, form, q_weight):
    """CSR values of a P1 mesh by plain torch (differentiable), canonical order."""
    X = pts[el]
    J = X[:, 1:] - X[:, :1]
    inv = torch.linalg.inv(J)
    P = torch.cat([-inv.sum(2, keepdim=True), inv], 2).transpose(1, 2)       # [E, B, D]
    c = kappa * q_weight * torch.linalg.det(J).abs()
    dot = P @ P.transpose(1, 2)
    N = pts.shape[0]
    if form == "laplace":
        Ke = c[:, None, None] * dot
    else:
        lam, mu = tg.forms.reference_lame(1.0, 0.3)
        D = P.shape[2]
        Ke = lam * torch.einsum("eai,ebj->eaibj", P, P) + mu * torch.einsum("eaj,ebi->eaibj", P, P)
        Ke = Ke + mu * torch.einsum("eab,ij->eaibj", dot, torch.eye(D, dtype=pts.dtype, device=pts.device))
        Ke = (c[:, None, None, None, None] * Ke).reshape(el.shape[0], el.shape[1] * D, -1)
        el = (el[:, :, None] * D + torch.arange(D, device=el.device)).reshape(el.shape[0], -1)
        N = N * D
    uniq, inv = torch.unique((el[:, :, None] * N + el[:, None, :]).reshape(-1), return_inverse=True)
    return torch.zeros(uniq.shape[0], dtype=pts.dtype, device=pts.device).index_add(0, inv, Ke.reshape(-1))


@pytest.mark.parametrize("etype,n", [("triangle", 1), ("triangle", 9), ("tetra", 1), ("tetra", 5)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("data", ["element_data", "point_data"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_p1_gradients_match_torch(etype, n, form, data, dtype):
    """Points and coefficient gradients of <G, values> against torch autograd
    in float64: within 1e-11 (float64; native FP64 of 200 to 700 operations)
    and 1e-4 (float32) of the largest gradient."""
    pts, el = ragged(etype, n, n + 1)
    el = torch.tensor(el, device=DEV)
    x = torch.tensor(pts, device=DEV, dtype=dtype)
    k = torch.exp(torch.randn(el.shape[0] if data == "element_data" else x.shape[0], device=DEV,
                              generator=torch.Generator(DEV).manual_seed(n), dtype=torch.float64)).to(dtype)
    asm = FORMS[form].from_mesh(tg.Mesh(points=x, cells={etype: el}), 2)
    xg, kg = x.clone().requires_grad_(True), k.clone().requires_grad_(True)
    vals = asm(xg, **{data: {"kappa": kg}}).values
    G = torch.randn(vals.shape[0], device=DEV, generator=torch.Generator(DEV).manual_seed(5), dtype=torch.float64)
    got = torch.autograd.grad(vals, (xg, kg), G.to(dtype))
    xr, kr = x.double().requires_grad_(True), k.double().requires_grad_(True)
    per_el = kr if data == "element_data" else kr[el].mean(1)
    ref = torch.autograd.grad(torch_values(xr, el, per_el, form, 0.5 if etype == "triangle" else 1 / 6), (xr, kr),
                              G.to(dtype).double())
    for a, b in zip(got, ref):
        err = float((a.double() - b).abs().max() / b.abs().max())
        assert err <= (1e-11 if dtype == torch.float64 else 1e-4), err
    again = torch.autograd.grad(asm(xg, **{data: {"kappa": kg}}).values, (xg, kg), G.to(dtype))
    assert all(torch.equal(a, b) for a, b in zip(got, again))


# -- streams -------------------------------------------------------------------------
@pytest.mark.parametrize("etype,n,H", [("triangle", 5, 1), ("tetra", 4, 1), ("tetra", 4, 3), ("tetra10", 2, 1)])
def test_lists_are_complete_when_they_become_visible(etype, n, H, monkeypatch):
    """The stream that built the lists is idle when ``struct`` returns, even
    where the last kernels of the build take long: a call on any other stream
    may read them at once."""
    pts, el = (curved if etype == "tetra10" else ragged)(etype, n, 3)
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV), cells={etype: torch.tensor(el, device=DEV)})
    topo = KappaLaplace.from_mesh(mesh).topology
    plan = tg.plan.GatherPlan(topo.elements, mesh.points, topo.pattern)
    inner, fills = tg._lib.call, []

    def slow_fill(name, *args):
        inner(name, *args)
        if name in ("tm_group_fill", "tm_gather_fill"):
            fills.append(name)
            torch.cuda._sleep(100_000_000)

    monkeypatch.setattr(tg._lib, "call", slow_fill)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        assert plan.struct(H) is not None
        assert fills and side.query()


@pytest.mark.parametrize("etype,n,form", [("tetra", 6, "laplace"), ("tetra", 6, "elasticity"), ("tetra10", 3, "laplace"),
                                          ("tetra10", 3, "elasticity")])
def test_first_calls_of_a_mesh_on_two_streams(etype, n, form):
    """A mesh's first call on one stream and its second on another, with no
    order between the two, give the values of a later call on the device's
    default stream."""
    pts, el = (curved if etype == "tetra10" else ragged)(etype, n, 5)
    x, k = torch.tensor(pts, device=DEV), torch.rand(el.shape[0], dtype=torch.float64, device=DEV) + 0.5
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        asm = FORMS[form].from_mesh(tg.Mesh(points=x, cells={etype: torch.tensor(el, device=DEV)}), 2)
    got = []
    for s in streams[::-1] + streams:
        with torch.cuda.stream(s):
            got.append(asm(x, element_data={"kappa": k}).values)
    torch.cuda.synchronize()
    ref = asm(x, element_data={"kappa": k}).values
    assert all(torch.equal(v, ref) for v in got)


# -- alignment ---------------------------------------------------------------------
@pytest.mark.parametrize("word", [1, 2, 3])
def test_connectivity_at_an_odd_address(word):
    """A tetrahedral connectivity that starts at any word of a larger array:
    loads, matrices and gradients are those of a connectivity of its own."""
    pts, el = ragged("tetra", 4, word)
    x, own = torch.tensor(pts, device=DEV), torch.tensor(el, device=DEV, dtype=torch.int32)
    flat = torch.zeros(own.numel() + word, dtype=torch.int32, device=DEV)
    flat[word:] = own.reshape(-1)
    view = flat[word:].view(-1, 4)
    load = tg.const_node_assembler(2.0)
    assert torch.equal(load.from_elements(x, {"tetra": view}, 2, DEV, torch.float64)(x),
                       load.from_elements(x, {"tetra": own}, 2, DEV, torch.float64)(x))
    k = torch.rand(el.shape[0], dtype=torch.float64, device=DEV) + 0.5
    got = []
    for cells in (view, own):
        xg = x.clone().requires_grad_(True)
        v = KappaLaplace(tg.assemble.topology_for(cells, x, "tetra"), x, 2)(xg, element_data={"kappa": k}).values
        got.append((v, *torch.autograd.grad(v.square().sum(), xg)))
    assert all(torch.equal(a, b) for a, b in zip(*got))


# -- limits ------------------------------------------------------------------------
def test_block_groups_of_too_many_entries_are_marked():
    """34 rows of a regular mesh have about 510 entries, 64 of them about 960:
    the count refuses what a CTA of 512 threads does not hold."""
    mesh = tg.Mesh.gen_unit_cube(8, device=DEV)
    topo = KappaLaplace.from_mesh(mesh).topology
    g, pat = topo.gather, topo.pattern
    for rows, quads, refused in ((64, 0, 1), (16, 0, 0), (64, 1, 0)):
        sizes = torch.empty((-(-topo.n_points // rows), 3), dtype=torch.int32, device=DEV)
        cnt, bad = torch.empty(pat.nnz, dtype=torch.int32, device=DEV), torch.empty(1, dtype=torch.int32, device=DEV)
        tg._lib.call("tm_group_count", 4, topo.n_points, rows, quads, g.order.data_ptr(), g.nptr.data_ptr(),
                     g.nrec.data_ptr(), pat.indptr.data_ptr(), pat.slots.data_ptr(), cnt.data_ptr(),
                     sizes.data_ptr(), bad.data_ptr(), tg._lib.stream_handle(torch.device(DEV)))
        assert int(bad) == refused


# -- elements outside the common exponent's window -----------------------------------
@pytest.mark.parametrize("etype,n,forms", [("tetra", 8, ("laplace", "mass", "elasticity")),
                                           ("triangle", 24, ("laplace", "mass", "elasticity")),
                                           ("tetra10", 4, ("laplace", "mass", "elasticity")),
                                           ("triangle6", 9, ("laplace",))])
def test_a_far_coefficient_changes_its_own_surroundings_only(etype, n, forms):
    """One element outside the window makes the rows near it add in native
    FP64; the others keep the bits they have without it."""
    base = tg.Mesh.gen_unit_square(n) if etype.startswith("tri") else tg.Mesh.gen_unit_cube(n)
    mesh = (base.to_p2() if etype in ("tetra10", "triangle6") else base).to(DEV)
    cells = mesh.cells[etype]
    g = torch.Generator(device=DEV).manual_seed(n)
    x = mesh.points + 0.1 / n * torch.rand(mesh.points.shape, generator=g, device=DEV, dtype=torch.float64)
    k = torch.exp(torch.randn(cells.shape[0], generator=g, device=DEV, dtype=torch.float64))
    far = k.clone()
    far[-1] *= 2.0 ** 70
    near = cells[-1].long()
    for form in forms:
        asm = FORMS[form].from_mesh(mesh, 2)
        a, b = (asm(x, element_data={"kappa": c}) for c in (k, far))
        H = a.shape[0] // x.shape[0]
        plan = asm.topology.gather
        group = torch.arange(x.shape[0], device=DEV)
        if plan.p1:
            group[plan.order.long()] = group.clone()
        group //= plan.struct(H).rows_per_cta
        rows = ~torch.isin(group, group[near]).repeat_interleave(H)[a.row]
        assert int(rows.sum()) > 500 and torch.equal(a.values[rows], b.values[rows])

    class PointLoad(tg.NodeAssembler):
        def forward(self, v, f):
            return v * f

    load, f = PointLoad.from_mesh(mesh, 2), torch.rand(x.shape[0], generator=g, device=DEV, dtype=torch.float64)
    f2 = f.clone()
    f2[cells[-1, 0].long()] *= 2.0 ** 70
    a, b = (load(x, point_data={"f": c}) for c in (f, f2))
    touched = torch.isin(cells, cells[-1, 0]).any(1)
    away = ~torch.isin(torch.arange(x.shape[0], device=DEV), cells[touched])
    assert int(away.sum()) > 100 and torch.equal(a[away], b[away])


# -- flat elements: native FP64, kept as doubles -----------------------------------------
FLAT = {"triangle": [[0, 0], [1, 0], [0.25, 1]], "tetra": [[0, 0, 0], [1, 0, 0], [0.5, 1, 0], [0.25, 0.25, 1]]}


def flat_mesh(etype, heights):
    """Disjoint elements of the given heights (their last coordinate's factor),
    every coordinate and edge a short dyadic number."""
    corners = np.array(FLAT["triangle" if etype.startswith("tri") else "tetra"])
    pts, el = [], []
    for i, h in enumerate(heights):
        x = corners * np.array([1.0] * (corners.shape[1] - 1) + [h])
        x[:, 0] += 4.0 * i
        pts.append(x)
        el.append(np.arange(len(x)) + i * len(x))
    mesh = tg.Mesh(points=torch.tensor(np.concatenate(pts)),
                   cells={"triangle" if corners.shape[1] == 2 else "tetra": torch.tensor(np.array(el))})
    mesh = mesh.to_p2() if etype in ("triangle6", "tetra10") else mesh
    return mesh.points.numpy(), mesh.cells[etype].numpy()


def longdouble_elements(pts, el, etype, form, q, coef, lam=0.0, mu=0.0):
    """Element matrices (load: vectors) in extended precision from the double
    tables, weights and coefficients the kernels are given."""
    L = np.longdouble
    t = tg.element.kernel_tables(etype, q, torch.device("cpu")).double().numpy().astype(L)
    Q, B, D = tg.element.n_quadrature(etype, q), el.shape[1], pts.shape[1]
    w, N, dN = t[:Q], t[Q:Q + Q * B].reshape(Q, B), t[Q + Q * B:Q + Q * B + Q * B * D].reshape(Q, B, D)
    x = (pts[el] - pts[el[:, :1]]).astype(L)
    total = 0
    for k in range(Q):
        J = np.einsum("bi,ebj->eij", dN[k], x)
        if D == 2:
            adj = np.stack([np.stack([J[:, 1, 1], -J[:, 0, 1]], 1), np.stack([-J[:, 1, 0], J[:, 0, 0]], 1)], 1)
        else:
            adj = np.stack([np.cross(J[:, 1], J[:, 2]), np.cross(J[:, 2], J[:, 0]), np.cross(J[:, 0], J[:, 1])], 2)
        det = (J[:, 0] * adj[:, :, 0]).sum(1)
        g = np.einsum("bi,eji->ebj", dN[k], adj)
        s, v = coef.astype(L) * w[k] / abs(det), coef.astype(L) * w[k] * abs(det)
        if form == "load":
            total = total + v[:, None] * N[k]
        elif form == "mass":
            total = total + v[:, None, None] * (N[k][:, None] * N[k])
        elif form == "laplace":
            total = total + s[:, None, None] * np.einsum("eaj,ebj->eab", g, g)
        else:
            blk = L(lam) * np.einsum("eai,ebj->eaibj", g, g) + L(mu) * np.einsum("eaj,ebi->eaibj", g, g)
            blk = blk + L(mu) * np.einsum("eab,ij->eaibj", np.einsum("eaj,ebj->eab", g, g), np.eye(D))
            total = total + s[:, None, None, None, None] * blk
    return total


def element_values(pts, el, etype, form, q, coef):
    """(values [E, ...] of the disjoint elements as assembled, lam, mu)."""
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV), cells={etype: torch.tensor(el, device=DEV)})
    E, B, D = el.shape[0], el.shape[1], pts.shape[1]
    c = torch.tensor(coef, device=DEV)
    if form == "load":
        class PointLoad(tg.NodeAssembler):
            def forward(self, v, f):
                return v * f

        nodal = torch.zeros(pts.shape[0], dtype=torch.float64, device=DEV)
        nodal[mesh.cells[etype].long()] = c[:, None].expand(E, B)
        out = PointLoad.from_mesh(mesh, q)(mesh.points, point_data={"f": nodal})
        return out.cpu().numpy()[el], 0.0, 0.0
    asm = FORMS[form].from_mesh(mesh, q)
    K = asm(mesh.points, element_data={"kappa": c})
    f = next(iter(asm._form_cache.values()))
    H = D if form == "elasticity" else 1
    dense = torch.zeros(E, B * H, B * H, dtype=torch.float64, device=DEV)
    where = torch.empty(pts.shape[0], 2, dtype=torch.int64, device=DEV)
    where[mesh.cells[etype].long()] = torch.stack(torch.meshgrid(torch.arange(E, device=DEV), torch.arange(
        B, device=DEV), indexing="ij"), 2)
    r, s = where[K.row // H], where[K.col // H]
    dense[r[:, 0], r[:, 1] * H + K.row % H, s[:, 1] * H + K.col % H] = K.values
    dense = dense.cpu().numpy()
    return (dense.reshape(E, B, D, B, D) if H > 1 else dense), f.lam, f.mu


@pytest.mark.parametrize("etype,form", [("triangle", "laplace"), ("triangle", "elasticity"), ("tetra", "laplace"),
                                        ("tetra", "elasticity"), ("tetra", "mass"), ("tetra", "load"),
                                        ("tetra10", "laplace"), ("tetra10", "elasticity")])
def test_flat_elements_keep_the_bits_of_fp64(etype, form):
    """Flat elements of dyadic shape (heights 2^-8 .. 2^-30: all of them past
    the double-float bound): cofactors, determinants and their products are
    exact in FP64, which leaves a handful of roundings: eight units of 2^-53 of
    an element's largest entry (the order-1 tables of a tetrahedron are exact
    but for the weight)."""
    h = 2.0 ** -np.linspace(8, 30, 40).round()
    pts, el = flat_mesh(etype, h)
    coef = np.exp(np.random.default_rng(4).normal(size=len(h)))
    got, lam, mu = element_values(pts, el, etype, form, 1, coef)
    ref = longdouble_elements(pts, el, etype, form, 1, coef, lam, mu)
    big = np.abs(ref).reshape(len(h), -1).max(1).reshape([-1] + [1] * (ref.ndim - 1))
    assert float((np.abs(got - ref) / big).max()) <= 8 * 2.0 ** -53


@pytest.mark.parametrize("etype", ["triangle", "triangle6", "tetra", "tetra10"])
@pytest.mark.parametrize("form", ["laplace", "elasticity", "mass", "load"])
def test_values_of_flat_elements_outside_floats_range(etype, form):
    """Stiffness of heights near 1e-27 with large coefficients (values past
    1e38), mass and loads of heights near 1e-51 (below 1e-45): finite, and
    within 1e-12 of the element's largest entry.  The first element is regular
    and sets the common exponent."""
    stiff = form in ("laplace", "elasticity")
    h = np.array([1.0] + [2.0 ** -(90 if stiff else 170)] * 5)
    pts, el = flat_mesh(etype, h)
    coef = np.array([1.0] + [2.0 ** (59 if stiff else 0) * 1.1] * 5)
    got, lam, mu = element_values(pts, el, etype, form, 2, coef)
    ref = longdouble_elements(pts, el, etype, form, 2, coef, lam, mu)
    big = np.abs(ref).reshape(len(h), -1).max(1).reshape([-1] + [1] * (ref.ndim - 1))
    assert np.isfinite(got).all() and float((np.abs(got - ref) / big).max()) <= 1e-12


@pytest.mark.parametrize("etype", ["triangle", "tetra"])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("height", [20.0, 200.0, 3e5])
def test_slivers_of_p1_matrices(etype, form, height):
    """Fans of needles, most of them past the double-float bound, that share
    their rows: the element kernel's native branch."""
    ring = 30
    t = np.arange(ring) * 2 * np.pi / ring
    if etype == "tetra":
        pts = np.concatenate([[[0.0, 0.0, -height], [0.0, 0.0, height]],
                              np.stack([np.cos(t), np.sin(t), 0.1 * np.sin(3 * t)], 1)])
        el = np.array([[0, 2 + k, 2 + (k + 1) % ring, 1] for k in range(ring)], dtype=np.int64)
    else:
        pts = np.concatenate([[[0.0, height]], np.stack([np.cos(t), np.sin(t)], 1)])
        el = np.array([[0, 1 + k, 1 + (k + 1) % ring] for k in range(ring)], dtype=np.int64)
    check(pts, el, etype, form, np.exp(np.random.default_rng(ring).normal(size=ring)))


# -- accuracy against the patch kernels ---------------------------------------------------
def exact_values(x, cells, etype, form, q, k, asm):
    """CSR values in float64 by plain torch (form's Lame constants as given)."""
    w, N = tg.element.shape_values(etype, q)
    xi = tg.element.quadrature(etype, q)[1]
    dN = torch.tensor(tg.element.shape_tables(etype, xi)[1], device=x.device)
    N, D = torch.tensor(N, device=x.device), x.shape[1]
    X, total = x[cells], 0
    for i in range(len(w)):
        J = torch.einsum("bi,ebj->eij", dN[i], X - X[:, :1])
        g, det = torch.einsum("bi,eji->ebj", dN[i], torch.linalg.inv(J)), torch.linalg.det(J).abs()
        cw = (k * float(w[i]) * det)[:, None, None]
        if form == "mass":
            total = total + cw * (N[i][:, None] * N[i])
        elif form == "laplace":
            total = total + cw * (g @ g.transpose(1, 2))
        else:
            f = next(iter(asm._form_cache.values()))
            blk = f.lam * torch.einsum("eai,ebj->eaibj", g, g) + f.mu * torch.einsum("eaj,ebi->eaibj", g, g)
            blk = blk + f.mu * torch.einsum("eab,ij->eaibj", g @ g.transpose(1, 2), torch.eye(D, device=x.device).double())
            total = total + cw[..., None, None] * blk
    n = x.shape[0]
    if form == "elasticity":
        cells = (cells[:, :, None] * D + torch.arange(D, device=x.device)).reshape(cells.shape[0], -1)
        total, n = total.reshape(cells.shape[0], cells.shape[1], -1), n * D
    uniq, inv = torch.unique((cells[:, :, None] * n + cells[:, None, :]).reshape(-1), return_inverse=True)
    return torch.zeros(uniq.shape[0], dtype=x.dtype, device=x.device).index_add(0, inv, total.reshape(-1))


def both_routes(etype, n, form, q, monkeypatch):
    """Relative 2-norm errors of the float64 values, (all, diagonal), of the
    element-once and of the patch kernels, over four jittered meshes."""
    base = (tg.Mesh.gen_unit_square if etype.startswith("tri") else tg.Mesh.gen_unit_cube)(n)
    mesh = (base.to_p2() if etype in ("triangle6", "tetra10") else base).to(DEV)
    cells, err = mesh.cells[etype].long(), np.zeros((2, 2))
    move = 0.05 if etype in ("triangle6", "tetra10") else 0.2
    for seed in range(4):
        g = torch.Generator(device=DEV).manual_seed(seed)
        x = mesh.points + move / n * (2 * torch.rand(mesh.points.shape, generator=g, device=DEV, dtype=torch.float64) - 1)
        k = torch.exp(torch.randn(cells.shape[0], generator=g, device=DEV, dtype=torch.float64))
        asm = FORMS[form].from_mesh(mesh, q)
        for route, least in enumerate((0, 1 << 40)):
            monkeypatch.setattr("tensormesh_gb300.assemble._GATHER_MIN_ELEMENTS", {etype: least})
            assert asm.topology.element_once == (least == 0)
            K = asm(x, element_data={"kappa": k})
            ref = exact_values(x, cells, etype, form, q, k, asm)
            d, on = K.values - ref, K.row == K.col
            err[route] += float(d.norm() / ref.norm()), float(d[on].norm() / ref[on].norm())
    return err


@pytest.mark.parametrize("etype,n", [("triangle", 60), ("tetra", 12), ("triangle6", 24), ("tetra10", 6)])
@pytest.mark.parametrize("q", [1, 2])
def test_mass_matrices_are_as_accurate_as_the_patch_kernels(etype, n, q, monkeypatch):
    once, patch = both_routes(etype, n, "mass", q, monkeypatch)
    assert (once <= patch).all(), (once, patch)


@pytest.mark.parametrize("etype,n", [("triangle", 60), ("tetra", 12)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("q", [1, 2])
def test_p1_stiffness_is_as_accurate_as_the_patch_kernels(etype, n, form, q, monkeypatch):
    once, patch = both_routes(etype, n, form, q, monkeypatch)
    assert (once <= patch).all(), (once, patch)


@pytest.mark.parametrize("etype,n", [("triangle6", 24), ("tetra10", 6)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("q", [1, 2, 3])
def test_p2_stiffness_is_as_accurate_as_the_patch_kernels(etype, n, form, q, monkeypatch):
    once, patch = both_routes(etype, n, form, q, monkeypatch)
    assert (once <= patch).all(), (once, patch)


def on_regular_meshes(etype, sizes, form, q, monkeypatch):
    """Relative 2-norm errors of the float64 values, element-once and patch
    kernels, summed over regular meshes: the geometry's roundings are the same
    in all elements of one and average out over the sizes only."""
    err = np.zeros(2)
    for n in sizes:
        base = (tg.Mesh.gen_unit_square if etype.startswith("tri") else tg.Mesh.gen_unit_cube)(n)
        mesh = (base.to_p2() if etype in ("triangle6", "tetra10") else base).to(DEV)
        cells = mesh.cells[etype].long()
        g = torch.Generator(device=DEV).manual_seed(n)
        k = torch.exp(torch.randn(cells.shape[0], generator=g, device=DEV, dtype=torch.float64))
        asm = FORMS[form].from_mesh(mesh, q)
        for route, least in enumerate((0, 1 << 40)):
            monkeypatch.setattr("tensormesh_gb300.assemble._GATHER_MIN_ELEMENTS", {etype: least})
            values = asm(mesh.points, element_data={"kappa": k}).values
            ref = exact_values(mesh.points, cells, etype, form, q, k, asm)
            err[route] += float((values - ref).norm() / ref.norm())
    return err


@pytest.mark.parametrize("etype,sizes,q", [("triangle", (20, 27, 33, 47, 60, 100, 150, 255), 1),
                                           ("triangle", (20, 27, 33, 47, 60, 100, 150, 255), 2),
                                           ("triangle6", (10, 27, 39, 50, 51, 57, 75, 79), 2),
                                           ("tetra", (8, 10, 13, 17, 21, 28), 2), ("tetra10", (4, 5, 6, 7, 8, 10), 2)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
def test_stiffness_of_regular_meshes_is_as_accurate_as_the_patch_kernels(etype, sizes, q, form, monkeypatch):
    once, patch = on_regular_meshes(etype, sizes, form, q, monkeypatch)
    assert once <= patch, (once, patch)


@pytest.mark.parametrize("etype,sizes", [("triangle", (20, 31, 57, 100, 150, 255)), ("tetra", (8, 10, 13, 17, 21, 28))])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
def test_gradients_of_p1_matrices_are_as_accurate_as_the_patch_form(etype, sizes, form, monkeypatch):
    """float32 gradients of the coefficient and the points against float64
    ones, summed over regular meshes."""
    err = np.zeros((2, 2))
    struct = tg.plan.GatherPlan.struct
    for n in sizes:
        mesh = (tg.Mesh.gen_unit_square if etype == "triangle" else tg.Mesh.gen_unit_cube)(n).to(DEV)
        asm = FORMS[form].from_mesh(mesh, 2)
        g = torch.Generator(device=DEV).manual_seed(n)
        k32 = torch.exp(torch.randn(mesh.cells[etype].shape[0], generator=g, device=DEV))
        x32, G = mesh.points.float(), None

        def gradients(dtype, patch):
            nonlocal G
            monkeypatch.setattr(tg.plan.GatherPlan, "struct", lambda p, H: None if H == 0 and patch else struct(p, H))
            x, k = x32.to(dtype).requires_grad_(), k32.to(dtype).requires_grad_()
            K = asm(x, element_data={"kappa": k})
            if G is None:
                G = torch.randn(K.values.shape[0], generator=g, device=DEV)
            return torch.autograd.grad(K.values, (k, x), G.to(dtype))
        exact = gradients(torch.float64, True)
        for route in range(2):
            got = gradients(torch.float32, bool(route))
            err[route] += [float((a.double() - b).norm() / b.norm()) for a, b in zip(got, exact)]
    assert (err[0] <= err[1]).all(), err


@pytest.mark.parametrize("etype,n", [("triangle6", 9), ("tetra10", 4)])
@pytest.mark.parametrize("form", ["laplace", "mass", "elasticity"])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_edge_nodes_in_another_order(etype, n, form, dtype, monkeypatch):
    """Tables and connectivity with the nodes on the edges in another order
    than the framework's (a caller of the C entry may have one): the same
    matrix, whose Jacobians no longer start from the vertices alone."""
    base = tg.Mesh.gen_unit_square(n) if etype == "triangle6" else tg.Mesh.gen_unit_cube(n)
    mesh = base.to_p2().to(DEV)
    B, D = mesh.cells[etype].shape[1], mesh.points.shape[1]
    g = torch.Generator(device=DEV).manual_seed(n)
    x = (mesh.points + 0.05 / n * torch.rand(mesh.points.shape, generator=g, device=DEV, dtype=torch.float64)).to(dtype)
    k = torch.exp(torch.randn(mesh.cells[etype].shape[0], generator=g, device=DEV, dtype=torch.float64)).to(dtype)
    Q = tg.element.n_quadrature(etype, 2)
    order = torch.arange(B, device=DEV)
    order[D + 1:] = order[D + 1:].flip(0).roll(1)
    K = FORMS[form].from_mesh(mesh, 2)(x, element_data={"kappa": k})
    plain = tg.element.kernel_tables
    t = plain(etype, 2, torch.device(DEV))
    N, dN = t[Q:Q + Q * B].view(Q, B)[:, order], t[Q + Q * B:Q + Q * B + Q * B * D].view(Q, B, D)[:, order]
    other = torch.cat([t[:Q], N.reshape(-1), dN.reshape(-1)])
    turned = tg.Mesh(points=mesh.points, cells={etype: mesh.cells[etype][:, order].contiguous()})
    asm = FORMS[form].from_mesh(turned, 2)
    asm(x, element_data={"kappa": k})   # the form is recognised with the framework's tables
    monkeypatch.setattr(tg.element, "kernel_tables", lambda *a: other)
    L = asm(x, element_data={"kappa": k})
    assert asm.topology.element_once
    assert torch.equal(L.indptr, K.indptr) and torch.equal(L.indices, K.indices)
    # the same sums in another order and grouping: float64 within 1e-13 of the largest, float32 within 4e-6
    bar = 1e-13 if dtype == torch.float64 else 4e-6
    assert float((L.values - K.values).abs().max()) <= bar * float(K.values.abs().max())


# -- native FP64 -------------------------------------------------------------------
@pytest.mark.parametrize("how", ["instance", "class"])
@pytest.mark.parametrize("kind", ["matrix", "load"])
def test_the_first_native_call_can_be_captured(how, kind):
    """Its plan is there when the precision is chosen, so that the first call
    runs inside a CUDA graph (the tables come from an earlier call of any
    assembler of this order)."""
    pts, el = ragged("tetra", 5, 2)
    base = KappaLaplace if kind == "matrix" else tg.const_node_assembler(2.0)
    cls = type("Native", (base,), {"precision": "native"} if how == "class" else {})
    x = torch.tensor(pts, device=DEV)
    kw = {"element_data": {"kappa": torch.ones(el.shape[0], dtype=torch.float64, device=DEV)}} if kind == "matrix" else {}
    cells = lambda: {"tetra": torch.tensor(el, device=DEV)}  # noqa: E731
    values = lambda a: a(x, **kw).values if kind == "matrix" else a(x)  # noqa: E731
    emulated = values(base.from_mesh(tg.Mesh(points=x, cells=cells()), 2))
    asm = cls.from_mesh(tg.Mesh(points=x, cells=cells()), 2)
    if how == "instance":
        asm.precision = "native"
    if kind == "matrix":   # recognising the form runs host code, not kernels
        asm._resolve_form(None, kw["element_data"], {}, {})
    tg.set_input_checks(False)
    try:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = values(asm)
    finally:
        tg.set_input_checks(True)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(values(asm), out)
    assert float((out - emulated).abs().max()) <= 1e-12 * float(emulated.abs().max())


# -- units, position and coefficients of P1 stiffness ----------------------------------------
@pytest.mark.parametrize("etype,n", [("triangle", 7), ("tetra", 4)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("scale", [1e-9, 1e-3, 1e3, 1e9])
def test_units_of_p1_stiffness(etype, n, form, scale):
    pts, el = ragged(etype, n, 11)
    check(pts * scale, el, etype, form, np.exp(np.random.default_rng(n).normal(size=el.shape[0])))


@pytest.mark.parametrize("etype,n", [("triangle", 7), ("tetra", 4)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
def test_p1_stiffness_far_from_the_origin(etype, n, form):
    """The oracle works on the same coordinates moved back, an exact
    subtraction: its own Jacobian sums would cancel."""
    pts, el = ragged(etype, n, 12)
    shift = np.array([12345.0, -23456.0, 3456.0])[: pts.shape[1]]
    away = pts + shift
    kappa = np.exp(np.random.default_rng(n).normal(size=el.shape[0]))
    mesh = tg.Mesh(points=torch.tensor(away, device=DEV), cells={etype: torch.tensor(el, device=DEV)})
    asm = FORMS[form].from_mesh(mesh, quadrature_order=2)
    got = asm(mesh.points, element_data={"kappa": torch.tensor(kappa, device=DEV)}).values.cpu().numpy()
    ref = fem.assemble_csr(away - shift, el, etype, form, 2, coef=kappa)[2]
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("etype,n", [("triangle", 7), ("tetra", 4)])
@pytest.mark.parametrize("form", ["laplace", "elasticity"])
@pytest.mark.parametrize("size", [1e150, 1e-150])
def test_coefficients_of_p1_stiffness_beyond_float_range(etype, n, form, size):
    pts, el = ragged(etype, n, 13)
    kappa = np.exp(np.random.default_rng(n).normal(size=el.shape[0]))
    check(pts, el, etype, form, size * kappa)
    check(pts, el, etype, form, kappa * np.where(np.arange(el.shape[0]) % 97 == 0, 1e80, 1.0))


def test_block_patterns_are_complete_when_they_become_visible(monkeypatch):
    mesh = tg.Mesh.gen_unit_cube(4, device=DEV)
    topo = KappaLaplace.from_mesh(mesh).topology
    inner = tg.assemble.block_pattern

    def slow(*args):
        out = inner(*args)
        torch.cuda._sleep(100_000_000)
        return out

    monkeypatch.setattr("tensormesh_gb300.assemble.block_pattern", slow)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        topo.dof_pattern(3)
        assert side.query()


@pytest.mark.parametrize("etype,n", [("tetra", 8), ("triangle", 24), ("tetra10", 4), ("triangle6", 9)])
@pytest.mark.parametrize("first", [2.0 ** 70, 2.0 ** -70, 0.0])
def test_an_outlying_first_element_leaves_the_others_in_the_window(etype, n, first):
    """The first element's coefficient (load: its nodes') far from the others',
    or zero: rows that share no group with it keep the bits they have without
    it, that is, they still add in pairs."""
    base = tg.Mesh.gen_unit_square(n) if etype.startswith("tri") else tg.Mesh.gen_unit_cube(n)
    mesh = (base.to_p2() if etype in ("tetra10", "triangle6") else base).to(DEV)
    cells = mesh.cells[etype].long()
    g = torch.Generator(device=DEV).manual_seed(n)
    x = mesh.points + 0.1 / n * torch.rand(mesh.points.shape, generator=g, device=DEV, dtype=torch.float64)
    # coefficients of another scale than one, so that a window around one would miss them
    k = 2.0 ** 100 * torch.exp(torch.randn(cells.shape[0], generator=g, device=DEV, dtype=torch.float64))
    far = k.clone()
    far[0] *= first
    for form in ("laplace", "mass", "elasticity"):
        asm = FORMS[form].from_mesh(mesh, 2)
        a, b = (asm(x, element_data={"kappa": c}) for c in (k, far))
        H = a.shape[0] // x.shape[0]
        plan = asm.topology.gather
        group = torch.arange(x.shape[0], device=DEV)
        if plan.p1:
            group[plan.order.long()] = group.clone()
        group //= plan.struct(H).rows_per_cta
        rows = ~torch.isin(group, group[cells[0]]).repeat_interleave(H)[a.row]
        assert int(rows.sum()) > 500 and torch.equal(a.values[rows], b.values[rows])

    class PointLoad(tg.NodeAssembler):
        def forward(self, v, f):
            return v * f

    load = PointLoad.from_mesh(mesh, 2)
    f = 2.0 ** 100 * (torch.rand(x.shape[0], generator=g, device=DEV, dtype=torch.float64) + 0.5)
    f2 = f.clone()
    f2[cells[0]] *= first
    a, b = (load(x, point_data={"f": c}) for c in (f, f2))
    away = torch.ones(x.shape[0], dtype=torch.bool, device=DEV)
    away[cells[torch.isin(cells, cells[0]).any(1)]] = False
    assert int(away.sum()) > 100 and torch.equal(a[away], b[away])


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_nodes_too_full_for_the_smallest_group_keep_the_patch_kernels(dtype):
    """Two apexes of 242 neighbours side by side: no group of eight block rows
    that holds both has at most 512 entries, so elasticity takes the patches."""
    ring = 240
    t = np.arange(ring) * 2 * np.pi / ring
    rim = np.stack([np.cos(t), np.sin(t), 0.8 * np.sin(3 * t)], 1)
    pts = np.concatenate([[[-0.3, -0.2, 0.1], [-0.3, -0.2, 0.12]], rim])
    el = np.array([[0, 2 + k, 2 + (k + 1) % ring, 1] for k in range(ring)], dtype=np.int64)
    coef = np.exp(np.random.default_rng(ring).normal(size=ring))
    mesh = tg.Mesh(points=torch.tensor(pts, device=DEV), cells={"tetra": torch.tensor(el, device=DEV)})
    plan = KappaLaplace.from_mesh(mesh).topology.gather
    assert plan.struct(1) is not None and plan.struct(3) is None
    check(pts, el, "tetra", "elasticity", coef, dtype)
    check(pts, el, "tetra", "laplace", coef, dtype)
