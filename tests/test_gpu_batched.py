"""Batched persistent launch: many uneven 2D P1 Poisson meshes assembled
(float32) and Jacobi-PCG-solved in one launch, replayed from a CUDA graph;
checked per instance against the float64 oracle."""
import numpy as np
import pytest
import torch

import tensormesh_gb300 as tg
from oracle import fem
from tensormesh_gb300.batched import BatchedPoisson

pytestmark = pytest.mark.gpu
DEV = "cuda"


def make_batch(sizes, seed=0):
    meshes = [tg.Mesh.gen_unit_square(int(n), device=DEV) for n in sizes]
    g = torch.Generator().manual_seed(seed)
    kappas = [torch.exp(torch.randn(m.n_elements, generator=g, dtype=torch.float64)) for m in meshes]
    return meshes, kappas


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("cluster,big", [(1, None), (4, None), (2, (8, 2)), (2, (16, 1))])
def test_batched_matches_fp64_oracle(graph, cluster, big, tmp_path, monkeypatch):
    """big = (cluster_big, n_big): the largest instances run in a second,
    concurrent launch on larger clusters."""
    monkeypatch.setenv("TM_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    sizes = [5, 17, 32, 9, 24, 3]
    meshes, kappas = make_batch(sizes)
    cb, nbig = big if big else (None, 0)
    bp = BatchedPoisson(meshes, cluster=cluster, cluster_big=cb, n_big=nbig)
    assert bp.config["n_big"] == nbig
    k = torch.cat(kappas).to(DEV)
    u, info = bp(k, rtol=1e-6, graph=graph)
    torch.cuda.synchronize()
    assert info.status.cpu().tolist() == [0] * len(sizes)
    vals = bp.values.double().cpu().numpy()
    ip = bp.pattern.indptr.cpu().numpy()
    for i, m in enumerate(meshes):
        pts, el = m.points.cpu().numpy(), m.cells["triangle"].cpu().numpy()
        oip, oix, odv = fem.assemble_csr(pts, el, "triangle", "laplace", 1, coef=kappas[i].numpy())
        r0, r1 = bp.node_ptr[i], bp.node_ptr[i + 1]
        got = vals[ip[r0]:ip[r1]]
        assert np.max(np.abs(got - odv)) <= 1e-5 * np.max(np.abs(odv))
        bref = fem.assemble_load(pts, el, "triangle", 1, "const", 1.0)
        bd = m.boundary_mask.cpu().numpy()
        iptr, iind, ival, fi = fem.condense(oip, oix, odv, bd, None, bref)
        if iptr.shape[0] > 1:
            uref = fem.recover(fem.spsolve(iptr, iind, ival, fi), bd)
            uu = u[r0:r1].double().cpu().numpy()
            assert np.max(np.abs(uu - uref)) <= 5e-4 * np.max(np.abs(uref))


@pytest.mark.parametrize("big", [None, (8, 1)])
def test_batched_graph_replay_is_deterministic(big, tmp_path, monkeypatch):
    monkeypatch.setenv("TM_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    meshes, kappas = make_batch([12, 30, 7, 20], seed=1)
    cb, nbig = big if big else (None, 0)
    bp = BatchedPoisson(meshes, cluster=2, cluster_big=cb, n_big=nbig)
    k = torch.cat(kappas).to(DEV)
    u1, _ = bp(k)
    a = u1.clone()
    for _ in range(3):
        u2, _ = bp(k)
        assert torch.equal(u2, a)


def test_autotuner_picks_and_caches(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("TM_AUTOTUNE_CACHE", str(path))
    meshes, kappas = make_batch([10, 40, 25], seed=2)
    bp = BatchedPoisson(meshes)
    k = torch.cat(kappas).to(DEV)
    best = bp.autotune(k, clusters=(1, 2, 4), budgets=(512, 2048), reps=2, big=((None, 0), (8, 1)))
    assert best["cluster"] in (1, 2, 4) and best["slot_budget"] in (512, 2048)
    assert len(best["candidates"]) == 12
    assert path.exists()
    bp2 = BatchedPoisson(meshes)
    again = bp2.autotune(k, clusters=(1, 2, 4), budgets=(512, 2048), big=((None, 0), (8, 1)))
    assert again["cluster"] == best["cluster"] and bp2.config["slot_budget"] == best["slot_budget"]
    assert bp2.config["n_big"] == best["n_big"]
    u, info = bp2(k)
    assert int(info.status.max()) == 0


@pytest.mark.parametrize("exponent", [-60, 40])
def test_units_of_the_source_scale_the_solution_exactly(exponent):
    """The dot products are formed in float pairs on values scaled by powers of
    two, so a source in units 2^-60 or 2^40 gives the same bits, scaled."""
    from tensormesh_gb300.batched import BatchedPoisson
    meshes = [tg.Mesh.gen_unit_square(n, device=DEV) for n in (5, 20, 33)]
    kappa = torch.exp(torch.randn(sum(m.n_elements for m in meshes), device=DEV,
                                  generator=torch.Generator(DEV).manual_seed(2)))
    base, info = BatchedPoisson(meshes)(kappa)
    base, its = base.clone(), info.iterations.clone()
    x, info = BatchedPoisson(meshes, source=2.0 ** exponent)(kappa)
    assert bool((info.status == 0).all()) and torch.equal(info.iterations, its)
    assert torch.equal(x, base * 2.0 ** exponent)


@pytest.mark.parametrize("length", [1, 2, 7, 33, 64])
@pytest.mark.parametrize("kind", ["normal", "squares", "cancel", "small"])
def test_dot_products_of_a_thread_are_as_good_as_fp64(length, kind):
    """A thread's sum of products against the exact one: a unit in the last
    place of a double for the conversion, and the roundings of the third
    float, whose terms are below 2^-47 of the partial sums."""
    import math
    from tensormesh_gb300 import _lib
    rng = np.random.default_rng(length)
    n = 300
    a = rng.normal(size=(length, n)).astype(np.float32)
    b = rng.normal(size=(length, n)).astype(np.float32)
    if kind == "squares":
        b = a.copy()
    elif kind == "cancel":
        b[1::2], a[1::2] = b[:-1:2][:length // 2], -a[:-1:2][:length // 2] * np.float32(1 + 2.0 ** -20)
    elif kind == "small":
        a, b = a * np.float32(2.0 ** -30), b * np.float32(2.0 ** -20)
    out = torch.empty(n, dtype=torch.float64, device=DEV)
    ta, tb = torch.tensor(a, device=DEV), torch.tensor(b, device=DEV)
    _lib.call("tm_selftest_dot", n, length, ta.data_ptr(), tb.data_ptr(), out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    for t in range(n):
        terms = [float(x) * float(y) for x, y in zip(a[:, t], b[:, t])]   # exact: 48 bits
        exact, size = math.fsum(terms), math.fsum(abs(v) for v in terms)
        bound = 2.0 ** -52 * abs(exact) + length ** 2 * 2.0 ** -71 * size
        assert abs(float(out[t]) - exact) <= bound, (t, float(out[t]) - exact, bound)


@pytest.mark.parametrize("left", [2.0 ** -20, 2.0 ** -28, 2.0 ** -36, 0.0])
def test_dot_products_that_cancel_keep_what_is_left(left):
    """Every product is taken back in another order, then one small product is
    added: the bound of the test above, where s + c is no larger than d or
    vanishes."""
    import math
    from tensormesh_gb300 import _lib
    rng = np.random.default_rng(4)
    n, half = 300, 32
    h, g = (rng.normal(size=(half, n)).astype(np.float32) for _ in range(2))
    back = rng.permutation(half)
    last = np.full((1, n), left, np.float32)
    a, b = np.concatenate([h, -h[back], last]), np.concatenate([g, g[back], np.ones_like(last)])
    out = torch.empty(n, dtype=torch.float64, device=DEV)
    ta, tb = torch.tensor(a, device=DEV), torch.tensor(b, device=DEV)
    _lib.call("tm_selftest_dot", n, a.shape[0], ta.data_ptr(), tb.data_ptr(), out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    for t in range(n):
        terms = [float(x) * float(y) for x, y in zip(a[:, t], b[:, t])]   # exact: 48 bits
        exact, size = math.fsum(terms), math.fsum(abs(v) for v in terms)
        bound = 2.0 ** -52 * abs(exact) + a.shape[0] ** 2 * 2.0 ** -71 * size
        assert abs(float(out[t]) - exact) <= bound, (t, float(out[t]) - exact, bound)
