"""The SELL solver's launch modes (one cluster, a resident grid, streaming) and
its grid-wide sums: fixed-point sums against exact ones, a wait that runs out,
and systems whose rows are too uneven for a CTA's shared memory."""
import ctypes
import math

import numpy as np
import pytest
import torch

import tensormesh_gb300 as tg
from tensormesh_gb300 import _lib, solve as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


def grid_sum(vals, blocks, absent=0, rounds=3, spins=1 << 20):
    out = torch.zeros(2 * blocks, dtype=torch.float64, device=DEV)
    work = torch.empty(8192 + 64 * blocks, dtype=torch.uint8, device=DEV)
    status = ctypes.c_int32(-1)
    st = _lib.call_status("tm_selftest_grid_sum", blocks, absent, rounds, spins, vals.data_ptr(), out.data_ptr(),
                          ctypes.byref(status), work.data_ptr(), work.numel(),
                          torch.cuda.current_stream().cuda_stream)
    assert st == _lib.TM_OK
    return out.view(blocks, 2).cpu(), status.value


@pytest.mark.parametrize("blocks", [2, 5, 32, 33, 152])
@pytest.mark.parametrize("kind", ["normal", "squares", "wide", "cancel", "zeros", "powers"])
def test_grid_sums_against_exact(blocks, kind):
    """Every CTA holds the same bits, within three roundings of 2^-53 (a CTA's,
    the grid's and the truncations) of the exact sum, relative to the largest
    partial result."""
    rng = np.random.default_rng(blocks)
    n = blocks * 512
    v = rng.normal(size=n)
    if kind == "squares":
        v = v * v
    elif kind == "wide":
        v = v * np.exp(30 * rng.normal(size=n))
    elif kind == "cancel":
        v[1::2] = -v[::2] * (1 + 1e-9)
    elif kind == "zeros":
        v[rng.random(n) < 0.9] = 0.0
        v[:512] = 0.0
    elif kind == "powers":
        v = np.ldexp(1.0, rng.integers(-40, 40, size=n)) * rng.choice([-1, 1], size=n)
    out, status = grid_sum(torch.tensor(v, device=DEV), blocks)
    assert status == 0
    assert torch.equal(out, out[:1].expand(blocks, 2))
    parts = [math.fsum(c) for c in v.reshape(blocks, 512)]
    scale = max(max(abs(p) for p in parts), abs(math.fsum(v)), np.abs(v).max())
    assert abs(float(out[0, 0]) - math.fsum(v)) <= (blocks + 2) * 2.0 ** -53 * scale
    assert abs(float(out[0, 1]) + 0.5 * math.fsum(v)) <= (blocks + 2) * 2.0 ** -53 * scale


def test_grid_sum_of_nan_is_nan():
    v = torch.ones(4 * 512, dtype=torch.float64, device=DEV)
    v[700] = float("nan")
    out, _ = grid_sum(v, 4)
    assert bool(torch.isnan(out).all())


def test_grid_sum_times_out_and_the_context_survives():
    v = torch.ones(8 * 512, dtype=torch.float64, device=DEV)
    _, status = grid_sum(v, 8, absent=1, spins=1 << 14)
    assert status == _lib.TM_ERR_TIMEOUT
    out, status = grid_sum(v, 8)
    assert status == 0 and float(out[0, 0]) == 4096.0


def poisson(dim, n, dtype):
    mesh = (tg.Mesh.gen_unit_square if dim == 2 else tg.Mesh.gen_unit_cube)(n, device=DEV, dtype=dtype)
    K = tg.LaplaceElementAssembler.from_mesh(mesh, quadrature_order=1)(mesh.points)
    b = tg.const_node_assembler(1.0).from_mesh(mesh, quadrature_order=1)(mesh.points)
    return tg.Condenser(mesh.boundary_mask)(K, b)


# 2 to 16 rows; one cluster; both sides of its shared memory; the resident grid; streaming
@pytest.mark.parametrize("dim,n", [(2, 2), (2, 3), (2, 64), (2, 150), (2, 190), (3, 40), (2, 600), (3, 80)])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.filterwarnings("ignore:PCG did not converge")   # float32: the residual's floor, see below
def test_every_mode_solves(dim, n, dtype):
    K, f = poisson(dim, n, dtype)
    rtol = 1e-9 if dtype == torch.float64 else 1e-4
    u = K.solve(f, rtol=rtol)
    info = K.last_solve_info
    # the rounding of K x in the value type floors the residual that can be reached
    eps = torch.finfo(dtype).eps
    floor = eps * float(((K.with_values(K.values.abs()) @ u.abs()).norm() / f.norm()))
    assert info.status == 0 and info.residual <= rtol + 4 * floor
    assert torch.equal(K.solve(f, rtol=rtol), u)          # bitwise repeatable
    x = torch.zeros_like(f)
    S.LAYOUT = "csr"
    try:
        ref = S.pcg_jacobi_raw(K.indptr, K.indices, K.values, f, x, rtol, 0.0, 100000)
    finally:
        S.LAYOUT = "sell"
    if info.restarts == ref.restarts == 0:   # corrections at the floor are not comparable
        assert abs(ref.iterations - info.iterations) <= max(2, ref.iterations // 50)
    assert float((u - x).norm() / x.norm()) <= (1e-6 if dtype == torch.float64 else 5e-2)


@pytest.mark.parametrize("n", [3000, 60000])
def test_uneven_rows_fall_back_to_global_memory(n):
    """The first 320 rows hold 200 entries each, the others three: the share of
    the first CTA exceeds its shared memory's entries."""
    rng = np.random.default_rng(n)
    import scipy.sparse as sp
    rows = np.repeat(np.arange(320), 100)
    cols = rng.integers(320, n, size=rows.shape[0])
    A = sp.coo_matrix((rng.uniform(-1, 1, size=rows.shape[0]), (rows, cols)), shape=(n, n))
    A = A + A.T + sp.diags([np.full(n - 1, -1.0), np.full(n - 1, -1.0)], [1, -1])
    A = (A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 0.1)).tocsr()
    A.sort_indices()
    b = rng.normal(size=n)
    K = tg.SparseMatrix(torch.tensor(A.data, device=DEV), shape=(n, n),
                        indptr=torch.tensor(A.indptr.astype(np.int64), device=DEV),
                        indices=torch.tensor(A.indices.astype(np.int32), device=DEV))
    x = K.solve(torch.tensor(b, device=DEV), rtol=1e-11)
    assert np.linalg.norm(A @ x.cpu().numpy() - b) <= 1e-10 * np.linalg.norm(b)


def test_iteration_cap_zero_and_one():
    K, f = poisson(2, 20, torch.float64)
    for cap in (0, 1):
        with pytest.warns(UserWarning, match="did not converge"):
            K.solve(f, rtol=1e-10, maxiter=cap)
        assert K.last_solve_info.iterations == cap and K.last_solve_info.status == _lib.TM_ERR_MAXITER


@pytest.mark.parametrize("n", [600_001, 1_000_000, 1_500_033, 2_500_000, 3_800_001])
@pytest.mark.parametrize("far", [1000, 40_000])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_streaming_grid_sizes(n, far, dtype):
    """Systems too large for shared memory, with four to none of the own-row
    vectors held there, 16-bit and 32-bit columns: the residual, formed by
    torch in float64, against the tolerance asked for (condition number below
    nine, so float32 reaches 1e-4 with a rounding floor near 1e-6)."""
    i = torch.arange(n, device=DEV)
    offs = torch.tensor([-far, -1, 0, 1, far], device=DEV)
    cols = i[:, None] + offs
    inside = (cols >= 0) & (cols < n)
    g = torch.Generator(device=DEV).manual_seed(n)
    scale = torch.exp(torch.randn(n, generator=g, device=DEV, dtype=torch.float64))   # Jacobi undoes it
    base = torch.tensor([-1.0, -1.0, 5.0, -1.0, -1.0], device=DEV, dtype=torch.float64).expand(n, 5)
    vals = (base * (scale[:, None] * scale[cols.clamp(0, n - 1)]).sqrt())[inside].to(dtype)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(inside.sum(1), 0)
    K = tg.SparseMatrix(vals, shape=(n, n), indptr=indptr, indices=cols[inside].to(torch.int32))
    b = torch.randn(n, generator=g, device=DEV, dtype=torch.float64).to(dtype)
    rtol = 1e-9 if dtype == torch.float64 else 1e-4
    x = K.solve(b, rtol=rtol)
    assert K.last_solve_info.status == 0
    A = torch.sparse_csr_tensor(indptr, K.indices.long(), vals.double(), size=(n, n))
    res = b.double() - (A @ x.double()[:, None])[:, 0]
    assert float(res.norm() / b.double().norm()) <= rtol * (1.0 if dtype == torch.float64 else 1.1)
    assert torch.equal(K.solve(b, rtol=rtol), x)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 255, 257, 480, 511, 512, 513])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_clusters_with_ctas_that_own_no_rows(n, dtype):
    """Fewer slices than the cluster has CTAs, many launches in a row: the
    same bits each time, and the tridiagonal system's dense solution."""
    i = torch.arange(n, device=DEV)
    cols = i[:, None] + torch.tensor([-1, 0, 1], device=DEV)
    inside = (cols >= 0) & (cols < n)
    vals = torch.tensor([-1.0, 4.0, -1.0], device=DEV, dtype=dtype).expand(n, 3)[inside]
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(inside.sum(1), 0)
    K = tg.SparseMatrix(vals, shape=(n, n), indptr=indptr, indices=cols[inside].to(torch.int32))
    b = torch.randn(n, generator=torch.Generator(device=DEV).manual_seed(n), device=DEV, dtype=torch.float64).to(dtype)
    rtol = 1e-12 if dtype == torch.float64 else 1e-5
    x = K.solve(b, rtol=rtol)
    A = 4.0 * torch.eye(n, dtype=torch.float64, device=DEV)
    A -= torch.diag(torch.ones(n - 1, dtype=torch.float64, device=DEV), 1)
    A -= torch.diag(torch.ones(n - 1, dtype=torch.float64, device=DEV), -1)
    ref = torch.linalg.solve(A, b.double())
    # the residual's relative size times the condition number (below three), and the value type's rounding
    assert float((x.double() - ref).norm() / ref.norm()) <= 3 * rtol + 16 * torch.finfo(dtype).eps
    assert all(torch.equal(K.solve(b, rtol=rtol), x) for _ in range(20))


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def renorm(h, l):
    s = h + l
    return s, l - (s - h)


def pair_add(a, b):
    s, e = two_sum(a[0], b[0])
    return renorm(s, e + (a[1] + b[1]))


def pair_mul(a, b):
    def fma(x, y, z):
        return (x.astype(np.float64) * y.astype(np.float64) + z.astype(np.float64)).astype(np.float32)
    p = a[0] * b[0]
    return renorm(p, fma(a[1], b[0], fma(a[0], b[1], fma(a[0], b[0], -p))))


@pytest.mark.parametrize("n,per", [(1500, 7), (3000, 15), (60_000, 15), (900_000, 7)])
def test_row_sums_have_the_error_of_normalised_pairs(n, per):
    """b - A x0 of the kernel's first sweep (a solve of no iterations) where it
    is nothing but the rounding of the row sums: its norm is that of the same
    sums in normalised float pairs on the host.  The last bits of a conversion
    may differ: 5 %, where sums normalised only at the end are at 170 %."""
    rng = np.random.default_rng(n)
    far = min(n // per, 4000)
    cols = (np.arange(n)[:, None] + far * np.arange(per)) % n
    vals = np.exp(rng.normal(size=(n, per))) * rng.choice([-1.0, 1.0], (n, per))
    vals[:, 0] = 1.0                                    # the diagonal: the Jacobi scaling is the identity
    order = np.argsort(cols, 1)
    cols, vals = np.take_along_axis(cols, order, 1), np.take_along_axis(vals, order, 1)
    x = rng.normal(size=n)
    b = (vals.astype(np.longdouble) * x[cols]).sum(1).astype(np.float64)

    def pair(v):
        h = v.astype(np.float32)
        return h, (v - h).astype(np.float32)

    acc = (np.zeros(n, np.float32), np.zeros(n, np.float32))
    for j in range(per):
        acc = pair_add(acc, pair_mul(pair(vals[:, j]), pair(x[cols[:, j]])))
    r = pair_add(pair(b), (-acc[0], -acc[1]))
    expect = np.linalg.norm(r[0].astype(np.float64) + r[1]) / np.linalg.norm(b)
    K = tg.SparseMatrix(torch.tensor(vals.reshape(-1), device=DEV), shape=(n, n),
                        indptr=torch.arange(0, n * per + 1, per, device=DEV),
                        indices=torch.tensor(cols.reshape(-1).astype(np.int32), device=DEV))
    with pytest.warns(UserWarning, match="did not converge"):
        K.solve(torch.tensor(b, device=DEV), x0=torch.tensor(x, device=DEV), rtol=1e-18, maxiter=0)
    got = K.last_solve_info.recurrence_residual
    assert abs(got - expect) <= 0.05 * expect, (got, expect)


@pytest.mark.parametrize("dim,n", [(2, 20), (2, 250), (3, 70)])
def test_workspace_on_eight_bytes(dim, n):
    """A workspace that starts 8 bytes past a 16-byte boundary, in each launch
    mode: the bits of an aligned one."""
    K, f = poisson(dim, n, torch.float64)
    sp, n_pad, narrow = S.sell_plan(K.indptr, K.indices)
    rows = f.shape[0]
    need = _lib.load().tm_pcg_sell_workspace_bytes(_lib.TM_F64, rows, n_pad)
    out = []
    for shift in (0, 8):
        work = torch.empty(need + 16, dtype=torch.uint8, device=DEV)
        at = work.data_ptr() + shift
        assert work.data_ptr() % 16 == 0
        x = torch.zeros_like(f)
        stream = torch.cuda.current_stream().cuda_stream
        _lib.call("tm_pcg_jacobi_sell", _lib.TM_F64, rows, K.indptr.data_ptr(), K.indices.data_ptr(),
                  K.values.data_ptr(), sp.data_ptr(), n_pad, f.data_ptr(), x.data_ptr(), 1e-6, 0.0, 10000,
                  _lib.TM_PCG_STANDARD | (_lib.TM_PCG_NARROW if narrow else 0), at, need, stream)
        it, res, bn = ctypes.c_int32(0), ctypes.c_double(0.0), ctypes.c_double(0.0)
        assert _lib.load().tm_pcg_result(at, ctypes.byref(it), ctypes.byref(res), ctypes.byref(bn), stream) == 0
        out.append((x, it.value))
    assert torch.equal(out[0][0], out[1][0]) and out[0][1] == out[1][1] > 10
