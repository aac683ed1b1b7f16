"""Sparse solve levels with columns around the length that gives a column a CTA of its own, against
the elementwise backward-error bound of substitution."""
from __future__ import annotations

import numpy as np
import pytest

from glu_public_b200 import glu
from tests.test_gpu_dense_solve import check_solve
from tests.test_gpu_dense_steps import check_lu

pytestmark = pytest.mark.gpu
LENGTHS = (1, 31, 33, 64, 65, 128, 191, 192, 193, 500)


def long_columns(n, seed):
    """Columns of the LENGTHS below the diagonal (rows drawn from the last part, so that they do not
    all fill) and the same lengths above it, random short entries elsewhere; dense [n, n]."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    for k, length in enumerate(LENGTHS):
        a[rng.choice(np.arange(n - 520, n), length, replace=False), 3 + 2 * k] = 1.0
        a[rng.choice(np.arange(0, 520), length, replace=False), n - 3 - 2 * k] = 1.0
    short = rng.integers(0, n, (2, 2 * n))
    a[short[0], short[1]] = 1.0
    a *= rng.uniform(-1.0, 1.0, a.shape)
    a[np.arange(n), np.arange(n)] = np.abs(a).sum(0) + np.abs(a).sum(1) + 1.0
    return a


@pytest.mark.parametrize("deterministic", [0, 1])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nrhs,count", [(1, 2), (2, 2), (4, 2), (5, 2), (1, 200), (5, 100)])
def test_long_columns(nrhs, count, transpose, deterministic):
    import torch
    n = 1100
    a = long_columns(n, 7)
    col, row = np.nonzero(a.T)                # column order
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    # no dense block and no fronts: every column goes through the sparse levels
    plan = glu.Plan(sym, dense_threshold=2.0, front_min_w=0, deterministic=deterministic)
    assert plan.stat("nt") == 0
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, count)            # more than 200,000 rows in all: a launch per level
    scale = torch.linspace(1.0, 2.0, count, dtype=torch.float64, device="cuda")
    batch.load_lu_values(scale[:, None] * torch.as_tensor(sym.val, device="cuda"))
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal((count, nrhs, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    cp = sym.sym_c_ptr.astype(np.int64)
    for i in (0, count - 1):
        lu = np.zeros((n, n))                 # [column, row]
        lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        nl = np.diff(cp) - (sym.l_col_ptr.astype(np.int64) - cp[:-1]) - 1
        assert nl.max() >= 192 and (nl < 192).any()
        check_solve(torch, lu, b[i], x[i], transpose)


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nrhs,count", [(1, 1), (3, 2), (1, 250)])
def test_sparse_columns_beside_a_dense_block(nrhs, count, transpose):
    """L21 and the part of U above the dense block, with rows and columns of more and of fewer entries
    than give them a CTA."""
    import torch
    n = 1100
    a = long_columns(n, 5)
    a[n - 260:, n - 260:] += 0.01             # a dense block; row 50 and column 51 reach all of it
    a[50, n - 260:] = 0.02
    a[n - 260:, 51] = 0.03
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, front_min_w=0)
    assert 200 <= plan.stat("nt") < n
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, count)
    batch.load_lu_values(torch.as_tensor(sym.val, device="cuda").repeat(count, 1))
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal((count, nrhs, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    assert not batch.status().any()
    cp = sym.sym_c_ptr.astype(np.int64)
    lu = np.zeros((n, n))
    lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(count - 1).cpu().numpy()
    check_solve(torch, lu, b[count - 1], x[count - 1], transpose)


@pytest.mark.parametrize("options", [{}, dict(sparse_persistent=0), dict(sparse_persistent=0, level_warps_per_sm=0),
                                     dict(sparse_warps_per_col=1, sparse_col_lanes=8),
                                     dict(sparse_warps_per_col=1, sparse_col_lanes=16, sparse_persistent=0),
                                     dict(sparse_warps_per_col=8, sparse_persistent=0),
                                     dict(sparse_warps_per_col=2, sparse_persistent=0),
                                     dict(dense_threshold=0.5)])
def test_long_and_short_pairs(options):
    """Factors of columns with few long pairs, many short ones and both (pairs of a column shared in
    pieces or four at a time), |L U - A| <= 4 n u |L| |U|."""
    import torch
    n = 1100
    a = long_columns(n, 3)
    a[40, 600:] = -0.01                       # long rows of U: many pairs of short columns
    a[41, 41:90] = 0.02
    a[500:900, 41] = 0.03                     # few long pairs
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, **{"dense_threshold": 2.0, "front_min_w": 0, **options})
    batch = glu.Batch(plan, 3)
    batch.load_lu_values(torch.as_tensor(np.stack([sym.val * s for s in (1.0, 2.0, -1.0)]),
                                         device="cuda"))
    batch.refactor(0.0)
    cp = sym.sym_c_ptr.astype(np.int64)
    for i, s in enumerate((1.0, 2.0, -1.0)):
        lu = np.zeros((n, n))                 # [column, row]
        lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_lu(torch, lu, np.ascontiguousarray(a.T * s)[None])


@pytest.mark.parametrize("pairs", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("options", [{}, dict(sparse_persistent=0, sparse_warps_per_col=8, level_warps_per_sm=0),
                                     dict(sparse_persistent=0, sparse_warps_per_col=1, sparse_col_lanes=8)])
def test_a_pair_to_itself(pairs, options):
    """Columns of the LENGTHS with about a pair for each group of lanes that shares them: a pair alone
    takes its rows four at a time.  |L U - A| <= 4 n u |L| |U|."""
    import torch
    n = 1100
    a = long_columns(n, 13)
    for k in range(len(LENGTHS)):
        a[3 + 2 * k, 60 + 20 * k:60 + 20 * k + pairs] = 0.02
    a[np.arange(n), np.arange(n)] += 1.0
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, **{"dense_threshold": 2.0, "front_min_w": 0, **options})
    batch = glu.Batch(plan, 2)
    batch.load_lu_values(torch.as_tensor(np.stack([sym.val, -3.0 * sym.val]), device="cuda"))
    batch.refactor(0.0)
    cp = sym.sym_c_ptr.astype(np.int64)
    for i, s in enumerate((1.0, -3.0)):
        lu = np.zeros((n, n))                 # [column, row]
        lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_lu(torch, lu, np.ascontiguousarray(a.T * s)[None])


@pytest.mark.parametrize("transpose", [False, True])
def test_residual_of_long_rows(transpose):
    """r = b - op(A) x with rows of 63 to 1,100 entries: within 2 n u |A| |x| of numpy's."""
    import torch
    n = 1100
    a = np.diag(np.linspace(1.0, 2.0, n))
    for k, length in enumerate((63, 64, 65, 66, 127, 128, 129, 600, n)):
        a[7 + 40 * k, :length] = np.sin(np.arange(length) + k)
        a[:length, 11 + 40 * k] = np.cos(np.arange(length) + k)
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym)
    plan.set_original_pattern(row, col)
    batch = glu.Batch(plan, 1)
    rng = np.random.default_rng(0)
    x, b = rng.standard_normal((2, 1, 1, n))
    op = a.T if transpose else a
    val = torch.as_tensor(a[row, col][None], device="cuda")
    got = batch.residual(val, torch.as_tensor(b, device="cuda"), torch.as_tensor(x, device="cuda"),
                         transpose=transpose).item()
    r = np.abs(b[0, 0] - op @ x[0, 0]).max()
    den = np.abs(op).sum(1).max() * np.abs(x).max() + np.abs(b).max()
    slack = 2 * n * 2.0 ** -53 * (np.abs(op) @ np.abs(x[0, 0])).max() / den
    assert abs(got - r / den) <= slack + 4 * n * 2.0 ** -53 * r / den


@pytest.mark.parametrize("count", [2, 24])
def test_assembly_of_the_dense_block(count):
    """Columns of the dense block built from the entries and the sparse columns' products, a CTA each
    (count 2) or a warp each (24), beside instances loaded in the filled-pattern order:
    |L U - A| <= 4 n u |L| |U|."""
    import torch
    n, tail = 1100, 300
    rng = np.random.default_rng(9)
    a = np.zeros((n, n))
    a[n - tail:, n - tail:] = rng.uniform(-1.0, 1.0, (tail, tail))
    for c in range(0, n - tail, 7):           # 1 to 100 rows of L21, up to 40 columns of U12 each
        a[rng.choice(np.arange(n - tail, n), 1 + c % 100, replace=False), c] = 0.1
        a[c, rng.choice(np.arange(n - tail, n), 1 + c % 40, replace=False)] = -0.2
    a[np.arange(n), np.arange(n)] = np.abs(a).sum(0) + np.abs(a).sum(1) + 1.0
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, front_min_w=0, hub_min_frac=0.9)
    nt = plan.stat("nt")
    assert 200 <= nt < n and 0 < plan.stat("pull_entries") <= 64 * nt
    assert (plan.stat("ntp") * count >= 32 * 148) == (count == 24)
    plan.set_ingest(sym.positions(row.astype(np.uint32), ap))
    batch = glu.Batch(plan, count)
    scale = np.linspace(1.0, 2.0, count)
    val = torch.as_tensor(scale[:, None] * a[row, col][None], device="cuda")
    batch.load_values(val)
    lu1 = torch.as_tensor(scale[1] * sym.val[None], device="cuda")
    batch.load_lu_values(lu1, first=1)
    batch.refactor(0.0)
    cp = sym.sym_c_ptr.astype(np.int64)
    for i in (0, 1, count - 1):
        lu = np.zeros((n, n))                 # [column, row]
        lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_lu(torch, lu, np.ascontiguousarray(a.T * scale[i])[None])


def test_workspace_of_many_vectors():
    """Vectors solved level by level hold one copy of themselves in the workspace and nothing for the
    dataflow, which fewer of them take: these find room in the same workspace, also under capture."""
    import torch
    n, nrhs = 1100, 40000
    a = long_columns(n, 7)
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, dense_threshold=2.0, front_min_w=0)
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, 1)
    batch.load_lu_values(torch.as_tensor(sym.val[None], device="cuda"))
    batch.refactor(0.0)
    gen = torch.Generator(device="cuda").manual_seed(1)
    b = torch.randn((1, nrhs, n), dtype=torch.float64, device="cuda", generator=gen)
    x = torch.empty_like(b)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    batch.solve(b, out=x)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 8 * n * nrhs + (64 << 20)
    cp = sym.sym_c_ptr.astype(np.int64)
    lu = np.zeros((n, n))
    lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(0).cpu().numpy()
    check_solve(torch, lu, b[0, -9:], x[0, -9:], False)
    for k in (1, 9, 727, 729):
        few, y = b[:, :k].contiguous(), torch.empty_like(b[:, :k])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            batch.solve(few, out=y)
        graph.replay()
        torch.cuda.synchronize()
        check_solve(torch, lu, few[0], y[0], False)


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("count", [1, 30, 150])
def test_rows_whose_waits_give_up(count, transpose):
    """The rows' dataflow with a bound of a nanosecond: every instance is flagged, and NaN, or right."""
    import torch
    n = 1100
    a = long_columns(n, 7)
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, dense_threshold=2.0, front_min_w=0, sparse_persistent=0, level_wait_ms=1e-6)
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, count)
    batch.load_lu_values(torch.as_tensor(sym.val, device="cuda").repeat(count, 1))
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(3).standard_normal((count, 1, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    flagged = batch.status()
    assert not (flagged & ~8).any()
    assert bool(x[torch.as_tensor(flagged != 0, device="cuda")].isnan().all())
    cp = sym.sym_c_ptr.astype(np.int64)
    lu = np.zeros((n, n))
    lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(0).cpu().numpy()
    good = np.flatnonzero(flagged == 0)
    if good.size:
        check_solve(torch, lu, b[good, 0], x[good, 0], transpose)
