"""Solves through fronts of widths around whole 64-row blocks (row blocks as a dataflow, outside
products in pieces, U rows pulled), against the elementwise backward-error bound of substitution."""
from __future__ import annotations

import numpy as np
import pytest

from glu_public_b200 import glu
from tests.test_gpu_dense_solve import check_solve

pytestmark = pytest.mark.gpu
WIDTHS = (16, 63, 64, 65, 129, 200)


def fronts_matrix(seed, tail=330):
    """Dense diagonal blocks of the WIDTHS, each coupled to its own part of a tail, with single
    columns between them; dense [n, n]."""
    rng = np.random.default_rng(seed)
    n = sum(WIDTHS) + 20 * len(WIDTHS) + tail
    a = np.zeros((n, n))
    at = 0
    for k, w in enumerate(WIDTHS):
        rows = np.sort(rng.choice(np.arange(n - tail, n), (30, 60, 65, 128, 257, 300)[k], replace=False))
        cols = np.sort(rng.choice(np.arange(n - tail, n), (300, 257, 65, 64, 63, 20)[k], replace=False))
        a[at:at + w, at:at + w] = 1.0
        a[np.ix_(rows, np.arange(at, at + w))] = 1.0
        a[np.ix_(np.arange(at, at + w), cols)] = 1.0
        nxt = slice(at + w + 20, at + w + 20 + WIDTHS[k + 1]) if k + 1 < len(WIDTHS) else None
        if nxt and k % 2:
            a[at:at + w, nxt] = 1.0           # entries above the next front's rows ...
        elif nxt:
            a[nxt, at:at + w] = 1.0           # ... or left of its columns
        at += w
        for s in range(20):                   # single columns, coupled to the tail
            a[at + s, rng.integers(n - tail, n, 3)] = 1.0
            a[rng.integers(n - tail, n, 3), at + s] = 1.0
        if nxt:                               # and one to the whole next front
            a[at + 3, nxt] = 1.0
            a[nxt, at + 5] = 1.0
        at += 20
    a[n - tail:, n - tail:][rng.random((tail, tail)) < 0.05] = 1.0
    a *= rng.uniform(-1.0, 1.0, a.shape)
    a[np.arange(n), np.arange(n)] = np.abs(a).sum(0) + np.abs(a).sum(1) + 1.0
    return a


@pytest.mark.parametrize("dense_threshold", [0.9, 2.0])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 5])
def test_front_solves(nrhs, transpose, dense_threshold):
    import torch
    a = fronts_matrix(11)
    n = a.shape[0]
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, dense_threshold=dense_threshold, front_min_flops=1.0)
    assert plan.stat("fronts") >= len(WIDTHS) - 1 and plan.stat("front_w_max") >= 200
    assert (plan.stat("nt") > 0) == (dense_threshold < 1)
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, 2)
    batch.load_lu_values(torch.as_tensor(np.stack([sym.val, -0.5 * sym.val]), device="cuda"))
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal((2, nrhs, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    assert not batch.status().any()
    cp = sym.sym_c_ptr.astype(np.int64)
    for i in range(2):
        lu = np.zeros((n, n))                 # [column, row]
        lu[np.repeat(np.arange(n), np.diff(cp)), sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_solve(torch, lu, b[i], x[i], transpose)


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_front_solves_of_many_instances(nrhs, transpose):
    """More row blocks than the GPU takes at once: a CTA has several, of different instances."""
    import torch
    a = fronts_matrix(12)
    n, count = a.shape[0], 150
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, dense_threshold=2.0, front_min_flops=1.0)
    assert plan.stat("front_w_max") >= 200    # four row blocks at least
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, count)
    batch.load_lu_values(torch.as_tensor(np.linspace(1.0, 2.0, count)[:, None] * sym.val[None],
                                         device="cuda"))
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal((count, nrhs, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    assert not batch.status().any()
    col = np.repeat(np.arange(n), np.diff(sym.sym_c_ptr.astype(np.int64)))
    for i in range(0, count, 7):
        lu = np.zeros((n, n))                 # [column, row]
        lu[col, sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_solve(torch, lu, b[i], x[i], transpose)


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("count", [24, 40, 57])
def test_instances_behind_a_wait_that_gave_up(count, transpose):
    """A front of eleven row blocks in more instances than the GPU takes at once, with a bound of a
    nanosecond: the first instance's rows cannot be divided by their diagonals in advance, so that
    its blocks take long and the waits for them give up.  Whatever a CTA that gave up had left to
    do belongs to other instances too: each is flagged or right."""
    import torch
    w, n = 700, 760
    rng = np.random.default_rng(4)
    a = np.eye(n)
    a[:w, :w] = a[720:740, :w] = a[:w, 710:730] = 1.0
    a *= rng.uniform(-1.0, 1.0, a.shape)
    a[np.arange(n), np.arange(n)] = np.abs(a).sum(0) + np.abs(a).sum(1) + 1.0
    col, row = np.nonzero(a.T)
    ap = np.searchsorted(col, np.arange(n + 1)).astype(np.uint32)
    sym = glu.SymbolicMatrix(n).analyze(row.astype(np.uint32), ap, a[row, col])
    plan = glu.Plan(sym, dense_threshold=2.0, front_min_flops=1.0, level_wait_ms=1e-6)
    assert plan.stat("front_w_max") == w
    idx, one = np.arange(n, dtype=np.uint32), np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    batch = glu.Batch(plan, count)
    b = torch.as_tensor(rng.standard_normal((count, 1, n)), device="cuda")
    col = np.repeat(np.arange(n), np.diff(sym.sym_c_ptr.astype(np.int64)))
    val = np.repeat(sym.val[None], count, 0)
    val[0] *= np.where(col == sym.sym_r_idx, 2.0 ** 700, 2.0 ** -400)
    batch.load_lu_values(torch.as_tensor(val, device="cuda"))
    batch.refactor(0.0)
    x = batch.solve(b, transpose=transpose)
    flagged = batch.status() & 8
    assert flagged[0]
    for i in np.flatnonzero(flagged == 0):
        lu = np.zeros((n, n))                 # [column, row]
        lu[col, sym.sym_r_idx] = batch.get_lu(i).cpu().numpy()
        check_solve(torch, lu, b[i], x[i], transpose)
