"""Triangular solves with the dense block (L then U, U^T then L^T) as a dataflow over 64-row blocks:
block edges, vector groups, one CTA or several per vector, pivots at the edge of the exponent range
and the bounded waits, against the elementwise backward-error bound of substitution."""
from __future__ import annotations

import numpy as np
import pytest

from glu_public_b200 import glu
from tests.test_gpu_dense_steps import U, dense_symbolic, matrices

pytestmark = pytest.mark.gpu


def plan_for(n, **options):
    plan = glu.Plan(dense_symbolic(n), dense_min=1, **options)
    idx = np.arange(n, dtype=np.uint32)
    one = np.ones(n)
    plan.set_solve_maps(glu.NicsluArrays(n, idx, idx, idx, idx, one, one, 0))
    return plan


def check_solve(torch, lu, b, x, transpose):
    """|b - op(L U) x| <= 8 n u |op(L U)| |x|: n u (plus one rounding of each entry of U) for each
    substitution, the rest for the products formed here."""
    n = x.shape[-1]
    m = torch.as_tensor(lu, device="cuda").reshape(n, n).T
    lo = torch.tril(m, -1) + torch.eye(n, dtype=m.dtype, device=m.device)
    up = torch.triu(m)
    f, g = (up.T, lo.T) if transpose else (lo, up)
    r = b.T - f @ (g @ x.T)
    bound = 8 * n * U * (f.abs() @ (g.abs() @ x.abs().T))
    assert bool((r.abs() <= bound).all())


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("n,count,nrhs", [(1, 1, 1), (63, 2, 2), (64, 1, 3), (65, 2, 1), (129, 1, 4),
                                          (200, 3, 5), (449, 1, 9), (1100, 2, 33), (130, 700, 1)])
def test_dense_solve_elementwise(n, count, nrhs, transpose):
    import torch
    batch = glu.Batch(plan_for(n), count)
    a = matrices(n, count, n + nrhs)
    batch.load_lu_values(torch.as_tensor(a.reshape(count, -1), device="cuda"))
    batch.refactor(0.0)
    rng = np.random.default_rng(n)
    b = torch.as_tensor(rng.standard_normal((count, nrhs, n)), device="cuda")
    x = batch.solve(b, transpose=transpose)
    assert not batch.status().any()
    for i in sorted({0, count // 2, count - 1}):
        check_solve(torch, batch.get_lu(i).cpu().numpy(), b[i], x[i], transpose)


@pytest.mark.parametrize("transpose", [False, True])
def test_pivots_at_the_edge_of_the_exponent_range(transpose):
    """A row scaled to the bottom of the normal range takes the triangle that divides pivot by
    pivot; scaling by a power of two changes no digit of the solution."""
    import torch
    n, k = 140, 70
    a = matrices(n, 1, 3)[0]
    a = np.where(np.arange(n)[:, None] >= np.arange(n)[None, :], a, 0.0)   # column j, row i <= j
    rng = np.random.default_rng(1)
    b = rng.standard_normal((1, 1, n))
    xs = []
    for scale in (1.0, 2.0 ** -965):
        s, bs = a.copy(), b.copy()
        s[:, k] *= scale
        if not transpose:
            bs[0, 0, k] *= scale
        batch = glu.Batch(plan_for(n), 1)
        batch.load_lu_values(torch.as_tensor(s.reshape(1, -1), device="cuda"))
        batch.refactor(0.0)
        x = batch.solve(torch.as_tensor(bs, device="cuda"), transpose=transpose)[0, 0].cpu().numpy()
        if transpose:
            x[k] *= scale
        xs.append(x)
    assert np.isfinite(xs[1]).all()
    cond = np.abs(a).sum() / np.abs(np.diag(a)).min()
    np.testing.assert_allclose(xs[1], xs[0], rtol=8 * n * U * cond, atol=0)


# (diagonal, entry, x of the entry's column, right-hand side, solution) of a row with one entry
EXTREME = {
    "quotient_overflows": (2.0 ** -900, 2.0 ** 200, 0.0, 2.0 ** -899, 2.0),
    "cancels_before_the_division": (2.0 ** -900, 2.0 ** 200, 1.0, 2.0 ** 200, 0.0),
    "quotient_underflows": (2.0 ** 900, 2.0 ** -200, 2.0 ** 150, 0.0, -2.0 ** -950),
    "reciprocal_overflows": (3e-310, 2.0 ** -3, 0.0, 6e-310, 2.0),
    "infinite": (np.inf, 1.0, 1.0, 3.0, 0.0),
}


@pytest.mark.parametrize("case", EXTREME)
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("front", [False, True])
@pytest.mark.parametrize("k,j", [(10, 50), (70, 100), (129, 139)])
def test_rows_of_extreme_exponents(case, transpose, front, k, j):
    """A row of U whose division by its diagonal overflows or underflows, or has no reciprocal, beside
    ordinary rows and beside a right-hand side of NaN: the row's solution is exact, the others'
    within 8 n u cond."""
    import torch
    n = 140
    d, entry, xj, bk, xk = EXTREME[case]
    a = matrices(n, 1, 3)[0]
    m = np.where(np.arange(n)[:, None] <= np.arange(n)[None, :], a.T, 0.0)   # upper, row, column
    if transpose:
        k, j = j, k                           # row k of U^T: column k of U
    for p in (k, j):
        m[p, :] = m[:, p] = 0.0
    m[j, j] = 1.0
    rest = np.delete(np.arange(n), [k, j])
    cond = np.abs(m).sum() / np.abs(np.diag(m))[rest].min()
    m[(j, k) if transpose else (k, j)] = entry
    m[k, k] = d
    rng = np.random.default_rng(2)
    b = rng.standard_normal((1, 3, n))
    b[0, :, k], b[0, :, j] = bk, xj
    b[0, 1] = np.nan
    sub = (m.T if transpose else m)[np.ix_(rest, rest)]
    want = np.linalg.solve(sub, b[0][:, rest].T).T
    size = n + 30 if front else n             # the rows and columns of a front and some outside it
    full = np.eye(size)
    full[:n, :n] = m
    if front:
        pattern = np.eye(size)
        pattern[:n, :n] = pattern[[n + 9, n + 19], :n] = pattern[:n, [n + 4, n + 14]] = 1.0
        col, row = np.nonzero(pattern.T)
        sym = glu.SymbolicMatrix(size).analyze(
            row.astype(np.uint32), np.searchsorted(col, np.arange(size + 1)).astype(np.uint32))
        plan = glu.Plan(sym, dense_threshold=2.0, front_min_flops=1.0)
        idx, one = np.arange(size, dtype=np.uint32), np.ones(size)
        plan.set_solve_maps(glu.NicsluArrays(size, idx, idx, idx, idx, one, one, 0))
        assert plan.stat("front_w_max") == n
    else:
        plan = plan_for(n)
    batch = glu.Batch(plan, 1)
    col = np.repeat(np.arange(size), np.diff(plan.sym.sym_c_ptr.astype(np.int64)))
    batch.load_lu_values(torch.as_tensor(full[plan.sym.sym_r_idx, col][None], device="cuda"))
    batch.refactor(0.0)
    b = np.concatenate([b, np.zeros((1, 3, size - n))], 2)
    x = batch.solve(torch.as_tensor(b, device="cuda"), transpose=transpose)[0].cpu().numpy()
    for v in (0, 2):
        assert x[v, k] == xk and x[v, j] == xj
        np.testing.assert_allclose(x[v, rest], want[v], rtol=8 * n * U * cond, atol=0)
    assert np.isnan(x[1, :n]).all()


def test_waits_of_the_dense_solve_are_bounded():
    """With a bound of a nanosecond a wait gives up: the instances are flagged, the launch ends and
    the context stays usable."""
    import torch
    n = 700
    a = matrices(n, 1, 2)
    val = torch.as_tensor(a.reshape(1, -1), device="cuda")
    b = torch.ones((1, 1, n), dtype=torch.float64, device="cuda")
    batch = glu.Batch(plan_for(n, level_wait_ms=1e-6), 1)
    batch.load_lu_values(val)
    batch.refactor(0.0)
    batch.solve(b)
    assert batch.status()[0] & 8
    good = glu.Batch(plan_for(n), 1)
    good.load_lu_values(val)
    good.refactor(0.0)
    x = good.solve(b)
    assert not good.status().any()
    check_solve(torch, good.get_lu(0).cpu().numpy(), b[0], x[0], False)


def test_a_solve_that_gave_up_is_no_solution():
    """Its vectors are NaN, also after a refinement; the flag goes with the next solve, whose waits
    (none: a CTA per group of right-hand sides) are met."""
    import torch
    n = 700
    a = matrices(n, 1, 2)
    plan = plan_for(n, level_wait_ms=1e-6)
    col = np.repeat(np.arange(n), n)
    plan.set_original_pattern(np.tile(np.arange(n), n), col)
    batch = glu.Batch(plan, 1)
    val = torch.as_tensor(a.reshape(1, -1), device="cuda")
    batch.load_lu_values(val)
    batch.refactor(0.0)
    b = torch.as_tensor(np.random.default_rng(0).standard_normal((1, 800, n)), device="cuda")
    one = b[:, :1].contiguous()
    x = batch.solve(one)
    assert batch.status()[0] == 8 and bool(x.isnan().all())
    batch.refine(val, one, x)
    assert batch.status()[0] == 8 and bool(x.isnan().all())
    x = batch.solve(b)
    assert batch.status()[0] == 0
    check_solve(torch, batch.get_lu(0).cpu().numpy(), b[0], x[0], False)
