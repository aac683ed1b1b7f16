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
