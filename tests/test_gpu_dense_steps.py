"""Dense blocks factored panel by panel (diagonal block, L21 / U12, update with the next diagonal
block) at the edges of tiles, groups and dispatch rules, against the elementwise error bound of LU."""
from __future__ import annotations

import numpy as np
import pytest

from glu_public_b200 import glu

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def dense_symbolic(n):
    ap = np.arange(0, n * n + 1, n, dtype=np.uint32)
    ai = np.tile(np.arange(n, dtype=np.uint32), n)
    return glu.SymbolicMatrix(n).analyze(ai, ap)


def matrices(n, count, seed):
    """[count, n, n] column-major (A[i][j] = column j) diagonally dominant values with zeros."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, (count, n, n))
    a[rng.random(a.shape) < 0.2] = 0.0
    a[:, np.arange(n), np.arange(n)] = rng.uniform(0.5, 1.5, (count, n)) * (0.3 * n + 2)
    return a


def check_lu(torch, lu, a):
    """|L U - A| <= 4 n u |L| |U|: n u per accumulated entry for the factorization, the same for
    quotients within an ulp, and n u each for the two products formed here."""
    n = a.shape[-1]
    m = torch.as_tensor(lu, device="cuda").reshape(-1, n, n).transpose(1, 2)   # rows, columns
    lo = torch.tril(m, -1) + torch.eye(n, dtype=m.dtype, device=m.device)
    up = torch.triu(m)
    err = (lo @ up - torch.as_tensor(a, device="cuda").transpose(1, 2)).abs()
    assert bool((err <= 4 * n * U * (lo.abs() @ up.abs())).all())


# one panel, remainders around whole panels, several panels; then more than 1,200 row tiles (the
# other kernels), and more than 5,000 tiles in few row tiles (groups of panels)
@pytest.mark.parametrize("n,count", [(1, 1), (8, 2), (63, 1), (64, 3), (65, 1), (127, 2), (128, 1),
                                     (129, 3), (200, 1), (449, 2), (129, 401), (2250, 4)])
def test_dense_block_elementwise(n, count):
    import torch
    sym = dense_symbolic(n)
    plan = glu.Plan(sym, dense_min=1)
    assert plan.stat("nt") == n
    batch = glu.Batch(plan, count)
    a = matrices(n, count, n)
    batch.load_lu_values(torch.as_tensor(a.reshape(count, -1), device="cuda"))
    batch.refactor(0.0)
    assert not batch.status().any()
    for i in sorted({0, count // 2, count - 1}):
        check_lu(torch, batch.get_lu(i).cpu().numpy(), a[i:i + 1])


@pytest.mark.parametrize("pivot", [0, 7, 8, 63, 64, 100])
def test_bad_and_perturbed_pivots_of_a_panel(pivot):
    """A zero pivot and a NaN flag their instance only; with perturbation the clamped pivot is
    exact."""
    import torch
    n = 130
    sym = dense_symbolic(n)
    batch = glu.Batch(glu.Plan(sym, dense_min=1), 3)
    a = matrices(n, 3, 5)
    a[1, pivot, :] = 0.0                  # column `pivot` empty: its pivot stays zero
    a[2, pivot, pivot] = np.nan
    val = torch.as_tensor(a.reshape(3, -1), device="cuda")
    batch.load_lu_values(val)
    batch.refactor(0.0)
    st = batch.status()
    assert st[0] == 0 and st[1] & 1 and st[2] & 2
    check_lu(torch, batch.get_lu(0).cpu().numpy(), a[:1])
    batch.load_lu_values(val)
    batch.refactor(1e-3)
    st = batch.status()
    assert st[0] == 0 and st[1] == 4 and st[2] & 2
    lu = batch.get_lu(1).cpu().numpy().reshape(n, n)
    assert lu[pivot, pivot] == 1e-3 and not lu[pivot, pivot + 1:].any()
    a[1, pivot, pivot] = 1e-3
    check_lu(torch, lu[None], a[1:2])


def lone_pivot(n, count, k, value, below):
    """`matrices` with pivot k of `value`: nothing left of it or above it, `below` under it."""
    a = matrices(n, count, 11)
    a[:, :k, k] = 0.0
    a[:, k, :k] = 0.0
    a[:, k, k] = value
    a[:, k, k + 1:] = below(n - k - 1)
    return a


@pytest.mark.parametrize("n,count,pivot", [(40, 1, 0), (64, 2, 9), (64, 1, 37), (130, 1, 3), (130, 2, 70),
                                           (129, 401, 20)])
def test_pivot_without_a_finite_reciprocal(n, count, pivot):
    """1 / d overflows for a pivot below 2^-1024; the quotients with it, of the block and of the rows
    below, are ordinary numbers: |L(i, k) - a / d| <= u |a / d| and |L U - A| <= 4 n u |L| |U|, each
    plus a subnormal's rounding."""
    import torch
    d = 3e-310
    rng = np.random.default_rng(0)
    a = lone_pivot(n, count, pivot, d, lambda m: rng.uniform(-1.0, 1.0, m) * d)
    batch = glu.Batch(glu.Plan(dense_symbolic(n), dense_min=1), count)
    batch.load_lu_values(torch.as_tensor(a.reshape(count, -1), device="cuda"))
    batch.refactor(0.0)
    assert not batch.status().any()
    lu = batch.get_lu(count - 1).cpu().numpy().reshape(n, n)
    want = a[-1, pivot, pivot + 1:] / d
    assert (np.abs(lu[pivot, pivot + 1:] - want) <= 2 * U * np.abs(want)).all()
    m = torch.as_tensor(lu, device="cuda").T
    lo, up = torch.tril(m, -1) + torch.eye(n, dtype=m.dtype, device=m.device), torch.triu(m)
    err = (lo @ up - torch.as_tensor(a[-1], device="cuda").T).abs()
    assert bool((err <= 4 * n * U * (lo.abs() @ up.abs()) + 2 * n * 2.0 ** -1074).all())


@pytest.mark.parametrize("n,pivot", [(40, 0), (64, 37), (130, 3), (130, 70)])
def test_infinite_pivot(n, pivot):
    """Quotients with an infinite pivot are zero, so the other pivots' factors are those of the matrix
    without its row and column; the instance is flagged."""
    import torch
    a = lone_pivot(n, 1, pivot, np.inf, lambda m: np.linspace(1.0, 2.0, m))
    batch = glu.Batch(glu.Plan(dense_symbolic(n), dense_min=1), 1)
    batch.load_lu_values(torch.as_tensor(a.reshape(1, -1), device="cuda"))
    batch.refactor(0.0)
    assert batch.status()[0] == 2
    lu = batch.get_lu(0).cpu().numpy().reshape(n, n)
    assert not lu[pivot, pivot + 1:].any()
    rest = np.delete(np.arange(n), pivot)
    check_lu(torch, lu[np.ix_(rest, rest)][None], a[:, rest][:, :, rest])
