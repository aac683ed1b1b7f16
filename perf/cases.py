"""Performance cases of the GLU numeric phase: what users of the package have it do.

A circuit simulator analyses a pattern once (ordering, symbolic analysis, plan) and then, for
every Newton iteration, time step or Monte Carlo sample, loads new values, refactors and solves.
The cases are those passes through the public entry points (:class:`glu.Plan`, :class:`glu.Batch`,
:class:`glu.Group`, ``autograd.sparse_solve``), each on the patterns of the benchmark and the tests
(netlist MNA matrices and two-layer power grids of ``gen.py``).

A case is a dict of plain values:

======== =======================================================================================
pattern  ``"mna"`` (netlist, order ``size``) or ``"grid"`` (power grid, ``size`` nodes a side)
seed     seed of the generated pattern
call     ``newton`` load + refactor + solve (+ refinement), ``graph`` the same as one CUDA graph
         replay, ``solve`` triangular solves on kept factors, ``factor`` factors in and out in
         the filled-pattern layout (the LUonDevice flow), ``grad`` forward and backward of the
         differentiable solve, ``group`` two patterns in one graph
count    value instances of the pattern, nrhs: right-hand sides of each, refine: refinement rounds
transpose, perturb, deterministic   the options of the same names
======== =======================================================================================

The fixtures ``tests/golden/nicslu_*.npz`` hold the reference preprocessing's permutations and
scalings of the benchmark's patterns; other sizes get a minimum-degree or nested-dissection order
and a diagonal scaling of the same form here.
"""
from __future__ import annotations

import functools
import heapq
import math
import os

import numpy as np
import torch

from glu_public_b200 import autograd, gen, glu

_GOLDEN = os.path.join("tests", "golden")
_DEFAULTS = dict(pattern="mna", size=2000, seed=3, call="newton", count=1, nrhs=1, refine=0,
                 transpose=False, perturb=False, deterministic=False)


def _case(name, **kw):
    return dict(_DEFAULTS, name=name, **kw)


def listed():
    return [
        # the inner loop of a transient simulation of a small circuit: latency of one matrix
        _case("newton_n2000", size=2000, seed=3),
        # one matrix of the plain benchmark workload, refined
        _case("newton_n4960", size=4960, seed=0, refine=1),
        # one large netlist matrix
        _case("newton_n20000", size=20000, seed=2, refine=1),
        # Monte Carlo of a small circuit, replayed as one graph
        _case("montecarlo_n2000_x256", call="graph", size=2000, seed=3, count=256, refine=1),
        # the benchmark's Monte Carlo batch, with the instances of a part of a GPU's memory
        _case("montecarlo_n20000_x64", size=20000, seed=2, count=64, refine=1),
        # power-grid analysis: one small mesh, one load vector
        _case("mesh_128", pattern="grid", size=128, seed=1),
        # power-grid analysis at the benchmark's size, four load vectors
        _case("mesh_512_rhs4", pattern="grid", size=512, seed=1, nrhs=4, refine=1),
        # many load vectors against factors that are kept
        _case("solve_n20000_rhs32", call="solve", size=20000, seed=2, nrhs=32),
        # the sensitivity (adjoint) solve of one system on kept factors
        _case("adjoint_solve_n20000", call="solve", size=20000, seed=2, transpose=True),
        # LUonDevice's own flow with the static-pivot perturbation: factors in and out
        _case("factor_n4960_perturbed", call="factor", size=4960, seed=0, perturb=True),
        # training through the solve: forward, adjoint and the gradient over A's nonzeros
        _case("gradient_n4960_x16", call="grad", size=4960, seed=0, count=16, refine=1),
        # bit-identical repeat runs
        _case("deterministic_n4960_x4", size=4960, seed=0, count=4, refine=1, deterministic=True),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))

    call = rng.choice(["newton", "newton", "newton", "graph", "solve", "solve", "factor", "grad",
                       "group"])
    grid = call in ("newton", "graph", "solve") and rng.random() < 0.35
    seed = rng.randrange(1000)
    if grid:
        size = spread(24, 200)
        count = spread(1, max(1, 4 * (200 // size)))
    else:
        size = spread(300, 7000)
        if call in ("newton", "solve") and rng.random() < 0.2:
            size, seed = 20000, 2
        # count * size^2.3 about constant, one matrix as likely as a batch
        most = max(1, int(256 * (2000.0 / size) ** 2.3))
        count = 1 if call in ("newton", "solve", "factor") and rng.random() < 0.5 else \
            spread(1, min(most, 1000))
    nrhs = 1 if call in ("grad", "group", "factor") or rng.random() < 0.5 else spread(1, 40)
    nrhs = max(1, min(nrhs, 2000 // count))
    return dict(_DEFAULTS, pattern="grid" if grid else "mna", size=size, seed=seed, call=call,
                count=1 if call == "factor" else count, nrhs=nrhs,
                refine=0 if call in ("solve", "factor") else rng.choice([0, 1]) if size < 3000 else 1,
                transpose=call == "solve" and rng.random() < 0.5,
                perturb=call == "factor" and rng.random() < 0.5,
                deterministic=call == "newton" and not grid and rng.random() < 0.2)


# ---------------------------------------------------------------------------------------------
# patterns
# ---------------------------------------------------------------------------------------------

def _minimum_degree(n, indptr, indices):
    """Approximate minimum-degree order of the symmetrized graph (quotient graph with element
    absorption); the nodes left when the remaining graph is nearly complete keep their order."""
    col = np.repeat(np.arange(n), np.diff(indptr))
    adj = [set() for _ in range(n)]
    for r, c in zip(indices.tolist(), col.tolist()):
        if r != c:
            adj[r].add(c)
            adj[c].add(r)
    els = [set() for _ in range(n)]          # elements (eliminated pivots) next to a variable
    elem = {}                                # element -> its variables
    deg = [len(a) for a in adj]
    heap = [(d, v) for v, d in enumerate(deg)]
    heapq.heapify(heap)
    done = [False] * n
    order = []
    while heap:
        d, p = heapq.heappop(heap)
        if done[p] or d != deg[p]:
            continue
        if d >= 0.8 * (n - len(order) - 1):
            break
        done[p] = True
        order.append(p)
        lp = set(adj[p])
        for e in els[p]:
            lp |= elem.pop(e)
        lp.discard(p)
        gone = els[p]
        elem[p] = lp
        outside = {}
        for v in lp:
            els[v] -= gone
            for e in els[v]:
                outside[e] = outside.get(e, len(elem[e])) - 1
        for v in lp:
            adj[v] -= lp
            adj[v].discard(p)
            els[v] = {e for e in els[v] if outside[e] > 0}
            nd = len(adj[v]) + len(lp) - 1 + sum(outside[e] for e in els[v])
            els[v].add(p)
            deg[v] = min(nd, n - len(order) - 1)
            heapq.heappush(heap, (deg[v], v))
        for e, left in outside.items():
            if left == 0:
                elem.pop(e, None)
        adj[p] = set()
    return np.array(order + [v for v in range(n) if not done[v]], np.int64)


def _nested_dissection(n, side, layers, hubs, pad_of):
    """Geometric nested dissection of the layered grid; a supply pad's row sits with its node,
    nodes tied to the whole grid come last."""
    node = np.arange(n)
    at = node.copy()
    at[layers * side * side:] = pad_of
    r, c = (at % (side * side)) // side, at % side
    box = [np.zeros(n, np.int64), np.full(n, side), np.zeros(n, np.int64), np.full(n, side)]
    key = np.zeros(n, np.int64)
    live = np.ones(n, bool)
    while live.any():
        h, w = box[1] - box[0], box[3] - box[2]
        tall = h >= w
        x = np.where(tall, r, c)
        lo, hi = np.where(tall, box[0], box[2]), np.where(tall, box[1], box[3])
        mid = (lo + hi) // 2
        digit = np.where(x < mid, 0, np.where(x > mid, 1, 2))
        key = key * 3 + np.where(live, digit, 0)
        live &= (digit != 2) & (np.maximum(h, w) > 1)
        nlo, nhi = np.where(digit == 0, lo, mid + 1), np.where(digit == 0, mid, hi)
        box[0], box[1] = np.where(tall, nlo, box[0]), np.where(tall, nhi, box[1])
        box[2], box[3] = np.where(tall, box[2], nlo), np.where(tall, box[3], nhi)
    key[hubs] = np.iinfo(np.int64).max
    return np.lexsort((node, key))


@functools.lru_cache(maxsize=None)
def _pattern(kind, size, seed):
    """(circuit, preprocessing arrays, symbolic analysis) of one pattern."""
    if kind == "mna":
        c = gen.mna_netlist(size, seed)
    else:                                    # small meshes with the tests' pads and hubs
        c = gen.power_grid(size, seed, **(dict(pads=16, hubs=4) if size < 128 else {}))
    path = os.path.join(_GOLDEN, f"nicslu_{kind}{size}_s{seed}.npz")
    if os.path.exists(path):
        nic = glu.NicsluArrays.from_npz(path)
    else:
        n = c.n
        cols = np.repeat(np.arange(n), np.diff(c.indptr))
        match = np.arange(n)                 # row that column's pivot sits in
        if kind == "mna":
            order = _minimum_degree(n, c.indptr, c.indices)
        else:
            nn = 2 * size * size
            pad_of = np.array([c.indices[c.indptr[p]] for p in range(nn, n)], np.int64)
            match[pad_of], match[nn:] = np.arange(nn, n), pad_of
            deg = np.diff(c.indptr)
            hubs = np.flatnonzero(deg > max(64, 0.002 * nn))
            order = _nested_dissection(n, size, 2, hubs, pad_of)
        hit = c.indices == match[cols]
        piv = np.ones(n)
        piv[cols[hit]] = np.abs(c.data[hit])
        scale = 1.0 / np.sqrt(piv)
        row_perm, col_perm = order, match[order]
        rpi, cpi = np.empty(n, np.int64), np.empty(n, np.int64)
        rpi[row_perm], cpi[col_perm] = np.arange(n), np.arange(n)
        u32 = np.uint32
        nic = glu.NicsluArrays(n, row_perm.astype(u32), rpi.astype(u32), col_perm.astype(u32),
                               cpi.astype(u32), scale, scale[row_perm], 1)
    ap, ai, _ = nic.preprocess(c.indptr, c.indices, c.data)
    return c, nic, glu.SymbolicMatrix(c.n).analyze(ai, ap)


@functools.lru_cache(maxsize=None)
def _plan(kind, size, seed, deterministic):
    """The plan a program keeps for one pattern."""
    c, nic, sym = _pattern(kind, size, seed)
    plan = glu.Plan(sym, **(dict(deterministic=1) if deterministic else {}))
    plan.set_ingest_from_nicslu(c.indptr, c.indices, nic)
    plan.set_solve_maps(nic)
    plan.set_original_csc(c.indptr, c.indices)
    return plan


def _patterns_of(case):
    """(kind, size, seed, count) of every pattern of the case: a group adds a mesh."""
    one = [(case["pattern"], case["size"], case["seed"], case["count"])]
    if case["call"] == "group":
        one.append(("grid", 32, case["seed"] + 1, 2))
    return one


def _inputs(case, seed, kind, size, pseed, count):
    """Monte Carlo values of the pattern and right-hand sides (node currents), on the host."""
    c = _pattern(kind, size, pseed)[0]
    vals = c.instance_values_indexed(0, count, int(seed))
    rng = np.random.default_rng((int(seed), 77))
    return vals, rng.standard_normal((count, case["nrhs"], c.n))


# ---------------------------------------------------------------------------------------------
# the pass
# ---------------------------------------------------------------------------------------------

def prepare(case, seed):
    call = case["call"]
    s = dict(case=case, parts=[])
    for kind, size, pseed, count in _patterns_of(case):
        plan = _plan(kind, size, pseed, case["deterministic"])
        vals, B = _inputs(case, seed, kind, size, pseed, count)
        p = dict(plan=plan, a=torch.as_tensor(vals, device="cuda"))
        if call == "factor":
            # the input of LUonDevice: the preprocessed values in the filled pattern
            c, nic, sym = _pattern(kind, size, pseed)
            ap, ai, ax = nic.preprocess(c.indptr, c.indices, vals[0])
            val = np.zeros((1, sym.nnz))
            val[0, _positions(kind, size, pseed)] = ax
            p["a"] = torch.as_tensor(val, device="cuda")
        p["B"] = torch.as_tensor(B, device="cuda")
        if call == "grad":
            p["a"].requires_grad_(True)
            p["B"].requires_grad_(True)
            p["G"] = torch.as_tensor(np.random.default_rng((int(seed), 78)).standard_normal(B.shape),
                                     device="cuda")
        else:
            p["batch"] = glu.Batch(plan, count)
        if call == "solve":
            p["batch"].load_values(p["a"])
            p["batch"].refactor(0.0)
        if call in ("graph", "group"):
            p["X"] = torch.empty_like(p["B"])
            _newton(p, case)                 # allocates the workspaces before the capture
        s["parts"].append(p)
    if call == "graph":
        p = s["parts"][0]
        torch.cuda.synchronize()
        s["stream"] = torch.cuda.Stream()
        p["batch"].capture(p["a"], p["B"], p["X"], refine=case["refine"], stream=s["stream"])
        torch.cuda.synchronize()
    if call == "group":
        torch.cuda.synchronize()
        s["stream"] = torch.cuda.Stream()
        s["group"] = glu.Group([p["batch"] for p in s["parts"]], [p["a"] for p in s["parts"]],
                               [p["B"] for p in s["parts"]], [p["X"] for p in s["parts"]],
                               refine=case["refine"], stream=s["stream"])
        torch.cuda.synchronize()
    return s


def _newton(p, case):
    b = p["batch"]
    b.load_values(p["a"])
    b.refactor(-1.0 if case["perturb"] else 0.0)
    X = b.solve(p["B"])
    if case["refine"]:
        b.refine(p["a"], p["B"], X, steps=case["refine"])
    return X


def run(s):
    case = s["case"]
    p = s["parts"][0]
    call = case["call"]
    if call == "newton":
        return _newton(p, case)
    if call == "graph":
        p["batch"].replay()
        return p["X"]
    if call == "group":
        s["group"].launch()
        return [q["X"] for q in s["parts"]]
    if call == "solve":
        return p["batch"].solve(p["B"], transpose=case["transpose"])
    if call == "factor":
        b = p["batch"]
        b.load_lu_values(p["a"])
        b.refactor(-1.0 if case["perturb"] else 0.0)
        return b.get_lu(0)
    X = autograd.sparse_solve(p["a"], p["B"], p["plan"], refine=case["refine"])
    ga, gb = torch.autograd.grad(X, (p["a"], p["B"]), p["G"])
    return [X.detach(), ga, gb]


def work(case):
    nbytes = flops = 0.0
    for kind, size, pseed, count in _patterns_of(case):
        c, _, sym = _pattern(kind, size, pseed)
        vec = 8.0 * c.n * count * case["nrhs"]
        solve = 2.0 * sym.nnz * count * case["nrhs"]
        if case["call"] == "solve":          # factors and right-hand sides in, solutions out
            nbytes += 8.0 * sym.nnz * count + 2 * vec
            flops += solve
        elif case["call"] == "factor":       # filled values in, factors out
            nbytes += 16.0 * sym.nnz
            flops += sym.flops()
        else:                                # values and right-hand sides in, factors and X out
            nbytes += 8.0 * count * (c.nnz + sym.nnz) + 2 * vec
            flops += sym.flops() * count + solve * (1 + case["refine"])
            if case["call"] == "grad":       # cotangents in, both gradients out
                nbytes += 8.0 * count * c.nnz + 2 * vec
                flops += solve * (1 + case["refine"]) + 2.0 * c.nnz * count * case["nrhs"]
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------------------------
# the same in plain torch / numpy
# ---------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _positions(kind, size, seed):
    """Position of every preprocessed entry in the filled pattern."""
    c, nic, sym = _pattern(kind, size, seed)
    ap, ai, _ = nic.preprocess(c.indptr, c.indices, c.data)
    return sym.positions(ai, ap)


def _product(rows, cols, vals, x, n):
    """A x for vectors x [k, n] in extended precision."""
    order = np.argsort(rows, kind="stable")
    start = np.searchsorted(rows[order], np.arange(n))
    t = vals[order].astype(np.longdouble) * x[:, cols[order]]
    return np.add.reduceat(t, start, axis=1)


def _dense_solve(rows, cols, vals, B, transpose=False, rounds=3):
    """op(A)^-1 B by a dense pivoted LU, refined with extended-precision residuals."""
    n = B.shape[1]
    if transpose:
        rows, cols = cols, rows
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.zeros((n, n), dtype=torch.float64, device=dev)
    A[torch.as_tensor(rows, device=dev), torch.as_tensor(cols, device=dev)] = \
        torch.as_tensor(vals, device=dev)
    lu, piv = torch.linalg.lu_factor(A)
    del A

    def solve(R):
        return torch.linalg.lu_solve(lu, piv, torch.as_tensor(R.astype(np.float64), device=dev).T
                                     .contiguous()).T.cpu().numpy()

    x = solve(B).astype(np.longdouble)
    for _ in range(rounds):
        x = x + solve(B - _product(rows, cols, vals, x, n))
    return x


def _dense_factors(n, rows, cols, vals, perturb, nb=64):
    """L and U (one array) of the LU factorization without pivoting, by blocks."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    A = torch.zeros((n, n), dtype=torch.float64, device=dev)
    A[torch.as_tensor(rows, device=dev), torch.as_tensor(cols, device=dev)] = \
        torch.as_tensor(vals, device=dev)
    pert = 3.45e-4 * float(A.abs().sum(0).max()) if perturb else 0.0
    for k in range(0, n, nb):
        e = min(n, k + nb)
        d = A[k:e, k:e].cpu().numpy()
        below = A[e:, k:e]
        for i in range(e - k):
            has_l = bool((d[i + 1:, i] != 0).any()) or bool((below[:, i] != 0).any()) \
                if pert > 0 and abs(d[i, i]) < pert else False
            if has_l:
                d[i, i] = pert
            d[i + 1:, i] /= d[i, i]
            d[i + 1:, i + 1:] -= np.outer(d[i + 1:, i], d[i, i + 1:])
        t = torch.as_tensor(d, device=dev)
        A[k:e, k:e] = t
        if e < n:
            A[e:, k:e] = torch.linalg.solve_triangular(torch.triu(t), A[e:, k:e], upper=True,
                                                       left=False)
            A[k:e, e:] = torch.linalg.solve_triangular(torch.tril(t), A[k:e, e:], upper=False,
                                                       unitriangular=True)
            A[e:, e:] -= A[e:, k:e] @ A[k:e, e:]
    return A


def exact(case, seed):
    cost = sum(((2 * size * size) if kind == "grid" else size) ** 3 * float(count)
               for kind, size, _, count in _patterns_of(case))
    if cost > 4e13:
        return None
    if case["call"] == "factor":
        kind, size, pseed, _ = _patterns_of(case)[0]
        c, nic, sym = _pattern(kind, size, pseed)
        vals, _ = _inputs(case, seed, kind, size, pseed, 1)
        ap, ai, ax = nic.preprocess(c.indptr, c.indices, vals[0])
        A = _dense_factors(c.n, ai.astype(np.int64), np.repeat(np.arange(c.n), np.diff(ap)), ax,
                           case["perturb"])
        r = torch.as_tensor(sym.sym_r_idx.astype(np.int64), device=A.device)
        j = torch.as_tensor(np.repeat(np.arange(c.n), np.diff(sym.sym_c_ptr.astype(np.int64))),
                            device=A.device)
        return A[r, j].cpu().numpy()
    out = []
    for kind, size, pseed, count in _patterns_of(case):
        c = _pattern(kind, size, pseed)[0]
        vals, B = _inputs(case, seed, kind, size, pseed, count)
        rows = c.indices.astype(np.int64)
        cols = np.repeat(np.arange(c.n), np.diff(c.indptr))
        X = [_dense_solve(rows, cols, vals[i], B[i], case["transpose"]) for i in range(count)]
        if case["call"] == "grad":
            G = np.random.default_rng((int(seed), 78)).standard_normal(B.shape)
            lam = [_dense_solve(rows, cols, vals[i], G[i], True) for i in range(count)]
            ga = [-(lam[i][:, rows] * X[i][:, cols]).sum(0) for i in range(count)]
            return [np.stack(v).astype(np.float64) for v in (X, ga, lam)]
        out.append(np.stack(X).astype(np.float64))
    return out if case["call"] == "group" else out[0]
