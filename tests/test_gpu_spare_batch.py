"""A destroyed batch's buffers taken over by the plan's next batch of the same count."""
from __future__ import annotations

import gc
import threading

import numpy as np
import pytest

from glu_public_b200 import glu
from tests.test_gpu_dense_solve import check_solve, plan_for
from tests.test_gpu_dense_steps import check_lu, dense_symbolic, matrices

pytestmark = pytest.mark.gpu


def test_batches_of_one_plan_in_turn():
    """Batches made and destroyed on changing streams with work still in flight, of two counts: every
    one starts unloaded and unflagged and gives its own matrices' factors."""
    import torch
    n = 300
    plan = plan_for(n)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    kept = []
    for k in range(8):
        count = 2 + k % 3 // 2
        a = matrices(n, count, k)
        if k == 3:
            a[0, 10, :] = 0.0                 # flags instance 0 of this batch only
        val = torch.as_tensor(a.reshape(count, -1), device="cuda")
        b = torch.ones((count, 1, n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        batch = glu.Batch(plan, count)
        assert not batch.status().any()
        with pytest.raises(glu.GluError):
            batch.refactor(0.0)               # nothing loaded
        with torch.cuda.stream(streams[k % 2]):
            batch.load_lu_values(val)
            batch.refactor(0.0)
            x = batch.solve(b)
            lu = batch.get_lu(count - 1)
        kept.append((a, lu, b, x, val))
        del batch                             # its work may still be running
    torch.cuda.synchronize()
    for a, lu, b, x, _ in kept:
        check_lu(torch, lu.cpu().numpy(), a[-1:])
        check_solve(torch, lu.cpu().numpy(), b[-1], x[-1], False)


def test_memory_is_given_back_with_the_plan():
    import torch
    torch.cuda.synchronize()
    gc.collect()
    n = 2000
    plan = plan_for(n)
    free0 = torch.cuda.mem_get_info()[0]
    batch = glu.Batch(plan, 16)               # 512 MB
    del batch
    batch = glu.Batch(plan, 40)               # over the bound: not kept
    del batch
    del plan
    gc.collect()
    assert torch.cuda.mem_get_info()[0] >= free0


@pytest.mark.parametrize("call", ["solve", "refine", "plan", "batch"])
def test_memory_is_given_back_when_an_allocation_needs_it(call):
    """With little but a destroyed batch's memory left on the device, every allocation of the library
    finds it: solve and refinement workspaces, plans, batches."""
    import torch
    n = 2000
    plan, other = plan_for(n), plan_for(n)
    col = np.repeat(np.arange(n), n)
    other.set_original_pattern(np.tile(np.arange(n), n), col)
    val = torch.as_tensor(matrices(n, 1, 0).reshape(1, -1), device="cuda")
    batch = glu.Batch(other, 1)
    batch.load_lu_values(val)
    batch.refactor(0.0)
    b = torch.ones((1, 6000, n), dtype=torch.float64, device="cuda")
    few = b[:, :9].contiguous()               # the kernels are on the device before it is full
    batch.refine(val, few, batch.solve(few))
    torch.cuda.synchronize()
    spare = glu.Batch(plan, 16)               # 512 MB
    if call == "refine":
        x = batch.solve(b)
    before = torch.cuda.mem_get_info()[0]
    del spare
    assert torch.cuda.mem_get_info()[0] < before + (256 << 20)    # kept
    x = torch.empty_like(b)
    leave = {"solve": 160, "refine": 64, "plan": 64, "batch": 64}[call] << 20
    rest = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    assert torch.cuda.mem_get_info()[0] <= leave
    try:
        if call == "solve":
            batch.solve(b, out=x)             # 290 MB
        elif call == "refine":
            batch.refine(val, b, x)           # 96 MB
        elif call == "plan":
            glu.Plan(dense_symbolic(2800), dense_min=1)   # over 90 MB
        else:
            glu.Batch(other, 4)               # 128 MB
        torch.cuda.synchronize()
    finally:
        del rest
        torch.cuda.empty_cache()


def test_a_batch_made_while_another_thread_captures():
    """Taking over a destroyed batch's buffers waits for their last use only: a capture in another
    thread goes on, and its graph runs."""
    import torch
    n = 200
    plan = plan_for(n)
    a = matrices(n, 2, 4)
    val = torch.as_tensor(a.reshape(2, -1), device="cuda")
    b = torch.ones((2, 1, n), dtype=torch.float64, device="cuda")
    x, s = torch.empty_like(b), torch.cuda.Stream()
    ones = torch.ones(8, device="cuda")

    def use():
        batch = glu.Batch(plan, 2)
        batch.load_lu_values(val, stream=s)
        batch.refactor(0.0, stream=s)
        batch.solve(b, out=x, stream=s)
        s.synchronize()
        return batch

    use()                                     # destroyed: its buffers are there for the next
    x.zero_()
    made = []
    thread = threading.Thread(target=lambda: made.append(use()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="thread_local"):
        twice = ones * 2.0
        thread.start()
        thread.join()
        twice = twice + 1.0
    graph.replay()
    torch.cuda.synchronize()
    assert bool((twice == 3.0).all())
    check_solve(torch, made[0].get_lu(1).cpu().numpy(), b[1], x[1], False)


def test_a_captured_batch_is_not_taken_over():
    """A graph of a batch's work may still run after the batch: the plan's next batch has buffers of
    its own."""
    import torch
    n = 200
    plan = plan_for(n)
    a = matrices(n, 2, 5)
    val = torch.as_tensor(a.reshape(2, -1), device="cuda")
    b = torch.ones((2, 1, n), dtype=torch.float64, device="cuda")
    x, y = torch.empty_like(b), torch.empty_like(b)
    batch = glu.Batch(plan, 2)
    batch.load_lu_values(val)
    batch.refactor(0.0)
    batch.solve(b, out=x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        batch.solve(b, out=x)
    for _ in range(20):
        graph.replay()
    del batch                                 # with the graph's solves under way
    batch = glu.Batch(plan, 2)
    batch.load_lu_values(2.0 * val)
    batch.refactor(0.0)
    batch.solve(b, out=y)
    torch.cuda.synchronize()
    torch.testing.assert_close(y, 0.5 * x, rtol=1e-12, atol=0.0)
    check_solve(torch, batch.get_lu(1).cpu().numpy(), b[1], y[1], False)


def test_a_batch_outlives_its_plan():
    """A plan destroyed before its batch (the order of a garbage collection) stays until the batch
    goes; nothing of it is kept for another plan."""
    import torch
    n, count = 300, 16
    torch.cuda.synchronize()
    gc.collect()
    a = matrices(n, count, 6)
    val = torch.as_tensor(a.reshape(count, -1), device="cuda")
    b = torch.ones((count, 1, n), dtype=torch.float64, device="cuda")
    for k in range(3):
        plan = plan_for(n + 64 * k)
        batch = glu.Batch(plan, count)
        assert glu.lib().glu_plan_destroy(plan.h) == 0
        plan.h = None
        if k == 0:
            batch.load_lu_values(val)
            batch.refactor(0.0)
            x = batch.solve(b)
            check_solve(torch, batch.get_lu(3).cpu().numpy(), b[3], x[3], False)
        assert glu.lib().glu_batch_destroy(batch.h) == 0
        batch.h = None
