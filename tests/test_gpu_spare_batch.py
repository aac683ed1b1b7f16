"""A destroyed batch's buffers taken over by the plan's next batch of the same count."""
from __future__ import annotations

import gc

import numpy as np
import pytest

from glu_public_b200 import glu
from tests.test_gpu_dense_solve import check_solve, plan_for
from tests.test_gpu_dense_steps import check_lu, matrices

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
