"""The first call on a new layout: its host work grows with the number of
matrices and of tiles, no faster."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["reconstruct", "correct", "native"])
def test_first_call_on_many_matrices(ctx, msq, what):
    """30000 matrices: milliseconds of host work per list of tiles, seconds and
    more if a pass over the batch were made for each matrix."""
    import torch
    n = {"reconstruct": 5, "correct": 6, "native": 7}[what]  # a layout of its own
    b = msq.Batch.from_orders([n] * 30000)
    v = torch.zeros(b.total, device="cuda")
    w = torch.ones(int(b.n.sum()), device="cuda")
    hi, lo = torch.zeros_like(v), torch.zeros_like(v)
    ws = torch.empty(2 * b.total, device="cuda")
    torch.cuda.synchronize()
    start = time.perf_counter()
    if what == "reconstruct":
        ctx.reconstruct_factor(msq.PLAN_FP32, v, b, hi)
    elif what == "correct":
        ctx.sylvester_sweep(msq.FP32, v, w, v, b, hi, lo, ws)
    else:
        ctx.native_sylvester_sweep(msq.FP32, v, v, w, v, b, hi, lo)
    ctx.synchronize()
    assert time.perf_counter() - start < 1.0
    assert not np.any(hi.cpu().numpy())
