"""One context used on two streams in turn: the calls share its workspaces and
must give the bits that they give one after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _symmetric(msq, orders, seed):
    import torch
    rng = np.random.default_rng(seed)
    b = msq.Batch.from_orders(orders)
    mats = []
    for n in orders:
        x = rng.standard_normal((n, n)) / np.sqrt(n)
        mats.append((x + x.T + 4.0 * np.eye(n)).astype(np.float32))
    return b, torch.from_numpy(b.pack(mats)).cuda()


def _calls(ctx, msq, b, x):
    import torch
    w = torch.linspace(0.5, 1.5, int(b.n.sum()), device="cuda")
    zero = torch.zeros_like(x)

    def correct():
        hi, lo = x.clone(), torch.zeros_like(x)
        ctx.sylvester_sweep(msq.FP32, x, w, x, b, hi, lo)
        return hi, lo

    return {"residual": lambda: ctx.residual(zero, x, None, b),
            "features": lambda: (ctx.features(x, b),),
            "reconstruct": lambda: (ctx.reconstruct_factor(msq.PLAN_FP32, x, b),
                                    ctx.reconstruct_factor(msq.PLAN_BF16, x, b)),
            "correct": correct}


@pytest.mark.parametrize("what", ["residual", "features", "reconstruct", "correct"])
def test_calls_on_two_streams(ctx, msq, what):
    """A long call on one stream, short ones on another right behind it."""
    import torch
    home = ctx.stream
    large, small = (_calls(ctx, msq, *_symmetric(msq, orders, 7)) for orders in ([1000] * 4 + [70] * 40, [130, 900]))
    want = [[t.cpu() for t in c[what]()] for c in (large, small)]
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        got = []
        for _ in range(5):
            for stream, c in ((one, large), (two, small)):
                with torch.cuda.stream(stream):
                    ctx.set_stream(stream)
                    got.append(c[what]())
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(home)
    for i, out in enumerate(got):
        # a float sum of norms may be added in another order
        for x, y in zip(out, want[i % 2]):
            if x.dtype == torch.float64:
                assert torch.allclose(x.cpu(), y, rtol=1e-13, atol=0.0)
            else:
                assert torch.equal(x.cpu(), y)


def test_solve_behind_a_call_on_another_stream(ctx, msq):
    """A replayed solve on one stream behind a long correction on another."""
    import torch
    home = ctx.stream
    b, x = _symmetric(msq, [300, 64, 65], 3)
    plans = [msq.plan(msq.PLAN_BF16, 1)] * 3
    out = torch.empty_like(x)
    side = torch.cuda.Stream()
    try:
        # on the side stream from the start: the graph belongs to its stream
        ctx.set_stream(side)
        torch.cuda.synchronize()
        for _ in range(3):
            ctx.solve_batched(x, b, plans, out=out)
        want = out.cpu()
        ctx.set_stream(home)
        big, y = _symmetric(msq, [700] * 6, 5)
        zero, hi, lo = torch.zeros_like(y), y.clone(), torch.zeros_like(y)
        w = torch.ones(int(big.n.sum()), device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):
            ctx.set_stream(home)
            ctx.sylvester_sweep(msq.BF16, y, w, zero, big, hi, lo)
            ctx.set_stream(side)
            ctx.solve_batched(x, b, plans, out=out)
            assert torch.equal(out.cpu(), want)
    finally:
        torch.cuda.synchronize()
        ctx.set_stream(home)
    assert torch.equal(hi, y)  # the correction of a zero residual is zero
