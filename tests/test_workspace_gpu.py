"""Workspaces that grow with the batch: work in several runs over one arena, and
the paths that need none when the device has no memory left for it (refused by
msq_debug_scratch_limit, not by filling the GPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def refuse(msq):
    yield lambda size: msq.lib().msq_debug_scratch_limit(size)
    msq.lib().msq_debug_scratch_limit(0)


def _batch(msq, orders, seed=0):
    import torch
    b = msq.Batch.from_orders(orders)
    g = torch.Generator("cuda").manual_seed(seed)
    flat = torch.zeros(b.total, device="cuda")
    for n, o in zip(b.n.tolist(), b.offset.tolist()):
        x = torch.randn(n, n, device="cuda", generator=g) / n**0.5
        flat[o:o + n * n] = ((x + x.T) / 2 + 2 * torch.eye(n, device="cuda")).reshape(-1)
    return b, flat


def _members(msq, b, flat):
    for n, o in zip(b.n.tolist(), b.offset.tolist()):
        yield msq.Batch.from_orders([n]), flat[o:o + n * n]


def test_residual_of_more_digits_than_are_kept_at_a_time(ctx, msq):
    """45 matrices of order 2048 have 3 GB of digits: two runs, each matrix as
    alone (its norms as sums in another order)."""
    import torch
    orders = [2048] * 20 + [64, 70] + [2048] * 25
    b, x = _batch(msq, orders)
    a = x.clone()
    held = torch.cuda.mem_get_info()[0]
    fresh = msq.Context(0)
    try:
        r, norms = fresh.residual(a, x, None, b)
        fresh.synchronize()
        assert held - torch.cuda.mem_get_info()[0] < (2 << 30) + 4 * b.total + (64 << 20)  # digits, R, lists
    finally:
        fresh.close()
    for i, (one, xi) in enumerate(_members(msq, b, x)):
        if i % 9 and i not in (20, 21):
            continue
        ri, ni = ctx.residual(xi.contiguous(), xi.contiguous(), None, one)
        o, n = int(b.offset[i]), int(b.n[i])
        assert torch.equal(r[o:o + n * n], ri)
        assert torch.allclose(norms[2 * i:2 * i + 2], ni, rtol=1e-13, atol=0.0)


@pytest.mark.parametrize("orders", [[65], [130, 64, 300, 20]])
def test_residual_without_memory_for_digits(ctx, msq, refuse, orders):
    """The CUDA-core kernel's residual: off by n 2^-48 ||X||^2 at most, rounded."""
    import torch
    b, x = _batch(msq, orders)
    a = x * 0.5
    assert refuse(1) == 0
    r, norms = ctx.residual(a, x, None, b)
    ctx.synchronize()
    refuse(0)
    norms = norms.cpu().numpy()
    for i, ((_, xi), ri) in enumerate(zip(_members(msq, b, x), b.unpack(r.cpu().numpy()))):
        n = int(b.n[i])
        xi = xi.reshape(n, n).double().cpu().numpy()
        ref = 0.5 * xi - xi @ xi
        floor = 8 * n * 2.0**-48 * np.linalg.norm(xi) ** 2
        assert np.linalg.norm(ri - ref) <= 2.0**-24 * np.linalg.norm(ref) + floor
        assert abs(np.sqrt(norms[2 * i]) - np.linalg.norm(ref)) <= 1e-12 * np.linalg.norm(ref) + floor


def test_solve_without_memory_for_workspaces(ctx, msq, refuse):
    """Direct (the launch shapes are tuned meanwhile), captured and replayed:
    accepted every time, with equal roots."""
    import torch
    b, x = _batch(msq, [200, 65, 130])
    a = torch.zeros_like(x)
    for n, o in zip(b.n.tolist(), b.offset.tolist()):
        m = x[o:o + n * n].view(n, n)
        a[o:o + n * n] = (m @ m).reshape(-1)
    plans = [msq.plan(msq.PLAN_BF16, 2, 1e-4)] * 3
    fresh = msq.Context(0)
    try:
        assert refuse(1) == 0
        out = torch.empty_like(a)
        roots = []
        for _ in range(8):
            _, res = fresh.solve_batched(a, b, plans, out=out)
            assert all(r.accepted == 1 for r in res)
            roots.append(out.clone())
        assert fresh.graph_launches > 0
        assert all(torch.equal(roots[0], r) for r in roots)
    finally:
        refuse(0)
        fresh.close()


def _correct(ctx, msq, fmt, b, v, w, r):
    import torch
    hi, lo = torch.zeros_like(v), torch.zeros_like(v)
    ctx.sylvester_sweep(fmt, v, w, r, b, hi, lo)
    return hi, lo


def test_products_of_more_pieces_than_are_kept_at_a_time(ctx, msq):
    """30 matrices of order 2048 have 3 GB of pieces: two runs, each matrix as
    alone."""
    import torch
    orders = [2048] * 12 + [70, 300] + [2048] * 18
    b, v = _batch(msq, orders)
    w = torch.linspace(0.5, 1.5, int(b.n.sum()), device="cuda")
    x = ctx.reconstruct_factor(msq.PLAN_FP32, v, b)
    hi, _ = _correct(ctx, msq, msq.FP32, b, v, w, v)
    eig = b.eig_offset
    for i, (one, vi) in enumerate(_members(msq, b, v)):
        n, o, k = int(b.n[i]), int(b.offset[i]), int(eig[i])
        if n < 2048 or i % 5:
            continue
        vi = vi.contiguous()
        assert torch.equal(x[o:o + n * n], ctx.reconstruct_factor(msq.PLAN_FP32, vi, one))
        assert torch.equal(hi[o:o + n * n], _correct(ctx, msq, msq.FP32, one, vi, w[k:k + n].contiguous(), vi)[0])


@pytest.mark.parametrize("orders", [[900], [512, 130, 700, 33, 300]])
def test_products_without_memory_for_pieces(ctx, msq, refuse, orders):
    """FMA chains: each of the four within sqrt(n) 2^-24 and a little of its terms'
    norms, as in test_gemm_tiles_gpu.py."""
    import torch
    b, v = _batch(msq, orders)
    w = torch.linspace(0.5, 1.5, int(b.n.sum()), device="cuda")
    assert refuse(1) == 0
    x = b.unpack(ctx.reconstruct_factor(msq.PLAN_FP32, v, b).cpu().numpy())
    hi = b.unpack(_correct(ctx, msq, msq.FP32, b, v, w, v)[0].cpu().numpy())
    refuse(0)
    for i, (_, vi) in enumerate(_members(msq, b, v)):
        n = int(b.n[i])
        m = vi.reshape(n, n).double().cpu().numpy()
        s = np.sqrt(w[int(b.eig_offset[i]):int(b.eig_offset[i]) + n].double().cpu().numpy())
        ref = m @ m
        assert np.linalg.norm(x[i] - ref) <= 8 * np.sqrt(n) * 2.0**-24 * np.linalg.norm(ref)
        h = 1.0 / (s[:, None] + s[None, :])
        e = m @ ((m @ m @ m) * h) @ m
        size = np.linalg.norm(np.abs(m) @ ((np.abs(m) @ np.abs(m) @ np.abs(m)) * h) @ np.abs(m))
        assert np.linalg.norm(hi[i] - (e + e.T) / 2) <= 8 * np.sqrt(n) * 2.0**-24 * size


def test_split_products_with_six_buffers(ctx, msq, refuse):
    """V and its transpose take the same buffers in turn: the same bits."""
    import torch
    b, v = _batch(msq, [300, 64, 129])
    w = torch.linspace(0.5, 1.5, int(b.n.sum()), device="cuda")
    want = _correct(ctx, msq, msq.BF16, b, v, w, v)
    assert refuse(1) == 0
    got = _correct(ctx, msq, msq.BF16, b, v, w, v)
    refuse(0)
    assert all(torch.equal(x, y) for x, y in zip(got, want))
