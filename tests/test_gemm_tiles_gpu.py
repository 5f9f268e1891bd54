"""The FP32 GEMM behind reconstruction and correction at the edges of its
tiles (32, 64, 128) and K steps, against FP64 products of the same operands.

Tolerance: an n-long FP32 FMA chain of random-sign terms has a relative
Frobenius error of about sqrt(n) 2^-24; a correction passes through four of
them, and 8 sqrt(n) 2^-24 leaves a factor of two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orders", [
    [1], [31], [32, 33], [63, 64, 65], [127, 128, 129], [300], [256] * 20,  # 32- and 64-tiles
    [24] * 300 + [100] * 80,                                               # both in one call
    [1000, 1001, 1023, 1025], [1409, 40]])                                 # 128-tiles
def test_reconstruction_and_correction_at_tile_edges(ctx, msq, orders):
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(len(orders) + orders[0])
    mats = [(rng.standard_normal((n, n)) / np.sqrt(n)).astype(np.float32) for n in orders]
    res = [(rng.standard_normal((n, n)) * 1e-3).astype(np.float32) for n in orders]
    lam = rng.uniform(0.1, 1.0, int(b.n.sum())).astype(np.float32)
    f = torch.from_numpy(b.pack(mats)).cuda()
    x = ctx.reconstruct_factor(msq.PLAN_FP32, f, b)
    hi, lo = torch.zeros_like(f), torch.zeros_like(f)
    ctx.sylvester_sweep(msq.FP32, f, torch.from_numpy(lam).cuda(),
                        torch.from_numpy(b.pack(res)).cuda(), b, hi, lo)
    torch.cuda.synchronize()
    at = 0
    for n, v, r, xg, eg in zip(orders, mats, res, b.unpack(x.cpu().numpy()),
                               b.unpack(hi.cpu().numpy())):
        tol = 8 * np.sqrt(n) * 2.0**-24
        v, r, s = v.astype(np.float64), r.astype(np.float64), np.sqrt(lam[at:at + n].astype(np.float64))
        at += n
        ref = v.T @ v
        assert np.linalg.norm(xg - ref) <= tol * np.linalg.norm(ref)
        assert np.array_equal(xg, xg.T)
        # the kernel reads the residual as R^T (equal for the symmetric R of a solve)
        c = (v.T @ r.T @ v) / (s[:, None] + s[None, :])
        e = v @ c @ v.T
        e = 0.5 * (e + e.T)
        assert np.linalg.norm(eg - e) <= tol * np.linalg.norm(e)


@pytest.mark.parametrize("orders", [
    [1, 31, 33], [63, 64, 65] * 30,             # 32- and 64-tiles
    [1000, 1001, 1023, 1025], [1409, 40]])      # 128-tiles
@pytest.mark.parametrize("trans", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("mode", ["plain", "same", "roots"])
def test_general_products_at_tile_edges(ctx, msq, orders, trans, mode):
    """msq_gemm, which is FMA chains at every order: every layout of the operands,
    an operand with itself (mirrored where the layouts agree) and the division by
    the sums of roots.  An element is within n 2^-24 sum |a_k b_k|, and the roots,
    their sum and the quotient round four times."""
    import ctypes
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(len(orders))
    am = [rng.standard_normal((n, n)).astype(np.float32) for n in orders]
    bm = am if mode == "same" else [rng.standard_normal((n, n)).astype(np.float32) for n in orders]
    lam = rng.uniform(0.1, 1.0, int(b.n.sum())).astype(np.float32)
    a = torch.from_numpy(b.pack(am)).cuda()
    bb = a if mode == "same" else torch.from_numpy(b.pack(bm)).cuda()
    w, c = torch.from_numpy(lam).cuda(), torch.zeros_like(a)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    ctx.check(msq.lib().msq_gemm(
        ctypes.c_void_p(ctx.handle.value), trans[0], trans[1], ptr(a), ptr(bb), ctypes.c_void_p(b.n.ctypes.data),
        ctypes.c_void_p(b.offset.ctypes.data), b.count, ptr(w) if mode == "roots" else None, ptr(c)), "msq_gemm")
    ctx.synchronize()
    at = 0
    for n, x, y, got in zip(orders, am, bm, b.unpack(c.cpu().numpy())):
        x, y = (m.astype(np.float64).T if t else m.astype(np.float64) for m, t in zip((x, y), trans))
        s = np.sqrt(lam[at:at + n].astype(np.float64))
        at += n
        h = 1.0 / (s[:, None] + s[None, :]) if mode == "roots" else 1.0
        bound = (n + 4) * 2.0**-24 * (np.abs(x) @ np.abs(y)) * h
        assert (np.abs(got - (x @ y) * h) <= bound).all()
        if mode == "same" and trans[0] != trans[1]:
            assert np.array_equal(got, got.T)


def test_batches_of_small_orders(ctx, msq):
    """Orders 1 .. 32 in a batch large enough for the one-step products and the
    kernels without shared memory, bit for bit what the same matrices give
    beside one of order 33 in a small batch."""
    import ctypes
    import torch
    orders = list(range(1, 33))
    many, few = msq.Batch.from_orders(orders * 10), msq.Batch.from_orders(orders + [33])
    rng = np.random.default_rng(32)
    vm, rm = ([rng.standard_normal((n, n)).astype(np.float32) for n in orders + [33]] for _ in range(2))
    lam = rng.uniform(0.1, 1.0, int(few.n.sum())).astype(np.float32)
    own = int(sum(orders))

    def run(b, times):
        pick = (lambda m: m) if times == 1 else (lambda m: m[:-1] * times)
        v, r = (torch.from_numpy(b.pack(pick(m))).cuda() for m in (vm, rm))
        w = torch.from_numpy(lam if times == 1 else np.tile(lam[:own], times)).cuda()
        out = [ctx.make_factor(v, w, b), ctx.reconstruct_factor(msq.PLAN_FP32, v, b)]
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        for ta, tb in ((0, 0), (1, 0), (0, 1), (1, 1)):
            c = torch.zeros_like(v)
            ctx.check(msq.lib().msq_gemm(
                ctypes.c_void_p(ctx.handle.value), ta, tb, ptr(v), ptr(r), ctypes.c_void_p(b.n.ctypes.data),
                ctypes.c_void_p(b.offset.ctypes.data), b.count, ptr(w), ptr(c)), "msq_gemm")
            out.append(c)
        hi, lo = out[1].clone(), torch.zeros_like(v)
        ctx.sylvester_sweep(msq.FP32, v, w, r, b, hi, lo)
        ctx.synchronize()
        return [b.unpack(t.cpu().numpy()) for t in out + [hi, lo]]

    for got, ref in zip(run(many, 10), run(few, 1)):
        for i, g in enumerate(got):
            assert np.array_equal(g, ref[i % len(orders)]), g.shape
