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
