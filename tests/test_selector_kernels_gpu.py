"""The selector's kernels at the sizes where they can go wrong: features of
matrices of ragged orders, alignments and extreme scales, forward and
backward at row counts around a CTA's rows, against FP64.

Tolerances: features are FP32 results of sums good to 2^-45 (rounding 2^-24,
a logarithm near zero absolutely); logits are chains of at most 64 FP32 FMAs
(64 2^-24 of the sums' terms); gradients sum over rows besides."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _features(a):
    n = a.shape[0]
    d = np.diag(a)
    off = np.abs(a - np.diag(d))
    rows = off.sum(1)
    mean, tiny = d.sum() / n, 1e-30
    fro2, off2 = (a * a).sum(), (off * off).sum()
    dmin, dmax = d.min(), d.max()
    lg = lambda x: np.log10(max(x, tiny))  # noqa: E731
    return np.array([
        np.log2(n), lg(mean), lg(np.sqrt(fro2) / n), lg(dmin), lg(dmax),
        np.log10(max(dmax, tiny) / max(dmin, tiny)),
        max(-10.0, min(1.0, (d - rows).min() / max(mean, tiny))),
        np.log10(max((d + rows).max(), tiny) / max(mean, tiny)),
        np.sqrt(off2) / max(np.sqrt(fro2), tiny), min(100.0, rows.max() / max(dmin, tiny)),
        (off.sum() / (n * (n - 1.0))) / max(mean, tiny) if n > 1 else 0.0,
        lg(fro2 * n / max(d.sum() ** 2, tiny)),
        np.sqrt(max((d * d).sum() / n - mean * mean, 0.0)) / max(mean, tiny),
        (d > rows).mean(), 0.0, 1.0])


@pytest.mark.parametrize("orders", [[1], [2, 3, 31], [32, 33, 64, 65, 128], [257, 500, 16]])
@pytest.mark.parametrize("scale", [1.0, 1e-22, 1e22, 1e16, 1e17])
def test_features_against_fp64(ctx, msq, orders, scale):
    import torch
    b = msq.Batch.from_orders(orders)
    mats = [(O.wishart(n, seed=n) * scale).astype(np.float32) for n in orders]
    mats[0] = np.diag(np.diag(mats[0]))  # no off-diagonal entry at all
    f = ctx.features(torch.from_numpy(b.pack(mats)).cuda(), b).cpu().numpy()
    for m, got in zip(mats, f):
        np.testing.assert_allclose(got, _features(m.astype(np.float64)), rtol=4e-7, atol=4e-7)


@pytest.mark.parametrize("rows", [1, 3, 4, 5, 255, 1021])
def test_forward_and_backward_rows(ctx, msq, rows):
    import torch
    rng = np.random.default_rng(rows)
    p = (rng.standard_normal(msq.MLP_PARAMS) * 0.2).astype(np.float32)
    x = rng.standard_normal((rows, msq.MLP_IN)).astype(np.float32)
    y = (rng.random((rows, msq.MLP_OUT)) < 0.5).astype(np.float32)
    dev = lambda v: torch.from_numpy(v).cuda()  # noqa: E731
    z = ctx.mlp_forward(dev(p), dev(x)).cpu().numpy()
    z_ref, _ = O.mlp_forward(p, x.astype(np.float64))
    np.testing.assert_allclose(z, z_ref, rtol=0, atol=3 * 64 * 2.0**-24 * max(1.0, np.abs(z_ref).max()))
    grad = torch.zeros(msq.MLP_PARAMS, device="cuda")
    loss = ctx.mlp_backward(dev(p), dev(x), dev(y), grad)
    loss_ref, grad_ref = O.mlp_loss_and_grad(p, x, y)
    assert abs(float(loss.item()) - loss_ref) <= 1e-5 * loss_ref
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - grad_ref) <= 1e-5 * np.linalg.norm(grad_ref)


@pytest.mark.parametrize("n", [33, 100, 500])
@pytest.mark.parametrize("spread", [1e-3, 1e-5, 1e-6])
def test_features_of_a_nearly_constant_diagonal(ctx, msq, n, spread):
    """Feature 12 is the difference of two sums that agree to spread^2, feature 11
    the logarithm of their quotient.  An FP64 sum is off by some sqrt(n / 32 + 5)
    roundings of 0.3 2^-53 and less; with the squares and the mean's, 1.5 2^-53 of
    the sums: twice that, over 200 matrices, and the rounding to FP32."""
    import torch
    count = 200
    rng = np.random.default_rng(n)
    b = msq.Batch.from_orders([n] * count)
    mats = [np.diag(1.0 + spread * rng.standard_normal(n)).astype(np.float32) for _ in range(count)]
    got = ctx.features(torch.from_numpy(b.pack(mats)).cuda(), b).cpu().numpy().astype(np.float64)
    err = np.zeros((count, 2))
    for k, m in enumerate(mats):
        d = np.diag(m).astype(np.longdouble)
        mean = d.mean()
        var = ((d - mean) ** 2).mean() / mean**2
        err[k, 0] = got[k, 12] / float(np.sqrt(var)) - 1.0
        err[k, 1] = got[k, 11] / float(np.log1p(var) / np.log(np.longdouble(10))) - 1.0
    assert (np.sqrt((err**2).mean(0)) <= np.array([1, 2]) * (2.0**-24 + 3 * 2.0**-53 / spread**2)).all()


@pytest.mark.parametrize("n", [40, 300])
def test_features_where_columns_cancel_the_diagonal(ctx, msq, n):
    """Diagonal entries within FP32 rounding of their columns' sums: n terms of
    FP64 rounding are left of the difference, and it is rounded to FP32."""
    import torch
    rng = np.random.default_rng(n)
    a = np.abs(rng.standard_normal((n, n))).astype(np.float32)
    a = np.triu(a, 1) + np.triu(a, 1).T
    sums = a.astype(np.float64).sum(0)
    np.fill_diagonal(a, np.float32(sums))
    b = msq.Batch.from_orders([n])
    got = ctx.features(torch.from_numpy(b.pack([a])).cuda(), b).cpu().numpy()[0].astype(np.float64)
    d = np.diag(a).astype(np.float64)
    off = np.abs(a.astype(np.longdouble)).sum(0) - np.abs(d.astype(np.longdouble))
    low = (d - off).astype(np.float64)
    assert got[13] == np.float32((low > 0).mean())
    assert abs(got[6] - low.min() / d.mean()) <= 2.0**-23 * abs(low.min() / d.mean()) + n * 2.0**-53


def test_loss_is_summed_beyond_fp32(ctx, msq):
    """The mean of rows x 8 terms: each term rounds a few times at 2^-24 of its
    size (the terms' errors average), the sum of 64 CTAs' parts 64 times at half
    of 2^-24 at most."""
    import torch
    rows = 20000
    rng = np.random.default_rng(0)
    p = (rng.standard_normal(msq.MLP_PARAMS) * 0.2).astype(np.float32)
    x = rng.standard_normal((rows, msq.MLP_IN)).astype(np.float32)
    y = (rng.random((rows, msq.MLP_OUT)) < 0.5).astype(np.float32)
    dev = lambda v: torch.from_numpy(v).cuda()  # noqa: E731
    loss = ctx.mlp_backward(dev(p), dev(x), dev(y), torch.zeros(msq.MLP_PARAMS, device="cuda"))
    ref, _ = O.mlp_loss_and_grad(p, x, y)
    assert abs(float(loss.item()) - ref) <= 64 * 2.0**-25 * ref
