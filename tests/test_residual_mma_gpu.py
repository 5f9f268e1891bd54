"""The residual on the tensor cores (digits of X, exact products) at the
edges of its tiles, K chunks and of the orders it takes, against FP64.

Tolerance: R is rounded to FP32 once (2^-24 of each entry); what the digits
drop and the FP64 reference rounds is below n 2^-53 ||X||^2 each, and a factor
of eight covers both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _root(n, rng, spread):
    """A symmetric float-float X whose columns span `spread` decades."""
    x = rng.standard_normal((n, n)) / np.sqrt(n) + np.eye(n)
    d = 10.0 ** rng.uniform(-spread, 0.0, n)
    x = d[:, None] * (x + x.T) * d[None, :]
    hi = x.astype(np.float32)
    return hi, (x - hi).astype(np.float32)


def _check(n, r, norms, a, a_lo, hi, lo):
    x = hi.astype(np.float64) + (0.0 if lo is None else lo.astype(np.float64))
    a64 = a.astype(np.float64) + (0.0 if a_lo is None else a_lo.astype(np.float64))
    ref = a64 - x @ x
    floor = 8 * n * 2.0**-53 * np.linalg.norm(x)**2
    assert np.linalg.norm(r - ref) <= 2.0**-24 * np.linalg.norm(ref) + floor
    assert abs(np.sqrt(norms[0]) - np.linalg.norm(ref)) <= 1e-12 * np.linalg.norm(ref) + floor
    assert abs(norms[1] - np.sum(a64 * a64)) <= 1e-12 * norms[1]


@pytest.mark.parametrize("orders", [[65, 66], [96], [127, 128, 129], [191, 192, 193, 20], [512, 513],
                                    [1, 640, 100, 33, 1025], [2047]])
@pytest.mark.parametrize("words", [(True, False), (False, False), (True, True)])
def test_residual_against_fp64(ctx, msq, orders, words):
    import torch
    rng = np.random.default_rng(sum(orders))
    b = msq.Batch.from_orders(orders)
    xs = [_root(n, rng, 0.0 if i % 2 == 0 else 3.0) for i, n in enumerate(orders)]
    mats = []
    for hi, lo in xs:
        e = rng.standard_normal(hi.shape) * 1e-6
        x = hi.astype(np.float64) + lo
        mats.append(x @ x + e + e.T)
    a = [m.astype(np.float32) for m in mats]
    a_lo = [(m - h).astype(np.float32) for m, h in zip(mats, a)]
    dev = lambda ms: torch.from_numpy(b.pack(ms)).cuda()  # noqa: E731
    with_lo, with_a_lo = words
    r, norms = ctx.residual(dev(a), dev([h for h, _ in xs]), dev([l for _, l in xs]) if with_lo else None,
                            b, a_lo=dev(a_lo) if with_a_lo else None)
    ctx.synchronize()
    norms = norms.cpu().numpy()
    for i, (n, rg) in enumerate(zip(orders, b.unpack(r.cpu().numpy()))):
        if n < 65:
            continue  # the CUDA-core kernel's, held to its own bound in test_pipeline_gpu.py
        _check(n, rg, norms[2 * i:2 * i + 2], a[i], a_lo[i] if with_a_lo else None, xs[i][0],
               xs[i][1] if with_lo else None)


@pytest.mark.parametrize("n", [130])
def test_extreme_columns_and_non_finite_entries(ctx, msq, n):
    """Columns scaled from 2^-60 to 2^60, an empty column, and the columns
    that a NaN or an infinity reaches."""
    import torch
    rng = np.random.default_rng(n)
    d = 2.0 ** rng.integers(-60, 60, n)
    d[3] = 0.0
    hi = (rng.standard_normal((n, n)) * np.sqrt(d[:, None] * d[None, :])).astype(np.float32)
    hi = np.triu(hi) + np.triu(hi, 1).T
    a = np.zeros((n, n), np.float32)
    b = msq.Batch.from_orders([n])
    dev = lambda m: torch.from_numpy(b.pack([m])).cuda()  # noqa: E731
    r, _ = ctx.residual(dev(a), dev(hi), None, b)
    ctx.synchronize()
    x = hi.astype(np.float64)
    size = np.abs(x).max(0)
    err = np.abs(b.unpack(r.cpu().numpy())[0] + x.T @ x)
    assert np.all(err <= 2.0**-23 * np.abs(x.T @ x) + n * 2.0**-50 * size[:, None] * size[None, :])
    for bad in (np.nan, np.inf):
        y = hi.copy()
        y[5, 7] = y[7, 5] = bad
        r, norms = ctx.residual(dev(a), dev(y), None, b)
        ctx.synchronize()
        rg = b.unpack(r.cpu().numpy())[0]
        hit = np.zeros(n, bool)
        hit[[5, 7]] = True
        assert not np.isfinite(rg[hit]).any() and not np.isfinite(rg[:, hit]).any()
        assert np.isfinite(rg[np.ix_(~hit, ~hit)]).all()
        assert not np.isfinite(norms.cpu().numpy()[0])
