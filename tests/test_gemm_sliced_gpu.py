"""FP32 reconstruction and correction as sliced products on the tensor cores:
orders around tiles of 128, K steps of 32 and the 1024 of one exact sum, beside
small matrices that keep the FMA chains, against FP64.

Tolerances.  An element is exact sums, cut off below 2^-27 of the two vectors'
largest entries and rounded once: relative Frobenius 2 2^-24 for a product of
matrices of random entries, four of them (and what each rounding does to the
next) 8 2^-24; the chains' 8 sqrt(n) 2^-24 for the small ones.  For graded
matrices element (i, j) is off by at most 2 sqrt(n) 2^-27 + 2^-24 of the two
vectors' norms, doubled for the bound on the largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLICED = 256  # smallest order that may be sliced


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


@pytest.mark.parametrize("orders", [[870], [256] * 40, [384, 33, 385, 700, 1, 701, 255, 257], [1025], [2049]])
def test_products_against_fp64(ctx, msq, orders):
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(orders[0])
    mats = [(rng.standard_normal((n, n)) / np.sqrt(n)).astype(np.float32) for n in orders]
    res = [(rng.standard_normal((n, n)) * 1e-3).astype(np.float32) for n in orders]
    lam = rng.uniform(0.1, 1.0, int(b.n.sum())).astype(np.float32)
    f = _dev(b.pack(mats))
    x = ctx.reconstruct_factor(msq.PLAN_FP32, f, b)
    hi, lo = torch.zeros_like(f), torch.zeros_like(f)
    ctx.sylvester_sweep(msq.FP32, f, _dev(lam), _dev(b.pack(res)), b, hi, lo)
    torch.cuda.synchronize()
    at = 0
    for n, v, r, xg, eg in zip(orders, mats, res, b.unpack(x.cpu().numpy()), b.unpack(hi.cpu().numpy())):
        v, r, s = v.astype(np.float64), r.astype(np.float64), np.sqrt(lam[at:at + n].astype(np.float64))
        at += n
        scale = 4 * np.sqrt(n) if n < SLICED else 1.0
        ref = v.T @ v
        assert np.linalg.norm(xg - ref) <= 2 * scale * 2.0**-24 * np.linalg.norm(ref), n
        assert np.array_equal(xg, xg.T)
        c = (v.T @ r.T @ v) / (s[:, None] + s[None, :])
        e = v @ c @ v.T
        e = 0.5 * (e + e.T)
        assert np.linalg.norm(eg - e) <= 8 * scale * 2.0**-24 * np.linalg.norm(e), n


def test_graded_and_extreme_columns(ctx, msq):
    import torch
    n = 900
    b = msq.Batch.from_orders([n])
    rng = np.random.default_rng(1)
    f = np.diag(10.0 ** (-3 * np.arange(n) / n)) + 1e-3 * rng.standard_normal((n, n))
    f = f * 2.0 ** rng.integers(-40, 41, n)[None, :]  # columns of very different sizes
    f[:, 7] = 0.0
    f = f.astype(np.float32)
    x = ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b)
    torch.cuda.synchronize()
    got = b.unpack(x.cpu().numpy())[0]
    f64 = f.astype(np.float64)
    norm = np.linalg.norm(f64, axis=0)
    bound = 2 * (2 * np.sqrt(n) * 2.0**-27 + 2.0**-24) * np.outer(norm, norm)
    assert (np.abs(got - f64.T @ f64) <= bound).all()


def test_a_nan_stays_in_its_row_and_column(ctx, msq):
    import torch
    n, i = 900, 321
    b = msq.Batch.from_orders([n])
    f = (np.random.default_rng(2).standard_normal((n, n)) / 30).astype(np.float32)
    clean = b.unpack(ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b).cpu().numpy())[0]
    f[5, i] = np.nan
    got = b.unpack(ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b).cpu().numpy())[0]
    assert np.isnan(got[i]).all() and np.isnan(got[:, i]).all()
    rest = np.delete(np.arange(n), i)
    assert np.array_equal(got[np.ix_(rest, rest)], clean[np.ix_(rest, rest)])


def test_result_is_symmetric_where_sums_cancel(ctx, msq):
    """Columns of two kinds, even ones odd and odd ones even under an exchange of
    the neighbours in K, so that all but the smallest parts of their product
    cancel.  (i, j) and (j, i) add the parts in another order; one of the two is
    stored twice."""
    import torch
    n = 1024
    rng = np.random.default_rng(n)
    sign = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    odd = np.arange(n)[None, :] % 2 == 0  # by column: the first three digits change sign
    first = [np.repeat(d, 2, axis=0) for d in (np.full((n // 2, n), 60.0), rng.integers(-60, 61, (n // 2, n)),
                                               rng.integers(-60, 61, (n // 2, n)))]
    y = sum(d * 128.0**-p for p, d in enumerate(first))
    f = np.where(odd, sign[:, None] * y + 56 * 128.0**-3, y + sign[:, None] * 56 * 128.0**-3) / 64
    assert np.array_equal(f, f.astype(np.float32))
    b = msq.Batch.from_orders([n])
    x = ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b)
    torch.cuda.synchronize()
    xg = b.unpack(x.cpu().numpy(), np.float32)[0]
    assert np.array_equal(xg, xg.T)


def _weak(n, rng, eps):
    """Weakly coupled unit vectors: every column large in one place, the rest
    spread over four decades below eps."""
    return np.eye(n) + eps * 10.0 ** rng.uniform(-4, 0, (n, n)) * rng.standard_normal((n, n))


def _blocks(n, rng, eps):
    """Two groups of columns, each large where the other is small."""
    group = np.arange(n) % 2
    return rng.standard_normal((n, n)) * np.where(group[:, None] == group[None, :], 1.0, eps)


@pytest.mark.parametrize("make,eps", [(_weak, 1e-6), (_weak, 1e-8), (_blocks, 1e-6)])
@pytest.mark.parametrize("orders", [[900], [512, 130, 513, 640, 385, 700]])
def test_small_entries_keep_their_bits(ctx, msq, orders, make, eps):
    """Element by element within the bound of an FMA chain, n 2^-24 sum |a_k b_k|
    (a correction: of four chains with three roundings between them)."""
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(len(orders))
    mats = [make(n, rng, eps).astype(np.float32) for n in orders]
    res = [(1e-3 * make(n, rng, eps)).astype(np.float32) for n in orders]
    lam = rng.uniform(0.1, 1.0, int(b.n.sum())).astype(np.float32)
    f = _dev(b.pack(mats))
    x = ctx.reconstruct_factor(msq.PLAN_FP32, f, b)
    hi, lo = torch.zeros_like(f), torch.zeros_like(f)
    ctx.sylvester_sweep(msq.FP32, f, _dev(lam), _dev(b.pack(res)), b, hi, lo)
    torch.cuda.synchronize()
    at = 0
    for n, v, r, xg, eg in zip(orders, mats, res, b.unpack(x.cpu().numpy()), b.unpack(hi.cpu().numpy())):
        v, r, s = v.astype(np.float64), r.astype(np.float64), np.sqrt(lam[at:at + n].astype(np.float64))
        at += n
        assert (np.abs(xg - v.T @ v) <= n * 2.0**-24 * (np.abs(v.T) @ np.abs(v))).all(), n
        h = 1.0 / (s[:, None] + s[None, :])
        e = v @ ((v.T @ r.T @ v) * h) @ v.T
        m = np.abs(v) @ ((np.abs(v.T) @ np.abs(r.T) @ np.abs(v)) * h) @ np.abs(v.T)
        assert (np.abs(eg - 0.5 * (e + e.T)) <= 4 * (n + 3) * 2.0**-24 * 0.5 * (m + m.T)).all(), n


def test_single_products(ctx, msq):
    """A permuted diagonal matrix: one product per element, of which the pairs
    left out are 2^-25 and the two roundings of its sum 2^-24 and 2^-32."""
    n = 900
    rng = np.random.default_rng(3)
    f = np.zeros((n, n), np.float32)
    f[rng.permutation(n), np.arange(n)] = rng.standard_normal(n).astype(np.float32)
    b = msq.Batch.from_orders([n])
    x = b.unpack(ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b).cpu().numpy())[0]
    d = f.astype(np.float64).T @ f.astype(np.float64)
    assert (np.abs(x - d) <= (2.0**-24 + 2.0**-25 + 2.0**-31) * np.abs(d)).all()


def test_an_infinity_stays_one(ctx, msq):
    """As in FP32: infinite where it meets a nonzero finite entry."""
    n, i = 900, 321
    b = msq.Batch.from_orders([n])
    f = (np.random.default_rng(2).standard_normal((n, n)) / 30).astype(np.float32)
    f[5, i] = np.inf
    got = b.unpack(ctx.reconstruct_factor(msq.PLAN_FP32, _dev(b.pack([f])), b).cpu().numpy(), np.float32)[0]
    want = np.copysign(np.float32(np.inf), f[5])
    assert np.array_equal(got[i], want) and np.array_equal(got[:, i], want)
