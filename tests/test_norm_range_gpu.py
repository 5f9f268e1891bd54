"""Norms of the residual, and what the solver decides from them, for matrices
in small and in large units.

A scaled by 4^k and X by 2^k give R and both norms scaled exactly, so each is
held to FP64 at every scale.  Tolerance: as test_residual_mma_gpu.py, 1e-12 of
a norm for sums of squares carried to 2^-48 and more, beside the rounding of
the digits and of the reference (8 n 2^-53 ||X||^2 of the residual's norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCALES = [-45, -35, -32, -12, 0, 12, 32, 35, 45]  # of X; of A twice that: R and its low words stay normal numbers


def _case(n, rng):
    x = rng.standard_normal((n, n)) / np.sqrt(n)
    x = (x + x.T) / 2 + 2.0 * np.eye(n)
    hi = x.astype(np.float32)
    lo = (x - hi).astype(np.float32)
    full = hi.astype(np.float64) + lo
    e = rng.standard_normal((n, n))
    a = (full @ full + 1e-3 * (e + e.T)).astype(np.float32)
    return a, hi, lo


def _norms(ctx, msq, b, a, hi, lo):
    import torch
    dev = lambda m: torch.from_numpy(b.pack([m])).cuda()  # noqa: E731
    _, norms = ctx.residual(dev(a), dev(hi), dev(lo), b)
    ctx.synchronize()
    return norms.cpu().numpy()


def _hold(norms, a, hi, lo):
    x = hi.astype(np.float64) + lo
    r = a.astype(np.float64) - x @ x
    floor = 8 * len(a) * 2.0**-53 * np.linalg.norm(x)**2
    assert abs(np.sqrt(norms[0]) - np.linalg.norm(r)) <= 1e-12 * np.linalg.norm(r) + floor
    assert abs(np.sqrt(norms[1]) - np.linalg.norm(a.astype(np.float64))) <= 1e-12 * np.sqrt(norms[1])


@pytest.mark.parametrize("n", [64, 65, 130, 512])
def test_norms_at_extreme_scales(ctx, msq, n):
    b = msq.Batch.from_orders([n])
    a, hi, lo = _case(n, np.random.default_rng(n))
    for k in SCALES:
        s = np.float32(2.0**k)
        sa, sh, sl = a * s * s, hi * s, lo * s
        _hold(_norms(ctx, msq, b, sa, sh, sl), sa, sh, sl)


@pytest.mark.parametrize("n", [129, 260])
def test_norms_of_blocks_in_different_units(ctx, msq, n):
    """The two halves of the matrix 2^80 apart: each tile at its own scale."""
    rng = np.random.default_rng(n)
    a, hi, lo = _case(n, rng)
    h = n // 2
    for m in (a, hi, lo):
        m[:h, h:] = m[h:, :h] = 0.0
    a[:h, :h] *= np.float32(2.0**-80)
    hi[:h, :h] *= np.float32(2.0**-40)
    lo[:h, :h] *= np.float32(2.0**-40)
    b = msq.Batch.from_orders([n])
    _hold(_norms(ctx, msq, b, a, hi, lo), a, hi, lo)
    a[h:, h:] = hi[h:, h:] = lo[h:, h:] = 0.0
    _hold(_norms(ctx, msq, b, a, hi, lo), a, hi, lo)
    z = np.zeros_like(a)
    assert np.all(_norms(ctx, msq, b, z, z, z) == 0.0)
    norms = _norms(ctx, msq, b, a, z, z)  # X = 0: R = A
    assert abs(norms[0] - norms[1]) <= 1e-12 * norms[1] and norms[1] > 0.0


@pytest.mark.parametrize("n", [65, 129, 260])
def test_norms_of_sparse_matrices(ctx, msq, n):
    """Tiles, rows and residuals of zeros beside single entries whose squares FP32
    does not hold: X a diagonal of powers of two, A its square and one such entry."""
    x = np.diag(2.0 ** np.random.default_rng(n).integers(-3, 4, n)).astype(np.float32)
    z = np.zeros_like(x)
    b = msq.Batch.from_orders([n])
    for small in (0.0, 2.0**-100, 1.0):
        a = x * x
        a[n - 1, 1] = a[1, n - 1] = np.float32(small)
        norms = _norms(ctx, msq, b, a, x, z)
        want = 2.0 * float(np.float32(small))**2
        assert abs(norms[0] - want) <= 1e-12 * want
        full = np.sum(a.astype(np.float64)**2)
        assert abs(norms[1] - full) <= 1e-12 * full


@pytest.mark.parametrize("n", [64, 65, 130])
def test_acceptance_does_not_depend_on_units(ctx, msq, n):
    """An MXFP4 root without a correction misses 1e-5 and falls back at every
    scale, and the FP32 root that replaces it meets it."""
    import torch
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, 2 * n))
    a = (g @ g.T / (2 * n)).astype(np.float32)
    b = msq.Batch.from_orders([n])
    for k in (0, -35, 33):
        s = np.float32(2.0**(2 * k))
        _, res = ctx.solve_batched(torch.from_numpy(b.pack([a * s])).cuda(), b,
                                   plans=[msq.plan(msq.PLAN_MXFP4, 0)], tolerance=1e-5)
        assert res[0].fallback == 1 and res[0].plan_residual > 1e-5
        assert 0.0 < res[0].final_residual <= 1e-5
