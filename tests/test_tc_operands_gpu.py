"""The operand packs and the mirrored tiles of the tensor-core products at the
edges of tiles, of 32-element blocks and of vector alignment (an odd order
before an even one), against FP64 products of the oracle's quantized factor.

Tolerances (relative Frobenius): FP32 accumulation of exact products, 2e-6;
the split-BF16 correction drops a term of 2^-18 and rounds two second pieces
at 2^-18 in each of its four products, 12 2^-18 and four accumulations; the
factor is two square roots and a product, each rounded once (2^-22)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

ACC = 2e-6
ORDERS = [[1, 2, 31], [33, 64, 128], [127, 129, 34, 255], [257, 256, 63, 130], [640]]


def _dev(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


def _quantized(fmt, f):
    n = f.shape[0]
    row = n if fmt == 8 else 0
    cols = [O.decode(fmt, *O.encode(fmt, np.ascontiguousarray(f[:, i]), row_length=row), n, row_length=row)
            for i in range(n)]
    return np.stack(cols, axis=1).astype(np.float64)


@pytest.mark.parametrize("orders", ORDERS)
@pytest.mark.parametrize("plan,fmt", [(1, 1), (2, 8), (3, 7)])
def test_reconstruction_from_the_factor(ctx, msq, orders, plan, fmt):
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(orders[0])
    fs = []
    for n in orders:
        f = rng.standard_normal((n, n)) * 2.0 ** rng.integers(-12, 1, (n, n))
        f[: n // 2, n // 3] = 0.0  # zero blocks of a row
        fs.append(f.astype(np.float32))
    x = ctx.reconstruct_factor(plan, _dev(b.pack(fs)), b)
    torch.cuda.synchronize()
    for f, xg in zip(fs, b.unpack(x.cpu().numpy())):
        q = _quantized(fmt, f)
        ref = q.T @ q
        assert np.linalg.norm(xg - ref) <= ACC * np.linalg.norm(ref), f.shape
        assert np.array_equal(xg, xg.T)


@pytest.mark.parametrize("orders", ORDERS)
def test_factor_and_split_correction(ctx, msq, orders):
    import torch
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(orders[-1])
    mats = [(rng.standard_normal((n, n)) / np.sqrt(n)).astype(np.float32) for n in orders]
    res = [rng.standard_normal((n, n)) * 1e-3 for n in orders]
    res = [(r + r.T).astype(np.float32) for r in res]
    lam = rng.uniform(0.1, 1.0, int(b.n.sum())).astype(np.float32)
    v = _dev(b.pack(mats))
    f = ctx.make_factor(v, _dev(lam), b)
    hi, lo = torch.zeros_like(v), torch.zeros_like(v)
    ctx.sylvester_sweep(msq.BF16, v, _dev(lam), _dev(b.pack(res)), b, hi, lo)
    torch.cuda.synchronize()
    at = 0
    for n, m, r, fg, eg in zip(orders, mats, res, b.unpack(f.cpu().numpy()), b.unpack(hi.cpu().numpy())):
        m, r, s = m.astype(np.float64), r.astype(np.float64), np.sqrt(lam[at:at + n].astype(np.float64))
        at += n
        np.testing.assert_allclose(fg, (m * np.sqrt(s)).T, rtol=2.0**-22, atol=0)
        c = (m.T @ r @ m) / (s[:, None] + s[None, :])
        e = m @ c @ m.T
        e = 0.5 * (e + e.T)
        assert np.linalg.norm(eg - e) <= (12 * 2.0**-18 + 4 * ACC) * np.linalg.norm(e), n


@pytest.mark.parametrize("plan", [1, 2, 3])
def test_mirrored_tiles_are_the_computed_ones(ctx, msq, plan):
    """A batch of more tiles than SMs (its lower tiles mirrored) against the
    same matrices one at a time (every tile computed), bit for bit."""
    import torch
    orders = [257, 130, 33, 600] * 5  # 39 tiles a group
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(plan)
    fs = [rng.standard_normal((n, n)).astype(np.float32) for n in orders]
    x = ctx.reconstruct_factor(plan, _dev(b.pack(fs)), b)
    torch.cuda.synchronize()
    for f, xg in zip(fs, b.unpack(x.cpu().numpy())):
        one = msq.Batch.from_orders([f.shape[0]])
        alone = ctx.reconstruct_factor(plan, _dev(one.pack([f])), one)
        assert np.array_equal(xg, one.unpack(alone.cpu().numpy())[0]), f.shape


@pytest.mark.parametrize("source", ["bf16", "fp8", "mxfp4", "bf16 codes", "fp8 codes", "mxfp4 flat codes",
                                    "mxfp4 codes", "mxfp8 codes"])
def test_packs_of_many_tiles(ctx, msq, source):
    """More operand tiles than four per SM (CTAs of four warps) against the
    matrices one at a time (of eight), bit for bit."""
    import torch
    aligned = source in ("mxfp4 codes", "mxfp8 codes")
    orders = ([256, 128, 32, 608] if aligned else [257, 130, 33, 600]) * 30
    b = msq.Batch.from_orders(orders)
    rng = np.random.default_rng(len(source))
    flat = _dev((rng.standard_normal(b.total) * 2.0 ** rng.integers(-12, 1, b.total)).astype(np.float32))
    fmt = {"bf16 codes": 1, "fp8 codes": 8, "mxfp8 codes": 4}.get(source, 7)
    if fmt == 8:  # row scales: matrix by matrix
        values, scales = torch.zeros(b.total, dtype=torch.uint8, device="cuda"), []
        for n, o in zip(b.n.tolist(), b.offset.tolist()):
            v, sc = ctx.copy_to_storage(fmt, flat[o:o + n * n].clone(), n)
            values[o:o + n * n] = v.view(torch.uint8).reshape(-1)
            scales.append(sc.view(torch.float32).reshape(-1))
        scales = torch.cat(scales)
    elif "codes" in source:
        values, scales = ctx.copy_to_storage(fmt, flat)

    def run(batch, first):
        out = torch.zeros_like(flat)
        if "codes" not in source:
            return ctx.reconstruct_factor({"bf16": 1, "fp8": 2, "mxfp4": 3}[source], flat, batch, out)
        return ctx.reconstruct(fmt, values, scales[first:] if fmt == 8 else scales, batch, out)

    x = b.unpack(run(b, 0).cpu().numpy())
    for i in [*range(4), *range(len(orders) - 4, len(orders))]:
        one = msq.Batch(b.n[i:i + 1].copy(), b.offset[i:i + 1].copy(), b.total)
        alone = one.unpack(run(one, int(b.eig_offset[i])).cpu().numpy())[0]
        assert np.abs(alone).max() > 0.0 and np.array_equal(x[i], alone), orders[i]


@pytest.mark.parametrize("n", [5, 33, 130])
def test_fp8_factor_with_an_infinity_and_a_nan(ctx, msq, n):
    """Words of four codes with an entry that the hardware conversion would not
    code as the codec does."""
    import torch
    b = msq.Batch.from_orders([n])
    f = np.random.default_rng(n).standard_normal((n, n)).astype(np.float32)
    f[2, 1], f[3, n - 1] = np.inf, np.nan
    x = b.unpack(ctx.reconstruct_factor(2, _dev(b.pack([f])), b).cpu().numpy())[0]
    torch.cuda.synchronize()
    q = _quantized(8, f)
    ref = q.T @ q
    assert np.array_equal(np.isnan(x), np.isnan(ref))
    ok = np.isfinite(ref)
    assert np.linalg.norm(x[ok] - ref[ok]) <= ACC * np.linalg.norm(ref[ok])
