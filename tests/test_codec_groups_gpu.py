"""The codec kernels' groups of eight elements where their paths divide: tails,
buffers 4, 16 and 32 bytes aligned, rows shorter and longer than a warp's
groups, and groups with infinities, NaN, zeros, subnormals and ties among
ordinary values.  Codes and values equal the oracle's, byte for byte."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

ALIGN = 8  # floats of slack before a buffer's first element


def _values(n, seed):
    """Random bit patterns, ties and small integers, and runs of plain values
    (so that some groups of eight and some blocks hold only finite ones)."""
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal(n) * 4.0).astype(np.float32)
    bits = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32).view(np.float32)
    ties = (rng.integers(-64, 65, n) / 16.0).astype(np.float32)
    kind = np.repeat(rng.integers(0, 6, n // 40 + 1), 40)[:n]
    x = np.where(kind == 1, bits, np.where(kind == 2, ties, x)).astype(np.float32)
    x[kind == 3] *= np.float32(2.0**-140)
    x[kind == 4] *= np.float32(2.0**120)
    x[rng.random(n) < 0.01] = 0.0
    return x


def _placed(torch, data, dtype, shift):
    buf = torch.empty(ALIGN + shift + data.size + ALIGN, dtype=dtype, device="cuda")
    view = buf[ALIGN + shift:ALIGN + shift + data.size]
    view.copy_(torch.from_numpy(data))
    return view


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("n", [1, 8, 9, 41, 256, 4103])
@pytest.mark.parametrize("fmt", [1, 2, 3, 4, 5, 6, 7])
def test_groups_equal_the_oracle(ctx, msq, fmt, n, shift):
    import torch
    x = _values(n, 10 * n + shift)
    dev = _placed(torch, x, torch.float32, shift)
    v_ref, s_ref = O.encode(fmt, x)
    v, s = ctx.copy_to_storage(fmt, dev)
    assert np.array_equal(v.cpu().numpy().view(np.uint8).ravel()[:len(v_ref)], v_ref)
    if s_ref is not None and len(s_ref):
        assert np.array_equal(s.cpu().numpy().view(np.uint8).ravel()[:len(s_ref)], s_ref)
    got = ctx.storage_values(fmt, v, s, n).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), O.decode(fmt, v_ref, s_ref, n).astype(np.float32).view(np.uint32))
    w_ref, _ = O.encode_stochastic(fmt, x, 7, 3)
    w, _ = ctx.copy_to_storage_stochastic(fmt, dev, 7, 3)
    assert np.array_equal(w.cpu().numpy().view(np.uint8).ravel()[:len(w_ref)], w_ref)


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("row", [1, 3, 8, 24, 40, 100, 256, 264, 2048])
def test_rows_equal_the_oracle(ctx, msq, row, shift):
    import torch
    rows = 37
    x = _values(rows * row, row + shift)
    dev = _placed(torch, x, torch.float32, shift)
    v_ref, s_ref = O.encode(8, x, row_length=row)
    v, s = ctx.copy_to_storage(8, dev, row)
    assert np.array_equal(v.cpu().numpy().view(np.uint8).ravel(), v_ref)
    assert np.array_equal(s.cpu().numpy().view(np.uint32).ravel(), np.ascontiguousarray(s_ref).view(np.uint32).ravel())
    got = ctx.storage_values(8, v, s, rows * row, row).cpu().numpy()
    ref = O.decode(8, v_ref, s_ref, rows * row, row_length=row).astype(np.float32)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    w_ref, _ = O.encode_stochastic(8, x, 7, 3, row_length=row)
    w, _ = ctx.copy_to_storage_stochastic(8, dev, 7, 3, row)
    assert np.array_equal(w.cpu().numpy().view(np.uint8).ravel(), w_ref)


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("n", [7, 256, 264, 511, 4103])
@pytest.mark.parametrize("fmt,row", [(1, 0), (2, 0), (3, 0), (4, 0), (5, 0), (6, 0), (7, 0), (8, 1), (8, 11)])
def test_decoding_into_a_shifted_buffer(ctx, msq, fmt, row, n, shift):
    """Outputs 4, 16 and 32 bytes aligned, of whole warps and with tails; what
    lies before and behind the output stays as it was."""
    import ctypes
    import torch
    n = n // row * row if row else n
    if n == 0:
        return
    x = _values(n, n + shift)
    kw = {"row_length": row} if row else {}
    v_ref, s_ref = O.encode(fmt, x, **kw)
    want = O.decode(fmt, v_ref, s_ref, n, **kw).astype(np.float32)
    v, s = ctx.copy_to_storage(fmt, torch.from_numpy(x).cuda(), row)
    buf = torch.full((ALIGN + shift + n + ALIGN,), 3.0, device="cuda")
    out = buf[ALIGN + shift:]
    ctx.check(msq.lib().msq_decode(
        ctypes.c_void_p(ctx.handle.value), fmt, ctypes.c_void_p(v.data_ptr()),
        ctypes.c_void_p(s.data_ptr()) if s is not None else None, n, row, ctypes.c_void_p(out.data_ptr())), "decode")
    ctx.synchronize()
    got = buf.cpu().numpy()
    at = ALIGN + shift
    assert np.array_equal(got[at:at + n].view(np.uint32), want.view(np.uint32))
    assert (got[:at] == 3.0).all() and (got[at + n:] == 3.0).all()


@pytest.mark.parametrize("row", [31, 32, 33, 127, 128, 129])
def test_row_lengths_around_a_lanes_first_elements(ctx, msq, row):
    import torch
    x = _values(row * 19, row)
    v_ref, s_ref = O.encode(8, x, row_length=row)
    v, s = ctx.copy_to_storage(8, _placed(torch, x, torch.float32, 1), row)
    assert np.array_equal(v.cpu().numpy().view(np.uint8).ravel()[:len(v_ref)], v_ref)
    assert np.array_equal(s.cpu().numpy().view(np.uint8).ravel()[:len(s_ref)], s_ref)
