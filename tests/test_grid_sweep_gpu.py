"""The grid Jacobi's sweep kernel at the edges of its layouts: padded orders,
rows of V and rotations in shared memory (n <= about 2300), rotations only
(n <= about 6500), neither; and its barrier's bounded wait.

Against the FP64 spectrum and orthogonality where the CPU restatement of the
blocked order would take minutes; tolerances as in the other tests of the
eigensolver (n u ||A|| with u = 2^-24, a few times over)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _toeplitz(n):
    """Equal diagonal entries (ties of the rotation angle), a band of exact
    zeros (pairs that are not rotated)."""
    d = np.abs(np.subtract.outer(np.arange(n), np.arange(n)))
    return np.where(d < 9, 0.5 ** d, 0.0)


@pytest.mark.parametrize("n,family", [(291, "spd"), (304, "spd"), (328, "toeplitz"), (617, "spd")])
def test_bit_exact_against_cpu_restatement(ctx, msq, n, family):
    import torch
    a = _toeplitz(n) if family == "toeplitz" else O.spd_loguniform(n, 1e3, seed=n)
    b = msq.Batch.from_orders([n])
    assert msq.jacobi_route([n])[0] == 1
    w_o, v_o, _, _, a_o = O.jacobi_blocked(a, 0.0, 2, with_matrix=True)
    t = torch.from_numpy(b.pack([a])).cuda()
    v, w, sweeps, off = ctx.jacobi(t, b, 0.0, 2)
    ctx.synchronize()
    assert np.array_equal(w.cpu().numpy(), w_o)
    assert np.array_equal(b.unpack(v.cpu().numpy(), np.float32)[0], v_o)
    assert np.array_equal(b.unpack(t.cpu().numpy(), np.float32)[0], a_o)


@pytest.mark.parametrize("n", [2300, 2600, 6600])
def test_layouts_of_large_orders(ctx, msq, n):
    """Two sweeps are a similarity transform: V orthogonal, V^T A V equal to
    the rotated matrix, the trace kept."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, n, generator=g, device="cuda")
    a = (x + x.T) / np.sqrt(8.0 * n)
    b = msq.Batch.from_orders([n])
    t = torch.zeros(b.total, device="cuda")
    t[:n * n] = a.reshape(-1)
    v, w, sweeps, off = ctx.jacobi(t, b, 0.0, 2)
    ctx.synchronize()
    vm = v[:n * n].view(n, n).T.double()  # column-major
    rot = t[:n * n].view(n, n).double()
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    # 2 (m - 1) rotations per row, each rounding to u: about sqrt(4 n) u per
    # entry direction, ten times over
    tol = 10 * np.sqrt(4.0 * n) * 2.0**-24
    assert float((vm.T @ vm - eye).norm()) <= tol * np.sqrt(n)
    ref = vm.T @ a.double() @ vm
    assert float((ref - rot).norm()) <= tol * float(a.double().norm())


def test_expired_barrier_is_reported_and_the_context_recovers(ctx, msq):
    import torch
    n = 300
    a = O.spd_loguniform(n, 1e2, seed=1).astype(np.float32)
    b = msq.Batch.from_orders([n])
    lib = msq.lib()
    ctx.synchronize()
    assert lib.msq_debug_expire_waits(1) == 0
    try:
        ctx.jacobi(torch.from_numpy(b.pack([a])).cuda(), b, 1e-7, 2)
        with pytest.raises(msq.MsqError, match="wait expired"):
            ctx.synchronize()
    finally:
        assert lib.msq_debug_expire_waits(0) == 0
    v, w, sweeps, off = ctx.jacobi(torch.from_numpy(b.pack([a])).cuda(), b, 1e-7, 15)
    ctx.synchronize()
    ref = np.linalg.eigvalsh(a.astype(np.float64))
    np.testing.assert_allclose(np.sort(w.cpu().numpy()), ref, rtol=0, atol=3 * n * 2.0**-24)


def test_report_of_an_earlier_call_does_not_stop_the_sweeps(ctx, msq):
    """A status word left by another call (a log-spectrum that is not positive)
    is reported by the next check, and the matrix is solved all the same, bit
    for bit."""
    import torch
    n = 1040
    assert msq.jacobi_route([n])[0] == 1
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    a = ((a + a.T) / 2).astype(np.float32)
    b = msq.Batch.from_orders([n])
    dev = torch.from_numpy(b.pack([a])).cuda()
    want = [t.cpu() for t in ctx.jacobi(dev.clone(), b, 1e-6, 15)]
    ctx.synchronize()
    ctx.copy_spectrum_to_storage(msq.FP8_E4M3FN, torch.full((8,), -1.0, device="cuda"))
    got = [t.cpu() for t in ctx.jacobi(dev, b, 1e-6, 15)]
    with pytest.raises(msq.MsqError, match="log-spectrum"):
        ctx.synchronize()
    assert want[2][0] > 1 and all(torch.equal(x, y) for x, y in zip(got, want))
