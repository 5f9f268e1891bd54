"""Workloads that the speed of the framework is judged on.

Each case is one thing that a program does with the framework through its
public Python entry points: the codecs of a stored basis, the whole solve of
one matrix or of a batch, and the stages that a program with its own loop
calls (factor and reconstruction, residual and correction, the
native-quantized correction, the learned plan selector).  `listed` names the
cases, `draw` gives others of the same ranges, `prepare` makes what a program
has in hand before the call, `run` is the call.
"""
from __future__ import annotations

import importlib
import math
import os

import numpy as np
import torch

msq = importlib.import_module("mixed-mlx_gb300")
selector = importlib.import_module("mixed-mlx_gb300.selector")

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(msq.__file__)), "selector_weights.npz")
FORMATS = {"bf16": msq.BF16, "fp8_e4m3fn": msq.FP8_E4M3FN, "fp8_e5m2": msq.FP8_E5M2,
           "mxfp8_e4m3fn": msq.MXFP8_E4M3FN, "mxfp8_e5m2": msq.MXFP8_E5M2,
           "fp4_e2m1": msq.FP4_E2M1, "mxfp4_e2m1": msq.MXFP4_E2M1,
           "fp8_e4m3fn_rowscale": msq.FP8_E4M3FN_ROWSCALE, "fp32": msq.FP32}
# stored bits per value, scale bits among them
BITS = {"bf16": 16, "fp8_e4m3fn": 8, "fp8_e5m2": 8, "mxfp8_e4m3fn": 8.25, "mxfp8_e5m2": 8.25,
        "fp4_e2m1": 4, "mxfp4_e2m1": 4.25, "fp8_e4m3fn_rowscale": 8, "fp32": 32}
PLANS = {"fp32": msq.PLAN_FP32, "bf16": msq.PLAN_BF16, "fp8": msq.PLAN_FP8,
         "mxfp4": msq.PLAN_MXFP4}


def listed():
    return [
        # a 256 x 256 eigenbasis stored in FP8 with a scale per row and read
        # back: what one small solve stores; latency
        {"name": "codec_rowscale_256", "kind": "codec", "format": "fp8_e4m3fn_rowscale",
         "elements": 256 * 256, "row": 256, "stochastic": False},
        # the MXFP4 codec on a large tensor, both directions; bandwidth
        {"name": "codec_mxfp4_64m", "kind": "codec", "format": "mxfp4_e2m1",
         "elements": 1 << 26, "row": 0, "stochastic": False},
        # stochastic rounding of a basis of order 2047 (a ragged last block)
        {"name": "codec_stochastic_mxfp8", "kind": "codec", "format": "mxfp8_e4m3fn",
         "elements": 2047 * 2047, "row": 0, "stochastic": True},
        # the plain FP32 solve of one matrix of order 256, condition 1e3:
        # the single-matrix benchmark, and the smallest whole call
        {"name": "solve_one_256_fp32", "kind": "solve_one", "n": 256, "cond": 1e3,
         "plan": "fp32"},
        # one large matrix with the BF16 basis and two corrections (the
        # low-bit sweep of the single-matrix benchmark)
        {"name": "solve_one_2048_bf16", "kind": "solve_one", "n": 2048, "cond": 1e2,
         "plan": "bf16"},
        # the headline: 4096 Wishart covariances, orders log-uniform in
        # [16, 512], with the plan that the learned selector picks for them
        {"name": "solve_wishart_4096_bf16", "kind": "solve_batch", "count": 4096, "lo": 16,
         "hi": 512, "plan": "bf16"},
        # the plain FP32 path on a batch of a few hundred, as a program
        # without low-bit plans runs it
        {"name": "solve_wishart_300_fp32", "kind": "solve_batch", "count": 300, "lo": 16,
         "hi": 512, "plan": "fp32"},
        # factor and reconstruction with block-scaled MXFP4 operands at the
        # largest order of the MXFP4 benchmark
        {"name": "reconstruct_8192_mxfp4", "kind": "reconstruct", "count": 1, "lo": 8192,
         "hi": 8192, "plan": "mxfp4"},
        # residual and FP32 correction of four matrices of order 1000
        {"name": "correct_1000_fp32", "kind": "correct", "count": 4, "lo": 1000, "hi": 1000,
         "gemm": "fp32"},
        # residual and tensor-core correction of an uneven batch
        {"name": "correct_uneven_bf16", "kind": "correct", "count": 96, "lo": 64, "hi": 512,
         "gemm": "bf16"},
        # the native-quantized correction, every stage stored in the basis
        # format, on eight matrices of order 384
        {"name": "native_384_mxfp8", "kind": "native", "count": 8, "lo": 384, "hi": 384,
         "format": "mxfp8_e4m3fn"},
        # the learned selector on 256 matrices: features, predictions, and
        # one training step (backward and Adam) on them
        {"name": "selector_256", "kind": "selector", "count": 256, "lo": 64, "hi": 512},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _log_orders(rng, lo, hi, most):
    """An order range within [lo, hi] and a batch size that keeps the sum of
    n^2 below `most`."""
    a, b = sorted((_log_int(rng, lo, hi), _log_int(rng, lo, hi)))
    return a, b, _log_int(rng, 1, max(1, min(4096, most // (b * b))))


def draw(rng):
    kind = rng.choice(["codec", "solve_one", "solve_batch", "reconstruct", "correct", "native",
                       "selector"])
    if kind == "codec":
        form = rng.choice(sorted(f for f in FORMATS if f != "fp32"))
        stochastic = rng.random() < 0.25
        row = _log_int(rng, 16, 4096) if form == "fp8_e4m3fn_rowscale" else 0
        elements = _log_int(rng, 1 << 10, 1 << (24 if stochastic else 26))
        if row:
            elements = max(1, elements // row) * row
        return {"kind": kind, "format": form, "elements": elements, "row": row,
                "stochastic": stochastic}
    if kind == "solve_one":
        return {"kind": kind, "n": _log_int(rng, 32, 1600),
                "cond": 10.0 ** rng.choice([1.0, 2.0, 3.0]), "plan": "fp32"}
    if kind == "solve_batch":
        lo, hi, count = _log_orders(rng, 16, 512, 1 << 26)
        return {"kind": kind, "count": count, "lo": lo, "hi": hi,
                "plan": rng.choice(["bf16", "fp32"])}
    if kind == "reconstruct":
        lo, hi, count = _log_orders(rng, 64, 4096, 1 << 24)
        return {"kind": kind, "count": min(count, 256), "lo": lo, "hi": hi,
                "plan": rng.choice(sorted(PLANS))}
    if kind == "correct":
        lo, hi, count = _log_orders(rng, 64, 1536, 1 << 23)
        return {"kind": kind, "count": min(count, 128), "lo": lo, "hi": hi,
                "gemm": rng.choice(["fp32", "bf16"])}
    if kind == "native":
        lo, hi, count = _log_orders(rng, 64, 1024, 1 << 22)
        return {"kind": kind, "count": min(count, 64), "lo": lo, "hi": hi,
                "format": rng.choice(["bf16", "mxfp8_e4m3fn", "mxfp4_e2m1", "fp32"])}
    lo, hi, count = _log_orders(rng, 16, 1024, 1 << 26)
    return {"kind": kind, "count": max(16, min(count, 1024)), "lo": lo, "hi": hi}


# ---- inputs ---------------------------------------------------------------

_CONTEXT = None


def _context():
    """One context for the process, as a program keeps it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = msq.Context(0)
    return _CONTEXT


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _orders(case):
    """The case's orders: log-uniform in [lo, hi], the same for every seed
    (a program keeps its batch layout and gets new matrices)."""
    if case["lo"] == case["hi"]:
        return np.full(case["count"], case["lo"], dtype=np.int32)
    rng = np.random.default_rng(case["count"])
    u = rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["count"])
    return np.clip(np.floor(np.exp(u)), case["lo"], case["hi"]).astype(np.int32)


def _members(flat, batch):
    """Views of a packed batch's matrices (all symmetric, or taken as
    stored: element (r, c) of a column-major matrix at [c, r])."""
    for n, at in zip(batch.n, batch.offset):
        n, at = int(n), int(at)
        yield flat[at:at + n * n].view(n, n)


def _gaps(batch):
    """Positions between the matrices of a packed batch (up to three floats
    after a matrix of odd order, which nothing defines)."""
    n2 = batch.n.astype(np.int64) ** 2
    at = [np.arange(o + k, (o + k + 3) // 4 * 4) for o, k in zip(batch.offset, n2) if k % 4]
    return torch.from_numpy(np.concatenate(at)).cuda() if at else None


def _wishart(batch, seed):
    """Covariances X^T X / m + 1e-6 I, X ~ N(0, 1) of m = 2n rows."""
    g = _generator(seed)
    flat = torch.zeros(batch.total, device="cuda")
    for a in _members(flat, batch):
        n = a.shape[0]
        x = torch.randn(2 * n, n, generator=g, device="cuda")
        w = x.T @ x
        torch.add(w, w.T, out=a)
        a.mul_(0.25 / n)
        a.diagonal().add_(1e-6)
    return flat


def _basis(n, g, dtype):
    """A random orthonormal basis: Q of the QR of a Gaussian matrix."""
    return torch.linalg.qr(torch.randn(n, n, generator=g, device="cuda", dtype=dtype))[0]


def _spectrum(n, cond, g, dtype):
    """Eigenvalues log-uniform in [1 / cond, 1]."""
    return torch.exp(torch.rand(n, generator=g, device="cuda", dtype=dtype) * -math.log(cond))


def _eigen(case, seed, dtype):
    """(batch, [(Q, lambda)]) of matrices with condition up to 1e3; bases of
    equal order are drawn together."""
    batch = msq.Batch.from_orders(_orders(case))
    g = _generator(seed)
    by_order, out = {}, [None] * batch.count
    for i, n in enumerate(batch.n):
        by_order.setdefault(int(n), []).append(i)
    for n, ids in by_order.items():
        for i in ids:
            out[i] = (_basis(n, g, dtype), _spectrum(n, 1e3, g, dtype))
    return batch, out


def _pack(batch, mats):
    flat = torch.zeros(batch.total, device="cuda")
    for dst, a in zip(_members(flat, batch), mats):
        dst.copy_(a.T)  # column-major storage
    return flat


def _source(case, seed):
    """Values of a stored basis: entries of an orthonormal basis of order n
    are close to N(0, 1 / n)."""
    n = math.isqrt(case["elements"])
    return torch.randn(case["elements"], generator=_generator(seed), device="cuda") / math.sqrt(n)


def _correction_inputs(case, seed):
    """A, its eigenbasis and spectrum, and a root X0 of 16-bit accuracy to be
    corrected, as the reconstruction of a quantized basis leaves it."""
    batch, eig = _eigen(case, seed, torch.float32)
    a = _pack(batch, [(q * lam) @ q.T for q, lam in eig])
    for m in _members(a, batch):
        m.copy_(0.5 * (m + m.T))
    x0 = _pack(batch, [((q * lam.sqrt()) @ q.T).bfloat16().float() for q, lam in eig])
    for m in _members(x0, batch):
        m.copy_(torch.triu(m) + torch.triu(m, 1).T)
    v = _pack(batch, [q for q, _ in eig])
    return batch, a, v, torch.cat([lam for _, lam in eig]), x0


def _plan(name, jacobi_tolerance=1e-2):
    # the plans that the selector and the benchmark use: two corrections of a
    # BF16 root (Jacobi to 1e-2 in the batch, to 1e-3 for one large matrix),
    # one FP32 correction of an FP32 one
    return msq.plan(PLANS[name], 2, jacobi_tolerance, 15) if name == "bf16" else \
        msq.plan(msq.PLAN_FP32, 1, 1e-7, 15)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ctx": _context(), "case": case}
    if kind == "codec":
        s.update(x=_source(case, seed), fmt=FORMATS[case["format"]], seed=seed & 0xffff)
    elif kind == "solve_one":
        g = _generator(seed)
        q, lam = _basis(case["n"], g, torch.float64), _spectrum(case["n"], case["cond"], g, torch.float64)
        batch = msq.Batch.from_orders([case["n"]])
        a = _pack(batch, [(q * lam) @ q.T])
        for m in _members(a, batch):
            m.copy_(0.5 * (m + m.T))
        s.update(batch=batch, a=a, out=torch.zeros_like(a), plans=[_plan(case["plan"], 1e-3)])
    elif kind == "solve_batch":
        batch = msq.Batch.from_orders(_orders(case))
        a = _wishart(batch, seed)
        s.update(batch=batch, a=a, out=torch.zeros_like(a), gaps=_gaps(batch),
                 plans=[_plan(case["plan"])] * batch.count)
    elif kind == "reconstruct":
        batch = msq.Batch.from_orders(_orders(case))
        g = _generator(seed)
        # entries of an orthonormal basis (its values, not its exact
        # orthogonality, are what the products see)
        v = torch.randn(batch.total, generator=g, device="cuda")
        for m in _members(v, batch):
            m.div_(math.sqrt(m.shape[0]))
        lam = torch.exp(torch.rand(int(batch.n.sum()), generator=g, device="cuda") * -math.log(1e4))
        s.update(batch=batch, v=v, lam=lam, plan=PLANS[case["plan"]], out=torch.zeros_like(v))
    elif kind == "correct":
        batch, a, v, lam, x0 = _correction_inputs(case, seed)
        s.update(batch=batch, a=a, v=v, lam=lam, x0=x0, gemm=FORMATS[case["gemm"]],
                 work=torch.empty(2 * batch.total, device="cuda"))
    elif kind == "native":
        batch, a, v, lam, x0 = _correction_inputs(case, seed)
        fmt, ctx = FORMATS[case["format"]], s["ctx"]
        # the stored basis and its transpose, quantized matrix by matrix
        vq, vtq = torch.zeros_like(v), torch.zeros_like(v)
        for src, dst, dst_t in zip(_members(v, batch), _members(vq, batch), _members(vtq, batch)):
            for x, y in ((src, dst), (src.T.contiguous(), dst_t)):
                codes, scales = ctx.copy_to_storage(fmt, x.reshape(-1), x.shape[0])
                y.copy_(ctx.storage_values(fmt, codes, scales, x.numel(), x.shape[0]).view_as(y))
        r, _ = ctx.residual(a, x0, None, batch)
        s.update(batch=batch, v=vq, vt=vtq, roots=lam.sqrt(), x0=x0, r=r, fmt=fmt)
    elif kind == "selector":
        batch = msq.Batch.from_orders(_orders(case))
        a = _wishart(batch, seed)
        net, _, _ = selector.load(msq, torch, s["ctx"], WEIGHTS)
        targets = (torch.rand(batch.count, msq.MLP_OUT, generator=_generator(seed + 1),
                              device="cuda") < 0.5).float()
        s.update(batch=batch, a=a, net=net, targets=targets, grad=torch.zeros_like(net.params))
    else:
        raise ValueError(kind)
    return s


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "codec":
        case, x, fmt = s["case"], s["x"], s["fmt"]
        if case["stochastic"]:
            codes, scales = ctx.copy_to_storage_stochastic(fmt, x, s["seed"], 1, case["row"])
        else:
            codes, scales = ctx.copy_to_storage(fmt, x, case["row"])
        values = ctx.storage_values(fmt, codes, scales, x.numel(), case["row"])
        if scales is None:
            return {"codes": codes, "values": values}
        if fmt == msq.FP8_E4M3FN_ROWSCALE:
            scales = scales.view(torch.float32)
        return {"codes": codes, "scales": scales, "values": values}
    if kind in ("solve_one", "solve_batch"):
        root, results = ctx.solve_batched(s["a"], s["batch"], s["plans"], 1e-5, s["out"])
        # what the caller reads of the results (the residuals themselves are
        # rounding noise of the accepted root)
        table = np.ctypeslib.as_array(results)
        if s.get("gaps") is not None:
            root.index_fill_(0, s["gaps"], 0.0)
        return {"root": root, "accepted": table["accepted"], "fallback": table["fallback"],
                "jacobi_sweeps": table["jacobi_sweeps"]}
    if kind == "reconstruct":
        f = ctx.make_factor(s["v"], s["lam"], s["batch"])
        return {"root": ctx.reconstruct_factor(s["plan"], f, s["batch"], s["out"])}
    if kind == "correct":
        x_hi, x_lo = s["x0"].clone(), torch.zeros_like(s["x0"])
        r, norms = ctx.residual(s["a"], x_hi, x_lo, s["batch"])
        ctx.sylvester_sweep(s["gemm"], s["v"], s["lam"], r, s["batch"], x_hi, x_lo, s["work"])
        # the corrected root's high word (the low word is below its last
        # place and has no digits that can be compared by themselves)
        return {"root": x_hi, "residual": list(_members(r, s["batch"]))[-1], "norms": norms}
    if kind == "native":
        x_hi, x_lo = s["x0"].clone(), torch.zeros_like(s["x0"])
        ctx.native_sylvester_sweep(s["fmt"], s["v"], s["vt"], s["roots"], s["r"], s["batch"],
                                   x_hi, x_lo)
        return {"root": x_hi}
    net, batch = s["net"], s["batch"]
    feats = selector.features(ctx, torch, batch, s["a"], 1e-5)
    x = net.normalise(feats).contiguous()
    logits = ctx.mlp_forward(net.params, x)
    s["grad"].zero_()
    loss = ctx.mlp_backward(net.params, x, s["targets"], s["grad"])
    net.step += 1
    ctx.mlp_step(net.params, s["grad"], net.m, net.v, net.step, 3e-4)
    return {"features": feats, "logits": logits, "loss": loss, "grad": s["grad"],
            "params": net.params}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "codec":
        stored = BITS[case["format"]] / 8.0
        return {"bytes": case["elements"] * (8.0 + 2.0 * stored), "flops": 0.0}
    if kind == "solve_one":
        n = np.asarray([case["n"]], dtype=np.float64)
    else:
        n = _orders(case).astype(np.float64)
    n2, n3 = float((n ** 2).sum()), float((n ** 3).sum())
    if kind in ("solve_one", "solve_batch"):
        low = case["plan"] == "bf16"
        # about 6 Jacobi sweeps to 1e-2 and 9 to 1e-7, each 4 n^3 FMA-flops on
        # the triangle of A and 4 n^3 on V; the reconstruction and per
        # correction 4 products; residuals 2 n^3 each
        sweeps, corrections = (6, 2) if low else (9, 1)
        return {"bytes": 8.0 * n2, "flops": (8.0 * sweeps + 2.0 + corrections * 8.0 +
                                             (corrections + 1) * 2.0) * n3}
    if kind == "reconstruct":
        return {"bytes": 8.0 * n2, "flops": 2.0 * n3}
    if kind == "correct":
        return {"bytes": 20.0 * n2, "flops": 10.0 * n3}
    if kind == "native":
        return {"bytes": 20.0 * n2, "flops": 8.0 * n3}
    rows, params = float(len(n)), float(msq.MLP_PARAMS)
    return {"bytes": 4.0 * n2 + rows * 4.0 * (msq.MLP_IN + 2 * msq.MLP_OUT) + 28.0 * params,
            "flops": 8.0 * rows * params}


# ---- the same in 64 bits -----------------------------------------------------

def _sqrt_newton(a):
    """Principal roots of a batch of well-conditioned SPD matrices (coupled
    Newton-Schulz iteration from A scaled to norm below 1)."""
    c = a.abs().sum(-1).amax(-1)[:, None, None]
    y, z = a / c, torch.eye(a.shape[-1], dtype=a.dtype, device=a.device).expand_as(a)
    eye3 = 3.0 * z
    for _ in range(24):
        t = 0.5 * (eye3 - z @ y)
        y, z = y @ t, t @ z
        if float((t - eye3 / 3.0).abs().amax()) < 1e-13:
            break
    return y * c.sqrt()


def _exact_roots(a, batch):
    out = torch.zeros(batch.total, dtype=torch.float64, device="cuda")
    views = list(_members(out, batch))
    mats = list(_members(a, batch))
    ids = sorted(range(batch.count), key=lambda i: int(batch.n[i]))
    group = 0
    while group < len(ids):
        n_max, part = 0, []
        while group < len(ids) and len(part) < 64:
            n = int(batch.n[ids[group]])
            if part and n > 1.2 * int(batch.n[part[0]]) + 8:
                break
            n_max = max(n_max, n)
            part.append(ids[group])
            group += 1
        # orders of a group padded with a unit diagonal
        stack = torch.eye(n_max, dtype=torch.float64, device="cuda").repeat(len(part), 1, 1)
        for k, i in enumerate(part):
            n = int(batch.n[i])
            stack[k, :n, :n] = mats[i].double()
        roots = _sqrt_newton(stack)
        for k, i in enumerate(part):
            n = int(batch.n[i])
            views[i].copy_(roots[k, :n, :n])
    return out


def _e2m1_rows(f):
    """MXFP4 values of the rows of f: blocks of 32 with a power-of-two scale
    that puts the block's largest value in the top binade, each value rounded
    to the nearest of 0, 0.5, 1, 1.5, 2, 3, 4, 6 (ties to the even code)."""
    rows, n = f.shape
    pad = -n % 32
    x = torch.nn.functional.pad(f, (0, pad)).view(rows, -1, 32)
    top = x.abs().amax(-1, keepdim=True)
    exponent = torch.floor(torch.log2(top.double())) - 2
    scale = torch.where(top > 0, torch.exp2(exponent), torch.ones_like(exponent))
    y = (x.double() / scale).abs().clamp(max=6.0)
    step = torch.where(y < 2.0, 0.5, torch.where(y < 4.0, 1.0, 2.0))
    q = (torch.round(y / step) * step).clamp(max=6.0)
    return (q * torch.sign(x.double()) * scale).reshape(rows, -1)[:, :n]


def exact(case, seed):
    kind = case["kind"]
    if kind == "codec":
        return None  # codes and what they stand for: compared as they are
    if kind in ("solve_one", "solve_batch"):
        if kind == "solve_one" and case["n"] > 3000:
            return None
        s = prepare(case, seed)
        if kind == "solve_batch":
            root = _exact_roots(s["a"], s["batch"])
        else:
            n = case["n"]
            lam, q = torch.linalg.eigh(next(_members(s["a"], s["batch"])).double())
            root = torch.zeros(s["batch"].total, dtype=torch.float64, device="cuda")
            root[:n * n] = ((q * lam.clamp(min=0).sqrt()) @ q.T).reshape(-1)
        return {"root": root, "accepted": None, "fallback": None, "jacobi_sweeps": None}
    if kind == "reconstruct":
        if case["plan"] == "fp8":
            return None  # 8-bit codes of FP32 quotients: no 64-bit value of their own
        s = prepare(case, seed)
        root = torch.zeros(s["batch"].total, dtype=torch.float64, device="cuda")
        at = 0
        for v, dst in zip(_members(s["v"], s["batch"]), _members(root, s["batch"])):
            n = v.shape[0]
            # row i of W: v is stored with [k, i] = V_ik; the stored factor is
            # its FP32 value
            quarter = s["lam"][at:at + n].sqrt().sqrt()
            w = (v * quarter[:, None]).T.contiguous()
            at += n
            if case["plan"] == "bf16":
                w = w.bfloat16()
            w = _e2m1_rows(w) if case["plan"] == "mxfp4" else w.double()
            dst.copy_(w @ w.T)
        return {"root": root}
    if kind == "correct":
        s = prepare(case, seed)
        root = torch.zeros(s["batch"].total, dtype=torch.float64, device="cuda")
        norms, at, r = [], 0, None
        for a, v, x, dst in zip(*(_members(t, s["batch"]) for t in (s["a"], s["v"], s["x0"], root))):
            n = a.shape[0]
            a, v, x = a.double(), v.double().T, x.double()
            root_lam = s["lam"][at:at + n].double().sqrt()
            at += n
            r = a - x @ x
            norms += [(r * r).sum(), (a * a).sum()]
            c = (v.T @ r @ v) / (root_lam[:, None] + root_lam[None, :])
            e = v @ c @ v.T
            dst.copy_(x + 0.5 * (e + e.T))
        return {"root": root, "residual": r, "norms": torch.stack(norms)}
    if kind == "native":
        if case["format"] not in ("fp32", "bf16"):
            return None
        s = prepare(case, seed)
        root = torch.zeros(s["batch"].total, dtype=torch.float64, device="cuda")
        at = 0

        def stored(x):
            return x.bfloat16().double() if case["format"] == "bf16" else x
        for r, v, vt, x, dst in zip(*(_members(t, s["batch"])
                                      for t in (s["r"], s["v"], s["vt"], s["x0"], root))):
            n = r.shape[0]
            r, v, vt = (t.double().T for t in (r, v, vt))
            roots = s["roots"][at:at + n].double()
            at += n
            w = stored(stored(vt @ stored(r)) @ v)
            c = stored(w / (roots[:, None] + roots[None, :]))
            e = stored(stored(v @ c) @ vt)
            dst.copy_(x.double() + 0.5 * (e + e.T))
        return {"root": root}
    s = prepare(case, seed)
    feats = torch.stack([_features(a.double()) for a in _members(s["a"], s["batch"])])
    net = s["net"]
    x = (feats - net.mean.double()) / net.std.double()
    p = net.params
    sizes, weights, at = ((64, 16), (64, 64), (8, 64)), [], 0
    for rows, cols in sizes:
        w = p[at:at + rows * cols].bfloat16().double().view(rows, cols).requires_grad_()
        b = p[at + rows * cols:at + rows * cols + rows].bfloat16().double().requires_grad_()
        weights.append((w, b))
        at += rows * cols + rows
    h = x
    for k, (w, b) in enumerate(weights):
        h = h @ w.T + b
        h = torch.relu(h) if k < 2 else h
    loss = torch.nn.functional.binary_cross_entropy_with_logits(h, s["targets"].double())
    loss.backward()
    grad = torch.cat([t.grad.reshape(-1) for pair in weights for t in pair])
    # the first Adam step from zero moments
    step = 3e-4 * grad / (grad.abs() + 1e-8)
    return {"features": feats, "logits": h.detach(), "loss": loss.detach().reshape(1),
            "grad": grad, "params": p.double() - step}


def _features(a):
    """The selector's 16 features of one matrix."""
    n = a.shape[0]
    d = a.diagonal()
    off = (a - torch.diag(d)).abs()
    rows = off.sum(1)
    mean, tiny = d.sum() / n, 1e-30
    fro2, off2 = (a * a).sum(), (off * off).sum()
    log10 = lambda t: torch.log10(torch.clamp(t, min=tiny))  # noqa: E731
    one = torch.ones((), dtype=a.dtype, device=a.device)
    return torch.stack([
        math.log2(n) * one, log10(mean), log10(fro2.sqrt() / n), log10(d.min()), log10(d.max()),
        log10(d.max() / d.min()), torch.clamp((d - rows).min() / mean, -10.0, 1.0),
        log10((d + rows).max() / mean), off2.sqrt() / fro2.sqrt(),
        torch.clamp(rows.max() / torch.clamp(d.min(), min=tiny), max=100.0),
        off.sum() / max(1, n * (n - 1)) / mean, log10(fro2 * n / (d.sum() ** 2)),
        torch.clamp((d * d).sum() / n - mean * mean, min=0.0).sqrt() / mean,
        (d > rows).double().mean(), -5.0 * one, one])
