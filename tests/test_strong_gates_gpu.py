"""Gates at the far end of what a caller can pass, forward and backward, against the recurrences in fp64: raw 16-bit logits
whose exponential overflows fp32, log-gates of -inf, of a type's lowest value, far outside the range that a segment's factored
form covers, and growing ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu
# relative 2-norm errors: results are rounded to the type once or twice on the way (2^-9, 2^-12)
TOL = {torch.float32: 1e-5, torch.bfloat16: 1e-2, torch.float16: 2e-3}


def _inputs(dtype, B, H, L, dk, dv, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda d: torch.randn(B, H, L, d, generator=gen, device="cuda")  # noqa: E731
    return [t.to(dtype) for t in (rand(dk), rand(dk), rand(dv))], [rand(dk), rand(dk)], rand(dv).to(dtype)


def _scan64(q, k, v, g, c, reverse, d_out):
    """One direction in fp64: (o, dq, dk, dv, d log-gate)."""
    B, H, L, dk = k.shape
    order = list(range(L - 1, -1, -1) if reverse else range(L))
    S = torch.zeros(B, H, dk, v.shape[-1], dtype=torch.float64, device=k.device)
    Z, a = torch.zeros_like(S), g.exp()
    o, dq, dkk, dvv = torch.empty_like(v), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    for t in order:
        S = S * a[:, :, t, :, None] + k[:, :, t, :, None] * v[:, :, t, None, :]
        o[:, :, t] = c * (q[:, :, t, :, None] * S).sum(2)
        dq[:, :, t] = c * (S * d_out[:, :, t, None, :]).sum(3)
    for t in reversed(order):
        D = c * q[:, :, t, :, None] * d_out[:, :, t, None, :] + Z
        dkk[:, :, t], dvv[:, :, t] = (D * v[:, :, t, None, :]).sum(3), (D * k[:, :, t, :, None]).sum(2)
        Z = D * a[:, :, t, :, None]
    e = dq * q - dkk * k
    return o, dq, dkk, dvv, e.cumsum(2) if reverse else e.flip(2).cumsum(2).flip(2)


def _reference(q, k, v, xf, xb, d_out, out_scale, norm):
    """Both directions: [o, dq, dk, dv, dx_fwd, dx_bwd]; x: raw logits (norm > 0) or log-gates."""
    q, k, v, d_out = (t.double() for t in (q, k, v, d_out))
    total, dxs = None, []
    for reverse, x in ((False, xf.double()), (True, xb.double())):
        g = torch.nn.functional.logsigmoid(x) / norm if norm else x
        *parts, dg = _scan64(q, k, v, g, q.shape[-1] ** -0.5 * out_scale, reverse, d_out)
        dxs.append(dg * torch.sigmoid(-x) / norm if norm else dg)
        total = parts if total is None else [a + b for a, b in zip(total, parts)]
    return total + dxs


def _run(ins, d_out, **kw):
    import vig_b200
    leaves = [t.detach().requires_grad_(True) for t in ins]
    o = vig_b200.bi_gla(*leaves, out_scale=0.5, **kw)
    return [o.detach(), *torch.autograd.grad(o, leaves, d_out)]


def _errors(got, ref):
    return [float((a.double() - b).norm() / b.norm()) for a, b in zip(got, ref)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dk,dv", [(16, 32), (32, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("L", [50, 196, 600, 3000])
def test_raw_logits_whose_exponential_overflows(dtype, dk, dv, L):
    """exp(100) and exp(1000) leave fp32, the gates logsigmoid(-100) / 16 and logsigmoid(-1000) / 16 do not; in the first, a
    middle and the last segment of a sequence of one segment, a cluster of segments, and segments scanned by a launch of
    their own."""
    import vig_b200
    (q, k, v), (xf, xb), d_out = _inputs(dtype, 1, 3, L, dk, dv, seed=L)
    for i, at in enumerate((3, L // 2, L - 2)):
        xf[0, 0, at, 1] = xb[0, 0, at, 2] = -100.0
        xf[0, 1, at, i] = xb[0, 2, at, i] = -1000.0
    xf, xb = xf.to(dtype), xb.to(dtype)
    errs = _errors(_run((q, k, v, xf, xb), d_out, gate_logit_normalizer=16.0), _reference(q, k, v, xf, xb, d_out, 0.5, 16.0))
    assert all(e < TOL[dtype] for e in errs), errs
    vig_b200.check_status()


@pytest.mark.parametrize("dk,dv", [(16, 32), (32, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("L,norm", [(49, 0.0), (196, 16.0), (1500, 0.0)])
def test_fp32_is_as_exact_as_the_recurrence_in_fp32(dk, dv, L, norm):
    """Ordinary gates, outputs and all gradients.  Token by token in fp32 the outputs and the gradients of q, k, v are 2.8e-7 ..
    3.1e-7 from fp64 (sums of about 20 remembered tokens, 2^-24 each step), the gate gradients 5e-7 .. 3e-6."""
    (q, k, v), (xf, xb), d_out = _inputs(torch.float32, 2, 3, L, dk, dv, seed=L + dk)
    if not norm:
        xf, xb = (torch.nn.functional.logsigmoid(x) / 16 for x in (xf, xb))
    errs = _errors(_run((q, k, v, xf, xb), d_out, gate_logit_normalizer=norm), _reference(q, k, v, xf, xb, d_out, 0.5, norm))
    assert all(e < 2.8e-7 for e in errs[:4]) and all(e < 5e-7 for e in errs[4:]), errs


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("dk,dv,L", [(16, 32, 100), (64, 64, 300)])
def test_fp32_gate_gradients_of_16_bit_inputs(dtype, dk, dv, L):
    """``bi_gla_backward`` returns them in fp32 whatever the inputs' type, through the library call as through Python: sums of fp32
    products (1e-6), the other gradients rounded once."""
    import vig_b200
    from vig_b200 import _lib
    (q, k, v), (xf, xb), d_out = _inputs(dtype, 1, 3, L, dk, dv, seed=L + dk)
    gf, gb = ((torch.nn.functional.logsigmoid(x) / 16).to(dtype) for x in (xf, xb))
    ref = _reference(q, k, v, gf, gb, d_out, 0.5, 0.0)[1:]
    got = vig_b200.bi_gla_backward(q, k, v, gf, gb, d_out, out_scale=0.5)
    lib, outs = _lib.lib(), [torch.empty(*t.shape, dtype=torch.float32 if i > 2 else dtype, device="cuda") for i, t in enumerate(ref)]
    ws = torch.empty(lib.vig_bigla_bwd_full_workspace_bytes(1, 3, L, dk, dv), dtype=torch.uint8, device="cuda")
    assert lib.vig_bigla_bwd_full(*map(_lib.ptr, (q, k, v, gf, gb, d_out, *outs)), 1, 1, 3, L, dk, dv, _lib.dtype_code(q), *[None] * 6, -1.0, 0.5, 0.0, float("nan"), 3,
                                  _lib.ptr(ws), ws.numel(), _lib.stream_ptr()) == 0
    for grads in (got, outs):
        errs = _errors(grads, ref)
        assert [g.dtype for g in grads] == [dtype] * 3 + [torch.float32] * 2
        assert all(e < 2e-6 for e in errs[3:]) and all(e < (2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12) for e in errs[:3]), errs


def _log_gates(kind, x):
    """Log-gates that a segment's factored form cannot take, made from normal numbers x [B, H, L, dk]."""
    g = torch.nn.functional.logsigmoid(x) / 16
    L = g.shape[2]
    if kind == "reset":                                                  # the state is dropped: exp(-inf) = 0
        for i, at in enumerate((min(3, L - 1), L // 2, L - 1)):
            g[0, i % g.shape[1], at, i::5] = -float("inf")
    elif kind == "lowest":                                               # masks of the lowest finite value, two in a row
        g[0, 0, L // 3:L // 3 + 2] = torch.finfo(torch.float16).min
    elif kind == "strong":
        g = g * 160
    elif kind == "growing":
        g[0, 0, :40, ::3] = 0.05                                         # 40 factors of the fast exponential, 2^-22 each: 1e-5
    return g


@pytest.mark.parametrize("kind", ["reset", "lowest", "strong", "growing"])
@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 16, 32), (torch.float32, 32, 32), (torch.float32, 32, 64), (torch.float32, 64, 64), (torch.bfloat16, 16, 32),
                                         (torch.bfloat16, 64, 64), (torch.float16, 32, 32), (torch.float16, 32, 64)])
@pytest.mark.parametrize("L", [5, 64, 150, 1000, 2500])
def test_segments_outside_the_range(dtype, dk, dv, L, kind):
    """Outputs in both directions and one, final and summed states, one launch (a lone segment, clusters) and three.  A segment
    is evaluated as the recurrence, so fp32 results carry its roundings only."""
    import vig_b200
    (q, k, v), (xf, xb), _ = _inputs(dtype, 1, 3, L, dk, dv, seed=L + dk)
    gf, gb = _log_gates(kind, xf).to(dtype), _log_gates(kind, xb).to(dtype)
    q64, k64, v64 = q.double(), k.double(), v.double()
    c = dk ** -0.5
    of, S = _forward64(q64, k64, v64, gf.double(), c, False)
    ob, _ = _forward64(q64, k64, v64, gb.double(), c, True)
    o, ex = vig_b200.bi_gla(q, k, v, gf, gb, output_final_state=True, output_logdecay=True, impl=vig_b200._lib.IMPL_SEG)
    one, state = vig_b200.fused_chunk_gla(q, k, v, gf, output_final_state=True) if dtype == torch.float32 or dv == 32 else (None, None)
    pairs = [(o, of + ob), (ex["final_fwd"], S), (torch.exp(ex["logdecay_fwd"]), torch.exp(gf.double().sum(2)))]
    if one is not None:
        pairs += [(one, of), (state, S)]
    for got, ref in pairs:
        tol = TOL[dtype] if got.dtype == dtype or dtype == torch.bfloat16 and dv == 64 else 1e-4
        assert float((got.double() - ref).norm()) <= tol * float(ref.norm()) + 1e-30, (kind, float((got.double() - ref).norm() / ref.norm()))


def _forward64(q, k, v, g, c, reverse):
    B, H, L, dk = k.shape
    S, o, a = torch.zeros(B, H, dk, v.shape[-1], dtype=torch.float64, device=k.device), torch.empty_like(v), g.exp()
    for t in range(L - 1, -1, -1) if reverse else range(L):
        S = S * a[:, :, t, :, None] + k[:, :, t, :, None] * v[:, :, t, None, :]
        o[:, :, t] = c * (q[:, :, t, :, None] * S).sum(2)
    return o, S


@pytest.mark.parametrize("kind", ["reset", "lowest", "strong", "growing"])
@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 16, 32), (torch.float32, 32, 64), (torch.float32, 64, 64), (torch.bfloat16, 32, 32), (torch.bfloat16, 64, 64),
                                         (torch.float16, 16, 32), (torch.float16, 32, 64)])
@pytest.mark.parametrize("L", [5, 64, 150, 1000])
def test_gradients_of_chunks_outside_the_range(dtype, dk, dv, L, kind):
    """One chunk and many: states of the chunk and its adjoint as recurrences, in both directions.  The gate gradients of decayed
    states are small differences of large sums of fp32 products, hence their wider bound."""
    (q, k, v), (xf, xb), d_out = _inputs(dtype, 1, 3, L, dk, dv, seed=L + dk)
    gf, gb = _log_gates(kind, xf).to(dtype), _log_gates(kind, xb).to(dtype)
    ref = _reference(q, k, v, gf, gb, d_out, 0.5, 0.0)
    errs = _errors(_run((q, k, v, gf, gb), d_out), ref)
    assert all(e < TOL[dtype] for e in errs[1:4]), errs
    assert all(e < max(1e-4, TOL[dtype]) for e in errs[4:]), errs


@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 32, 64), (torch.float32, 64, 64), (torch.bfloat16, 32, 32), (torch.float16, 16, 32)])
@pytest.mark.parametrize("L", [40, 150, 700])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_what_is_not_finite_stays_with_the_tokens_that_see_it(dtype, dk, dv, L, bad):
    """Causal, one token's q, k or v: tokens before it, and value columns beside it, are those of the clean call."""
    import vig_b200
    (q, k, v), (x, _), d_out = _inputs(dtype, 1, 3, L, dk, dv, seed=L)
    g = (torch.nn.functional.logsigmoid(x) / 16).to(dtype)
    at = 2 * L // 3
    clean, _ = vig_b200.fused_chunk_gla(q, k, v, g)
    for which in range(3):
        ins = [t.clone() for t in (q, k, v)]
        ins[which][0, 1, at, 5] = bad
        o, _ = vig_b200.fused_chunk_gla(*ins, g)
        same = torch.ones_like(o, dtype=torch.bool)
        same[0, 1, at:at + 1 if which == 0 else None] = False
        if which == 2:
            same[0, 1, at:] = torch.arange(dv, device="cuda") != 5
        scale = float(clean.float().abs().max())
        assert float((o.float() - clean.float())[same].abs().max()) <= TOL[dtype] * scale
        assert not torch.isfinite(o[0, 1, at, 5] if which == 2 else o[0, 1, at]).all()


@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 32, 64), (torch.bfloat16, 64, 64), (torch.float16, 16, 32)])
@pytest.mark.parametrize("L", [40, 150])
def test_gradients_of_tokens_that_do_not_see_what_is_not_finite(dtype, dk, dv, L):
    """Causal: d_out of one token is NaN.  The gradients of q before and after it, of k and v after it are those of the clean call."""
    import vig_b200
    (q, k, v), (x, _), d_out = _inputs(dtype, 1, 2, L, dk, dv, seed=L)
    leaves = [t.requires_grad_(True) for t in (q, k, v, (torch.nn.functional.logsigmoid(x) / 16).to(dtype))]
    at, spoilt = L // 2, d_out.clone()
    spoilt[0, 1, at, 3] = float("nan")
    o, _ = vig_b200.fused_chunk_gla(*leaves)
    clean = torch.autograd.grad(o, leaves, d_out, retain_graph=True)
    got = torch.autograd.grad(o, leaves, spoilt)
    for i, (a, b) in enumerate(zip(got[:3], clean)):
        same = torch.ones_like(a, dtype=torch.bool)
        if i == 0:
            same[0, 1, at] = False
        else:
            same[0, 1, :at + 1] = False
        assert float((a.float() - b.float())[same].abs().max()) <= TOL[dtype] * float(b.float().abs().max()), i
        assert torch.isnan(a[0, 1, at]).any()
