"""Tensor-core backward of bi-GLA (vig_bigla_bwd_full) where it can go wrong: chunk edges (64 tokens), a lone chunk, every
head size, chunks whose gates leave the factorisation's range (exact per-chunk form), unaligned strides (exact form)."""
import pytest
import torch

import oracle
from conftest import rel_err
from test_bigla_bwd_gpu import _reference_grads

pytestmark = pytest.mark.gpu
NAMES = ["dq", "dk", "dv", "dg_fwd", "dg_bwd"]


# fp32: operands carry 24 bits, what remains is the rounding of 64-token cumulative gates of up to 24 (2^-24 * 24 = 1.4e-6
# per factor) summed over a few factors; 16-bit types: the rounding of the results (2^-9, 2^-12) against the max norm.
TOL = {torch.float32: 2e-5, torch.bfloat16: 5e-3, torch.float16: 1e-3}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,dk,dv,dir_mask,strength", [(63, 64, 64, 3, 1.0), (64, 32, 64, 3, 1.0), (65, 64, 64, 3, 1.0), (128, 16, 32, 3, 1.0),
                                                        (193, 32, 32, 1, 1.0), (129, 64, 64, 2, 1.0), (150, 64, 64, 3, 60.0), (40, 32, 64, 3, 60.0)])
def test_gradients_at_chunk_edges(dtype, L, dk, dv, dir_mask, strength):
    import vig_b200
    q, k, v, gf, gb = oracle.make_bigla_inputs(2, 2, L, dk, dv, seed=L + dk)
    gf = gf * strength                                       # 60: every chunk of the forward direction leaves the range
    q, k, v, gf, gb = (t.to(dtype) for t in (q, k, v, gf, gb))
    d_out = torch.randn(2, 2, L, dv, generator=torch.Generator().manual_seed(1)).to(dtype)
    _, ref = _reference_grads(q.float(), k.float(), v.float(), gf.float(), gb.float(), d_out.float(), 0.5, dir_mask)
    got = vig_b200.bi_gla_backward(*[t.cuda() for t in (q, k, v, gf, gb, d_out)], out_scale=0.5, dir_mask=dir_mask)
    errs = {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref) if g is not None}
    assert all(e < TOL[dtype] for e in errs.values()), errs


def test_unaligned_rows_take_the_exact_form():
    import vig_b200
    B, H, L, d = 1, 2, 70, 32
    q, k, v, gf, gb = oracle.make_bigla_inputs(B, H, L, d, d, seed=4)
    d_out = torch.randn(B, H, L, d, generator=torch.Generator().manual_seed(2))
    _, ref = _reference_grads(q, k, v, gf, gb, d_out, 1.0, 3)
    odd = torch.zeros(B, H, L, d + 1, device="cuda")
    odd[..., 1:] = q.cuda()
    got = vig_b200.bi_gla_backward(odd[..., 1:], *[t.cuda() for t in (k, v, gf, gb, d_out)])
    errs = {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref)}
    assert all(e < 2e-5 for e in errs.values()), errs


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,dk,dv,norm", [(63, 64, 64, 0.0), (64, 32, 64, 16.0), (65, 64, 64, 16.0), (128, 16, 32, 0.0), (193, 32, 32, 16.0), (200, 64, 64, 16.0)])
def test_training_step_in_16_bits(dtype, L, dk, dv, norm):
    """The 16-bit kernels, as training runs them: gate gradients in the gates' type, log-gates or raw logits without a clamp."""
    import vig_b200
    gen = torch.Generator().manual_seed(L)
    q, k, v, xf, xb, d_out = [torch.randn(2, 2, L, d, generator=gen).to(dtype) for d in (dk, dk, dv, dk, dk, dv)]
    if not norm:
        xf, xb = ((torch.nn.functional.logsigmoid(x.float()) / 16).to(dtype) for x in (xf, xb))
    leaves = [t.cuda().requires_grad_() for t in (q, k, v, xf, xb)]
    o = vig_b200.bi_gla(*leaves, out_scale=0.5, gate_logit_normalizer=norm)
    got = torch.autograd.grad(o, leaves, d_out.cuda())
    gf, gb = (torch.nn.functional.logsigmoid(x.double()) / norm if norm else x.double() for x in (xf, xb))
    _, ref = _reference_grads(q.float(), k.float(), v.float(), gf, gb, d_out.float(), 0.5, 3)
    if norm:
        ref = [*ref[:3], *(g * torch.sigmoid(-x.double()) / norm for g, x in zip(ref[3:], (xf, xb)))]
    errs = {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref)}
    assert all(e < TOL[dtype] for e in errs.values()), errs


@pytest.mark.parametrize("dk,dv", [(16, 32), (32, 64), (64, 64)])
@pytest.mark.parametrize("which", ["fwd", "bwd"])
def test_a_chunk_that_one_direction_leaves(dk, dv, which):
    """The two directions of a chunk are two CTAs that add up their results: where one of them leaves the range, the exact form replaces what
    the other has written, and the chunks beside it are as they were."""
    import vig_b200
    q, k, v, gf, gb = oracle.make_bigla_inputs(2, 2, 200, dk, dv, seed=dk)
    (gf if which == "fwd" else gb)[0, 1, 64:128] *= 200
    d_out = torch.randn(2, 2, 200, dv, generator=torch.Generator().manual_seed(3))
    _, ref = _reference_grads(q, k, v, gf, gb, d_out, 0.5, 3)
    got = vig_b200.bi_gla_backward(*[t.cuda() for t in (q, k, v, gf, gb, d_out)], out_scale=0.5)
    errs = {n: rel_err(g, r) for n, g, r in zip(NAMES, got, ref)}
    assert all(e < TOL[torch.float32] for e in errs.values()), errs


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("L", [128, 256, 257, 384, 385])
@pytest.mark.parametrize("strong", [False, True])
def test_few_chunks_sum_their_states_themselves(dtype, L, strong):
    """Both sides of the lines behind which a launch forms the entering states (4 and 6 chunks), with a chunk for the exact form, which needs them too."""
    import vig_b200
    q, k, v, gf, gb = oracle.make_bigla_inputs(1, 2, L, 32, 64, seed=L)
    if strong:
        gf[0, 0, 64:128] *= 200
    q, k, v, gf, gb = (t.to(dtype) for t in (q, k, v, gf, gb))
    d_out = torch.randn(1, 2, L, 64, generator=torch.Generator().manual_seed(5)).to(dtype)
    _, ref = _reference_grads(q.float(), k.float(), v.float(), gf.float(), gb.float(), d_out.float(), 0.5, 3)
    leaves = [t.cuda().requires_grad_() for t in (q, k, v, gf, gb)]
    got = torch.autograd.grad(vig_b200.bi_gla(*leaves, out_scale=0.5), leaves, d_out.cuda())
    errs = {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref)}
    assert all(e < TOL[dtype] for e in errs.values()), errs


@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 64, 64), (torch.bfloat16, 64, 64), (torch.float16, 32, 64), (torch.bfloat16, 32, 32), (torch.bfloat16, 16, 32)])
@pytest.mark.parametrize("L", [130, 250, 384, 448])
@pytest.mark.parametrize("dirs", [3, 1, 2])
def test_every_chunk_left_to_the_exact_form(dtype, dk, dv, L, dirs):
    """The exact form's own sums of the states that other chunks contribute, with 3 to 6 chunks, and the launched ones with 7 (fp32: from 5)."""
    import vig_b200
    q, k, v, gf, gb = oracle.make_bigla_inputs(1, 2, L, dk, dv, seed=L + dk)
    ins = [t.to(dtype) for t in (q, k, v, gf * 25, gb * 25)]
    d_out = torch.randn(1, 2, L, dv, generator=torch.Generator().manual_seed(6)).to(dtype)
    _, ref = _reference_grads(*[t.float() for t in ins], d_out.float(), 0.5, dirs)
    if dirs == 3:
        leaves = [t.cuda().requires_grad_() for t in ins]
        got = torch.autograd.grad(vig_b200.bi_gla(*leaves, out_scale=0.5), leaves, d_out.cuda())
    else:
        got = vig_b200.bi_gla_backward(*[t.cuda() for t in (*ins, d_out)], out_scale=0.5, dir_mask=dirs)
    errs = {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref) if r is not None and g is not None}
    assert all(e < TOL[dtype] for e in errs.values()), errs


def test_exact_chunks_cost_the_same_with_and_without_a_launch_over_chunks():
    """Backward per chunk, gates of all chunks out of range: 4 chunks sum the contributions in the exact form itself, 5 have a launch for it.  1.06 of it, 1.33
    when each value was summed by itself."""
    import vig_b200

    def per_chunk(chunks):
        q, k, v, d_out = (torch.randn(64, 3, 64 * chunks, 64, device="cuda") for _ in range(4))
        g = torch.full_like(q, -4.0)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            vig_b200.bi_gla_backward(q, k, v, g, g, d_out)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times) / chunks
    folded, launched = per_chunk(4), per_chunk(5)
    assert folded < 1.2 * launched, (folded, launched)
