"""The segment form of the forward (mma.sync; fp32, dv = 32, short and medium 16-bit sequences): segment edges, one-launch
clusters of 1 to 16 segments and the three-launch form above, entering and final states, one direction, gates that leave the
factorisation's range, and rows only the token-by-token form can read."""
import pytest
import torch

import oracle
from conftest import rel_err

pytestmark = pytest.mark.gpu
# fp32: operands carry 24 bits; 64-token cumulative gates of up to 24 round to 2^-24 * 24 = 1.4e-6 per factor.  16-bit: the
# output's rounding (2^-9, 2^-12) in the max norm plus 2^-17 operand splits.
TOL = {torch.float32: 2e-5, torch.bfloat16: 5e-3, torch.float16: 1e-3}
DIMS = {torch.float32: [(16, 32), (32, 32), (32, 64), (64, 64)], torch.bfloat16: [(16, 32), (32, 32)], torch.float16: [(16, 32), (32, 32)]}


@pytest.mark.parametrize("dtype,dk,dv", [(t, *d) for t in DIMS for d in DIMS[t]])
@pytest.mark.parametrize("L,strength", [(1, 1.0), (63, 1.0), (64, 1.0), (65, 1.0), (200, 1.0), (150, 60.0)])
def test_forward_at_chunk_edges(dtype, dk, dv, L, strength):
    import vig_b200
    q, k, v, gf, gb = oracle.make_bigla_inputs(2, 2, L, dk, dv, seed=L + dk)
    ins = [t.to(dtype) for t in (q, k, v, gf * strength, gb)]
    ref = oracle.naive_bi_gla(*[t.float() for t in ins])
    assert rel_err(vig_b200.bi_gla(*[t.cuda() for t in ins]).float(), ref) < TOL[dtype]


@pytest.mark.parametrize("dtype,dk,dv", [(torch.bfloat16, 64, 64), (torch.bfloat16, 32, 64), (torch.float16, 64, 64)])
@pytest.mark.parametrize("B,L,strength", [(1, 64, 1.0), (1, 100, 1.0), (1, 513, 1.0), (40, 130, 1.0), (1, 1024, 1.0), (1, 1030, 1.0), (2, 2048, 1.0), (1, 2049, 1.0), (1, 300, 60.0)])
def test_forward_of_16_bit_heads(dtype, dk, dv, B, L, strength):
    """64- and 128-token segments, 1 to 16 of them in a cluster, more in three launches.  bf16 runs on bf16 operands (one
    term): three roundings of 2^-9 per product on random signs, in the max norm."""
    import vig_b200
    from vig_b200 import _lib
    q, k, v, gf, gb = oracle.make_bigla_inputs(B, 2, L, dk, dv, seed=L + dk)
    ins = [t.to(dtype) for t in (q, k, v, gf * strength, gb)]
    ref = oracle.naive_bi_gla(*[t.float() for t in ins])
    tol = 1.5e-2 if dtype == torch.bfloat16 else 2e-3
    assert rel_err(vig_b200.bi_gla(*[t.cuda() for t in ins], impl=_lib.IMPL_SEG).float(), ref) < tol


@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 64, 64), (torch.float16, 16, 32)])
@pytest.mark.parametrize("L", [64, 130, 1200])
def test_one_direction_continues_from_a_state(dtype, dk, dv, L):
    import vig_b200
    q, k, v, g, _ = [t.to(dtype) for t in oracle.make_bigla_inputs(1, 2, L, dk, dv, seed=3)]
    cut = L // 2
    full, h_full = vig_b200.fused_chunk_gla(*[t.cuda() for t in (q, k, v, g)], output_final_state=True)
    first = [t[:, :, :cut].cuda() for t in (q, k, v, g)]
    rest = [t[:, :, cut:].cuda() for t in (q, k, v, g)]
    _, h = vig_b200.fused_chunk_gla(*first, output_final_state=True)
    o, h_end = vig_b200.fused_chunk_gla(*rest, initial_state=h, output_final_state=True)
    ref, ref_h = oracle.naive_gla(*[t.float() for t in (q, k, v, g)])
    assert rel_err(full.float(), ref) < TOL[dtype] and rel_err(h_full, ref_h) < 1e-4
    assert rel_err(o.float(), ref[:, :, cut:]) < TOL[dtype] and rel_err(h_end, ref_h) < 1e-4


def test_unaligned_rows_take_the_exact_form():
    import vig_b200
    ins = oracle.make_bigla_inputs(1, 2, 70, 32, 32, seed=4)
    odd = torch.zeros(1, 2, 70, 33, device="cuda")
    odd[..., 1:] = ins[0].cuda()
    assert rel_err(vig_b200.bi_gla(odd[..., 1:], *[t.cuda() for t in ins[1:]]), oracle.naive_bi_gla(*ins)) < 2e-5


def test_a_call_without_workspace_runs_where_one_segment_needs_none():
    """vig_bigla_fwd leaves the form to the library: 16-bit sequences of up to 256 tokens with an output need no workspace."""
    from vig_b200 import _lib
    B, H, L, d = 1, 3, 196, 64
    ins = [t.bfloat16() for t in oracle.make_bigla_inputs(B, H, L, d, d, seed=8)]
    dev, o = [t.cuda() for t in ins], torch.empty(B, H, L, d, device="cuda", dtype=torch.bfloat16)
    st = _lib.lib().vig_bigla_fwd(*map(_lib.ptr, dev), _lib.ptr(o), B, H, L, d, d, _lib.dtype_code(o), *[None] * 6, -1.0, 1.0, 0.0, float("nan"), *[None] * 6, 3, 0,
                                  None, 0, None, _lib.stream_ptr())
    assert st == 0
    assert rel_err(o.float(), oracle.naive_bi_gla(*[t.float() for t in ins])) < 1.5e-2
    f32 = [t.float().cuda() for t in ins]
    st = _lib.lib().vig_bigla_fwd(*map(_lib.ptr, f32), _lib.ptr(o), B, H, L, d, d, 0, *[None] * 6, -1.0, 1.0, 0.0, float("nan"), *[None] * 6, 3, 0, None, 0, None,
                                  _lib.stream_ptr())
    assert st == -5                                                      # fp32 has no such form: refused before any launch


@pytest.mark.parametrize("dk,B,H,L", [(64, 1, 3, 196), (64, 4, 6, 450), (32, 4, 3, 1000)])
def test_bf16_rounds_no_more_often_than_the_tcgen05_form(dk, B, H, L):
    """Errors against fp64 of the two forms that share these calls: the same operands rounded once each, so the same error but
    for the sums' order (10 % of it)."""
    import vig_b200
    from vig_b200 import _lib
    ins = [t.bfloat16() for t in oracle.make_bigla_inputs(B, H, L, dk, 64, seed=12)]
    ref = oracle.chunked_bi_gla_f64(*[t.double() for t in ins])
    err = {impl: float((vig_b200.bi_gla(*[t.cuda() for t in ins], impl=impl).double().cpu() - ref).norm() / ref.norm()) for impl in (_lib.IMPL_SEG, _lib.IMPL_TC_SPLIT)}
    assert err[_lib.IMPL_SEG] < 1.1 * err[_lib.IMPL_TC_SPLIT], err


@pytest.mark.parametrize("dtype,dk,dv", [(torch.float32, 64, 64), (torch.float32, 32, 64), (torch.float16, 64, 64), (torch.bfloat16, 16, 32)])
@pytest.mark.parametrize("L", [65, 96, 97, 480, 512])
def test_small_calls_in_segments_of_32(dtype, dk, dv, L):
    """Up to 16 segments of 32 tokens a cluster, states at both ends, a direction out of the factorised range in the middle; a workspace for
    64-token segments, which earlier callers hold, gives the same."""
    import vig_b200
    from vig_b200 import _lib
    q, k, v, gf, gb = oracle.make_bigla_inputs(1, 2, L, dk, dv, seed=L)
    gb[:, 1, 32:64] *= 200
    ins = [t.to(dtype) for t in (q, k, v, gf, gb)]
    ref = oracle.naive_bi_gla(*[t.float() for t in ins])
    dev = [t.cuda() for t in ins]
    tol = 2e-3 if dtype == torch.float16 else TOL[dtype]
    assert rel_err(vig_b200.bi_gla(*dev, impl=_lib.IMPL_SEG).float(), ref) < tol
    need = [_lib.lib().vig_bigla_workspace_bytes(1, 2, L, dk, dv, _lib.dtype_code(dev[0]), i) for i in (_lib.IMPL_SEG, _lib.IMPL_SIMT)]
    assert need[0] > need[1] or (dtype == torch.float16 and L > 256)
    ws, o = torch.empty(need[1], dtype=torch.uint8, device="cuda"), torch.empty(1, 2, L, dv, device="cuda", dtype=dtype)
    st = _lib.lib().vig_bigla_fwd(*map(_lib.ptr, dev), _lib.ptr(o), 1, 2, L, dk, dv, _lib.dtype_code(o), *[None] * 6, -1.0, 1.0, 0.0, float("nan"), *[None] * 6, 3,
                                  _lib.IMPL_SEG, _lib.ptr(ws), need[1], None, _lib.stream_ptr())
    assert st == 0 and rel_err(o.float(), ref) < tol


def _shapes(f, tmp_path):
    """(Segments of a sequence, threads a CTA) of the segment kernels that ``f`` launches; three times, the profiler may lose one"""
    import json
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(3):
            f()
            torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.load(open(tmp_path / "trace.json"))["traceEvents"]
    return {(e["args"]["grid"][0], e["args"]["block"][0]) for e in events if e.get("cat") == "kernel" and "bigla_seg_kernel" in e["name"]}


@pytest.mark.parametrize("dtype,dk", [(torch.bfloat16, 32), (torch.bfloat16, 64), (torch.float16, 32)])
@pytest.mark.parametrize("L", [1, 17, 49, 64])
@pytest.mark.parametrize("more", [0, 1])
def test_sequences_of_one_segment_around_one_an_sm(dtype, dk, L, more, tmp_path):
    """Up to one sequence an SM two warps share 16 rows; beyond that the scores are not formed twice.  Both with a sequence whose gates leave the
    factorisation's range, and with final states."""
    import vig_b200
    B, H = torch.cuda.get_device_properties(0).multi_processor_count + more, 1
    q, k, v, gf, gb = oracle.make_bigla_inputs(B, H, L, dk, 64, seed=L)
    gb[B // 2] *= 200
    ins = [t.to(dtype) for t in (q, k, v, gf, gb)]
    ref = oracle.naive_bi_gla(*[t.float() for t in ins])
    dev = [t.cuda() for t in ins]
    tol = 1.5e-2 if dtype == torch.bfloat16 else 2e-3
    assert rel_err(vig_b200.bi_gla(*dev).float(), ref) < tol
    assert _shapes(lambda: vig_b200.bi_gla(*dev), tmp_path) == {(1, 128 if more else 256)}
    o, h = vig_b200.fused_chunk_gla(*dev[:3], dev[4], output_final_state=True)
    want, state = oracle.naive_gla(*[t.float() for t in (*ins[:3], ins[4])])
    assert rel_err(o.float(), want) < tol and rel_err(h, state) < (1e-2 if dtype == torch.bfloat16 else 1e-4)


@pytest.mark.parametrize("dtype,dk,dv,L,plain,finals", [(torch.float16, 64, 64, 100, 4, 2), (torch.float16, 32, 64, 256, 8, 4), (torch.float32, 64, 64, 256, 8, 8), (torch.float32, 64, 64, 257, 9, 5),
                                                        (torch.bfloat16, 16, 32, 512, 16, 8), (torch.bfloat16, 64, 64, 512, 8, 8), (torch.bfloat16, 64, 64, 700, 11, 6),
                                                        (torch.float16, 32, 64, 1024, 16, 8)])
def test_final_states_are_summed_over_fewer_segments(dtype, dk, dv, L, plain, finals, tmp_path):
    """A stream continued from a state, as fine as a call without final states only where that is the faster form."""
    import vig_b200
    q, k, v, g, _ = [t.to(dtype) for t in oracle.make_bigla_inputs(1, 3, L, dk, dv, seed=L)]
    h0 = torch.randn(1, 3, dk, dv, generator=torch.Generator().manual_seed(1))
    dev = [t.cuda() for t in (q, k, v, g)]
    with torch.no_grad():
        o, h = vig_b200.fused_chunk_gla(*dev, initial_state=h0.cuda(), output_final_state=True)
        assert {s[0] for s in _shapes(lambda: vig_b200.fused_chunk_gla(*dev), tmp_path)} == {plain}
        assert {s[0] for s in _shapes(lambda: vig_b200.fused_chunk_gla(*dev, initial_state=h0.cuda(), output_final_state=True), tmp_path)} == {finals}
    ref, ref_h = oracle.naive_gla(*[t.float() for t in (q, k, v, g)], initial_state=h0)
    tol = {torch.float32: 2e-5, torch.bfloat16: 1.5e-2, torch.float16: 2e-3}[dtype]
    assert rel_err(o.float(), ref) < tol and rel_err(h, ref_h) < max(tol, 1e-4)
