"""Convolution + stacked input projection of a small call in one launch (vig_conv_proj_fwd) against the two operations it stands for, at the edges
of its 16-token tiles, of images and of batches."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
# the same convolution, bit for bit; products of bf16 / fp16 values summed in fp32 in another order, then rounded once: 2^-9, 2^-12 of the largest value
TOL = {torch.bfloat16: 4e-3, torch.float16: 5e-4}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C,N", [(96, 384), (192, 768), (192, 1152)])
@pytest.mark.parametrize("B,h,w,act,biased", [(1, 1, 1, 1, True), (1, 3, 5, 0, True), (1, 4, 4, 1, False), (2, 1, 17, 1, True), (3, 17, 1, 1, True), (2, 14, 14, 1, True), (1, 7, 7, 0, False)])
def test_one_launch_equals_convolution_and_projection(dtype, C, N, B, h, w, act, biased):
    from vig_b200 import _lib, ops
    gen = torch.Generator(device="cuda").manual_seed(B * 100 + h)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    x, taps, cb, W, b = rand(B, h * w, C), rand(9, C) / 3, rand(C), rand(N, C) / C ** 0.5, rand(N)
    if not biased:
        cb = b = None
    xs, z = torch.empty_like(x), torch.empty(B, h * w, N, device="cuda", dtype=dtype)
    st = _lib.lib().vig_conv_proj_fwd(_lib.ptr(x), _lib.ptr(taps), _lib.ptr(cb), _lib.ptr(W), _lib.ptr(b), _lib.ptr(xs), _lib.ptr(z), B, h, w, C, N, act, _lib.dtype_code(x),
                                      _lib.stream_ptr())
    assert st == 0
    ref = ops.dwconv3x3(x, taps, cb, (h, w), bool(act))
    assert torch.equal(xs, ref)
    assert rel_err(z.float(), torch.nn.functional.linear(ref.float(), W.float(), None if b is None else b.float())) < TOL[dtype]
    assert _lib.lib().vig_conv_proj_supported(B * h * w, 384, N, _lib.dtype_code(x)) == 0 and _lib.lib().vig_conv_proj_preferred(1 << 20, C, N, _lib.dtype_code(x)) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("side", [4, 8, 14])
def test_overlapping_launches_give_the_same_bits(dtype, side):
    """Convolution + projection, scan and block tail over and over through the same buffers, each launch let in before the one ahead has ended, and one
    by one: whatever is read too early holds the values of a layer before.  16 and 64 tokens in one segment, 196 in segments of 64 (bf16) or 32 (fp16)."""
    from vig_b200 import _lib, ops
    lib, P, C, H, dk, dv, I, L = _lib.lib(), _lib.ptr, 192, 3, 32, 64, 512, side * side
    kd, vd = H * dk, H * dv
    N = 4 * kd + 2 * vd
    assert lib.vig_conv_proj_preferred(L, C, N, _lib.dtype_code(torch.empty(0, dtype=dtype)))
    gen = torch.Generator(device="cuda").manual_seed(side)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    layers = [dict(taps=rand(9, C) / 3, cb=rand(C) * 0.1, w=rand(N, C) / C ** 0.5, b=rand(N) * 0.1, wo=rand(C, C) / C ** 0.5, wg=rand(2 * I, C) / C ** 0.5, wd=rand(C, I) / I ** 0.5)
              for _ in range(4)]
    one, head = torch.ones(C, device="cuda", dtype=dtype), torch.ones(dv, device="cuda", dtype=dtype)
    x, xs, z, o = rand(1, L, C), torch.empty(1, L, C, device="cuda", dtype=dtype), torch.empty(1, L, N, device="cuda", dtype=dtype), torch.empty(1, L, H, dv, device="cuda", dtype=dtype)
    part = lambda col, d: z.as_strided((1, H, L, d), (L * N, d, N, 1), col)  # noqa: E731

    def forward(on):
        h, r, outs = x[0], x[0], []
        was = lib.vig_chain_launches(on)
        for i in range(24):
            p = layers[i % 4]
            assert lib.vig_conv_proj_fwd(*map(P, (h, p["taps"], p["cb"], p["w"], p["b"], xs, z)), 1, side, side, C, N, 1, _lib.dtype_code(x), _lib.stream_ptr()) == 0
            ops.bi_gla(part(0, dk), part(kd, dk), part(2 * kd, dv), part(2 * kd + 2 * vd, dk), part(3 * kd + 2 * vd, dk), gate_logit_normalizer=16.0, out_scale=0.5,
                       out=o.permute(0, 2, 1, 3))
            h, r = ops.block_tail(o.view(L, C), xs[0], z[0, :, 2 * kd + vd:2 * kd + 2 * vd], head, head, p["wo"], r, one, p["wg"], p["wd"], one)
            outs.append(h)
        lib.vig_chain_launches(was)
        torch.cuda.synchronize()
        return outs
    apart = forward(0)
    assert bool(apart[-1].isfinite().all())
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(forward(1), apart))


@pytest.mark.parametrize("more", [0, 1])
def test_scans_of_more_segments_than_sms_wait_for_the_launch_ahead(more, tmp_path):
    """A chained scan begins under the end of the launch ahead of it only while each segment has an SM of its own."""
    import json
    from vig_b200 import _lib, ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x, taps = torch.randn(128, 64, 192, device="cuda").bfloat16(), torch.randn(9, 192, device="cuda").bfloat16()
    q, k, gf, gb = (torch.randn(sms + more, 1, 64, 32, device="cuda").bfloat16() for _ in range(4))
    v = torch.randn(sms + more, 1, 64, 64, device="cuda").bfloat16()
    o, graph = torch.empty_like(v), torch.cuda.CUDAGraph()

    def both():
        y = ops.dwconv3x3(x, taps, None, (8, 8), True)
        was = _lib.lib().vig_chain_launches(1)
        ops.bi_gla(q, k, v, gf, gb, gate_logit_normalizer=16.0, out=o)
        _lib.lib().vig_chain_launches(was)
        return y
    both()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        both()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(5):
            graph.replay()
            torch.cuda.synchronize()
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    events = sorted((e for e in json.load(open(tmp_path / "trace.json"))["traceEvents"] if e.get("cat") == "kernel"), key=lambda e: e["ts"])
    ahead = [b["ts"] < a["ts"] + a["dur"] - 0.05 for a, b in zip(events, events[1:]) if "dwconv" in a["name"] and "bigla_seg" in b["name"]]
    assert ahead and any(ahead) == (not more), ahead          # the profiler may lose a replay


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("L", [40, 100])
def test_overlapping_scans_continue_from_each_others_states(dtype, L):
    """Each call begins under the end of the one that writes the state it starts from, in one of two buffers in turn."""
    import vig_b200
    from vig_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(L)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    q, k, v = (rand(2, 3, L, 64).to(dtype) for _ in range(3))
    g = (torch.nn.functional.logsigmoid(rand(2, 3, L, 64)) / 16).to(dtype)
    start = rand(2, 3, 64, 64)

    def stream(on):
        h, outs = start, []
        was = _lib.lib().vig_chain_launches(on)
        with torch.no_grad():
            for _ in range(30):
                o, h = vig_b200.fused_chunk_gla(q, k, v, g, initial_state=h, output_final_state=True)   # h: a buffer that the call before last has read
                outs.append(o)
        _lib.lib().vig_chain_launches(was)
        torch.cuda.synchronize()
        return outs
    apart = stream(0)
    assert all(all(torch.equal(a, b) for a, b in zip(stream(1), apart)) for _ in range(10))
