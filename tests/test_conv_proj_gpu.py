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
