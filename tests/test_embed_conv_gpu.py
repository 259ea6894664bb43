"""First embedding convolution + bias + LayerNorm + GELU as one kernel against the fp32 steps with the same roundings: odd sides
(clipped window at the far edges), pixel counts that do not fill a tile of 16, every channel count."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,W,O,bias,gelu", [(1, 1, 1, 32, True, True), (2, 7, 9, 48, False, True), (3, 32, 64, 48, True, True), (1, 33, 30, 64, True, False),
                                               (2, 224, 224, 48, True, True)])
def test_embed_conv_ln(dtype, B, H, W, O, bias, gelu):
    from vig_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(H + O)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x, w, b = rnd(B, 3, H, W).to(dtype), (rnd(O, 3, 3, 3) / 27 ** 0.5).to(dtype), (0.1 * rnd(O)).to(dtype) if bias else None
    lw, lb = (1 + 0.1 * rnd(O)).to(dtype), (0.1 * rnd(O)).to(dtype)
    got = ops.embed_conv_ln(x, w, b, lw, lb, 1e-5, gelu)
    y = F.conv2d(x.double(), w.double(), None, 2, 1).to(dtype)
    y = (y.float() + b.float().view(1, -1, 1, 1)).to(dtype) if bias else y
    y = F.layer_norm(y.double().permute(0, 2, 3, 1), (O,), lw.double(), lb.double(), 1e-5).to(dtype)
    y = F.gelu(y.double()).to(dtype) if gelu else y
    # the same roundings; sums in another order flip some of them, by one unit in the last place of a stored value
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    d = (got.double() - y.double()).abs()
    assert got.shape == y.shape and float(d.max()) <= 4 * ulp * float(y.double().abs().max()) and float(d.norm() / y.double().norm()) < ulp
