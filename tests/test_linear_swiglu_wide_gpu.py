"""Weight-stationary gate projection + SwiGLU at K above 192 (64 features a CTA, x boxes streamed): around the row count from
which it is taken, with ragged rows and a K that does not fill the ring evenly."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,I", [(9088, 384, 1024), (9089, 384, 1024), (9217, 384, 1024), (25088, 384, 1024), (37700, 320, 192), (9001, 256, 768)])
def test_linear_swiglu_wide(dtype, M, K, I):
    from vig_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(2 * I, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    a, b = (x.double() @ w.double().t()).chunk(2, -1)
    ref = a * torch.sigmoid(a) * b
    got = ops.linear_swiglu(x, w)
    ops.check_status()
    # one rounding of the result (2^-9, 2^-12) and the sigmoid through tanh.approx (2^-11 relative)
    tol = 4e-3 if dtype == torch.bfloat16 else 1e-3
    assert float((got.double() - ref).norm() / ref.norm()) < tol
