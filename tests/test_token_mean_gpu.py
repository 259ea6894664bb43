"""Mean over tokens: one, few and many tokens a CTA, one to eight CTAs of a cluster, channel counts that do not fill 64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,L,C", [(1, 1, 64), (2, 49, 768), (3, 129, 192), (2, 300, 200), (1, 836, 96), (2, 5000, 192)])
def test_token_mean(dtype, B, L, C):
    from vig_b200 import ops
    x = torch.randn(B, L, C, generator=torch.Generator(device="cuda").manual_seed(L), device="cuda").to(dtype) + 1
    got, ref = ops.token_mean(x), x.double().mean(1)
    # fp32 sums in blocks of a few dozen, one rounding to the type
    tol = {torch.float32: 1e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert float((got.double() - ref).abs().max()) <= tol * float(ref.abs().max())


def test_many_small_images_at_once():
    """Thousands of clusters at a time, of one CTA to eight: the first CTA of each runs before the others write its memory (a
    cluster barrier on entry; a missing one would show as lost parts of the sums)."""
    from vig_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(3)
    for B, L in ((4000, 129), (2000, 513), (900, 1025)):
        x = torch.randn(B, L, 64, generator=gen, device="cuda").bfloat16()
        ref = x.float().mean(dim=1)
        for _ in range(3):
            # one rounding of the mean (bf16: 8 significant bits, 2^-8 at most) and the order of fp32 sums; a lost part: L / S of L
            assert float((ops.token_mean(x).float() - ref).abs().max()) <= 2 ** -8 * float(ref.abs().max()) + 1e-6


def test_more_images_than_a_launch_takes():
    from vig_b200 import ops
    x = torch.randn(65535 * 2 + 3, 2, 32, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda").half()
    assert float((ops.token_mean(x).double() - x.double().mean(1)).abs().max()) <= 2.0 ** -11 * float(x.abs().max())
