"""The row-local half of a block as one kernel (vig_block_tail_fwd) against the separate kernels it stands for, at the edges of
its 16-, 32- and 64-token tiles, of the clusters of 4 and 2 that share one, and of the rule that picks them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,I,out_act", [(1, 512, True), (16, 64, False), (17, 512, True), (196, 512, True), (2368, 512, False), (2369, 512, True),
                                         (256, 512, False), (257, 512, True), (512, 448, True), (513, 512, False), (1024, 128, True), (1025, 512, True), (100, 256, True), (2401, 128, True), (4736, 512, True), (4737, 512, True), (9999, 512, False)])
def test_block_tail_equals_the_separate_kernels(dtype, M, I, out_act):
    import vig_b200
    from vig_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M + I)
    rnd = lambda *s, k=1.0: (k * torch.randn(*s, generator=g, device="cuda")).to(dtype)  # noqa: E731
    C = 192
    o, local, res, wide = rnd(M, C), rnd(M, C), rnd(M, C), rnd(M, 3 * C)
    gl = wide[:, C:2 * C]
    gw, lw = 1 + rnd(64, k=0.1), 1 + rnd(64, k=0.1)
    n1, n2 = 1 + rnd(C, k=0.1), 1 + rnd(C, k=0.1)
    wo, wg, wd = rnd(C, C, k=C ** -0.5), rnd(2 * I, C, k=C ** -0.5), rnd(C, I, k=I ** -0.5)
    h, r = ops.block_tail(o, local, gl, gw, lw, wo, res, n1, wg, wd, n2, out_act=out_act)
    ops.check_status()
    y = ops.gate_inject(o.view(1, M, 3, 64).permute(0, 2, 1, 3), local.view(1, M, C), gl.unsqueeze(0), gw, lw, 1e-6, out_act)[0]
    r1 = (torch.nn.functional.linear(y, wo).float() + res.float()).to(dtype)
    h1 = vig_b200.add_rmsnorm(r1, n1)
    z = ops.swiglu(*torch.nn.functional.linear(h1, wg).chunk(2, -1))
    r2 = (torch.nn.functional.linear(z, wd).float() + r1.float()).to(dtype)
    h2 = vig_b200.add_rmsnorm(r2, n2)
    # same roundings; sums in another order flip some of them: a few units in the last place (2^-8, 2^-11) of single values
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for got, ref in ((r, r2), (h, h2)):
        d = (got.float() - ref.float())
        assert float(d.norm() / ref.float().norm()) < ulp and float(d.abs().max()) < 6 * ulp * float(ref.float().abs().max())
