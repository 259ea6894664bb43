"""Products on pairs of CTAs (tcgen05, cta_group::2) against fp64: rows around the 128 of a CTA and the 256 of a pair, features that do not
fill the last tile of 128, one and many k boxes, W streamed (K = 448 and up, few row tiles) and kept for the launch, leading dimensions."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
# one rounding of the result (2^-9, 2^-12, uniform: over sqrt(3)) and, for SwiGLU, the sigmoid through tanh.approx (2^-11)
TOL = {torch.bfloat16: 2.5e-3, torch.float16: 6e-4}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,I", [(1, 64, 64), (127, 192, 512), (129, 384, 192), (255, 448, 128), (257, 768, 320), (1000, 1024, 2816), (9473, 384, 1024),
                                   (19200, 320, 1024), (20001, 64, 128), (37500, 192, 320)])
def test_swiglu(dtype, M, K, I):
    import vig_b200
    g = torch.Generator(device="cuda").manual_seed(M + K + I)
    x = torch.randn(M, 2 * K, generator=g, device="cuda").to(dtype)[:, :K]          # rows of a wider matrix
    w = (torch.randn(2 * I, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    out = torch.full((M, I + 8), 7.0, device="cuda", dtype=dtype)
    lib, ptr = vig_b200._lib.lib(), vig_b200._lib.ptr
    assert lib.vig_linear_swiglu_supported(M, K, I, vig_b200._lib.dtype_code(x))
    assert lib.vig_linear_swiglu_fwd(ptr(x), 2 * K, ptr(w), ptr(out), I + 8, M, K, I, vig_b200._lib.dtype_code(x), None, vig_b200._lib.stream_ptr()) == 0
    rows = torch.cat([torch.arange(min(M, 3000)), torch.arange(max(0, M - 3000), M)]).cuda()
    a, b = (x[rows].double() @ w.double().t()).chunk(2, -1)
    ref = a * torch.sigmoid(a) * b
    assert float((out[rows, :I].double() - ref).norm() / ref.norm()) < TOL[dtype]
    assert torch.equal(out[:, I:], torch.full_like(out[:, I:], 7.0))                # nothing past the last feature


def test_a_hooked_projection_runs_by_itself():
    """A hook on the gate projection sees its output also where the fused kernel would take its place."""
    import vig_b200
    mlp = vig_b200.modules.GLAMLP(384).cuda().bfloat16()
    x = torch.randn(1, 4096, 384, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        fused, seen = mlp(x), []
        mlp.gate_proj.register_forward_hook(lambda m, i, o: seen.append(o))
        hooked = mlp(x)
    assert len(seen) == 1 and seen[0].shape[-1] == 2 * mlp.intermediate_size
    assert float((fused.float() - hooked.float()).norm() / hooked.float().norm()) < 1e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N,with_res", [(1, 64, 256, True), (129, 704, 256, False), (257, 384, 384, True), (19201, 128, 384, True), (300, 2048, 768, True),
                                            (9473, 192, 768, True), (20000, 320, 768, False)])
def test_projection_add_norm(dtype, M, K, N, with_res):
    """Rows of 256, 384 and 768 (two pairs a row): the sum against fp64 with the projection rounded as the separate kernels round it, the
    norm against fp64 of the sum that was returned; one and several tiles a cluster, ragged rows."""
    import vig_b200
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    res = torch.randn(M, N, generator=g, device="cuda").to(dtype) if with_res else None
    nw = (1 + 0.1 * torch.randn(N, generator=g, device="cuda")).to(dtype)
    h, r = vig_b200.ops.linear_add_rmsnorm(x, w, res, nw, 1e-6)
    vig_b200.check_status()
    ref = x.double() @ w.double().t()
    if with_res:
        ref = ref + res.double()
    rd = r.double()
    norm = rd * torch.rsqrt((rd * rd).mean(-1, keepdim=True) + 1e-6) * nw.double()
    # the sum: two roundings, of values of up to its own size; the norm: one
    assert float((rd - ref).norm() / ref.norm()) < 2 * TOL[dtype]
    assert float((h.double() - norm).norm() / norm.norm()) < TOL[dtype]


@pytest.mark.parametrize("name", ["vig_t", "vig_s"])
@pytest.mark.parametrize("pick", [lambda m: m.blocks[0].mlp_norm, lambda m: m.blocks[1].attn.o_proj, lambda m: m.blocks[1].mlp, lambda m: m.blocks[0].attn,
                                  lambda m: m.norm, lambda m: m.patch_embed], ids=["mlp_norm", "o_proj", "mlp", "attn", "norm", "patch_embed"])
def test_a_hooked_module_runs_by_itself(name, pick):
    """A hook on a module that one kernel would stand for sees what the module gives, and what it returns instead is taken."""
    import vig_b200
    model = vig_b200.ViG(depth=3, **vig_b200.vig._PRESETS[name], num_classes=10).cuda().bfloat16().eval()
    x = torch.randn(2, 3, 64, 64, device="cuda").bfloat16()
    seen = []

    def turn(m, i, o):                                        # (a factor would cancel in the norms)
        first = o[0] if isinstance(o, tuple) else o
        seen.append(first.float())
        return (first.roll(1, -1), *o[1:]) if isinstance(o, tuple) else first.roll(1, -1)

    with torch.no_grad():
        plain = model(x)
        pick(model).register_forward_hook(turn)
        got = model(x)
        model.fuse_norm_epilogues = False
        want = model(x)
    assert len(seen) == 2 and float((seen[0] - seen[1]).norm() / seen[1].norm()) < 2e-2
    assert float((got.float() - want.float()).norm() / want.float().norm()) < 2e-2 and not torch.equal(got, plain)


def _off16(t):
    """The same values two bytes off a 16-byte boundary, as a view into a flat buffer has them."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return flat[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("name,size,batch", [("vig_t", 64, 2), ("vig_t", 224, 52), ("vig_s", 224, 106), ("vig_b", 64, 2)])
def test_matrices_off_16_bytes(name, size, batch):
    """Matrices that TMA cannot read go to the library's GEMM, from the modules and from the C++ forward, one at a time."""
    import vig_b200
    from vig_b200 import native
    model = vig_b200.ViG(depth=1, **vig_b200.vig._PRESETS[name], num_classes=10).cuda().bfloat16().eval().requires_grad_(False)
    x = torch.randn(batch, 3, size, size, device="cuda").bfloat16()
    blk = model.blocks[0]
    with torch.no_grad():
        ref = model(x).float()
        for linear in (blk.attn.o_proj, blk.mlp.gate_proj, blk.mlp.down_proj):
            keep = linear.weight.data
            linear.weight.data = _off16(keep)
            assert linear.weight.data_ptr() % 16
            got = native.vig_forward(model, x)
            assert got is not None
            for y in (got, model.head(model.forward_features(x))):
                assert float((y.float() - ref).norm() / ref.norm()) < 1e-2
            linear.weight.data = keep


def test_rows_off_16_bytes():
    """Inputs of an MLP by itself that TMA cannot read: off 16 bytes, an odd row stride, one row for all."""
    import vig_b200
    mlp = vig_b200.modules.GLAMLP(384).cuda().bfloat16().requires_grad_(False)
    x = torch.randn(2, 2048, 384, device="cuda").bfloat16()
    wide = torch.empty(2, 2048, 387, device="cuda", dtype=torch.bfloat16)
    wide[..., :384] = x
    with torch.no_grad():
        ref = mlp(x).float()
        for y in (_off16(x), wide[..., :384]):
            assert float((mlp(y).float() - ref).norm() / ref.norm()) < 1e-2
        one = mlp(x[:1, :1].expand(1, 4096, 384)).float()
        assert float((one - ref[:1, :1]).norm() / one.norm()) < 1e-2
        row = torch.randn(192, 1, device="cuda").bfloat16().t()                     # one row, "contiguous" with a row stride of 1
        narrow = vig_b200.modules.GLAMLP(192).cuda().bfloat16().requires_grad_(False)
        assert row.stride(0) == 1 and float((narrow(row) - narrow(row.clone(memory_format=torch.contiguous_format))).norm()) < 1e-2 * float(narrow(row).norm())


@pytest.mark.parametrize("N,K", [(256, 256), (256, 704), (384, 384), (384, 1024), (768, 768), (768, 2048)])
def test_long_rows_are_counted_in_rounds(N, K):
    """The one kernel works on as many tiles of 256 rows at a time as there are pairs of SMs (clusters of four for rows of 768): while rounds
    are few it is taken for full ones and not for a single tile more; many rounds always are."""
    import math

    import vig_b200
    lib = vig_b200._lib.lib()
    bf16 = vig_b200._lib.dtype_code(torch.empty(0, dtype=torch.bfloat16))
    takes = lambda tiles: bool(lib.vig_linear_add_rmsnorm_preferred(tiles * 256, K, N, bf16))  # noqa: E731
    most = torch.cuda.get_device_properties(0).multi_processor_count // (4 if N == 768 else 2)
    given_up = [t for t in range(1, 4 * most + 1) if takes(t) and not takes(t + 1)]
    full = math.gcd(*given_up)
    assert given_up and 0.75 * most <= full <= most
    assert not takes(1) and all(takes(t) for t in range(40 * most, 44 * most))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,I", [(300, 384, 192), (38000, 192, 128), (19200, 384, 1024), (700, 768, 320)])
def test_swiglu_infinities_stay_in_their_rows(dtype, M, K, I):
    """Infinities and NaN in a few rows of x, the last one among them: the other rows keep their bits."""
    import vig_b200
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(2 * I, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    clean = vig_b200.ops.linear_swiglu(x, w)
    bad = torch.tensor([0, 127, 130, M // 2, M - 1], device="cuda")
    x[bad, torch.tensor([0, K - 1, 5, 63, 64 % K], device="cuda")] = torch.tensor([float("inf"), float("nan"), -float("inf"), float("nan"), float("inf")], device="cuda").to(dtype)
    out = vig_b200.ops.linear_swiglu(x, w)
    vig_b200.check_status()
    rest = torch.ones(M, dtype=torch.bool, device="cuda")
    rest[bad] = False
    assert torch.equal(out[rest], clean[rest]) and not bool(out[bad].isfinite().all(-1).any())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N", [(300, 512, 192), (300, 256, 256), (19201, 384, 384), (600, 2048, 768), (9473, 768, 768)])
def test_projection_add_norm_infinities_stay_in_their_rows(dtype, M, K, N):
    """Infinities and NaN in rows of x and of the residual, in either half of a row that two pairs share: the other rows keep their bits."""
    import vig_b200
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    w = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(dtype)
    res = torch.randn(M, N, generator=g, device="cuda").to(dtype)
    nw = (1 + 0.1 * torch.randn(N, generator=g, device="cuda")).to(dtype)
    clean = vig_b200.ops.linear_add_rmsnorm(x, w, res, nw)
    x[0, 3], x[130, K - 1] = float("nan"), float("inf")
    res[127, 0], res[M // 2, N - 1], res[M - 1, N // 2] = float("inf"), float("nan"), -float("inf")
    got = vig_b200.ops.linear_add_rmsnorm(x, w, res, nw)
    vig_b200.check_status()
    bad = torch.tensor([0, 127, 130, M // 2, M - 1], device="cuda")
    rest = torch.ones(M, dtype=torch.bool, device="cuda")
    rest[bad] = False
    for a, b in zip(got, clean):
        assert torch.equal(a[rest], b[rest]) and not bool(a[bad].isfinite().all(-1).any())


@pytest.mark.parametrize("M,K,N", [(20000, 512, 192), (300, 256, 256), (19201, 384, 384), (9473, 768, 768)])
def test_projection_add_norm_in_place(M, K, N):
    """The sum may be written over the residual."""
    import vig_b200
    from vig_b200 import _lib
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = (torch.randn(N, K, device="cuda") / K ** 0.5).bfloat16()
    res, nw = torch.randn(M, N, device="cuda").bfloat16(), torch.randn(N, device="cuda").bfloat16()
    want_h, want_r = vig_b200.ops.linear_add_rmsnorm(x, w, res, nw, 1e-6)
    h = torch.empty_like(res)
    assert _lib.lib().vig_linear_add_rmsnorm_fwd(_lib.ptr(x), K, _lib.ptr(w), _lib.ptr(res), _lib.ptr(nw), _lib.ptr(res), _lib.ptr(h), M, K, N, 1e-6, _lib.dtype_code(x),
                                                 None, _lib.stream_ptr()) == 0
    assert torch.equal(h, want_h) and torch.equal(res, want_r)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N,biased", [(1, 64, 8, True), (255, 192, 264, True), (257, 384, 256, False), (19000, 192, 768, True), (19001, 384, 520, True), (2500, 768, 1544, True), (20000, 320, 2304, False)])
def test_pair_linear(dtype, M, K, N, biased):
    """x W^T + bias on CTA pairs: W streamed and kept, partial tiles on every side, strided rows.  One rounding of fp32 sums: 2^-9, 2^-12 of the largest."""
    from vig_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(M)
    rand = lambda *s: torch.randn(*s, generator=gen, device="cuda").to(dtype)  # noqa: E731
    x, w, b = rand(M, K + 8)[:, :K], rand(N, K) / K ** 0.5, rand(N) if biased else None
    out = torch.full((M, N + 8), 7.0, device="cuda", dtype=dtype)
    st = _lib.lib().vig_linear_pair_fwd(_lib.ptr(x), K + 8, _lib.ptr(w), _lib.ptr(b), _lib.ptr(out), N + 8, M, K, N, _lib.dtype_code(x), None, _lib.stream_ptr())
    assert st == 0 and bool((out[:, N:] == 7).all())
    ref = torch.nn.functional.linear(x.float(), w.float(), None if b is None else b.float())
    assert rel_err(out[:, :N].float(), ref) < (4e-3 if dtype == torch.bfloat16 else 5e-4)
    assert _lib.lib().vig_linear_pair_fwd(_lib.ptr(x), K + 8, _lib.ptr(w), _lib.ptr(b), _lib.ptr(out), N + 8, M, K - 8, N, _lib.dtype_code(x), None, _lib.stream_ptr()) == -2


def test_linear_bias_refuses_what_it_refused():
    """``vig_linear_bias_fwd`` takes up to 192 columns for each SM; ``vig_linear_pair_fwd`` any number."""
    from vig_b200 import _lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M, K, N = 256 * sms, 64, 192 * sms + 8
    x, w, out = (torch.empty(*s, device="cuda", dtype=torch.bfloat16) for s in ((M, K), (N, K), (M, N)))
    call = lambda n: _lib.lib().vig_linear_bias_fwd(_lib.ptr(x), K, _lib.ptr(w), None, _lib.ptr(out), N, M, K, n, _lib.dtype_code(x), None, _lib.stream_ptr())  # noqa: E731
    assert call(N) == -2 and call(N - 8) == 0
