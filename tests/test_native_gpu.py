"""The C++ forward of the models against the Python modules it stands for (same kernels, so the same bits), and its plan's
staleness: changed parameters and attributes are seen, hooks and overridden forwards send the call to the modules."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


def _model(kind, dtype):
    import vig_b200
    torch.manual_seed(1)
    if kind == "hier":
        m = vig_b200.HierViG(depths=[1, 1, 1, 1], dims=64, num_heads=[2, 4, 8, 16], norm_layer="ln2d", patchembed_version="v2", downsample_version="v3",
                             gmlp=True, num_classes=12)
    elif kind == "hier_mlp":
        m = vig_b200.HierViG(depths=[1, 1, 1, 1], dims=64, num_heads=[2, 4, 8, 16], num_classes=12, expand_k=1.0)
    else:
        m = vig_b200.ViG(depth=2, num_classes=12, **vig_b200.vig._PRESETS[kind])
    return m.to("cuda", dtype).eval().requires_grad_(False)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind,size", [("vig_t", (224, 224)), ("vig_t", (80, 112)), ("vig_s", (64, 96)), ("hier", (64, 96)), ("hier_mlp", (96, 64))])
def test_native_forward_equals_the_modules(kind, size, dtype):
    from vig_b200 import native
    m = _model(kind, dtype)
    x = torch.randn(2, 3, *size, device="cuda").to(dtype)
    with torch.no_grad():
        run = native.hier_forward if kind.startswith("hier") else native.vig_forward
        got = run(m, x)
        assert got is not None
        handle = m.register_forward_hook(lambda *a: None)               # a hook anywhere: the modules run
        assert run(m, x) is None
        ref = m(x)
        handle.remove()
        assert run(m, x) is not None                                    # and no longer
    rel = float((got.float() - ref.float()).norm() / ref.float().norm())
    # hier: the branch's add is fused into the next norm; vig_t: the row-local half of a block is one kernel whose sums run in
    # another order, which flips roundings (2^-9) of stored activations
    assert rel < (1e-6 if kind == "vig_s" else 1e-2), rel


def test_plan_follows_the_model():
    from vig_b200 import native
    m = _model("vig_t", torch.bfloat16)
    x = torch.randn(1, 3, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        a = m(x)
        assert native._plans.get(m)
        m.blocks[1].mlp.down_proj.weight.mul_(2.0)                      # in place
        b = m(x)
        m.blocks[0].attn.out_scale = 0.5                                # attribute
        c = m(x)
        m.blocks[0].attn_norm.weight = torch.nn.Parameter(m.blocks[0].attn_norm.weight * 1.5, requires_grad=False)   # replaced
        d = m(x)
        m.blocks[0].forward = lambda *a, **k: None
        assert native.vig_forward(m, x) is None
    outs = [a, b, c, d]
    assert all(not torch.equal(outs[i], outs[i + 1]) for i in range(3))


def test_small_forwards_are_replayed_and_stay_independent():
    """From the second call of a shape a small forward is a replayed graph: results of earlier calls stay what they were, other
    shapes, strides and streams get their own, and a changed weight reaches the next call."""
    from vig_b200 import native
    m = _model("vig_t", torch.bfloat16)
    xs = [torch.randn(1, 3, 64, 64, device="cuda").bfloat16() for _ in range(3)]
    wide = torch.randn(2, 3, 64, 96, device="cuda").bfloat16()
    with torch.no_grad():
        ref = []
        for x in (*xs, wide):
            native._plans.clear()
            ref.append(m(x))                                            # first call of a plan: launched one by one
        for _ in range(3):
            got = [m(x) for x in (*xs, wide)]
            assert all(torch.equal(a, b) for a, b in zip(got, ref))
        assert torch.equal(m(xs[0].contiguous(memory_format=torch.channels_last)), ref[0])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            outs = [m(xs[i % 3]) for i in range(6)]
        torch.cuda.current_stream().wait_stream(side)
        assert all(torch.equal(o, ref[i % 3]) for i, o in enumerate(outs))
        m.head.bias.add_(1.0)
        assert torch.equal(m(xs[0]), m(xs[0])) and not torch.equal(m(xs[0]), ref[0])


@pytest.mark.parametrize("kind", ["vig_t", "vig_s", "hier", "hier_mlp"])
def test_replay_reads_the_images_of_its_call(kind):
    """The kernel in front of the replayed part (8 x 8 cells, with or without a border, the embedding's first convolution, the
    change to channels-last) writes its input from the images at hand, whatever their strides: same kernels, same bits.  Forwards
    of another size in between, and memory that they give back and others fill, change nothing."""
    m = _model(kind, torch.float16)
    xs = [torch.randn(2, 3, 64, 96, device="cuda").half() for _ in range(2)]
    xs.append(torch.randn(2, 3, 64, 192, device="cuda").half()[..., ::2])
    other = torch.randn(1, 3, 96, 32, device="cuda").half()
    with torch.no_grad():
        from vig_b200 import native
        ref = []
        for x in xs:
            native._plans.clear()
            ref.append(m(x))
        for _ in range(3):
            assert all(torch.equal(m(x), r) for x, r in zip(xs, ref))
            m(other)
            filled = [torch.full((n,), float("nan"), device="cuda", dtype=torch.float16) for n in (1024, 4608, 9216, 18432, 73728) for _ in range(8)]
            del filled


def test_shapes_that_push_each_other_out_are_not_captured_for_ever():
    """Two shapes that do not fit the graphs' budget together, in pairs: after a few exchanges both run without a capture, more
    and more rarely interrupted by one; shapes seen once take no room; results stay what launches one by one give."""
    from vig_b200 import native
    m = _model("vig_t", torch.bfloat16)
    small, big = [torch.randn(b, 3, 512, 1024, device="cuda").bfloat16() for b in (60, 120)]       # 23.6 M and 47.2 M of 64 M elements
    once = [torch.randn(1, 3, 64, 64 + 16 * i, device="cuda").bfloat16() for i in range(12)]
    held = []
    with torch.no_grad():
        m.replay_graphs = False
        ref = {t: m(t) for t in (small, big)}
        assert native._plans[m].graphs() == 0
        m.replay_graphs = True
        for _ in range(2):
            assert torch.equal(m(small), ref[small])
        for t in once:                                                   # seen once: the graph stays
            m(t)
        assert native._plans[m].graphs() == 1
        for t in (big, big, small, small) * 8:
            before = native._plans[m].captures()
            assert torch.equal(m(t), ref[t])
            held.append(native._plans[m].captures() - before)
        assert sum(held[:16]) >= 1 and sum(held) <= 8, held


def test_graphs_own_the_scratch_their_gemms_write():
    """Replays of two models on two streams at the same time, without waits between them, give what they give alone; and giving
    back torch's GEMM workspaces takes nothing from a graph (tensors that then get that memory stay as they were)."""
    from vig_b200 import native
    models = [_model("vig_s", torch.bfloat16), _model("vig_s", torch.bfloat16)]
    xs = [torch.randn(2, 3, 224, 224, device="cuda").bfloat16() for _ in models]
    streams = [torch.cuda.Stream() for _ in models]
    with torch.no_grad():
        ref = [m(x) for m, x in zip(models, xs)]
        torch.cuda.synchronize()
        for m, x, s in zip(models, xs, streams):
            with torch.cuda.stream(s):
                for _ in range(3):
                    m(x)
            torch.cuda.synchronize()
        assert all(native._plans[m].graphs() == 1 for m in models)
        outs = []
        for _ in range(50):
            for m, x, s in zip(models, xs, streams):
                with torch.cuda.stream(s):
                    outs.append(m(x))
        torch.cuda.synchronize()
        assert all(torch.equal(o, ref[i % 2]) for i, o in enumerate(outs))
        torch._C._cuda_clearCublasWorkspaces()
        bystanders = [torch.full((1 << 20,), float(i), device="cuda") for i in range(64)]
        with torch.cuda.stream(streams[0]):
            again = models[0](xs[0])
        torch.cuda.synchronize()
        assert torch.equal(again, ref[0]) and all(bool((b == i).all()) for i, b in enumerate(bystanders))


def test_a_refusal_lasts_as_long_as_its_reason():
    """A call in training mode, a hook on a submodule, an overridden forward: the modules run while it lasts, the plan after it."""
    from vig_b200 import native
    x = torch.randn(1, 3, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        m = _model("vig_t", torch.bfloat16).train()
        assert native.vig_forward(m, x) is None and native.vig_forward(m, x) is None
        m.eval()
        ref = native.vig_forward(m, x)
        assert ref is not None
        handle = m.blocks[1].mlp.register_forward_pre_hook(lambda *a: None)
        assert native.vig_forward(m, x) is None and native.vig_forward(m, x) is None
        handle.remove()
        assert torch.equal(native.vig_forward(m, x), ref)
        m.blocks[0].forward = m.blocks[0].forward
        assert native.vig_forward(m, x) is None and native.vig_forward(m, x) is None
        del m.blocks[0].forward
        assert torch.equal(native.vig_forward(m, x), ref)


def test_global_hooks_see_every_module():
    """Hooks registered for all modules: before the first forward, between forwards, one in another's place."""
    x = torch.randn(1, 3, 64, 64, device="cuda").bfloat16()
    names = []
    see = lambda mod, args, out=None: names.append(type(mod).__name__)  # noqa: E731
    with torch.no_grad():
        m = _model("vig_t", torch.bfloat16)
        for register in (nn.modules.module.register_module_forward_hook, nn.modules.module.register_module_forward_pre_hook):
            for warm in (False, True):
                if warm:
                    m(x), m(x), m(x)
                for _ in range(2):
                    handle = register(see)
                    names.clear()
                    m(x)
                    handle.remove()
                    assert names.count("GatedLinearAttention") == 2, names
                names.clear()
                m(x)
                assert not names


def test_parameters_of_other_strides_and_convolutions_of_other_kinds():
    """Transposed and strided parameters, also where address, version and identity stay the same, and a convolution that pads
    otherwise: the modules' results."""
    from vig_b200 import native
    x = torch.randn(1, 3, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        m = _model("vig_t", torch.bfloat16)
        ref = m(x)
        w = m.blocks[0].attn.o_proj.weight
        w.data = w.data.t().contiguous().t()                            # the same values, column by column
        assert native.vig_forward(m, x) is None and float((m(x) - ref).norm() / ref.norm()) < 1e-2
        w.data = w.data.contiguous()
        assert native.vig_forward(m, x) is not None
        before = w.data_ptr()
        w.data = w.data.t()                                             # square: other values at the same address
        assert w.data_ptr() == before
        turned = m(x)
        w.data = w.data.contiguous()
        fresh = m(x)
        assert float((turned - fresh).norm() / fresh.norm()) < 1e-2 < float((turned - ref).norm() / ref.norm())
        h = _model("hier", torch.float16)
        y = x.half()
        assert native.hier_forward(h, y) is not None
        h.layers[0].downsample[1].padding_mode = "circular"
        assert native.hier_forward(h, y) is None


@pytest.mark.parametrize("kind", ["vig_t", "hier", "hier_mlp"])
def test_weights_written_without_a_trace(kind):
    """Writes through .data leave a parameter's version alone; what needs no derived form -- filters of the strided convolutions,
    projections, norms -- is read where it lies, also by a replayed graph."""
    m, fresh = _model(kind, torch.float16), _model(kind, torch.float16)
    x = torch.randn(2, 3, 64, 96, device="cuda").half()
    convs = [m.patch_embed.proj[3]] if kind == "vig_t" else [c for c in m.modules() if isinstance(c, nn.Conv2d) and c.groups == 1]
    with torch.no_grad():
        for _ in range(3):
            m(x)
        for part in (convs, [l for l in m.modules() if isinstance(l, nn.LayerNorm)]):
            for c in part:
                c.weight.data.mul_(1.25)
        changed = m(x)
        fresh.load_state_dict(m.state_dict())
        assert torch.equal(changed, fresh(x))


def test_an_error_is_reported_once():
    """A bit in the device's error word, seen by a forward's copy of it: the next forward or ``check_status`` reports it, not both."""
    import vig_b200
    m = _model("vig_t", torch.bfloat16)
    x = torch.randn(1, 3, 64, 64, device="cuda").bfloat16()
    word = vig_b200.ops.status_word("cuda").tensor

    def left_by_a_forward():
        word.fill_(2)
        m(x)
        torch.cuda.synchronize()

    with torch.no_grad():
        m(x)
        torch.cuda.synchronize()
        m(x)
        torch.cuda.synchronize()
        vig_b200.check_status()
        left_by_a_forward()
        with pytest.raises(RuntimeError, match="status 2"):
            vig_b200.check_status()
        for _ in range(3):
            m(x)
            torch.cuda.synchronize()
        left_by_a_forward()
        with pytest.raises(RuntimeError, match="status 2"):
            m(x)
        vig_b200.check_status()
        for _ in range(3):
            m(x)
            torch.cuda.synchronize()


def test_a_plan_is_replaced_while_the_caller_captures():
    """A change of the model inside the caller's own capture drops the plan and its graphs: the capture goes on."""
    from vig_b200 import native
    m = _model("vig_s", torch.bfloat16)
    x = torch.randn(2, 3, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        for _ in range(3):
            m(x)
        assert native._plans[m].graphs() == 1
        ref = m(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            m.replay_graphs = False
            y = m(x)
        assert native._plans[m].graphs() == 0
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, ref)


def test_dispatch_modes_see_the_forward():
    """A mode that watches torch's operators (operation counters, loggers) sees a forward's GEMMs, also once it is replayed."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Count(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen += "mm" in str(func)
            return func(*args, **(kwargs or {}))

    m = _model("vig_s", torch.bfloat16)
    x = torch.randn(2, 3, 64, 64, device="cuda").bfloat16()
    with torch.no_grad():
        for _ in range(3):
            ref = m(x)
        with Count() as c:
            y = m(x)
        assert c.seen >= 4 and torch.equal(y, ref) and torch.equal(m(x), ref)


@pytest.mark.parametrize("kind", ["vig_t", "hier"])
def test_changes_give_what_a_fresh_model_gives(kind):
    """After each kind of change -- a weight in place, a replaced parameter, an attribute, another precision -- the plan's logits
    are those of a model that was made with it."""
    m = _model(kind, torch.bfloat16 if kind == "vig_t" else torch.float16)
    x = torch.randn(2, 3, 64, 96, device="cuda").to(next(m.parameters()).dtype)
    attn = (lambda n: n.blocks[0].attn) if kind == "vig_t" else (lambda n: n.layers[1].blocks[0].op)

    def check():
        fresh = _model(kind, next(m.parameters()).dtype)
        fresh.load_state_dict(m.state_dict())
        attn(fresh).use_out_act = attn(m).use_out_act
        got = [m(x) for _ in range(3)]
        want = fresh(x)
        assert all(torch.equal(g, want) for g in got)
        return want

    with torch.no_grad():
        for p in m.parameters():                                         # weights at which every one of these changes shows in 16 bits
            if p.dim() > 1:
                p.normal_(0, p[0].numel() ** -0.5)
        outs = [check()]
        attn(m).qkv_proj.weight.mul_(1.5)
        outs.append(check())
        attn(m).gk_proj[1].weight = nn.Parameter(attn(m).gk_proj[1].weight * -2, requires_grad=False)
        outs.append(check())
        attn(m).in_proj[0].weight.add_(0.1)
        outs.append(check())
        attn(m).use_out_act = not attn(m).use_out_act
        outs.append(check())
        m.half() if kind == "vig_t" else m.bfloat16()
        x = x.to(next(m.parameters()).dtype)
        outs.append(check())
    assert all(not torch.equal(a.float(), b.float()) for a, b in zip(outs, outs[1:]))


@pytest.mark.parametrize("kind,size", [("vig_t", 64), ("vig_t", 512), ("hier", 64)])
def test_weights_made_on_the_way_are_complete_before_they_are_read(kind, size):
    """A plan's first forward makes the stacked weights between its launches: neither the launch behind them nor the last of the launches that make them
    overlaps, and the result is that of the second forward, also in memory that held something else."""
    from vig_b200 import _lib
    m, seen = _model(kind, torch.bfloat16), []
    attns = [a for a in m.modules() if hasattr(a, "_pack")]
    for a in attns:
        def pack(fold, own=a._pack):
            seen.append(_lib.lib().vig_chain_launches(0))
            _lib.lib().vig_chain_launches(seen[-1])
            return own(fold)
        a._pack = pack
    x = torch.randn(1, 3, size, size, device="cuda").bfloat16()
    with torch.no_grad():
        before = [torch.full((1 << n,), float("nan"), device="cuda", dtype=torch.bfloat16) for n in range(8, 20) for _ in range(8)]
        del before
        first = m(x)
        assert len(seen) == len(attns) and not any(seen)
        for _ in range(3):
            assert torch.equal(m(x), first)
    assert len(seen) == len(attns)
