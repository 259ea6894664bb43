"""What a model's forward calls: the fused path, which hands every residual add and norm to the step in front of it, stands for calls of
the modules only while these are what the constructors made.  The operators are replaced by plain stand-ins, so that it runs anywhere."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

import vig_b200
from torch.utils._python_dispatch import TorchDispatchMode, _disable_current_modes

from vig_b200 import modules, ops
from vig_b200.vig import V2PatchEmbed


def _kernel_product(x, w):
    """What a fused kernel makes of the bytes it is given; neither a tensor's own operators nor a mode sees it."""
    with _disable_current_modes(), torch._C.DisableTorchFunctionSubclass():
        return x @ w.as_subclass(torch.Tensor).t()


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


class _Status:
    def poll(self):
        pass

    def snapshot(self):
        pass


@pytest.fixture
def plain_ops(monkeypatch):
    def add_rmsnorm(x, weight, residual=None, eps=1e-6, prenorm=False):
        r = x if residual is None else x + residual
        return (_rms(r, weight, eps), r) if prenorm else _rms(r, weight, eps)

    def linear_add_rmsnorm(x, w, residual, norm_weight, eps=1e-6):
        return add_rmsnorm(_kernel_product(x, w), norm_weight, residual, eps, True)

    def linear_swiglu(x, w):
        gate, y = _kernel_product(x, w).chunk(2, -1)
        return F.silu(gate) * y

    def layernorm_act(x, weight, bias, eps=1e-5, act_swish=False, pre_bias=None, post_add=None, rms_weight=None, rms_eps=1e-6):
        y = F.layer_norm(x if pre_bias is None else x + pre_bias, x.shape[-1:], weight, bias, eps)
        y = F.silu(y) if act_swish else y
        y = y if post_add is None else (y.flatten(1, 2) + post_add).view(y.shape)
        return y if rms_weight is None else (y, _rms(y, rms_weight, rms_eps))

    def bi_gla(q, k, v, g_fwd, g_bwd, out=None, **kw):
        out.copy_(torch.tanh(q.sum(-1, keepdim=True) + k.mean(-1, keepdim=True) + g_fwd.mean(-1, keepdim=True) - g_bwd.mean(-1, keepdim=True)) * v)

    def gate_inject(o, local, gate_logits, w_gnorm, w_lnorm, eps, out_act):
        return o.permute(0, 2, 1, 3).flatten(2) * torch.sigmoid(gate_logits) + local

    monkeypatch.setattr(ops, "status_word", lambda device: _Status())
    monkeypatch.setattr(ops, "linear_add_rmsnorm_supported", lambda x, w, preferred=False: True)
    monkeypatch.setattr(ops, "linear_swiglu_supported", lambda x, w, preferred=False: True)
    monkeypatch.setattr(ops, "swiglu", lambda g, y: F.silu(g) * y)
    monkeypatch.setattr(ops, "dwconv3x3", lambda x, taps, bias, hw, act: F.silu(x * taps[4]))
    monkeypatch.setattr(ops, "token_mean", lambda x: x.mean(1))
    monkeypatch.setattr(ops, "stem_unfold", lambda x, s: F.pad(x.permute(0, 2, 3, 1), (0, 0, 1, s - 1, 1, s - 1)).unflatten(1, (-1, s)).unflatten(3, (-1, s))
                        .permute(0, 1, 3, 2, 4, 5).flatten(3))
    for f in (add_rmsnorm, linear_add_rmsnorm, linear_swiglu, layernorm_act, bi_gla, gate_inject):
        monkeypatch.setattr(ops, f.__name__, f)


def _hook(seen, pick):
    """A hook that keeps what it is given and puts something else in its place."""
    def attach(model):
        def see(module, args, out):
            first = out[0] if isinstance(out, tuple) else out
            seen.append(first.clone())
            other = first.roll(1, -1)                    # (a factor would cancel in the norms)
            return (other, *out[1:]) if isinstance(out, tuple) else other
        pick(model).register_forward_hook(see)
    return attach


class OwnMLP(modules.GLAMLP):
    def forward(self, x):
        return torch.zeros_like(x)


class OwnAttention(modules.GatedLinearAttention):
    def forward(self, x, **kwargs):
        return -x


class OwnBlock(modules.GLABlock):
    def forward_deferred(self, hidden_states, residual, **kwargs):
        return hidden_states * 0.5, hidden_states


class OwnEmbed(V2PatchEmbed):
    def forward(self, x, pos_fn=None):
        tokens, hw = super().forward(x, pos_fn=pos_fn)
        return tokens.roll(1, -1), hw


class Sign(nn.Module):
    def __init__(self, width):
        super().__init__()
        self.weight, self.eps = nn.Parameter(torch.ones(width)), 1e-6

    def forward(self, x, residual=None, prenorm=False):
        r = x if residual is None else x + residual
        return (torch.sign(r), r) if prenorm else torch.sign(r)


def _replace(owner, name, make):
    def put(model):
        parent = owner(model)
        new = make(model)
        if not isinstance(new, Sign):
            new.load_state_dict(getattr(parent, name).state_dict())
        if isinstance(parent, nn.ModuleList):
            parent[int(name)] = new
        else:
            setattr(parent, name, new)
    return put


class Doubled(torch.Tensor):
    """A weight with a product of its own."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        out = super().__torch_function__(func, types, args, kwargs or {})
        return (out * 2).as_subclass(torch.Tensor) if func is F.linear else out


def _own_product(pick):
    def put(model):
        linear = pick(model)
        linear.weight = nn.Parameter(linear.weight.detach().as_subclass(Doubled), requires_grad=False)
    return put


def _own_forward(model):
    mlp = model.blocks[0].mlp
    mlp.forward = lambda x: x * 0.25


REPLACED = {
    "mlp subclass": _replace(lambda m: m.blocks[0], "mlp", lambda m: OwnMLP(m.embed_dim)),
    "mlp forward": _own_forward,
    "attention subclass": _replace(lambda m: m.blocks[1], "attn", lambda m: OwnAttention(d_model=m.embed_dim, expand_k=0.5, expand_v=1, num_heads=m.config.num_attention_heads,
                                                                                       layernorm_eps=1e-6)),
    "block subclass": _replace(lambda m: m.blocks, "1", lambda m: OwnBlock(m.config)),
    "embedding subclass": _replace(lambda m: m, "patch_embed", lambda m: OwnEmbed(32, 16, 3, m.embed_dim)),
    "final norm": _replace(lambda m: m, "norm", lambda m: Sign(m.embed_dim)),
    "attention norm": _replace(lambda m: m.blocks[1], "attn_norm", lambda m: Sign(m.embed_dim)),
    "MLP norm": _replace(lambda m: m.blocks[1], "mlp_norm", lambda m: Sign(m.embed_dim)),
    "output weight": _own_product(lambda m: m.blocks[0].attn.o_proj),
    "gate weight": _own_product(lambda m: m.blocks[1].mlp.gate_proj),
    "down weight": _own_product(lambda m: m.blocks[1].mlp.down_proj),
}
HOOKED = {
    "attention": lambda m: m.blocks[0].attn, "output projection": lambda m: m.blocks[1].attn.o_proj, "mlp": lambda m: m.blocks[1].mlp,
    "gate projection": lambda m: m.blocks[0].mlp.gate_proj, "first norm": lambda m: m.blocks[0].attn_norm, "attention norm": lambda m: m.blocks[1].attn_norm,
    "MLP norm": lambda m: m.blocks[0].mlp_norm, "final norm": lambda m: m.norm, "embedding": lambda m: m.patch_embed,
}


def _model(width):
    torch.manual_seed(width)
    return vig_b200.ViG(img_size=32, depth=2, num_heads=width // 64, embed_dim=width, num_classes=10, expand_k=0.5).eval()


def _runs(width, change, x):
    """Logits of the model as it is and with the fused path switched off, after ``change``."""
    out = []
    for fuse in (True, False):
        model = _model(width)
        model.fuse_norm_epilogues = fuse
        change(model)
        out.append(model(x))
    return out


@pytest.mark.parametrize("width", [192, 256, 384, 768])
def test_replaced_modules_run(plain_ops, width):
    x = torch.randn(2, 3, 32, 48)
    with torch.no_grad():
        fused, steps = _runs(width, lambda m: None, x)
        torch.testing.assert_close(fused, steps, rtol=1e-4, atol=1e-5)           # fp32 sums in another order
        for name, change in REPLACED.items():
            got, want = _runs(width, change, x)
            assert float((want - steps).norm() / steps.norm()) > 1e-3, name      # the replacement shows
            torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-5, msg=name)


@pytest.mark.parametrize("width", [192, 256, 384, 768])
def test_hooks_see_and_replace_the_outputs(plain_ops, width):
    x = torch.randn(2, 3, 32, 48)
    with torch.no_grad():
        for name, pick in HOOKED.items():
            seen = []
            got, want = _runs(width, _hook(seen, pick), x)
            assert len(seen) == 2, name
            torch.testing.assert_close(seen[0], seen[1], rtol=1e-4, atol=1e-5, msg=name)
            torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-5, msg=name)


class Products(TorchDispatchMode):
    seen = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.seen += "mm" in str(func)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("width", [256, 384, 768])
def test_modes_see_the_products(plain_ops, width):
    """A mode that counts operators sees the four products of each block and the classifier's."""
    model = _model(width)
    x = torch.randn(2, 3, 32, 48)
    with torch.no_grad():
        ref = model(x)
        with Products() as p:
            y = model(x)
        assert p.seen >= 4 * 2 + 1
        torch.testing.assert_close(y, ref, rtol=1e-4, atol=1e-5)
        mlp = vig_b200.hier.gMlp(width)
        with Products() as p:
            mlp(torch.randn(2, 6, width))
        assert p.seen == 2
