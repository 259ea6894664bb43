"""Plans for the C++ forward of the models (``vig_b200/csrc/host_model.cpp``): what the Python modules hold, collected once.

``forward(model, images)`` runs the model's plan, building or rebuilding it when something it was built from has changed, and
answers ``None`` whenever the modules themselves have to run: a precision or configuration without a plan, subclassed or
hooked modules, an overridden ``forward``, replaced operators of ``vig_b200.ops``, gradients enabled, autocast."""
import math
import weakref

import torch
import torch.nn as nn

from . import _lib, hier, modules, ops, vig

_plans = weakref.WeakKeyDictionary()          # model -> plan, or refusal: why the model has none, for as long as that stands
_OPS = {n: getattr(ops, n) for n in ("bi_gla", "dwconv3x3", "gate_inject", "add_rmsnorm", "layernorm_act", "add_layernorm", "linear_swiglu",
                                     "linear_add_rmsnorm", "linear_bias", "swiglu", "token_mean", "stem_fold", "stem_unfold", "stem_conv_ln")}
_GLOBAL_HOOKS = ("_global_forward_hooks", "_global_forward_pre_hooks")
_CLASSES = (vig.ViG, vig.V2PatchEmbed, vig.LayerNorm2d, modules.GLABlock, modules.GatedLinearAttention, modules.GLAMLP, modules.RMSNorm,
            hier.HierViG, hier.VSSBlock, hier.GLA2D, hier.Mlp, hier.gMlp, nn.Linear, nn.Conv2d, nn.LayerNorm, nn.SiLU, nn.GELU, nn.Identity,
            nn.Sequential, nn.ModuleList)


def _status_seen(device):
    return lambda value: ops.status_word(device)._raise(value)


def _watch(plan, mods):
    """Everything whose change makes the plan stale (the C++ side compares identities, versions and sizes)."""
    plan.watch_modules(mods)
    for name in _GLOBAL_HOOKS:
        plan.watch_size(getattr(nn.modules.module, name))
    for name, fn in _OPS.items():
        plan.watch_item(ops.__dict__, name, fn)


def _norm(m):
    return dict(w=m.weight, b=getattr(m, "bias", None), eps=m.eps)


class _NoPlan(Exception):
    """The model has something that only its modules can evaluate."""


def _conv(m, weight=None, stride=None, pad=None):
    if len(set(m.stride)) != 1 or isinstance(m.padding, str) or len(set(m.padding)) != 1 or m.dilation != (1, 1) or m.groups != 1 or m.padding_mode != "zeros":
        raise _NoPlan
    # the parameter itself: what is written to it without a trace (through .data, by a replayed graph) reaches the next call
    return dict(w=m.weight if weight is None else weight, b=m.bias, stride=m.stride[0] if stride is None else stride, pad=m.padding[0] if pad is None else pad)


def _attn(a):
    if not a.fold_gate_bottleneck or a.own_in_proj_gemm or a.o_proj.bias is not None:
        return None
    return dict(pack=lambda: a._pack(True), conv_b=a.in_proj[0].bias, gn_w=a.g_norm.weight, ln_w=a.l_norm.weight, o_w=a.o_proj.weight,
                H=a.num_heads, dk=a.head_qk_dim, dv=a.head_v_dim, act_conv=bool(a.use_act_in_conv), out_act=bool(a.use_out_act), eps=a.g_norm.eps,
                out_scale=a.out_scale, norm=float(a.gate_logit_normalizer), clamp=math.nan if a.clamp_min is None else float(a.clamp_min))


def _vig(model):
    # every module is of a known class, without hooks or a forward of its own, but one may be in the place of another
    if not (type(model.patch_embed) is vig.V2PatchEmbed and type(model.norm) is modules.RMSNorm):
        return None
    pe, conv1 = model.patch_embed, model.patch_embed.proj[0]
    if pe.stride != 8 or conv1.weight.shape[1] != 3 or not isinstance(model.head, nn.Linear) or not len(model.blocks):
        return None
    blocks = []
    for b in model.blocks:
        if type(b) is not modules.GLABlock or "forward_deferred" in b.__dict__:
            return None
        a, mlp, n1, n2 = b.attn, b.mlp, b.attn_norm, b.mlp_norm
        if type(a) is not modules.GatedLinearAttention or type(mlp) is not modules.GLAMLP or type(n1) is not modules.RMSNorm or type(n2) is not modules.RMSNorm:
            return None
        gate, down = mlp.gate_proj, mlp.down_proj
        if not (type(a.o_proj) is type(gate) is type(down) is nn.Linear and gate.bias is None and down.bias is None):
            return None
        attn = _attn(a)
        if attn is None:
            return None
        blocks.append(dict(n1=n1.weight, e1=n1.eps, n2=n2.weight, e2=n2.eps, gate_w=gate.weight, down_w=down.weight, attn=attn))
    probe = model.head.weight.new_empty(1, 1, model.embed_dim)
    fused = bool(model.fuse_norm_epilogues and all(b.epilogues_fit(probe) for b in model.blocks))
    one_kernel = pe.fuse_conv1 and conv1.weight.shape[0] == 96
    ref = weakref.ref(model)
    return _lib.host().VigPlan(dict(
        head_w=model.head.weight, head_b=model.head.bias, on_status=_status_seen(model.head.weight.device), graphs=getattr(model, "replay_graphs", True), blocks=blocks, fused_norms=fused,
        w_gemm=pe._gemm_weight() if one_kernel else None, b1=conv1.bias, ln1=_norm(pe.proj[1]), ln2=_norm(pe.proj[4]),
        cells=_conv(conv1, weight=pe._block_weight(), stride=1, pad=0), conv2=_conv(pe.proj[3]), norm_w=model.norm.weight, norm_e=model.norm.eps,
        pos_fn=lambda hw: ref()._pos(hw)))


def _hier(model):
    embed, pe = [], list(model.patch_embed)
    for i, m in enumerate(pe):
        if isinstance(m, nn.Conv2d):
            rest = pe[i + 1:]
            rest = rest[:next((j for j, r in enumerate(rest) if isinstance(r, nn.Conv2d)), len(rest))]
            norm = next((r for r in rest if isinstance(r, nn.LayerNorm)), None)
            gelu = next((r for r in rest if isinstance(r, nn.GELU)), None)
            if gelu is not None and gelu.approximate != "none":
                return None
            embed.append(dict(conv=_conv(m), norm=None if norm is None else _norm(norm), act=0 if gelu is None else 2))
    c = pe[0]
    own = (tuple(c.kernel_size) == (3, 3) and tuple(c.stride) == (2, 2) and tuple(c.padding) == (1, 1) and c.weight.shape[1] == 3 and
           c.weight.shape[0] in (32, 48, 64) and c.groups == 1 and embed[0]["norm"] is not None)
    stages = []
    for layer in model.layers:
        blocks = []
        for b in layer.blocks:
            attn, gated = _attn(b.op), isinstance(b.mlp, hier.gMlp)
            if attn is None or not (gated or isinstance(b.mlp.act, nn.GELU) and b.mlp.act.approximate == "none"):
                return None
            blocks.append(dict(n1=_norm(b.norm), n2=_norm(b.norm2), attn=attn, gated=gated, fc1_w=b.mlp.fc1.weight, fc1_b=b.mlp.fc1.bias,
                               fc2_w=b.mlp.fc2.weight, fc2_b=b.mlp.fc2.bias))
        down = layer.downsample
        has = not isinstance(down, nn.Identity)
        stages.append(dict(blocks=blocks, conv=_conv(down[1]) if has else None, norm=_norm(down[3]) if has else None))
    head = model.classifier.head
    return _lib.host().HierPlan(dict(head_w=head.weight, head_b=head.bias, on_status=_status_seen(head.weight.device), graphs=getattr(model, "replay_graphs", True), embed=embed, stages=stages,
                                     first_w=c.weight if own else None,
                                     last=_norm(model.classifier.norm)))


def _build(model, make):
    mods = list(model.modules())
    plan = None
    if not (model.training or any(getattr(nn.modules.module, name) for name in _GLOBAL_HOOKS) or any(type(m) not in _CLASSES or "forward" in m.__dict__ or m._forward_hooks or m._forward_pre_hooks for m in mods)):
        params = [p for m in mods for p in m._parameters.values() if p is not None]
        # vectors and matrices go to kernels by address, filters to the library, which takes any strides
        if all(type(p) in (nn.Parameter, torch.Tensor) and p.dtype == params[0].dtype and p.device == params[0].device and (p.dim() == 4 or p.is_contiguous()) for p in params):
            try:
                with torch.no_grad():
                    plan = make(model)
            except _NoPlan:
                pass
    if plan is None:
        plan = _lib.host().Refusal()
    _watch(plan, mods)
    return plan


def _forward(model, images, head, make):
    if torch.is_grad_enabled() or head.dtype not in (torch.bfloat16, torch.float16) or type(images) is not torch.Tensor or not images.is_cuda:
        return None
    plan = _plans.get(model)
    if plan is not None:
        y = plan.forward(images)
        if y is not None or plan.valid():
            return y
    if any(ops.__dict__[n] is not fn for n, fn in _OPS.items()) or head.device != images.device:
        return None
    ops.status_word(images.device)
    plan = _plans[model] = _build(model, make)
    return plan.forward(images)


def vig_forward(model, images):
    head = model.head
    return _forward(model, images, head.weight, _vig) if isinstance(head, nn.Linear) else None


def hier_forward(model, images):
    return _forward(model, images, model.classifier.head.weight, _hier)
