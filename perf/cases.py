"""What a user of this package has it do, as a list of measurable cases: image classification with the ViG and HierViG
models, the bi-GLA operator called by itself, and the operator inside a training step (forward and backward).

``listed()`` names fixed cases, ``draw(rng)`` gives further ones of the same ranges; ``prepare`` makes what a program has
in hand before the call, ``run`` is one call through the public entry points, ``work`` the bytes and operations of it,
``tolerance`` how far two correct implementations may be apart."""
import math

import torch

import vig_b200

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BYTES = {"f32": 4, "bf16": 2, "f16": 2}
WIDTH = {"vig_t": 192, "vig_s": 384, "vig_b": 768}
HEADS = {"vig_t": 3, "vig_s": 6, "vig_b": 12}
DEPTH = 12
# the hierarchical model: widths, heads and depths of its four stages, gated MLP, strided 3x3 convolutions between stages
HIER_DIMS, HIER_HEADS, HIER_DEPTHS = (96, 192, 384, 768), (3, 6, 12, 24), (2, 2, 9, 2)
CLASSES = 1000


def _model(name, preset, height, width, batch, dtype, expand_k=0.5):
    return dict(name=name, kind="model", preset=preset, height=height, width=width, batch=batch, dtype=dtype, expand_k=expand_k)


def _op(name, kind, entry, B, H, L, dk, dv, dtype, layout="tokens", raw_gates=False):
    return dict(name=name, kind=kind, entry=entry, B=B, H=H, L=L, dk=dk, dv=dv, dtype=dtype, layout=layout, raw_gates=raw_gates)


def listed():
    return [
        # ---- models, eval forward from an image batch on the device to logits ----
        # one photo at a time through the smallest shipped model: latency of an interactive service
        _model("vig_t_224_b1", "vig_t", 224, 224, 1, "bf16"),
        # a batch server on standard crops
        _model("vig_s_224_b128", "vig_s", 224, 224, 128, "bf16", 1.0),
        # the benchmark's workload: high-resolution images, long token sequences
        _model("vig_t_1024_b64", "vig_t", 1024, 1024, 64, "bf16", 1.0),
        # the largest: 16384 tokens an image, wide projections
        _model("vig_b_2048_b8", "vig_b", 2048, 2048, 8, "bf16", 1.0),
        # a few photos of another aspect ratio (22 x 38 patches), half precision, shipped head size
        _model("vig_t_352x608_b3_f16", "vig_t", 352, 608, 3, "f16"),
        # the hierarchical model on a batch of standard crops: four stages of 3136 to 49 tokens
        _model("hier_224_b64_f16", "hier", 224, 224, 64, "f16"),
        # ---- the operator by itself ----
        # the reference's smallest check in full precision: one 14 x 14 patch grid
        _op("op_f32_196", "op", "bi", 2, 3, 196, 64, 64, "f32", "heads"),
        # the reference model's own call, both directions' gates stacked along the batch, a 56 x 56 grid
        _op("op_bid_3136", "op", "bid", 32, 3, 3136, 32, 64, "bf16"),
        # a causal stream continued from a state that an earlier call left, ragged length
        _op("op_causal_state_1000", "op", "causal", 4, 12, 1000, 64, 64, "f16"),
        # ---- the operator in training: forward and all gradients ----
        # a training batch of standard crops, raw gate logits
        _op("train_196_b128", "train", "bi", 128, 3, 196, 32, 64, "bf16", "tokens", True),
        # fine-tuning at high resolution
        _op("train_4096_b8", "train", "bi", 8, 6, 4096, 64, 64, "bf16", "tokens", True),
        # the reference's causal training operator in full precision, odd length
        _op("train_causal_f32_1021", "train", "causal", 4, 3, 1021, 32, 64, "f32", "heads"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["model", "model", "op", "train"])
    if kind == "model":
        preset = rng.choice(["vig_t", "vig_t", "vig_s", "vig_b", "hier"])
        dtype = "f16" if preset == "hier" else rng.choice(["bf16", "bf16", "f16"])
        if preset == "hier":
            height = 32 * _log_int(rng, 4, 14)
            width = 32 * _log_int(rng, 4, 14)
            batch = _log_int(rng, 1, max(1, 64 * 224 * 224 // (height * width)))
            expand_k = rng.choice([0.5, 1.0])
        else:
            height = 16 * _log_int(rng, 8, 128)
            width = min(2048, max(128, 16 * round(height * math.exp(rng.uniform(-0.5, 0.5)) / 16)))
            # at most the work of the largest listed case of the same width, and 64 images of 1024 x 1024 for the narrow ones
            most = {"vig_t": 64 << 20, "vig_s": 48 << 20, "vig_b": 32 << 20}[preset]
            batch = _log_int(rng, 1, max(1, min(256, most // (height * width))))
            expand_k = rng.choice([0.5, 1.0])
        c = _model(None, preset, height, width, batch, dtype, expand_k)
    else:
        entry = rng.choice(["bi", "bid", "causal"]) if kind == "op" else rng.choice(["bi", "causal"])
        dk, dv = rng.choice([(32, 64), (64, 64), (64, 64), (16, 32), (32, 32)])
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        L = _log_int(rng, 49, 16384)
        H = rng.choice([2, 3, 6, 12])
        # operator: at most 64 sequences x 3 heads of 4096 tokens; training and full precision: a quarter of that
        most = (64 if kind == "op" and dtype != "f32" else 16) * 3 * 4096
        B = _log_int(rng, 1, max(1, min(256, most // (H * L))))
        raw = kind == "train" and entry == "bi" and rng.random() < 0.7 or kind == "op" and entry == "bi" and rng.random() < 0.5
        c = _op(None, kind, entry, B, H, L, dk, dv, dtype, rng.choice(["tokens", "tokens", "heads"]), raw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------------------------
def _build_model(case):
    if case["preset"] == "hier":
        return vig_b200.HierViG(depths=HIER_DEPTHS, dims=list(HIER_DIMS), num_heads=HIER_HEADS, norm_layer="ln2d", patchembed_version="v2",
                                downsample_version="v3", gmlp=True, use_act_in_conv=False, use_out_act=False, num_classes=CLASSES,
                                expand_k=case["expand_k"])
    return vig_b200.build_vig(case["preset"], expand_k=case["expand_k"], num_classes=CLASSES)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    rand = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")  # noqa: E731
    if case["kind"] == "model":
        with torch.device("cuda"):
            model = _build_model(case)
        with torch.no_grad():
            for name, p in model.named_parameters():
                # norms near one, biases small, matrices and filters at the scale that keeps activations of order one
                if p.dim() == 1 and name.endswith("weight"):
                    p.copy_(1 + 0.1 * rand(*p.shape))
                elif p.dim() == 1:
                    p.copy_(0.02 * rand(*p.shape))
                elif name == "pos_embed":
                    p.copy_(0.2 * rand(*p.shape))
                else:
                    p.copy_(rand(*p.shape) / math.sqrt(p[0].numel()))
        model = model.to("cuda", dtype).eval().requires_grad_(False)
        images = rand(case["batch"], 3, case["height"], case["width"]).to(dtype)   # normalised pixels
        return dict(case=case, model=model, images=images)

    B, H, L, dk, dv = (case[n] for n in ("B", "H", "L", "dk", "dv"))

    def tensor(b, d):
        # "tokens": the [B, L, H*d] output of a projection seen as [B, H, L, d]; "heads": [B, H, L, d] as it is
        return rand(b, L, H, d).permute(0, 2, 1, 3) if case["layout"] == "tokens" else rand(b, H, L, d)

    q, k, v = tensor(B, dk).to(dtype), tensor(B, dk).to(dtype), tensor(B, dv).to(dtype)
    gates = [tensor(B, dk)] if case["entry"] == "causal" else [tensor(2 * B, dk)] if case["entry"] == "bid" else [tensor(B, dk), tensor(B, dk)]
    if not case["raw_gates"]:
        gates = [torch.nn.functional.logsigmoid(g) / 16 for g in gates]           # log-space gates as ViG computes them
    gates = [g.to(dtype) for g in gates]
    state = dict(case=case, inputs=[q, k, v, *gates])
    if case["kind"] == "train":
        for t in state["inputs"]:
            t.requires_grad_(True)
        state["d_out"] = rand(B, H, L, dv).to(dtype)
    elif case["entry"] == "causal":
        state["initial"] = rand(B, H, dk, dv)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "model":
        with torch.no_grad():
            return state["model"](state["images"])
    q, k, v, *gates = state["inputs"]
    if case["kind"] == "op":
        with torch.no_grad():
            if case["entry"] == "causal":
                return vig_b200.fused_chunk_gla(q, k, v, gates[0], initial_state=state["initial"], output_final_state=True)
            if case["entry"] == "bid":
                return vig_b200.bid_fused_recurrent_gla(q, k, v, gates[0])[0]
            return vig_b200.bi_gla(q, k, v, *gates, out_scale=0.5, gate_logit_normalizer=16.0 if case["raw_gates"] else 0.0)
    if case["entry"] == "causal":
        o, _ = vig_b200.fused_chunk_gla(q, k, v, gates[0])
    else:
        o = vig_b200.bi_gla(q, k, v, *gates, out_scale=0.5, gate_logit_normalizer=16.0 if case["raw_gates"] else 0.0)
    return (o.detach(), *torch.autograd.grad(o, state["inputs"], state["d_out"]))


# ---------------------------------------------------------------------------------------------------------------------
def _block(tokens, C, H, kd, inter):
    """(operations, weights) of one block on ``tokens`` tokens: conv, stacked projections, scan as a recurrence in both
    directions, output projection, gated MLP."""
    dk, dv = kd // H, C // H
    weights = 9 * C + C * (2 * kd + C) + C * C + C * 16 + 16 * 2 * kd + C * C + 3 * C * inter
    scan = 2 * 4 * dk * dv * H
    return tokens * (2 * weights + scan), weights


def work(case):
    e = BYTES[case["dtype"]]
    if case["kind"] == "model":
        pixels = case["batch"] * case["height"] * case["width"]
        if case["preset"] == "hier":
            flops, weights = 2 * pixels // 4 * 27 * HIER_DIMS[0] // 2 + 2 * pixels // 16 * 9 * HIER_DIMS[0] ** 2 // 2, 0
            for i, (C, H, depth) in enumerate(zip(HIER_DIMS, HIER_HEADS, HIER_DEPTHS)):
                tokens = pixels // (16 * 4 ** i)
                f, w = _block(tokens, C, H, int(C * case["expand_k"]), 32 * ((int(C * 8 / 3) + 31) // 32))
                flops, weights = flops + depth * f, weights + depth * w
                if i:
                    flops, weights = flops + 2 * tokens * 9 * C * HIER_DIMS[i - 1], weights + 9 * C * HIER_DIMS[i - 1]
            C = HIER_DIMS[-1]
        else:
            C, H = WIDTH[case["preset"]], HEADS[case["preset"]]
            tokens = pixels // 256
            f, w = _block(tokens, C, H, int(C * case["expand_k"]), 256 * ((int(C * 8 / 3) + 255) // 256))
            flops = DEPTH * f + 2 * tokens * (4 * 243 * C // 2 + 9 * C * C // 2)
            weights = DEPTH * w + 243 * C // 2 + 9 * C * C // 2
        head = C * CLASSES
        return dict(bytes=e * (3 * pixels + weights + head + case["batch"] * CLASSES), flops=flops + 2 * case["batch"] * head)
    B, H, L, dk, dv = (case[n] for n in ("B", "H", "L", "dk", "dv"))
    rows, dirs = B * H * L, 1 if case["entry"] == "causal" else 2
    ins = (2 + dirs) * dk + dv
    fwd = rows * dirs * 4 * dk * dv                        # state update and read-out of the recurrence
    if case["kind"] == "op":
        states = 2 * 4 * B * H * dk * dv if case["entry"] == "causal" else 0
        return dict(bytes=e * rows * (ins + dv) + states, flops=fwd)
    # training: inputs and the output's gradient in, output and all gradients out; the backward recurrences rebuild S,
    # run its adjoint and read dq, dk, dv out of them
    return dict(bytes=e * rows * (2 * ins + 2 * dv), flops=fwd + rows * dirs * 10 * dk * dv)


def tolerance(case):
    # An operator's operands and results are rounded to the type (bf16 2^-9, fp16 2^-12) a few times on the way, sums are
    # fp32.  In a model every stored activation of every block is, and the LayerNorm'd stages of the hierarchical one
    # amplify it: measured against the same weights in fp32, 3e-3 .. 1.2e-2 (ViG, bf16), 5e-4 (ViG, fp16), 8e-3 (HierViG,
    # fp16); two implementations are apart by up to 1.5 times that.
    if case["kind"] == "model":
        return {"rel": 1.5e-2 if case["preset"] == "hier" else {"bf16": 2e-2, "f16": 2.5e-3}[case["dtype"]]}
    return {"rel": {"f32": 1e-5, "bf16": 1e-2, "f16": 2e-3}[case["dtype"]]}
