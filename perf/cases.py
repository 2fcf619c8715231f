"""The work that a user of this package has it do, as timed cases.

Every kind below is one public entry point (a module, an operator, a launch group or the decoder), taken over the range
of sizes that its callers use: single tokens and full prompts, odd token counts, the widths of the shapes that the
package's own benchmark and tests name, each activation type, and the forward as well as the training direction.

`exact` gives the same results in 64 bits.  The int8 quantization of activations and the ternarization of weights are
part of the operation's definition (in the arithmetic of the input type), so they are carried out as defined, and all
that follows from them in 64 bits.
"""
from __future__ import annotations

import importlib
import math
from dataclasses import replace

import torch

from __graft_entry__ import load_package

wf = load_package()
DEV = "cuda"
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
EPS = 1e-5

# (N, K) of the projections: a 2B-like model, the 8B shape, a 135M-like model
SHAPES = [(2560, 2560), (6912, 2560), (2560, 6912), (4096, 4096), (14336, 4096), (4096, 14336), (576, 576), (1536, 576), (576, 1536)]


def listed():
    return [
        # one sequence, one token: a single projection in inference, the call that latency and launches decide
        dict(name="layer_m1", kind="layer", m=1, n=2560, k=2560, dtype="bf16", bias=False),
        # a prompt of odd length through a down projection in half precision
        dict(name="layer_m1237", kind="layer", m=1237, n=2560, k=6912, dtype="f16", bias=False),
        # a long prompt, or a batch of them, through an up projection
        dict(name="layer_m8192", kind="layer", m=8192, n=6912, k=2560, dtype="bf16", bias=False),
        # the serving plug-in on checkpoint bytes in the I2_S layout: a handful of sequences, float32 results
        dict(name="plugin_m7", kind="plugin", m=7, n=4096, k=4096, dtype="bf16", bias=True),
        # independent layers decoded with one token each, as one launch: the stream of packed weights
        dict(name="group_m1", kind="group", layers=60, m=1, n=6912, k=2560, dtype="bf16"),
        # stacks of layers with a batch of sequences each
        dict(name="stack_m16", kind="stack", layers=120, m=16, n=2560, k=2560, dtype="bf16"),
        dict(name="stack_m61", kind="stack", layers=30, m=61, n=2560, k=6912, dtype="bf16"),
        # training: the optimizer has just written the weights; forward and backward of one projection
        dict(name="train_m4096", kind="train", m=4096, n=6912, k=2560, dtype="bf16", bias=False),
        dict(name="train_m777", kind="train", m=777, n=1536, k=576, dtype="f32", bias=True),
        # conversion of a checkpoint: one large matrix to packed weights
        dict(name="pack", kind="pack", n=14336, k=4096, wtype="f32", mode="f32"),
        # attention of one new token per sequence over the cache
        dict(name="attention_b32", kind="attention", b=32, t=2048, pos=2031, nq=32, nkv=8, d=128),
        # a whole call of the small decoder: a prompt, then single tokens
        dict(name="decoder_135m", kind="decoder", layers=8, b=1, s=121, steps=12),
    ]


def _spread(rng, lo, hi):
    """A whole number of lo..hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "plugin", "group", "stack", "stack", "train", "train", "pack", "attention", "decoder"])
    n, k = rng.choice(SHAPES)
    if kind == "layer":
        if rng.random() < 0.3:
            n = n - rng.randrange(1, 130)  # widths that no tile divides
        most = max(1, 8192 * 6912 * 2560 // (n * k))
        return dict(kind=kind, m=_spread(rng, 1, min(8192, most)), n=n, k=k, dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), bias=rng.random() < 0.3)
    if kind == "plugin":
        n, k = rng.choice([s for s in SHAPES if s[1] % 128 == 0])
        return dict(kind=kind, m=_spread(rng, 1, 512), n=n, k=k, dtype=rng.choice(["bf16", "f16", "f32"]), bias=rng.random() < 0.5)
    if kind == "group":
        n, k = rng.choice(SHAPES[:5])
        return dict(kind=kind, layers=rng.randrange(2, max(3, min(120, 60 * 6912 * 2560 // (n * k)))), m=rng.randrange(1, 5), n=n, k=k,
                    dtype=rng.choice(["bf16", "bf16", "f16"]))
    if kind == "stack":
        n, k = rng.choice(SHAPES[:5])
        return dict(kind=kind, layers=rng.randrange(2, max(3, min(120, 60 * 6912 * 2560 // (n * k)))), m=_spread(rng, 8, 100), n=n, k=k, dtype="bf16")
    if kind == "train":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        n, k = rng.choice(SHAPES[:4] if dtype == "bf16" else SHAPES[6:])
        return dict(kind=kind, m=_spread(rng, 128, 4096), n=n, k=k, dtype=dtype, bias=rng.random() < 0.3)
    if kind == "pack":
        return dict(kind=kind, n=n, k=k, wtype=rng.choice(["f32", "f32", "bf16"]), mode=rng.choice(["f32", "bf16", "f16"]))
    if kind == "attention":
        nq, nkv, d = rng.choice([(32, 8, 128), (32, 8, 128), (9, 3, 64)])
        t = rng.randrange(256, 4096)
        return dict(kind=kind, b=_spread(rng, 1, min(64, 32 * 2048 // t)), t=t, pos=rng.randrange(t // 4, t), nq=nq, nkv=nkv, d=d)
    return dict(kind="decoder", layers=rng.randrange(1, 9), b=rng.randrange(1, 8), s=rng.randrange(5, 121), steps=rng.randrange(1, 13))


# ---------------------------------------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _activations(g, *shape):
    """Hidden states: normal, one in a thousand an outlier."""
    x = torch.randn(*shape, generator=g, device=DEV)
    far = torch.rand(*shape, generator=g, device=DEV) < 1e-3
    return torch.where(far, 20.0 * x.sign(), x)


def _weights(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV) * 0.02


def _model(case):
    """The decoder's configuration."""
    return replace(_decoder_module().SMOLLM2_135M, layers=case["layers"])


def _decoder_module():
    return importlib.import_module(wf.__name__ + ".decoder")


def _model_weights(case, seed):
    cfg, g, out = _model(case), _gen(seed), {}
    q, kv = cfg.n_q * cfg.head_dim, cfg.n_kv * cfg.head_dim
    sizes = {"self_attn.q_proj": (q, cfg.hidden), "self_attn.k_proj": (kv, cfg.hidden), "self_attn.v_proj": (kv, cfg.hidden),
             "self_attn.o_proj": (cfg.hidden, q), "mlp.gate_proj": (cfg.intermediate, cfg.hidden),
             "mlp.up_proj": (cfg.intermediate, cfg.hidden), "mlp.down_proj": (cfg.hidden, cfg.intermediate)}
    for i in range(cfg.layers):
        for name, size in sizes.items():
            out[f"transformer.layers.{i}.{name}.weight"] = _weights(g, *size)
    out["embed_tokens.weight"] = _weights(g, cfg.vocab, cfg.hidden)
    out["lm_head.weight"] = _weights(g, cfg.vocab, cfg.hidden)
    ids = torch.randint(0, cfg.vocab, (case["b"], case["s"] + case["steps"]), generator=g, device=DEV)
    return out, ids


def _tensors(case, seed):
    """The inputs of every kind but the decoder, from the seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind in ("layer", "plugin", "train"):
        dt = TYPES[case["dtype"]]
        t = dict(w=_weights(g, case["n"], case["k"]), x=_activations(g, case["m"], case["k"]).to(dt), b=None)
        if case["bias"]:
            t["b"] = _weights(g, case["n"])
        if kind == "train":
            t["dy"] = (_weights(g, case["m"], case["n"])).to(dt)
        return t
    if kind in ("group", "stack"):
        return dict(w=[_weights(g, case["n"], case["k"]) for _ in range(case["layers"])],
                    x=_activations(g, case["layers"], case["m"], case["k"]).to(TYPES[case["dtype"]]))
    if kind == "pack":
        return dict(w=_weights(g, case["n"], case["k"]).to(TYPES[case["wtype"]]))
    assert kind == "attention"
    b, t, nq, nkv, d = (case[v] for v in ("b", "t", "nq", "nkv", "d"))
    kc, vc = (torch.randn(b, nkv, t, d, generator=g, device=DEV).bfloat16() for _ in range(2))
    return dict(q=torch.randn(b, nq * d, generator=g, device=DEV).bfloat16(), kc=kc, vc=vc)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "decoder":
        weights, ids = _model_weights(case, seed)
        dec = _decoder_module().TernaryDecoder(_model(case), case["b"], case["s"] + case["steps"], torch.device(DEV), weights=weights)
        dec.capture()
        return dict(kind=kind, dec=dec, prompt=ids[:, :case["s"]].contiguous(), rest=ids[:, case["s"]:].contiguous())
    t = _tensors(case, seed)
    if kind in ("layer", "train"):
        layer = wf.BitLinear(case["k"], case["n"], bias=case["bias"], eps=EPS).to(DEV)
        with torch.no_grad():
            layer.weight.copy_(t["w"])
            if case["bias"]:
                layer.bias.copy_(t["b"])
        if kind == "layer":
            layer.packed_weight(t["x"].dtype)  # a model in inference packs its weights when it is loaded
            return dict(kind=kind, layer=layer, x=t["x"])
        return dict(kind=kind, layer=layer, x=t["x"].requires_grad_(True), dy=t["dy"], w=t["w"])
    if kind == "plugin":
        codes, scale = wf.pack_ternary(t["w"])
        method, layer = wf.BitNetLinearMethod(), torch.nn.Module()
        method.create_weights(layer, case["k"], [case["n"]], case["k"], case["n"], t["x"].dtype)
        layer.to(DEV)
        layer.qweight.data.copy_(wf.repack(codes, 0, case["n"], case["k"], 1))  # layout 1: I2_S
        layer.scale.data.copy_(scale[:1])
        method.process_weights_after_loading(layer)
        return dict(kind=kind, method=method, layer=layer, x=t["x"], b=t["b"])
    if kind == "group":
        problems = []
        for w, x in zip(t["w"], t["x"]):
            codes, scale = wf.pack_ternary(w, mode=x.dtype)
            problems.append(dict(x=x, codes=codes, w_scale=scale))
        return dict(kind=kind, group=wf.DecodeGroup(problems))
    if kind == "stack":
        packed = [wf.pack_ternary(w, mode=t["x"].dtype) for w in t["w"]]
        return dict(kind=kind, x=t["x"], codes=torch.stack([c for c, _ in packed]), scales=torch.stack([s for _, s in packed]))
    if kind == "pack":
        return dict(kind=kind, w=t["w"], mode=TYPES[case["mode"]])
    return dict(kind=kind, out=torch.empty_like(t["q"]), pos=torch.tensor(case["pos"], dtype=torch.long, device=DEV), **t)


# ---------------------------------------------------------------------------------------------- one pass


def run(state):
    kind = state["kind"]
    if kind == "layer":
        with torch.no_grad():
            return state["layer"](state["x"])
    if kind == "plugin":
        with torch.no_grad():
            return state["method"].apply(state["layer"], state["x"], state["b"])
    if kind == "group":
        return list(state["group"].run())
    if kind == "stack":
        return wf.bitlinear_batched(state["x"], state["codes"], state["scales"])
    if kind == "train":
        layer = state["layer"]
        with torch.no_grad():
            layer.weight.copy_(state["w"])  # the optimizer's write: new weights are ternarized and packed in this step
        y = layer(state["x"])
        wanted = [state["x"], layer.weight] + ([layer.bias] if layer.bias is not None else [])
        return [y.detach(), *torch.autograd.grad(y, wanted, state["dy"])]
    if kind == "pack":
        return list(wf.pack_ternary(state["w"], mode=state["mode"], eps=EPS))
    if kind == "attention":
        return wf.ops.attn_decode(state["q"], state["kc"], state["vc"], state["pos"], state["out"])
    dec, out = state["dec"], []
    out.append(dec.prefill(state["prompt"]))
    for i in range(state["rest"].shape[1]):  # the continuation is given, so every step scores the same tokens
        dec.tok.copy_(state["rest"][:, i])
        dec.decode(1)
        out.append(dec.logits.clone())
    return torch.stack(out, 1)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without


def work(case):
    kind = case["kind"]
    if kind == "decoder":
        cfg = _model(case)
        q, kv = cfg.n_q * cfg.head_dim, cfg.n_kv * cfg.head_dim
        layer = cfg.hidden * (2 * q + 2 * kv + 3 * cfg.intermediate)
        head, b, s, steps = cfg.vocab * cfg.hidden, case["b"], case["s"], case["steps"]
        cache = 4 * kv * cfg.layers * b  # bytes of one position
        bytes_ = (1 + steps) * (cfg.layers * layer // 4 + 2 * head + 2 * b * cfg.vocab) + cache * (2 * s + sum(s + i + 1 for i in range(steps)))
        flops = 2 * b * ((s + steps) * cfg.layers * layer + (1 + steps) * head) + 2 * b * cfg.layers * q * (s * s + 2 * steps * s)
        return dict(bytes=bytes_, flops=flops)
    if kind == "attention":
        b, t, nq, nkv, d = case["b"], case["pos"] + 1, case["nq"], case["nkv"], case["d"]
        return dict(bytes=4 * b * nkv * t * d + 4 * b * nq * d, flops=4 * b * nq * t * d)
    if kind == "pack":
        nk = case["n"] * case["k"]
        return dict(bytes=nk * (4 if case["wtype"] == "f32" else 2) + nk // 4 + 8, flops=2 * nk)
    m, n, k, size = case["m"], case["n"], case["k"], 4 if case["dtype"] == "f32" else 2
    if kind == "train":
        return dict(bytes=3 * n * k * 4 + 2 * size * m * (k + n), flops=6 * m * n * k)
    layers = case.get("layers", 1)
    return dict(bytes=layers * (n * k // 4 + 4 + size * m * k + (4 if kind == "plugin" else size) * m * n), flops=2 * layers * m * n * k)


def tolerance(case):
    kind = case["kind"]
    if kind == "pack":
        return "exact"  # bytes and two scales of a sum that is rounded once
    if kind == "decoder":
        return dict(rel=0.03, max=0.3)  # a change of rounding flips int8 codes of every later layer
    if kind == "attention":
        return dict(rel=8e-3, max=0.1)  # bf16 results and probabilities (measured against 64 bits: 2.1e-3)
    if kind == "train":
        # gradients: sums of thousands of products in another order (measured against 64 bits: 2.3e-3 in bf16, 6e-7 in f32)
        return dict(rel=8e-3, max=0.1) if case["dtype"] == "bf16" else dict(rel=2.5e-6, max=5e-5)
    # whole-number products and one rescale in 32 bits: what remains is where the result rounds (measured against 64 bits
    # rounded once: 1.2e-5 in bf16, 6e-8 in f32)
    return dict(rel={"bf16": 5e-5, "f16": 2e-5, "f32": 3e-7}["f32" if kind == "plugin" else case["dtype"]], max=0.05)


# ---------------------------------------------------------------------------------------------- the same in 64 bits


def _quantize(x):
    """Per-token absmax int8 in the arithmetic of x's type: (codes, multipliers), in 64 bits."""
    scale = x.abs().amax(-1, keepdim=True).clamp(min=EPS).reciprocal() * 127.0
    return (x * scale).round().clamp(-128, 127).double(), scale.double()


def _ternary(w, mode):
    """(codes, dequantization multiplier, quantization multiplier); the first two in 64 bits."""
    mean = w.to(mode).abs().double().mean().float()
    if mode == torch.float32:
        mean = mean.clamp(min=EPS)
        return (w.float() / mean).round().clamp(-1, 1).double(), mean.double(), mean
    mul = mean.to(mode).clamp(min=EPS).reciprocal()
    return (w.to(mode) * mul).round().clamp(-1, 1).double(), mul.reciprocal().double(), mul.float()


def _bitlinear(x, w, mode, bias=None):
    q, s = _quantize(x)
    c, dq, _ = _ternary(w, mode)
    y = (q @ c.t()) / s * dq
    return y if bias is None else y + bias.double()


def _exact_decoder(case, seed):
    weights, ids = _model_weights(case, seed)
    cfg, b, t, d = _model(case), case["b"], case["s"] + case["steps"], _model(case).head_dim
    inv = cfg.rope_theta ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
    ang = torch.arange(t, device=DEV, dtype=torch.float64)[:, None] * inv
    cos, sin = ang.cos(), ang.sin()
    bar = torch.full((t, t), float("-inf"), device=DEV, dtype=torch.float64).triu(1)

    def norm(v):
        return v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + cfg.eps)

    def project(v, name):
        return _bitlinear(v, weights.pop(name), torch.float32)

    def heads(v, rotate):
        v = v.view(b, t, -1, d).transpose(1, 2)
        if rotate:
            v0, v1 = v[..., 0::2], v[..., 1::2]
            v = torch.stack([v0 * cos - v1 * sin, v1 * cos + v0 * sin], -1).flatten(-2)
        return v

    h = weights.pop("embed_tokens.weight").bfloat16()[ids].double()
    for i in range(cfg.layers):
        pre = f"transformer.layers.{i}."
        v = norm(h)
        q = heads(project(v, pre + "self_attn.q_proj.weight"), True)
        key, val = (heads(project(v, pre + f"self_attn.{n}_proj.weight"), n == "k").repeat_interleave(cfg.n_q // cfg.n_kv, 1) for n in "kv")
        a = torch.softmax(q @ key.transpose(-1, -2) / math.sqrt(d) + bar, -1) @ val
        h = h + project(a.transpose(1, 2).reshape(b, t, -1), pre + "self_attn.o_proj.weight")
        v = norm(h)
        gate, up = (project(v, pre + f"mlp.{n}_proj.weight") for n in ("gate", "up"))
        h = h + project(torch.nn.functional.silu(gate) * up, pre + "mlp.down_proj.weight")
    return norm(h[:, case["s"] - 1:]) @ weights.pop("lm_head.weight").bfloat16().double().t()


def exact(case, seed):
    kind = case["kind"]
    if kind == "decoder":
        return _exact_decoder(case, seed)
    t = _tensors(case, seed)
    if kind == "layer":
        return _bitlinear(t["x"], t["w"], t["x"].dtype, t["b"])
    if kind == "plugin":
        return _bitlinear(t["x"], t["w"], torch.float32, t["b"])
    if kind == "group":
        return [_bitlinear(x, w, x.dtype) for x, w in zip(t["x"], t["w"])]
    if kind == "stack":
        return torch.stack([_bitlinear(x, w, x.dtype) for x, w in zip(t["x"], t["w"])])
    if kind == "train":
        q, s = _quantize(t["x"])
        c, dq, _ = _ternary(t["w"], t["x"].dtype)
        dy = t["dy"].double()
        y = (q @ c.t()) / s * dq
        out = [y if t["b"] is None else y + t["b"].double(), (dy @ c) * dq, dy.t() @ (q / s)]
        return out + ([dy.sum(0)] if t["b"] is not None else [])
    if kind == "pack":
        _, dq, mul = _ternary(t["w"], TYPES[case["mode"]])
        return [None, torch.stack([dq, mul.double()])]
    b, n, nq, nkv, d = case["b"], case["pos"] + 1, case["nq"], case["nkv"], case["d"]
    q = t["q"].double().view(b, nkv, nq // nkv, d)
    p = torch.softmax(q @ t["kc"][:, :, :n].double().transpose(-1, -2) / math.sqrt(d), -1)
    return (p @ t["vc"][:, :, :n].double()).reshape(b, nq * d)
