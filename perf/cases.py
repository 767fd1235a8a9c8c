"""The work that training runs of this framework spend their time on, through the entry points that models and trainers call.

Nine kinds of case, each a forward and backward pass (or an optimizer update) on one GPU in bf16:

  mlp        `models.common.GatedMLP`: three projections and the gated activation, tokens from a handful to a full sequence
  attention  `ops.attention`: packed causal documents, grouped heads, head sizes 64, 128 and 256
  norm       `ops.rms_norm` / `ops.add_rms_norm` over the residual stream
  layer      `models.qwen3.Qwen3DecoderLayer`: a dense decoder block over packed documents
  head       `ops.linear_cross_entropy_sum`: vocabulary projection and loss in chunks
  moe        `models.moe.MoE`: router, dispatch, grouped experts, combine
  gdn        `models.qwen3_5.GatedDeltaNet`: the linear-attention mixer of the Qwen3.5 family
  adamw      `ops.sq_norm` and `ops.adamw_step_` on one flat shard: gradient norm, clipping, update
  model      `models.qwen3.Qwen3ForCausalLM`: logits, loss and every gradient of a small dense model
"""
import math

import torch

DEV = "cuda"
BF16 = torch.bfloat16
EPS = 1e-6
IGNORE = -100


def listed():
    return [
        # the smallest call: the MLP of the 512-wide smoke configuration on a short validation batch, where launches count
        {"name": "mlp_small", "kind": "mlp", "tokens": 200, "hidden": 512, "inter": 1536},
        # the MLP of Qwen3-8B at its training length: most of that model's arithmetic
        {"name": "mlp_8b", "kind": "mlp", "tokens": 8192, "hidden": 4096, "inter": 12288},
        # Qwen3-8B's attention on one document that fills the sequence
        {"name": "attention_8k", "kind": "attention", "tokens": 8192, "docs": 1, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # packed documents of unequal, odd lengths with the head layout of Qwen3-30B-A3B
        {"name": "attention_packed", "kind": "attention", "tokens": 6007, "docs": 9, "heads": 32, "kv_heads": 4, "head_dim": 128},
        # the wide heads of Qwen3.5's full-attention layers
        {"name": "attention_wide", "kind": "attention", "tokens": 4096, "docs": 2, "heads": 16, "kv_heads": 4, "head_dim": 256},
        # residual addition and norm of Qwen3-8B, twice per layer
        {"name": "norm_8b", "kind": "norm", "tokens": 8192, "hidden": 4096, "residual": True},
        # one Qwen3-8B block on a ragged packed batch: every op of a dense layer in its place
        {"name": "layer_8b_ragged", "kind": "layer", "tokens": 3001, "docs": 3, "hidden": 4096, "inter": 12288, "heads": 32, "kv_heads": 8,
         "head_dim": 128},
        # vocabulary head and loss of Qwen3-8B on half a sequence, in two chunks
        {"name": "head_8b", "kind": "head", "tokens": 4096, "hidden": 4096, "vocab": 151936, "chunks": 2},
        # the sparse block of Qwen3-30B-A3B at its training length
        {"name": "moe_30b", "kind": "moe", "tokens": 4096, "hidden": 2048, "experts": 128, "top_k": 8, "inter": 768},
        # a gated delta-net mixer of the Qwen3.5 recipe among the examples
        {"name": "gdn_2k", "kind": "gdn", "tokens": 2048, "docs": 1, "hidden": 2048, "heads": 32, "key_heads": 16, "head_dim": 128},
        # the update of one Qwen3-8B block's parameters on a single shard rank
        {"name": "adamw_block", "kind": "adamw", "numel": 192946432, "grad": "bf16"},
        # a whole small model (the smoke configuration): many short launches one after another
        {"name": "model_small", "kind": "model", "tokens": 1024, "docs": 2, "layers": 2, "hidden": 512, "inter": 1536, "heads": 4, "kv_heads": 2,
         "head_dim": 128, "vocab": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "attention", "attention", "norm", "layer", "head", "moe", "gdn", "adamw", "model"])
    if kind == "mlp":
        hidden = 64 * _log(rng, 4, 64)
        return {"kind": kind, "tokens": _log(rng, 16, 8192), "hidden": hidden, "inter": min(12288, 8 * _log(rng, hidden // 4, hidden // 2))}
    if kind == "attention":
        hd = rng.choice([64, 128, 128, 256])
        kv = rng.choice([2, 4, 8] if hd < 256 else [2, 4])
        group = rng.choice([1, 2, 4, 8] if kv < 8 else [1, 2, 4])
        return {"kind": kind, "tokens": _log(rng, 128, 8192 if hd < 256 else 4096), "docs": rng.choice([1, 1, 2, 5, 11]),
                "heads": min(32 if hd < 256 else 16, kv * group), "kv_heads": kv, "head_dim": hd}
    if kind == "norm":
        return {"kind": kind, "tokens": _log(rng, 64, 16384), "hidden": 8 * _log(rng, 16, 640), "residual": rng.random() < 0.7}
    if kind == "layer":
        kv = rng.choice([2, 4, 8])
        hd = rng.choice([64, 128])
        hidden = 128 * _log(rng, 4, 32)
        return {"kind": kind, "tokens": _log(rng, 200, 4096), "docs": rng.choice([1, 2, 4, 7]), "hidden": hidden, "inter": 3 * hidden,
                "heads": kv * rng.choice([2, 4]), "kv_heads": kv, "head_dim": hd}
    if kind == "head":
        return {"kind": kind, "tokens": _log(rng, 200, 4096), "hidden": 256 * _log(rng, 2, 16), "vocab": 8 * _log(rng, 500, 18992),
                "chunks": rng.choice([1, 2, 4])}
    if kind == "moe":
        experts = rng.choice([8, 16, 64, 128])
        return {"kind": kind, "tokens": _log(rng, 128, 4096), "hidden": 256 * rng.randint(2, 8), "experts": experts,
                "top_k": rng.choice([2, 4, 8] if experts > 8 else [2, 4]), "inter": 64 * rng.randint(4, 12)}
    if kind == "gdn":
        heads = rng.choice([8, 16, 32])
        return {"kind": kind, "tokens": _log(rng, 256, 2048), "docs": rng.choice([1, 2, 3]), "hidden": 256 * rng.randint(2, 8), "heads": heads,
                "key_heads": heads // rng.choice([1, 2]), "head_dim": rng.choice([64, 128])}
    if kind == "adamw":
        return {"kind": kind, "numel": _log(rng, 100000, 150000000), "grad": rng.choice(["bf16", "fp32"])}
    kv = rng.choice([1, 2, 4])
    return {"kind": kind, "tokens": _log(rng, 100, 2048), "docs": rng.choice([1, 2, 4]), "layers": rng.choice([1, 2, 3]),
            "hidden": 128 * rng.randint(2, 8), "inter": 256 * rng.randint(2, 10), "heads": kv * 2, "kv_heads": kv,
            "head_dim": rng.choice([64, 128]), "vocab": 8 * _log(rng, 250, 4000)}


# ------------------------------------------------------------------------------------------------------------ inputs
class _Make:
    """Tensors of one seed, in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=BF16, grad=False):
        t = torch.empty(*shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=self.g).to(dtype)
        return t.requires_grad_(grad)

    def near_one(self, n, grad=False):
        return (1.0 + 0.1 * torch.randn(n, generator=self.g, device=DEV)).to(BF16).requires_grad_(grad)

    def integers(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device=DEV)


def _cuts(tokens, docs):
    """Cumulative document cuts of unequal lengths: the same for every seed, so that passes of one case do the same work."""
    weights = [1.0 + (0.73 * i * i) % 2.1 for i in range(docs)]
    total, cuts, acc = sum(weights), [0], 0.0
    for w in weights[:-1]:
        acc += w
        cuts.append(max(cuts[-1] + 1, int(tokens * acc / total)))
    return cuts + [tokens]


def _rope(tokens_in_docs, head_dim, theta=1e6):
    pos = torch.cat([torch.arange(b - a, device=DEV) for a, b in zip(tokens_in_docs[:-1], tokens_in_docs[1:])])
    inv = 1.0 / theta ** (torch.arange(0, head_dim, 2, dtype=torch.float32, device=DEV) / head_dim)
    ang = pos.float()[:, None] * inv[None, :]
    return pos, ang.cos(), ang.sin()


def _layer_weights(m, c, grad=False):
    D, F, d = c["hidden"], c["inter"], c["head_dim"]
    q, kv = c["heads"] * d, c["kv_heads"] * d
    return {"input_layernorm.weight": m.near_one(D), "self_attn.q_proj.weight": m.normal(q, D, std=0.02),
            "self_attn.k_proj.weight": m.normal(kv, D, std=0.02), "self_attn.v_proj.weight": m.normal(kv, D, std=0.02),
            "self_attn.o_proj.weight": m.normal(D, q, std=0.02), "self_attn.q_norm.weight": m.near_one(d),
            "self_attn.k_norm.weight": m.near_one(d), "post_attention_layernorm.weight": m.near_one(D),
            "mlp.gate_proj.weight": m.normal(F, D, std=0.02), "mlp.up_proj.weight": m.normal(F, D, std=0.02),
            "mlp.down_proj.weight": m.normal(D, F, std=0.02)}


def _qwen3_config(c):
    from torchllmtuner_b200.models.qwen3 import Qwen3Config
    return Qwen3Config(vocab_size=c.get("vocab", 128), hidden_size=c["hidden"], intermediate_size=c["inter"],
                       num_hidden_layers=c.get("layers", 1), num_attention_heads=c["heads"], num_key_value_heads=c["kv_heads"],
                       head_dim=c["head_dim"], rms_norm_eps=EPS)


def _load(module, weights):
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(weights[name])
    return module


def _inputs(c, seed):
    """Plain tensors of a case: what `prepare` wraps and what `exact` computes from."""
    m, kind = _Make(seed), c["kind"]
    if kind == "mlp":
        T, D, F = c["tokens"], c["hidden"], c["inter"]
        return {"x": m.normal(T, D), "dy": m.normal(T, D),
                "w": {"gate_proj.weight": m.normal(F, D, std=0.02), "up_proj.weight": m.normal(F, D, std=0.02),
                      "down_proj.weight": m.normal(D, F, std=0.02)}}
    if kind == "attention":
        T, H, K, d = c["tokens"], c["heads"], c["kv_heads"], c["head_dim"]
        return {"q": m.normal(T, H, d), "k": m.normal(T, K, d), "v": m.normal(T, K, d), "do": m.normal(T, H, d)}
    if kind == "norm":
        T, D = c["tokens"], c["hidden"]
        return {"x": m.normal(T, D), "res": m.normal(T, D, std=2.0), "w": m.near_one(D), "dy": m.normal(T, D), "ds": m.normal(T, D)}
    if kind == "layer":
        T, D = c["tokens"], c["hidden"]
        return {"x": m.normal(T, D), "dy": m.normal(T, D), "w": _layer_weights(m, c)}
    if kind == "head":
        T, D, V = c["tokens"], c["hidden"], c["vocab"]
        y = m.integers(0, V, T)
        y[::17] = IGNORE                        # padding and prompt tokens carry no loss
        return {"h": m.normal(T, D), "w": m.normal(V, D, std=0.02), "y": y}
    if kind == "moe":
        T, D, E, F = c["tokens"], c["hidden"], c["experts"], c["inter"]
        return {"x": m.normal(T, D), "dy": m.normal(T, D),
                "w": {"router.gate.weight": m.normal(E, D, std=0.02), "routed.experts.w1_EFD": m.normal(E, F, D, std=0.02),
                      "routed.experts.w3_EFD": m.normal(E, F, D, std=0.02), "routed.experts.w2_EDF": m.normal(E, D, F, std=0.02)}}
    if kind == "gdn":
        T, D, H, K, d = c["tokens"], c["hidden"], c["heads"], c["key_heads"], c["head_dim"]
        C = 2 * K * d + H * d
        u = torch.rand(H, generator=m.g, device=DEV)
        return {"x": m.normal(T, D), "dy": m.normal(T, D),
                "w": {"in_proj_qkv.weight": m.normal(C, D, std=0.02), "in_proj_z.weight": m.normal(H * d, D, std=0.02),
                      "in_proj_b.weight": m.normal(H, D, std=0.02), "in_proj_a.weight": m.normal(H, D, std=0.02),
                      "conv1d.weight": m.normal(C, 1, 4, std=0.3), "dt_bias": torch.ones(H, device=DEV), "A_log": (0.01 + 15.99 * u).log(),
                      "norm.weight": m.near_one(d), "out_proj.weight": m.normal(D, H * d, std=0.02)}}
    if kind == "adamw":
        n = c["numel"]
        gdt = BF16 if c["grad"] == "bf16" else torch.float32
        p = m.normal(n, std=0.02, dtype=torch.float32)
        return {"p": p, "p16": p.to(BF16), "g": m.normal(n, std=1e-3, dtype=gdt), "m": m.normal(n, std=1e-3, dtype=torch.float32),
                "v": m.normal(n, std=1e-3, dtype=torch.float32).square_()}
    T, D, V = c["tokens"], c["hidden"], c["vocab"]
    w = {"model.embed_tokens.weight": m.normal(V, D, std=0.5), "model.norm.weight": m.near_one(D), "lm_head.weight": m.normal(V, D, std=0.02)}
    for i in range(c["layers"]):
        w.update({f"model.layers.{i}.{k}": t for k, t in _layer_weights(m, c).items()})
    y = m.integers(0, V, T)
    y[::17] = IGNORE
    return {"tokens": m.integers(0, V, T), "y": y, "w": w}


def prepare(case, seed):
    from torchllmtuner_b200.ops import AttnMeta
    c, kind = case, case["kind"]
    s = _inputs(c, seed)
    s["case"] = c
    if kind == "mlp":
        from torchllmtuner_b200.models.common import GatedMLP
        s["module"] = _load(GatedMLP(c["hidden"], c["inter"], dtype=BF16, device=DEV), s.pop("w"))
    elif kind == "attention":
        s["meta"] = AttnMeta.build(_cuts(c["tokens"], c["docs"]), causal=True, device=DEV)
        for k in "qkv":
            s[k].requires_grad_()
    elif kind == "norm":
        for k in ("x", "res", "w"):
            s[k].requires_grad_()
    elif kind == "layer":
        from torchllmtuner_b200.models.qwen3 import ForwardContext, Qwen3DecoderLayer
        s["module"] = _load(Qwen3DecoderLayer(_qwen3_config(c), 0, dtype=BF16, device=DEV), s.pop("w"))
        cuts = _cuts(c["tokens"], c["docs"])
        _, cos, sin = _rope(cuts, c["head_dim"])
        s["ctx"] = ForwardContext(cos, sin, AttnMeta.build(cuts, causal=True, device=DEV))
    elif kind == "head":
        s["h"].requires_grad_()
        s["w"].requires_grad_()
    elif kind == "moe":
        from torchllmtuner_b200.models.moe import MoE
        s["module"] = _load(MoE(c["hidden"], c["experts"], c["top_k"], c["inter"], dtype=BF16, device=DEV), s.pop("w"))
    elif kind == "gdn":
        from torchllmtuner_b200.models.qwen3_5 import GatedDeltaNet, Qwen35Config, Qwen35Context
        cfg = Qwen35Config(hidden_size=c["hidden"], linear_num_value_heads=c["heads"], linear_num_key_heads=c["key_heads"],
                           linear_key_head_dim=c["head_dim"], linear_value_head_dim=c["head_dim"], rms_norm_eps=EPS)
        s["module"] = _load(GatedDeltaNet(cfg, dtype=BF16, device=DEV), s.pop("w"))
        cuts = _cuts(c["tokens"], c["docs"])
        pos, cos, sin = _rope(cuts, 64)
        s["ctx"] = Qwen35Context(cos, sin, AttnMeta.build(cuts, causal=True, device=DEV), positions=pos)
    elif kind == "model":
        from torchllmtuner_b200.models.qwen3 import Qwen3ForCausalLM
        s["module"] = _load(Qwen3ForCausalLM(_qwen3_config(c), dtype=BF16, device=DEV), s.pop("w"))
        cuts = _cuts(c["tokens"], c["docs"])
        s["positions"], s["meta"] = _rope(cuts, c["head_dim"])[0], AttnMeta.build(cuts, causal=True, device=DEV)
    if "x" in s and kind != "norm":
        s["x"].requires_grad_()
    return s


def _module_pass(s, y, extra):
    params = dict(s["module"].named_parameters())
    grads = torch.autograd.grad(y, [s["x"], *params.values()], s["dy"])
    return {"y": y.detach(), "x": grads[0], **dict(zip(params, grads[1:])), **extra}


def run(state):
    from torchllmtuner_b200 import ops
    s, kind = state, state["case"]["kind"]
    if kind == "mlp":
        return _module_pass(s, s["module"](s["x"]), {})
    if kind == "attention":
        o = ops.attention(s["q"], s["k"], s["v"], s["meta"])
        dq, dk, dv = torch.autograd.grad(o, [s["q"], s["k"], s["v"]], s["do"])
        return {"o": o.detach(), "q": dq, "k": dk, "v": dv}
    if kind == "norm":
        if s["case"]["residual"]:
            y, h = ops.add_rms_norm(s["x"], s["res"], s["w"], EPS)
            dx, dres, dw = torch.autograd.grad([y, h], [s["x"], s["res"], s["w"]], [s["dy"], s["ds"]])
            return {"y": y.detach(), "h": h.detach(), "x": dx, "res": dres, "w": dw}
        y = ops.rms_norm(s["x"], s["w"], EPS)
        dx, dw = torch.autograd.grad(y, [s["x"], s["w"]], s["dy"])
        return {"y": y.detach(), "x": dx, "w": dw}
    if kind in ("layer", "gdn"):
        return _module_pass(s, s["module"](s["x"], s["ctx"]), {})
    if kind == "head":
        loss = ops.linear_cross_entropy_sum(s["h"], s["w"], s["y"], s["case"]["chunks"])
        dh, dw = torch.autograd.grad(loss, [s["h"], s["w"]], torch.full_like(loss, 1.0 / s["case"]["tokens"]))
        return {"loss": loss.detach(), "h": dh, "w": dw}
    if kind == "moe":
        return _module_pass(s, s["module"](s["x"]), {"counts": s["module"].tokens_per_expert_E})
    if kind == "adamw":
        sq = ops.sq_norm([s["g"]])
        coef = (1.0 / (sq.sqrt() + 1e-6)).clamp(max=1.0).reshape(1)
        ops.adamw_step_(s["p"], s["g"], s["m"], s["v"], lr=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=100,
                        p_lowp=s["p16"], clip_coef=coef)
        return {"sq": sq, "p": s["p"], "p16": s["p16"], "m": s["m"], "v": s["v"]}
    model = s["module"]
    logits = model(s["tokens"], model.build_context(s["positions"], s["meta"]))
    loss = ops.cross_entropy_sum(logits, s["y"]) / s["case"]["tokens"]
    params = dict(model.named_parameters())
    grads = torch.autograd.grad(loss, list(params.values()))
    return {"logits": logits.detach(), "loss": loss.detach(), **dict(zip(params, grads))}


# ---------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(tokens, docs):
    """Visible (query, key) pairs of causal documents."""
    cuts = _cuts(tokens, docs)
    return sum((b - a) * (b - a + 1) / 2 for a, b in zip(cuts[:-1], cuts[1:]))


def _layer_work(c):
    T, D, F, d = c["tokens"], c["hidden"], c["inter"], c["head_dim"]
    weights = D * d * (2 * c["heads"] + 2 * c["kv_heads"]) + 3 * D * F
    return weights, 6 * T * weights + 14 * _pairs(T, c["docs"]) * c["heads"] * d


def work(case):
    c, kind = case, case["kind"]
    T, D = c.get("tokens"), c.get("hidden")
    if kind == "mlp":
        W = 3 * D * c["inter"]
        return {"bytes": 2 * (4 * T * D + 2 * W), "flops": 6 * T * W}
    if kind == "attention":
        return {"bytes": 4 * T * c["head_dim"] * (2 * c["heads"] + 2 * c["kv_heads"]),
                "flops": 14 * _pairs(T, c["docs"]) * c["heads"] * c["head_dim"]}
    if kind == "norm":
        return {"bytes": 2 * ((7 if c["residual"] else 4) * T * D + 2 * D), "flops": 12 * T * D}
    if kind == "layer":
        weights, flops = _layer_work(c)
        return {"bytes": 2 * (4 * T * D + 2 * weights), "flops": flops}
    if kind == "head":
        return {"bytes": 2 * (2 * T * D + 2 * D * c["vocab"]) + 8 * T, "flops": 6 * T * D * c["vocab"]}
    if kind == "moe":
        W = 3 * D * c["inter"]
        used = min(c["experts"], T * c["top_k"])
        return {"bytes": 2 * (4 * T * D + (used + c["experts"]) * W), "flops": 6 * T * (c["top_k"] * W + D * c["experts"])}
    if kind == "gdn":
        H, K, d = c["heads"], c["key_heads"], c["head_dim"]
        weights = D * (2 * K * d + 3 * H * d + 2 * H)
        return {"bytes": 2 * (4 * T * D + 2 * weights), "flops": 6 * T * weights + 3 * T * H * 8 * d * d}
    if kind == "adamw":
        return {"bytes": c["numel"] * (26 + (2 if c["grad"] == "bf16" else 4)), "flops": 15 * c["numel"]}
    weights, flops = _layer_work(c)
    V = c["vocab"]
    return {"bytes": 2 * (2 * c["layers"] * weights + 3 * V * D + T * V), "flops": c["layers"] * flops + 6 * T * V * D}


def tolerance(case):
    """About four times what the results are off from 64 bits (2-norm): 0.0036 mlp, 0.0030 attention, 0.0025 norm, 0.0082 layer,
    0.0027 head, 0.0088 moe (where a tie between two experts may also change a whole token), 0.011 gdn, 0.0073 model. The update is
    fp32 (1e-7) next to a bf16 copy whose last bit may differ where the fp32 value lies between two bf16 values."""
    return {"mlp": {"rel": 0.014}, "attention": {"rel": 0.012}, "norm": {"rel": 0.01}, "layer": {"rel": 0.03}, "head": {"rel": 0.011},
            "moe": {"rel": 0.03, "max": 0.99}, "gdn": {"rel": 0.03}, "adamw": {"rel": 1e-4}, "model": {"rel": 0.03}}[case["kind"]]


# -------------------------------------------------------------------------------------------------------- in 64 bits
def _d(t, grad=True):
    return t.detach().double().requires_grad_(grad and t.is_floating_point())


def _norm64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _attention64(q, k, v, cuts):
    """q [T, H, d], k / v [T, K, d] -> [T, H, d], causal inside each document."""
    g, scale, outs = q.shape[1] // k.shape[1], q.shape[-1] ** -0.5, []
    for a, b in zip(cuts[:-1], cuts[1:]):
        qi, ki, vi = (t[a:b].transpose(0, 1) for t in (q, k, v))
        ki, vi = ki.repeat_interleave(g, 0), vi.repeat_interleave(g, 0)
        hidden = torch.ones(b - a, b - a, dtype=torch.bool, device=q.device).triu(1)
        p = (qi @ ki.transpose(1, 2) * scale).masked_fill(hidden, float("-inf")).softmax(-1)
        outs.append((p @ vi).transpose(0, 1))
    return torch.cat(outs)


def _rotate64(x, cos, sin):
    a, b = x.chunk(2, -1)
    c, s = cos[:, None, :], sin[:, None, :]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _layer64(x, w, c, cuts, cos, sin, at=""):
    T, d = x.shape[0], c["head_dim"]
    h = _norm64(x, w[at + "input_layernorm.weight"])
    q, k, v = ((h @ w[f"{at}self_attn.{n}_proj.weight"].t()).view(T, -1, d) for n in "qkv")
    q, k = (_rotate64(_norm64(t, w[f"{at}self_attn.{n}_norm.weight"]), cos, sin) for n, t in (("q", q), ("k", k)))
    x = x + _attention64(q, k, v, cuts).reshape(T, -1) @ w[at + "self_attn.o_proj.weight"].t()
    h = _norm64(x, w[at + "post_attention_layernorm.weight"])
    return x + _mlp64(h, w, at + "mlp.")


def _mlp64(h, w, at=""):
    g, u = h @ w[at + "gate_proj.weight"].t(), h @ w[at + "up_proj.weight"].t()
    return (torch.nn.functional.silu(g) * u) @ w[at + "down_proj.weight"].t()


def _gdn64(x, w, c, cuts):
    """The gated delta rule token by token, all heads at once."""
    T, H, K, d = x.shape[0], c["heads"], c["key_heads"], c["head_dim"]
    F = torch.nn.functional
    mixed = x @ w["in_proj_qkv.weight"].t()
    taps, docs = w["conv1d.weight"][:, 0, :], []
    for a, b in zip(cuts[:-1], cuts[1:]):
        padded = F.pad(mixed[a:b], (0, 0, 3, 0))
        docs.append(F.silu(sum(padded[j:j + b - a] * taps[:, j] for j in range(4))))
    mixed = torch.cat(docs)
    q, k, v = mixed[:, :K * d].view(T, K, d), mixed[:, K * d:2 * K * d].view(T, K, d), mixed[:, 2 * K * d:].view(T, H, d)
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // K, 1), k.repeat_interleave(H // K, 1)
    beta = torch.sigmoid(x @ w["in_proj_b.weight"].t())
    decay = (-w["A_log"].exp() * F.softplus(x @ w["in_proj_a.weight"].t() + w["dt_bias"])).exp()
    outs = []
    qs, ks, vs, bs, ds = q.unbind(0), k.unbind(0), v.unbind(0), beta.unbind(0), decay.unbind(0)
    for a, b in zip(cuts[:-1], cuts[1:]):
        S = x.new_zeros(H, d, d)
        for t in range(a, b):
            S = S * ds[t][:, None, None]
            u = bs[t][:, None] * (vs[t] - torch.bmm(ks[t].unsqueeze(1), S).squeeze(1))
            S = torch.baddbmm(S, ks[t].unsqueeze(2), u.unsqueeze(1))
            outs.append(torch.bmm(qs[t].unsqueeze(1), S).squeeze(1))
    o = _norm64(torch.stack(outs), w["norm.weight"]) * F.silu((x @ w["in_proj_z.weight"].t()).view(T, H, d))
    return o.reshape(T, H * d) @ w["out_proj.weight"].t()


def _moe64(x, w, c):
    scores = (x @ w["router.gate.weight"].t()).softmax(-1)
    idx = scores.detach().topk(c["top_k"], -1).indices
    weight = scores.gather(-1, idx)
    weight = weight / weight.sum(-1, keepdim=True)
    parts, rows = [], []
    for e in range(c["experts"]):
        t, j = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            h = x[t]
            h = torch.nn.functional.silu(h @ w["routed.experts.w1_EFD"][e].t()) * (h @ w["routed.experts.w3_EFD"][e].t())
            parts.append((h @ w["routed.experts.w2_EDF"][e].t()) * weight[t, j, None])
            rows.append(t)
    counts = torch.bincount(idx.reshape(-1), minlength=c["experts"]).double()
    return torch.zeros_like(x).index_add(0, torch.cat(rows), torch.cat(parts)), counts


def exact(case, seed):
    c, kind = case, case["kind"]
    s = _inputs(c, seed)
    if kind == "adamw":
        sq = s["g"].double().square().sum()
        g = s["g"].double() * (1.0 / (sq.sqrt() + 1e-6)).clamp(max=1.0)
        m = s["m"].double().mul_(0.9).add_(g, alpha=0.1)
        v = s["v"].double().mul_(0.95).addcmul_(g, g, value=0.05)
        p = s["p"].double().mul_(1.0 - 3e-4 * 0.1)
        p -= 3e-4 * (m / (1.0 - 0.9 ** 100)) / ((v / (1.0 - 0.95 ** 100)).sqrt_() + 1e-8)
        return {"sq": sq, "p": p, "p16": p, "m": m, "v": v}
    if kind == "head":
        h, w, y = s["h"].double(), s["w"].double(), s["y"]
        loss, dh, dw = h.new_zeros(()), [], torch.zeros_like(w)
        for a in range(0, c["tokens"], 1024):
            z, yc = h[a:a + 1024] @ w.t(), y[a:a + 1024]
            live = (yc != IGNORE).nonzero().squeeze(1)
            lse = z.logsumexp(-1)
            loss = loss + (lse[live] - z[live, yc[live]]).sum()
            z = z.sub_(lse[:, None]).exp_()
            z[live, yc[live]] -= 1.0
            z[yc == IGNORE] = 0.0
            z /= c["tokens"]
            dh.append(z @ w)
            dw += z.t() @ h[a:a + 1024]
        return {"loss": loss, "h": torch.cat(dh), "w": dw}
    if kind == "attention":
        cuts, H, K = _cuts(c["tokens"], c["docs"]), c["heads"], c["kv_heads"]
        q, k, v, do = (s[n].double() for n in ("q", "k", "v", "do"))
        o, dq, dk, dv = torch.zeros_like(q), torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
        scale = c["head_dim"] ** -0.5
        for a, b in zip(cuts[:-1], cuts[1:]):
            hidden = torch.ones(b - a, b - a, dtype=torch.bool, device=DEV).triu(1)
            for h in range(H):
                r = h // (H // K)
                qi, ki, vi, di = q[a:b, h], k[a:b, r], v[a:b, r], do[a:b, h]
                p = (qi @ ki.t() * scale).masked_fill_(hidden, float("-inf")).softmax(-1)
                o[a:b, h] = p @ vi
                dv[a:b, r] += p.t() @ di
                ds = (di @ vi.t()).sub_((di * o[a:b, h]).sum(-1, keepdim=True)).mul_(p)
                dq[a:b, h] = ds @ ki * scale
                dk[a:b, r] += ds.t() @ qi * scale
        return {"o": o, "q": dq, "k": dk, "v": dv}
    if kind == "norm":
        x, res, w = _d(s["x"]), _d(s["res"]), _d(s["w"])
        if not c["residual"]:
            y = _norm64(x, w)
            dx, dw = torch.autograd.grad(y, [x, w], s["dy"].double())
            return {"y": y.detach(), "x": dx, "w": dw}
        h = x + res
        y = _norm64(h, w)
        dx, dres, dw = torch.autograd.grad([y, h], [x, res, w], [s["dy"].double(), s["ds"].double()])
        return {"y": y.detach(), "h": h.detach(), "x": dx, "res": dres, "w": dw}
    w = {n: _d(t) for n, t in s["w"].items()}
    cuts = _cuts(c["tokens"], c.get("docs", 1))
    if kind == "model":
        _, cos, sin = _rope(cuts, c["head_dim"])
        x = w["model.embed_tokens.weight"][s["tokens"]]
        for i in range(c["layers"]):
            x = _layer64(x, w, c, cuts, cos.double(), sin.double(), f"model.layers.{i}.")
        logits = _norm64(x, w["model.norm.weight"]) @ w["lm_head.weight"].t()
        loss = torch.nn.functional.cross_entropy(logits, s["y"], ignore_index=IGNORE, reduction="sum") / c["tokens"]
        grads = torch.autograd.grad(loss, list(w.values()))
        return {"logits": logits.detach(), "loss": loss.detach(), **dict(zip(w, grads))}
    x, extra = _d(s["x"]), {}
    if kind == "mlp":
        y = _mlp64(x, w)
    elif kind == "moe":
        y, extra["counts"] = _moe64(x, w, c)
    elif kind == "gdn":
        y = _gdn64(x, w, c, cuts)
    else:
        _, cos, sin = _rope(cuts, c["head_dim"])
        y = _layer64(x, w, c, cuts, cos.double(), sin.double())
    grads = torch.autograd.grad(y, [x, *w.values()], s["dy"].double())
    return {"y": y.detach(), "x": grads[0], **dict(zip(w, grads[1:])), **extra}
