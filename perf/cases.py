"""Timed workloads of the framework: what training, scoring and sampling spend their time in, through the public
entry points, at the shapes of the repository's own model presets (``moe-30b-a3b`` and ``dense-9b``).

A case is a dict with a ``kind`` and its sizes:

  model_decode   one sampling step of a whole dense decoder over its key/value cache: logits of every sequence
  attn_decode    one attention block in a sampling step with long, ragged caches (a rollout batch)
  moe_decode     router and routed experts for the few tokens of a sampling step
  mlp_decode     the dense feed-forward block for the few tokens of a sampling step
  attn_prefill   causal attention of packed prompts, forward only
  attn_train     q/k norm, rotary embedding and attention of a packed training row, forward and backward
  moe_train      router and routed experts of a training row, forward and backward
  ffn_train      residual add, RMSNorm and dense SwiGLU block, forward and backward
  head_loss      output head fused with the cross-entropy, loss and both gradients
  logprobs       token log-probabilities and entropies of a scored row (the scoring pass of RL)
  adamw          one optimizer step over a layer's parameters, with a clip coefficient
"""

from __future__ import annotations

import math

import numpy as np
import torch

from halo_b200.inference.generate import KVCache
from halo_b200.models.config import ModelConfig
from halo_b200.models.qwen3 import Attention, DenseMLP, ForwardContext, build_model
from halo_b200.ops import attention as attn_ops
from halo_b200.ops import gemm
from halo_b200.ops import moe as moe_ops
from halo_b200.ops.cross_entropy import fused_linear_cross_entropy, linear_logprobs
from halo_b200.ops.norm import add_rms_norm, rms_norm
from halo_b200.ops.rope import rope_table
from halo_b200.optim.adamw_bf16 import AdamWBF16

DEV = "cuda"
D = 128                      # head dimension of both presets
EPS = 1e-6
THETA = 1e6
VOCAB = 151936
EXPERTS, TOP_K, EXPERT_WIDTH, MOE_HIDDEN = 128, 8, 768, 2048


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # a few interactive generations: one step of a 4-layer slice of the 9B model, latency and launches count
        {"name": "model_decode_b4", "kind": "model_decode", "batch": 4, "cache": 700},
        # a rollout batch of 64 sequences, each several thousand tokens long, in one layer's attention
        {"name": "attn_decode_b64", "kind": "attn_decode", "batch": 64, "cache": 8000},
        # the same step's experts for 32 sequences: most experts see one or two rows
        {"name": "moe_decode_t32", "kind": "moe_decode", "tokens": 32},
        # the 9B feed-forward block for 16 sequences: bound by reading the weights
        {"name": "mlp_decode_t16", "kind": "mlp_decode", "tokens": 16, "hidden": 4096, "width": 12288},
        # packed prompts of 256 .. 16,384 tokens, odd total
        {"name": "attn_prefill_24k", "kind": "attn_prefill", "tokens": 24531, "kv_heads": 4, "doc_max": 16384, "window": 0},
        # the benchmark's row: 65,536 tokens of chat documents
        {"name": "attn_train_64k", "kind": "attn_train", "tokens": 65536, "kv_heads": 4, "doc_max": 4579, "window": 0},
        # a small ragged micro-batch through the experts
        {"name": "moe_train_3k", "kind": "moe_train", "tokens": 3001},
        # the benchmark's row through the experts
        {"name": "moe_train_64k", "kind": "moe_train", "tokens": 65536},
        # a row of the dense preset through its feed-forward half
        {"name": "ffn_train_8k", "kind": "ffn_train", "tokens": 8192, "hidden": 4096, "width": 12288},
        # the loss of 8,192 tokens over the whole vocabulary
        {"name": "head_loss_8k", "kind": "head_loss", "tokens": 8192, "hidden": 2048},
        # scoring one rollout of odd length
        {"name": "logprobs_2k", "kind": "logprobs", "tokens": 2047, "hidden": 2048},
        # the optimizer step of one dense layer
        {"name": "adamw_layer", "kind": "adamw", "hidden": 4096, "width": 12288},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model_decode", "attn_decode", "moe_decode", "mlp_decode", "attn_prefill", "attn_train", "moe_train",
                       "ffn_train", "head_loss", "logprobs", "adamw"])
    if kind == "model_decode":
        return {"kind": kind, "batch": rng.randint(1, 8), "cache": _log_int(rng, 128, 2048)}
    if kind == "attn_decode":
        return {"kind": kind, "batch": _log_int(rng, 2, 64), "cache": _log_int(rng, 500, 8000)}
    if kind == "moe_decode":
        return {"kind": kind, "tokens": _log_int(rng, 1, 300)}
    if kind == "mlp_decode":
        hidden, width = rng.choice([(4096, 12288), (2048, 6144)])
        return {"kind": kind, "tokens": _log_int(rng, 1, 300), "hidden": hidden, "width": width}
    if kind == "attn_prefill":
        return {"kind": kind, "tokens": _log_int(rng, 700, 24000), "kv_heads": rng.choice([4, 8]),
                "doc_max": _log_int(rng, 600, 16384), "window": rng.choice([0, 0, 1024])}
    if kind == "attn_train":
        return {"kind": kind, "tokens": _log_int(rng, 1500, 60000), "kv_heads": rng.choice([4, 8]), "doc_max": 4579,
                "window": rng.choice([0, 0, 1024])}
    if kind == "moe_train":
        return {"kind": kind, "tokens": _log_int(rng, 800, 60000)}
    if kind == "ffn_train":
        hidden, width = rng.choice([(4096, 12288), (2048, 6144)])
        return {"kind": kind, "tokens": _log_int(rng, 500, 8190), "hidden": hidden, "width": width}
    if kind == "head_loss":
        return {"kind": kind, "tokens": _log_int(rng, 500, 8190), "hidden": 2048}
    if kind == "logprobs":
        return {"kind": kind, "tokens": _log_int(rng, 200, 8190), "hidden": 2048}
    return {"kind": kind, "hidden": rng.choice([1024, 2048, 3072]), "width": rng.randint(1000, 12000)}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62))


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    out = torch.empty(*shape, device=DEV, dtype=dtype)
    return out.normal_(0.0, std, generator=g)


def _norm_weight(g, n):
    return (1.0 + 0.1 * torch.randn(n, device=DEV, generator=g)).to(torch.bfloat16)


def _doc_lengths(total, lo, hi, seed, chat):
    """Lengths of packed documents that fill ``total`` tokens: chat rows are log-normal around 990 tokens."""
    rng = np.random.default_rng(int(seed))
    out, left = [], total
    while left > 0:
        n = rng.lognormal(6.90, 0.6) if chat else math.exp(rng.uniform(math.log(lo), math.log(hi)))
        n = max(1, min(int(np.clip(n, lo, hi)), left))
        out.append(n)
        left -= n
    return out


def _attention_inputs(case, seed):
    T, hkv = case["tokens"], case["kv_heads"]
    chat = case["kind"] == "attn_train"
    lens = _doc_lengths(T, 64 if chat else min(256, case["doc_max"]), case["doc_max"], seed, chat)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    g = _gen(seed)
    qkv = _normal(g, T, (32 + 2 * hkv) * D)
    return cu, g, qkv


def _routing_logits(g, T):
    # experts are not equally popular: a per-expert offset beside the per-token scores
    offset = 0.5 * torch.randn(EXPERTS, device=DEV, generator=g)
    return torch.randn(T, EXPERTS, device=DEV, generator=g) + offset


def _decode_lengths(case, seed):
    rng = np.random.default_rng(int(seed) + 17)
    top = case["cache"]
    return torch.from_numpy(rng.integers(max(1, top // 4), top + 1, size=case["batch"])).to(DEV)


def _filled_cache(g, layers, case, hkv, lengths):
    cache = KVCache(layers, case["batch"], case["cache"] + 64, hkv, D, torch.bfloat16, torch.device(DEV))
    cache.k.normal_(0.0, 1.0, generator=g)
    cache.v.normal_(0.0, 1.0, generator=g)
    cache.lengths.copy_(lengths)
    return cache


def _moe_config():
    return ModelConfig(hidden_size=2048, num_hidden_layers=1, num_attention_heads=32, num_key_value_heads=4, head_dim=D,
                       intermediate_size=6144, moe_intermediate_size=EXPERT_WIDTH, num_experts=EXPERTS,
                       num_experts_per_tok=TOP_K)


def _dense_config(layers):
    return ModelConfig(hidden_size=4096, num_hidden_layers=layers, num_attention_heads=32, num_key_value_heads=8, head_dim=D,
                       intermediate_size=12288, num_experts=0, model_type="qwen3")


MODEL_LAYERS = 4


def _adamw_shapes(case):
    h, f = case["hidden"], case["width"]
    return {"self_attn.qkv_proj": (6144, h), "self_attn.o_proj": (h, 4096), "mlp.gate_up_proj": (2 * f, h), "mlp.down_proj": (h, f),
            "input_layernorm": (h,), "post_attention_layernorm": (h,)}


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind == "model_decode":
        model = build_model(_dense_config(MODEL_LAYERS), device=DEV, seed=int(seed) % 1000003).requires_grad_(False)
        lengths = _decode_lengths(case, seed)
        tokens = torch.randint(0, VOCAB, (case["batch"],), device=DEV, generator=g)
        return {"kind": kind, "model": model, "cache": _filled_cache(g, MODEL_LAYERS, case, 8, lengths), "tokens": tokens}
    if kind == "attn_decode":
        cfg = _moe_config()
        attn = Attention(cfg, torch.bfloat16, DEV).requires_grad_(False)
        for p in (attn.qkv_proj, attn.o_proj):
            p.normal_(0.0, 0.02, generator=g)
        attn.q_norm.copy_(_norm_weight(g, D))
        attn.k_norm.copy_(_norm_weight(g, D))
        lengths = _decode_lengths(case, seed)
        return {"kind": kind, "attn": attn, "x": _normal(g, case["batch"], cfg.hidden_size),
                "cache": _filled_cache(g, 1, case, 4, lengths)}
    if kind in ("moe_decode", "moe_train"):
        T, train = case["tokens"], kind == "moe_train"
        x = _normal(g, T, MOE_HIDDEN).requires_grad_(train)
        logits = _routing_logits(g, T).requires_grad_(train)
        w_gu = _normal(g, EXPERTS, 2 * EXPERT_WIDTH, MOE_HIDDEN, std=0.02).requires_grad_(train)
        w_dn = _normal(g, EXPERTS, MOE_HIDDEN, EXPERT_WIDTH, std=0.02).requires_grad_(train)
        return {"kind": kind, "x": x, "logits": logits, "w_gu": w_gu, "w_dn": w_dn, "dy": _normal(g, T, MOE_HIDDEN) if train else None,
                "transport": moe_ops.LocalTransport()}
    if kind in ("mlp_decode", "ffn_train"):
        T, H, train = case["tokens"], case["hidden"], kind == "ffn_train"
        mlp = DenseMLP(H, case["width"], torch.bfloat16, DEV).requires_grad_(False)
        mlp.gate_up_proj.normal_(0.0, 0.02, generator=g)
        mlp.down_proj.normal_(0.0, 0.02, generator=g)
        state = {"kind": kind, "mlp": mlp.requires_grad_(train), "x": _normal(g, T, H).requires_grad_(train)}
        if train:
            state["residual"] = _normal(g, T, H).requires_grad_(True)
            state["norm"] = _norm_weight(g, H).requires_grad_(True)
            state["dy"] = _normal(g, T, H)
            state["dr"] = _normal(g, T, H)
        return state
    if kind in ("attn_prefill", "attn_train"):
        cu, g, qkv = _attention_inputs(case, seed)
        plan = attn_ops.build_plan(cu, device=DEV, window=case["window"])
        pos = torch.from_numpy(np.concatenate([np.arange(n) for n in np.diff(cu)])).to(DEV)
        wq, wk = _norm_weight(g, D), _norm_weight(g, D)
        train = kind == "attn_train"
        return {"kind": kind, "qkv": qkv.requires_grad_(train), "wq": wq.requires_grad_(train), "wk": wk.requires_grad_(train),
                "table": rope_table(pos, D, THETA), "plan": plan, "hkv": case["kv_heads"],
                "do": _normal(g, case["tokens"], 32 * D) if train else None}
    if kind in ("head_loss", "logprobs"):
        T, H, train = case["tokens"], case["hidden"], kind == "head_loss"
        hidden = _normal(g, T, H).requires_grad_(train)
        weight = _normal(g, VOCAB, H, std=0.02).requires_grad_(train)
        labels = torch.randint(0, VOCAB, (T,), device=DEV, generator=g)
        labels[torch.rand(T, device=DEV, generator=g) < 0.1] = -100        # prompt tokens are not scored
        return {"kind": kind, "hidden": hidden, "weight": weight, "labels": labels}
    if kind == "adamw":
        params = []
        for name, shape in _adamw_shapes(case).items():
            p = torch.nn.Parameter(_normal(g, *shape, std=0.02))
            p.grad = _normal(g, *shape, std=1e-3)
            params.append((name, p))
        opt = AdamWBF16(params, lr=1e-4, weight_decay=0.01)
        opt.step()                                                         # a run in progress: the moments are filled
        return {"kind": kind, "opt": opt, "params": [p for _, p in params], "scale": torch.full((1,), 0.7, device=DEV)}
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "model_decode":
        m, cache = state["model"], state["cache"]
        with torch.no_grad():
            cache.begin_decode()
            ctx = ForwardContext(None, m.rope(cache.lengths), m.transport)
            ctx.positions = cache.lengths
            ctx.kv_cache = cache
            trunk = m.trunk_states(state["tokens"], ctx)
            h = rms_norm(trunk, m.norm, m.cfg.rms_norm_eps)
            logits = gemm.matmul(h, m.head_weight(), out_dtype=torch.float32)
        return {"trunk": trunk, "logits": logits}
    if kind == "attn_decode":
        cache, attn = state["cache"], state["attn"]
        with torch.no_grad():
            cache.begin_decode()
            ctx = ForwardContext(None, rope_table(cache.lengths, D, THETA), None)
            ctx.positions = cache.lengths
            ctx.kv_cache = cache
            return attn(state["x"], ctx)
    if kind == "moe_decode":
        with torch.no_grad():
            idx, w = moe_ops.router_topk(state["logits"], TOP_K, True)
            out = moe_ops.moe_experts(state["x"], idx, w, state["w_gu"], state["w_dn"], state["transport"])
        return {"out": out, "idx": idx, "w": w}
    if kind == "moe_train":
        idx, w = moe_ops.router_topk(state["logits"], TOP_K, True)
        out = moe_ops.moe_experts(state["x"], idx, w, state["w_gu"], state["w_dn"], state["transport"])
        dx, dlogits, dgu, ddn = torch.autograd.grad(out, [state["x"], state["logits"], state["w_gu"], state["w_dn"]], state["dy"])
        return {"out": out.detach(), "idx": idx, "dx": dx, "dlogits": dlogits, "dgu": dgu, "ddn": ddn}
    if kind == "mlp_decode":
        with torch.no_grad():
            return state["mlp"](state["x"])
    if kind == "ffn_train":
        mlp = state["mlp"]
        h, res = add_rms_norm(state["x"], state["residual"], state["norm"], EPS)
        y = mlp(h)
        grads = torch.autograd.grad([y, res], [state["x"], state["norm"], mlp.gate_up_proj, mlp.down_proj], [state["dy"], state["dr"]])
        return {"y": y.detach(), "res": res.detach(), "dx": grads[0], "dnorm": grads[1], "dgu": grads[2], "ddn": grads[3]}
    if kind == "attn_prefill":
        with torch.no_grad():
            return attn_ops.rope_attention(state["qkv"], state["wq"], state["wk"], state["table"], state["plan"], 32, state["hkv"], EPS)
    if kind == "attn_train":
        o = attn_ops.rope_attention(state["qkv"], state["wq"], state["wk"], state["table"], state["plan"], 32, state["hkv"], EPS)
        dqkv, dwq, dwk = torch.autograd.grad(o, [state["qkv"], state["wq"], state["wk"]], state["do"])
        return {"o": o.detach(), "dqkv": dqkv, "dwq": dwq, "dwk": dwk}
    if kind == "head_loss":
        loss = fused_linear_cross_entropy(state["hidden"], state["weight"], state["labels"])
        dh, dw = torch.autograd.grad(loss, [state["hidden"], state["weight"]])
        return {"loss": loss.detach(), "dh": dh, "dw": dw}
    if kind == "logprobs":
        with torch.no_grad():
            logp, ent = linear_logprobs(state["hidden"], state["weight"], state["labels"], want_entropy=True)
        return {"logp": logp, "entropy": ent}
    if kind == "adamw":
        opt = state["opt"]
        opt.defer_grad_scale(state["scale"])
        opt.step()
        return [t for p in state["params"] for t in (p.detach(), opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"])]
    raise ValueError(kind)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _visible_pairs(lens, window):
    """Query-key pairs of causal documents under a window (0: none)."""
    total = 0
    for n in lens:
        w = min(window, n) if window else n
        total += w * (w + 1) // 2 + (n - w) * w
    return total


def work(case):
    kind = case["kind"]
    if kind == "model_decode":
        B, cfg = case["batch"], _dense_config(MODEL_LAYERS)
        H, F = cfg.hidden_size, cfg.intermediate_size
        weights = MODEL_LAYERS * (6144 * H + H * 4096 + 3 * H * F) + VOCAB * H
        keys = MODEL_LAYERS * B * int(0.625 * case["cache"]) * 2 * 8 * D
        return {"bytes": 2.0 * (weights + keys + B * H) + 4.0 * B * VOCAB, "flops": 2.0 * B * weights}
    if kind == "attn_decode":
        B, H = case["batch"], 2048
        keys = B * int(0.625 * case["cache"])
        weights = 5120 * H + H * 4096
        return {"bytes": 2.0 * (weights + keys * 2 * 4 * D + 2 * B * H), "flops": 2.0 * B * weights + 4.0 * keys * 32 * D}
    if kind in ("moe_decode", "moe_train"):
        T, H, F = case["tokens"], MOE_HIDDEN, EXPERT_WIDTH
        products = 2.0 * T * TOP_K * 3 * H * F
        touched = EXPERTS * (1.0 - (1.0 - TOP_K / EXPERTS) ** T)
        weights = touched * 3 * H * F
        if kind == "moe_decode":
            return {"bytes": 2.0 * (weights + 2 * T * H) + 4.0 * T * (EXPERTS + 2 * TOP_K), "flops": products}
        return {"bytes": 2.0 * (3 * weights + 6 * T * H) + 8.0 * T * EXPERTS, "flops": 3 * products}
    if kind in ("mlp_decode", "ffn_train"):
        T, H, F = case["tokens"], case["hidden"], case["width"]
        if kind == "mlp_decode":
            return {"bytes": 2.0 * (3 * H * F + 2 * T * H), "flops": 6.0 * T * H * F}
        return {"bytes": 2.0 * (3 * 3 * H * F + 7 * T * H), "flops": 18.0 * T * H * F}
    if kind in ("attn_prefill", "attn_train"):
        T, hkv, chat = case["tokens"], case["kv_heads"], kind == "attn_train"
        lens = _doc_lengths(T, 64 if chat else min(256, case["doc_max"]), case["doc_max"], 1, chat)
        forward = 4.0 * D * 32 * _visible_pairs(lens, case["window"])
        if kind == "attn_prefill":
            return {"bytes": 2.0 * T * D * (2 * 32 + 2 * hkv), "flops": forward}
        return {"bytes": 2.0 * T * D * (4 * 32 + 4 * hkv), "flops": 3.5 * forward}
    if kind in ("head_loss", "logprobs"):
        T, H = case["tokens"], case["hidden"]
        if kind == "logprobs":
            return {"bytes": 2.0 * (VOCAB * H + T * H) + 16.0 * T, "flops": 2.0 * T * VOCAB * H}
        return {"bytes": 2.0 * (2 * VOCAB * H + 2 * T * H), "flops": 6.0 * T * VOCAB * H}
    n = sum(math.prod(s) for s in _adamw_shapes(case).values())
    return {"bytes": 14.0 * n, "flops": 20.0 * n}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        return "exact"
    # bf16 operands and results with fp32 sums; four times the error of the present path against 64 bits
    rel = {"model_decode": 0.03, "attn_decode": 0.018, "moe_decode": 0.016, "mlp_decode": 0.014, "attn_prefill": 0.018,
           "attn_train": 0.026, "moe_train": 0.016, "ffn_train": 0.022, "head_loss": 0.007, "logprobs": 0.0005}[kind]
    return {"rel": rel, "max": 0.5, "differ": 0.001}


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------
def _f(t):
    return t.detach().double()


def _rms(x, w):
    return _f(w) * (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS))


def _angles(pos):
    inv = THETA ** (-torch.arange(0, D // 2, device=DEV, dtype=torch.float32) * 2.0 / D)
    a = pos.to(DEV).float()[:, None] * inv
    return a.cos().bfloat16().double(), a.sin().bfloat16().double()


def _rotate(x, cos, sin):
    """x [T, heads, D]; cos / sin [T, D/2]."""
    a, b = x[..., : D // 2], x[..., D // 2:]
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _causal(q, k, v, window):
    """q [h, n, D], k / v [h, n, D] of one document."""
    n = q.shape[1]
    i = torch.arange(n, device=DEV)
    hidden = i[None, :] > i[:, None]
    if window:
        hidden = hidden | (i[None, :] <= i[:, None] - window)
    s = (q @ k.transpose(1, 2)) * D ** -0.5
    return torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ v


def _exact_attention(case, seed):
    T, hkv = case["tokens"], case["kv_heads"]
    cu, g, qkv = _attention_inputs(case, seed)
    wq, wk = _norm_weight(g, D), _norm_weight(g, D)
    train = case["kind"] == "attn_train"
    pos = torch.from_numpy(np.concatenate([np.arange(n) for n in np.diff(cu)]))
    cos, sin = _angles(pos)
    do = _f(_normal(g, T, 32 * D)) if train else None
    wqd, wkd = _f(wq).requires_grad_(train), _f(wk).requires_grad_(train)
    out = torch.empty(T, 32 * D, device=DEV, dtype=torch.float64)
    dqkv = torch.empty_like(qkv, dtype=torch.float64) if train else None
    rep = 32 // hkv
    for a, b in zip(cu[:-1], cu[1:]):
        n = int(b - a)
        x = _f(qkv[a:b]).requires_grad_(train)
        h = x.view(n, 32 + 2 * hkv, D)
        with torch.set_grad_enabled(train):
            q = _rotate(_norm_heads(h[:, :32], wqd), cos[a:b], sin[a:b]).transpose(0, 1)
            k = _rotate(_norm_heads(h[:, 32:32 + hkv], wkd), cos[a:b], sin[a:b]).transpose(0, 1)
            v = h[:, 32 + hkv:].transpose(0, 1)
            # the heads in groups small enough for the scores of a long document
            step = max(1, min(rep, int(6e8 // (n * n)) or 1))
            parts = []
            for i in range(0, 32, step):
                kv = i // rep
                parts.append(_causal(q[i:i + step], k[kv:kv + 1], v[kv:kv + 1], case["window"]))
            o = torch.cat(parts, 0).transpose(0, 1).reshape(n, 32 * D)
            if train:
                o.backward(do[a:b])
                dqkv[a:b] = x.grad
        out[a:b] = o.detach()
    if not train:
        return out
    return {"o": out, "dqkv": dqkv, "dwq": wqd.grad, "dwk": wkd.grad}


def _norm_heads(x, w):
    return w * (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS))


def _decode_step(x, attn, k_cache, v_cache, lengths, hkv):
    """One query per sequence against its cached keys and its own, in 64 bits."""
    B = x.shape[0]
    qkv = (x @ _f(attn.qkv_proj).t()).view(B, 32 + 2 * hkv, D)
    cos, sin = _angles(lengths)
    q = _rotate(_norm_heads(qkv[:, :32], _f(attn.q_norm)), cos, sin)
    k = _rotate(_norm_heads(qkv[:, 32:32 + hkv], _f(attn.k_norm)), cos, sin)
    v = qkv[:, 32 + hkv:]
    rep, outs = 32 // hkv, []
    for b in range(B):
        n = int(lengths[b])
        keys = torch.cat([_f(k_cache[b, :n]), k[b:b + 1]], 0).repeat_interleave(rep, 1)
        vals = torch.cat([_f(v_cache[b, :n]), v[b:b + 1]], 0).repeat_interleave(rep, 1)
        p = torch.softmax(torch.einsum("hd,shd->hs", q[b], keys) * D ** -0.5, -1)
        outs.append(torch.einsum("hs,shd->hd", p, vals).reshape(-1))
    return torch.stack(outs) @ _f(attn.o_proj).t()


def _swiglu(pre):
    f = pre.shape[-1] // 2
    return torch.nn.functional.silu(pre[..., :f]) * pre[..., f:]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("attn_prefill", "attn_train"):
        return _exact_attention(case, seed)
    if kind == "adamw":
        return None                        # a rounding that depends on the step's own noise: compared bit by bit
    state = prepare(case, seed)
    if kind == "model_decode":
        m, cache = state["model"], state["cache"]
        x = _f(m.embed_tokens)[state["tokens"]]
        for i, layer in enumerate(m.layers):
            x = x + _decode_step(_rms(x, layer.input_layernorm), layer.self_attn, cache.k[i], cache.v[i], cache.lengths, 8)
            h = _rms(x, layer.post_attention_layernorm)
            x = x + _swiglu(h @ _f(layer.mlp.gate_up_proj).t()) @ _f(layer.mlp.down_proj).t()
        return {"trunk": x, "logits": _rms(x, m.norm) @ _f(m.lm_head).t()}
    if kind == "attn_decode":
        cache = state["cache"]
        return _decode_step(_f(state["x"]), state["attn"], cache.k[0], cache.v[0], cache.lengths, 4)
    if kind == "mlp_decode":
        mlp = state["mlp"]
        return _swiglu(_f(state["x"]) @ _f(mlp.gate_up_proj).t()) @ _f(mlp.down_proj).t()
    if kind == "ffn_train":
        mlp = state["mlp"]
        x, w, gu, dn = (_f(t).requires_grad_(True) for t in (state["x"], state["norm"], mlp.gate_up_proj, mlp.down_proj))
        res = x + _f(state["residual"])
        h = w * (res * torch.rsqrt(res.pow(2).mean(-1, keepdim=True) + EPS))
        y = _swiglu(h @ gu.t()) @ dn.t()
        dx, dw, dgu, ddn = torch.autograd.grad([y, res], [x, w, gu, dn], [_f(state["dy"]), _f(state["dr"])])
        return {"y": y.detach(), "res": res.detach(), "dx": dx, "dnorm": dw, "dgu": dgu, "ddn": ddn}
    if kind in ("moe_decode", "moe_train"):
        train = kind == "moe_train"
        x = _f(state["x"])
        logits = _f(state["logits"]).requires_grad_(train)
        with torch.set_grad_enabled(train):
            probs = torch.softmax(logits, -1)
            idx = torch.topk(logits.detach(), TOP_K, -1).indices
            w = probs.gather(-1, idx)
            w = w / w.sum(-1, keepdim=True)
        out, dx = torch.zeros_like(x), torch.zeros_like(x)
        dw = torch.zeros_like(w)
        dgu = torch.zeros(state["w_gu"].shape, device=DEV, dtype=torch.float64) if train else None
        ddn = torch.zeros(state["w_dn"].shape, device=DEV, dtype=torch.float64) if train else None
        for e in range(EXPERTS):
            tok, slot = torch.where(idx == e)
            if not tok.numel():
                continue
            xe, we = x[tok].requires_grad_(train), w.detach()[tok, slot][:, None].requires_grad_(train)
            gu, dn = _f(state["w_gu"][e]).requires_grad_(train), _f(state["w_dn"][e]).requires_grad_(train)
            with torch.set_grad_enabled(train):
                y = we * (_swiglu(xe @ gu.t()) @ dn.t())
            out.index_add_(0, tok, y.detach())
            if train:
                gx, gw, dgu[e], ddn[e] = torch.autograd.grad(y, [xe, we, gu, dn], _f(state["dy"])[tok])
                dx.index_add_(0, tok, gx)
                dw[tok, slot] = gw[:, 0]
        if not train:
            return {"out": out, "idx": None, "w": w}
        return {"out": out, "idx": None, "dx": dx, "dlogits": torch.autograd.grad(w, logits, dw)[0], "dgu": dgu, "ddn": ddn}
    # the output head, in row chunks
    hidden, weight, labels = _f(state["hidden"]), _f(state["weight"]), state["labels"]
    scored = labels != -100
    count = scored.sum().clamp_min(1)
    loss, logps, ents = torch.zeros((), device=DEV, dtype=torch.float64), [], []
    dh, dw = torch.empty_like(hidden), torch.zeros_like(weight) if kind == "head_loss" else None
    for a in range(0, hidden.shape[0], 2048):
        lab, ok = labels[a:a + 2048].clamp_min(0)[:, None], scored[a:a + 2048]
        logp = torch.log_softmax(hidden[a:a + 2048] @ weight.t(), -1)
        picked = torch.where(ok, logp.gather(-1, lab)[:, 0], 0.0)
        if kind == "logprobs":
            logps.append(picked)
            ents.append(-(logp.exp() * logp).sum(-1))
            continue
        loss -= picked.sum()
        d = logp.exp_()
        d.scatter_add_(1, lab, torch.full_like(lab, -1.0, dtype=torch.float64))
        d *= (ok.double() / count)[:, None]
        dh[a:a + 2048] = d @ weight
        dw += d.t() @ hidden[a:a + 2048]
    if kind == "logprobs":
        return {"logp": torch.cat(logps), "entropy": torch.cat(ents)}
    return {"loss": loss / count, "dh": dh, "dw": dw}
