"""What this framework is timed on: its layers, blocks and whole steps, each through the entry point a program calls.

Every case is one pass of one kind of work (``KINDS``) at one size:

``attention``   the attention core on a packed QKV projection, forward and backward
``attn_block``  norm, QKV projection, rotary embedding, attention and output projection, forward and backward
``mlp_block``   residual add, norm, both linears and the activation, forward and backward
``head``        final norm, vocabulary projection and token loss, forward and backward
``embedding``   token lookup and its scatter-add gradient
``moe``         token dispatch, experts and weighted combine, forward and backward
``optimizer``   global-norm clipping and AdamW over one unit's flat buffers
``train_step``  a whole training step of a small model: gradients, clipping and the update
``generate``    a cached forward of a small stack: one decode token per sequence, or a prompt (prefill)

The modules are the ones a model is assembled from, wrapped in the sharded-parameter manager that gives them their
flat parameters and fp32 gradient buffers.  Sizes are those of the configurations in ``config/model_zoo`` (named by
``model``) at the sequence lengths and batches of training and generation, ragged ones among them.
"""
from __future__ import annotations

import math
import os

os.environ.setdefault("HG_QUIET", "1")   # no plan print-out for every model that is built

import torch
import torch.nn as nn
from torch.utils.checkpoint import checkpoint

from hetu_galvatron_b200 import ops
from hetu_galvatron_b200.config.schema import GalvatronRuntimeArgs
from hetu_galvatron_b200.models import inference
from hetu_galvatron_b200.models.modules import (GalvatronAttention, GalvatronCausalLMHead, GalvatronDecoderLayer,
                                                GalvatronEmbedding, GalvatronFinalNorm, GalvatronMLP)
from hetu_galvatron_b200.models.moe import GalvatronMoEMLP
from hetu_galvatron_b200.models.spec import LayerCtx, ModelSpec
from hetu_galvatron_b200.parallel.zero import ShardedUnit
from hetu_galvatron_b200.runtime.engine import build_model
from hetu_galvatron_b200.runtime.optimizer import ShardedAdamW

DEV = "cuda"
LP = torch.bfloat16

# hidden, heads, kv heads, head dim, ffn, vocab, norm, eps, activation, position, rotary base, bias, qkv bias
MODELS = {
    "gpt2-small": (768, 12, 12, 64, 3072, 50304, "LayerNorm", 1e-5, "gelu", "learned_absolute", 10000.0, True, True),
    "gpt2-xl": (1600, 25, 25, 64, 6400, 50304, "LayerNorm", 1e-5, "gelu", "learned_absolute", 10000.0, True, True),
    "llama2-7b": (4096, 32, 32, 128, 11008, 32000, "RMSNorm", 1e-6, "swiglu", "rope", 10000.0, False, False),
    "llama2-13b": (5120, 40, 40, 128, 13824, 32000, "RMSNorm", 1e-5, "swiglu", "rope", 10000.0, False, False),
    "qwen2.5-7b": (3584, 28, 4, 128, 18944, 152064, "RMSNorm", 1e-6, "swiglu", "rope", 1000000.0, False, True),
    "mixtral-8x7b": (4096, 32, 8, 128, 14336, 32000, "RMSNorm", 1e-5, "swiglu", "rope", 1000000.0, False, False),
}
DENSE = ["gpt2-small", "gpt2-xl", "llama2-7b", "llama2-13b", "qwen2.5-7b"]


def listed():
    return [
        # the attention core of the benchmark's training step, at its micro-batch
        {"name": "attention_7b_4096", "kind": "attention", "model": "llama2-7b", "seq": 4096, "batch": 2},
        # head dim 64: every layer of a gpt2-xl run at its full context
        {"name": "attention_gpt2xl_1024", "kind": "attention", "model": "gpt2-xl", "seq": 1024, "batch": 8},
        # grouped-query attention with QKV biases on a sequence that fills no tile
        {"name": "attn_block_qwen_1531", "kind": "attn_block", "model": "qwen2.5-7b", "seq": 1531, "batch": 1},
        # the MLP half of the benchmark's layer, at its micro-batch: the bulk of a training step
        {"name": "mlp_7b_4096x2", "kind": "mlp_block", "model": "llama2-7b", "seq": 4096, "batch": 2},
        # LayerNorm, biases and GELU at ragged sizes
        {"name": "mlp_gpt2xl_999x3", "kind": "mlp_block", "model": "gpt2-xl", "seq": 999, "batch": 3},
        # logits and loss of one micro-batch
        {"name": "head_7b_4096", "kind": "head", "model": "llama2-7b", "seq": 4096, "batch": 1},
        # lookup and gradient of one micro-batch, token frequencies as skewed as those of text
        {"name": "embedding_7b_4096x2", "kind": "embedding", "model": "llama2-7b", "seq": 4096, "batch": 2},
        # eight experts, top-2: the largest layer of the zoo that one GPU trains
        {"name": "moe_8x7b_4096", "kind": "moe", "model": "mixtral-8x7b", "seq": 4096, "batch": 1},
        # the optimizer's share of one 202 M parameter layer
        {"name": "optimizer_7b_layer", "kind": "optimizer", "hidden": 4096, "ffn": 11008},
        # a small model's whole step: many short kernels, where launches and host work count
        {"name": "train_step_small", "kind": "train_step", "hidden": 512, "head_dim": 128, "layers": 2, "seq": 512,
         "batch": 2},
        # one decode step: latency, weight and cache bandwidth
        {"name": "decode_7b_4x1000", "kind": "generate", "model": "llama2-7b", "layers": 4, "past": 1000, "new": 1,
         "batch": 4},
        # the prompt of such a batch
        {"name": "prefill_gqa_2x777", "kind": "generate", "model": "qwen2.5-7b", "layers": 2, "past": 0, "new": 777,
         "batch": 2},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["attention", "attn_block", "mlp_block", "head", "embedding", "moe", "optimizer", "train_step",
                       "generate", "generate"])
    if kind == "optimizer":
        hidden = 64 * _log_int(rng, 4, 60)
        return {"kind": kind, "hidden": hidden, "ffn": 8 * _log_int(rng, hidden // 8, 3 * hidden // 8)}
    if kind == "train_step":
        hd = rng.choice([64, 128])
        return {"kind": kind, "hidden": hd * rng.randint(4, 8), "head_dim": hd, "layers": rng.randint(1, 3),
                "seq": _log_int(rng, 64, 512), "batch": rng.randint(1, 4)}
    if kind == "generate":
        model = rng.choice(["llama2-7b", "qwen2.5-7b", "mixtral-8x7b"])
        batch = _log_int(rng, 1, 32)
        if rng.random() < 0.7:
            return {"kind": kind, "model": model, "layers": rng.randint(1, 2), "past": _log_int(rng, 16, 2000),
                    "new": 1, "batch": batch}
        return {"kind": kind, "model": model, "layers": 1, "past": 0,
                "new": _log_int(rng, 16, max(16, 2048 // batch)), "batch": batch}
    if kind == "moe":
        return {"kind": kind, "model": "mixtral-8x7b", "seq": _log_int(rng, 128, 2048), "batch": rng.randint(1, 2)}
    batch = rng.randint(1, 4)
    tokens = {"attention": 8192, "attn_block": 4096, "mlp_block": 4096, "head": 2048, "embedding": 8192}[kind]
    seq = _log_int(rng, 32, tokens // batch)
    models = ["llama2-7b", "llama2-13b", "qwen2.5-7b"] if kind in ("head", "embedding") else DENSE
    return {"kind": kind, "model": rng.choice(models), "seq": seq, "batch": batch}


# ---- shared pieces ----------------------------------------------------------------------------------------------
def _spec(model, layers=1, seq=0):
    h, nh, ng, hd, ffn, vocab, norm, eps, act, pos, base, bias, qkv_bias = MODELS[model]
    moe = model == "mixtral-8x7b"
    return ModelSpec(family="llama", hidden=h, layers=layers, heads=nh, kv_heads=ng, head_dim=hd, ffn=ffn, vocab=vocab,
                     padded_vocab=vocab, seq_len=seq, norm=norm, eps=eps, activation=act, pos=pos, rope_base=base,
                     bias=bias, qkv_bias=qkv_bias, experts=8 if moe else 0, moe_ffn=ffn if moe else 0)


def _optimizer_spec(case):
    h = case["hidden"]
    return ModelSpec(family="llama", hidden=h, layers=1, heads=h // 64, kv_heads=h // 64, head_dim=64, ffn=case["ffn"],
                     vocab=1024, padded_vocab=1024, seq_len=0)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _randn(g, *shape, std=1.0, dtype=LP):
    return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, std, generator=g).to(dtype)


def _fill_vectors(module, g):
    """Norm weights and biases away from their initial ones and zeros, as in a model that has been trained."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() == 1:
                scale = name.endswith("norm.weight")
                p.copy_((1.0 if scale else 0.0) + _randn(g, p.numel(), std=0.1 if scale else 0.02, dtype=torch.float32))


def _unit(module, seed, g):
    module.reset_parameters(int(seed), False)
    _fill_vectors(module, g)
    return ShardedUnit(module, "unit", None, 1)


def _zipf_ids(g, vocab, *shape):
    """Token ids with the skew of text: rank r with a frequency of about 1 / r."""
    u = torch.empty(shape, dtype=torch.float64, device=DEV).uniform_(0.0, 1.0, generator=g)
    return torch.exp(u * math.log(vocab)).long().clamp_(1, vocab) - 1


def _grads(unit):
    """The fp32 gradients of a unit's parameters once its backward is over, as the optimizer reads them."""
    unit.reduce_grads()
    return [p.main_grad for p in unit.params]


def _train_args(case):
    h, hd = case["hidden"], case["head_dim"]
    return GalvatronRuntimeArgs(
        parallel=dict(mixed_precision="bf16"),
        model=dict(model_size="llama-small", hidden_size=h, num_layers=case["layers"], num_attention_heads=h // hd,
                   ffn_hidden_size=h * 11 // 4 // 64 * 64, vocab_size=4096, normalization="RMSNorm",
                   activation_func="torch.nn.functional.silu", gated_linear_unit=True),
        train=dict(seq_length=case["seq"], global_batch_size=case["batch"], chunks=1, lr=1e-3, seed=1234))


def _generate_args(case, seed):
    h, nh, ng, hd, ffn, vocab, _, eps, _, _, base, _, qkv_bias = MODELS[case["model"]]
    return GalvatronRuntimeArgs(
        parallel=dict(mixed_precision="bf16"),
        model=dict(model_size="llama-generate", hidden_size=h, num_layers=case["layers"], num_attention_heads=nh,
                   num_query_groups=ng, ffn_hidden_size=ffn, vocab_size=vocab, normalization="RMSNorm",
                   norm_epsilon=eps, activation_func="torch.nn.functional.silu", gated_linear_unit=True,
                   add_qkv_bias=qkv_bias, rotary_base=int(base)),
        train=dict(seq_length=case["past"] + case["new"], global_batch_size=case["batch"], chunks=1, lr=1e-3,
                   seed=int(seed) + 1))


# ---- prepare ----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "train_step":
        model = build_model(_train_args(case), device=torch.device(DEV, torch.cuda.current_device()))
        tok = _zipf_ids(g, 4096, case["batch"], case["seq"] + 1)
        opt = ShardedAdamW(model.sharded_units, lr=1e-4, weight_decay=0.1, clip_grad=1.0, device=model.device)
        return {"kind": kind, "model": model, "opt": opt, "tok": tok[:, :-1].contiguous(),
                "labels": tok[:, 1:].contiguous()}
    if kind == "generate":
        model = build_model(_generate_args(case, seed), device=torch.device(DEV, torch.cuda.current_device()))
        for u in model.sharded_units:
            _fill_vectors(u.module, g)
        vocab = MODELS[case["model"]][5]
        ids = _zipf_ids(g, vocab, case["batch"], case["past"] + case["new"])
        ctx = inference.StaticInferenceContext(case["batch"], case["past"] + case["new"])
        if case["past"]:
            inference.forward_step(model, ids[:, :case["past"]], ctx)
        return {"kind": kind, "model": model, "ctx": ctx, "past": case["past"], "ids": ids,
                "new": ids[:, case["past"]:].contiguous()}

    if kind == "optimizer":
        unit = _unit(GalvatronDecoderLayer(_optimizer_spec(case), LayerCtx(), DEV, "layer"), seed, g)
        unit.reload_master()
        unit.exp_avg.normal_(0.0, 1e-3, generator=g)
        unit.exp_avg_sq.normal_(0.0, 1e-3, generator=g).square_()
        unit.step_count = 10
        unit.main_grad.normal_(0.0, 1e-3, generator=g)
        for p in unit.params:
            p.mg_fresh = False
        return {"kind": kind, "unit": unit,
                "opt": ShardedAdamW([unit], lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1, clip_grad=1.0)}

    S, B = case["seq"], case["batch"]
    spec = _spec(case["model"], seq=S)
    ctx = LayerCtx(seq_len=S)
    H = spec.hidden
    if kind == "attention":
        qkv = _randn(g, S * B, spec.qkv_out).requires_grad_()
        return {"kind": kind, "spec": spec, "S": S, "B": B, "qkv": qkv, "dout": _randn(g, S * B, spec.heads * spec.head_dim)}
    if kind == "attn_block":
        unit = _unit(GalvatronAttention(spec, ctx, DEV, "attn"), seed, g)
        return {"kind": kind, "unit": unit, "spec": spec, "x": _randn(g, S, B, H).requires_grad_(),
                "dout": _randn(g, S, B, H)}
    if kind == "mlp_block":
        unit = _unit(GalvatronMLP(spec, ctx, DEV, "ffn"), seed, g)
        return {"kind": kind, "unit": unit, "spec": spec, "attn": _randn(g, S, B, H).requires_grad_(),
                "x": _randn(g, S, B, H).requires_grad_(), "dout": _randn(g, S, B, H)}
    if kind == "head":
        module = nn.Module()
        module.prenorm = GalvatronFinalNorm(spec, ctx, DEV, "prenorm")
        module.head = GalvatronCausalLMHead(spec, ctx, DEV, "lm_head")
        module.prenorm.reset_parameters()
        module.head.reset_parameters(int(seed))
        _fill_vectors(module, g)
        return {"kind": kind, "unit": ShardedUnit(module, "unit", None, 1), "spec": spec,
                "x": _randn(g, S, B, H).requires_grad_(), "labels": _zipf_ids(g, spec.vocab, B, S)}
    if kind == "embedding":
        unit = _unit(GalvatronEmbedding(spec, ctx, DEV, "embedding"), seed, g)
        return {"kind": kind, "unit": unit, "spec": spec, "tok": _zipf_ids(g, spec.vocab, B, S),
                "dout": _randn(g, S, B, H)}
    if kind == "moe":
        unit = _unit(GalvatronMoEMLP(spec, ctx, DEV, "mlp"), seed, g)
        T = S * B
        # top-2 of skewed scores: some experts get several times the tokens of others
        scores = torch.softmax(_randn(g, T, spec.experts, dtype=torch.float32) +
                               0.7 * _randn(g, spec.experts, dtype=torch.float32), dim=-1)
        top = scores.topk(spec.topk, dim=-1)
        return {"kind": kind, "unit": unit, "spec": spec, "x": _randn(g, T, H).requires_grad_(),
                "probs": (top.values / top.values.sum(-1, keepdim=True)).requires_grad_(), "idx": top.indices,
                "dout": _randn(g, T, H)}
    raise KeyError(kind)


# ---- run --------------------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "attention":
        s, qkv = state["spec"], state["qkv"]
        out = ops.flash_attention_packed(qkv, state["S"], state["B"], s.heads, s.kv_heads, s.head_dim, causal=True)
        return [out, torch.autograd.grad(out, qkv, state["dout"])[0]]
    if kind == "generate":
        ctx = state["ctx"]
        ctx.sequence_len_offset = state["past"]
        return inference.forward_step(state["model"], state["new"], ctx)
    if kind == "optimizer":
        u = state["unit"]
        state["opt"].step()
        return [u.flat, u.master, u.exp_avg, u.exp_avg_sq]
    if kind == "train_step":
        model, opt = state["model"], state["opt"]
        opt.zero_grad()
        loss = model.forward_backward(state["tok"], 0, labels=state["labels"])
        opt.step()
        return {"loss": loss, "grads": [p.main_grad for u in model.sharded_units for p in u.params],
                "weights": [u.flat for u in model.sharded_units]}

    unit = state["unit"]
    unit.zero_grad()
    if kind == "attn_block":
        x = state["x"]
        x.grad = None
        out = unit.module(x)
        out.backward(state["dout"])
        return [out, x.grad, _grads(unit)]
    if kind == "mlp_block":
        a, x = state["attn"], state["x"]
        a.grad = x.grad = None
        out = unit.module(a, x)
        out.backward(state["dout"])
        return [out, a.grad, x.grad, _grads(unit)]
    if kind == "head":
        x = state["x"]
        x.grad = None
        loss = unit.module.head(unit.module.prenorm(x), state["labels"])
        loss.mean().backward()
        return [loss, x.grad, _grads(unit)]
    if kind == "embedding":
        out = unit.module(state["tok"])
        out.backward(state["dout"])
        return [out, _grads(unit)]
    x, probs = state["x"], state["probs"]   # moe
    x.grad = probs.grad = None
    out = unit.module(x, probs, state["idx"])
    out.backward(state["dout"])
    return [out, x.grad, probs.grad, _grads(unit)]


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "train_step":
        h, L, T = case["hidden"], case["layers"], case["seq"] * case["batch"]
        f = h * 11 // 4 // 64 * 64
        layer = 4 * h * h + 3 * h * f + 2 * h
        n = L * layer + 2 * 4096 * h + h
        fwd = 2.0 * T * (L * layer + 4096 * h) + L * 2.0 * T * case["seq"] * h
        # weights read once a direction, gradients written and read, optimizer state read and written, bf16 copy
        return {"flops": 3 * fwd, "bytes": n * (2 * 2 + 2 * 4 + 6 * 4 + 2) + 16.0 * T}
    if kind == "optimizer":
        n = _optimizer_spec(case).layer_params()
        return {"flops": 20.0 * n, "bytes": 34.0 * n}      # gradient twice (norm, update), 3 x 4 B read and written, bf16
    h, nh, ng, hd, ffn, vocab = MODELS[case["model"]][:6]
    qkv_out = (nh + 2 * ng) * hd
    gated = MODELS[case["model"]][8] != "gelu"
    attn_w = h * qkv_out + nh * hd * h
    mlp_w = (3 if gated else 2) * h * ffn
    if kind == "generate":
        B, new, past, L = case["batch"], case["new"], case["past"], case["layers"]
        T, keys = B * new, B * (past + new)
        flops = 2.0 * T * (L * (attn_w + mlp_w) + vocab * h) + L * 4.0 * nh * hd * T * (past + (new + 1) / 2)
        return {"flops": flops, "bytes": 2.0 * (L * (attn_w + mlp_w) + vocab * h + L * keys * 2 * ng * hd + T * (h + vocab))}
    S, B = case["seq"], case["batch"]
    T = float(S * B)
    core = 4.0 * nh * hd * T * (S + 1) / 2
    if kind == "attention":
        return {"flops": 3.5 * core, "bytes": 2.0 * T * (2 * qkv_out + 2 * nh * hd)}
    if kind == "attn_block":
        return {"flops": 6.0 * T * attn_w + 3.5 * core, "bytes": 6.0 * attn_w + 8.0 * T * h}
    if kind == "mlp_block":
        return {"flops": 6.0 * T * mlp_w, "bytes": 6.0 * mlp_w + 2.0 * 6 * T * h}
    if kind == "head":
        return {"flops": 6.0 * T * vocab * h, "bytes": 6.0 * vocab * h + 4.0 * T * h + 12.0 * T}
    if kind == "embedding":
        rows = min(T, vocab)
        return {"flops": T * h, "bytes": 2.0 * rows * h + 2.0 * T * h + 2.0 * T * h + 4.0 * vocab * h}
    return {"flops": 6.0 * 2 * T * 3 * h * ffn, "bytes": 6.0 * 8 * 3 * h * ffn + 8.0 * T * h}   # moe, top-2 of 8


def tolerance(case):
    # Measured against 64-bit arithmetic, worst output of each kind: attention 2.6e-3, attn_block 7.8e-3, mlp_block
    # 4.8e-3, head 2.3e-3, moe 4.2e-3 (one 16-bit rounding is 1.7e-3, and a block chains several); generate 1.8e-2 over
    # four layers; about four times that, or the most that a comparison allows.  Embedding gradients and optimizer
    # state are fp32 sums in any order (measured 1e-8 and 6e-8).
    return {
        "attention": {"rel": 1e-2, "max": 0.3},
        "attn_block": {"rel": 2e-2, "max": 0.5},
        "mlp_block": {"rel": 2e-2, "max": 0.5},
        "head": {"rel": 1e-2, "max": 0.5},
        "embedding": {"rel": 1e-5, "max": 1e-3},     # fp32 sums in any order
        "moe": {"rel": 2e-2, "max": 0.5},
        "optimizer": {"rel": 1e-5, "max": 2e-2},     # the bf16 copy of a weight may round the other way
        "train_step": {"rel": 3e-2, "max": 0.9},
        "generate": {"rel": 3e-2, "max": 0.5},
    }[case["kind"]]


# ---- 64-bit restatement -----------------------------------------------------------------------------------------
def _norm64(x, w, b, spec):
    if spec.norm == "RMSNorm":
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + spec.eps) * w
    return nn.functional.layer_norm(x, (x.shape[-1],), w, b, spec.eps)


def _rope64(t, spec):
    """t [S, B, heads, hd], rotate-half; angles in 32 bits, as the tables that every layer of a model shares."""
    half = spec.head_dim // 2
    inv = 1.0 / (spec.rope_base ** (torch.arange(0, spec.head_dim, 2, dtype=torch.float32) / spec.head_dim))
    ang = torch.outer(torch.arange(t.shape[0], dtype=torch.float32), inv)
    c, s = (f.to(DEV).double()[:, None, None, :] for f in (ang.cos(), ang.sin()))
    a, b = t[..., :half], t[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _head64(q, k, v, scale):
    s = (q @ k.transpose(-1, -2)) * scale
    s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=DEV).triu(1), float("-inf"))
    return torch.softmax(s, dim=-1) @ v


def _attention64(qkv, spec, rope):
    """qkv [S, B, P] packed per kv head -> [S, B, nh * hd]; one (sequence, kv head) at a time."""
    S, B = qkv.shape[:2]
    ng, qpg, hd = spec.kv_heads, spec.heads // spec.kv_heads, spec.head_dim
    t = qkv.view(S, B, ng, qpg + 2, hd)
    q, k, v = t[:, :, :, :qpg], t[:, :, :, qpg], t[:, :, :, qpg + 1]
    if rope:
        q = _rope64(q.reshape(S, B, spec.heads, hd), spec).view(S, B, ng, qpg, hd)
        k = _rope64(k, spec)
    rows = []
    for b in range(B):
        for g in range(ng):
            o = checkpoint(_head64, q[:, b, g].transpose(0, 1), k[:, b, g], v[:, b, g], 1.0 / math.sqrt(hd),
                           use_reentrant=False)
            rows.append(o.transpose(0, 1).reshape(S, qpg * hd))
    return torch.stack(rows, dim=1).view(S, B, spec.heads * hd)


def _linear64(x, lin):
    return nn.functional.linear(x, lin["weight"], lin.get("bias"))


def _act64(y, spec):
    if spec.activation == "gelu":
        return nn.functional.gelu(y, approximate="tanh")
    a, b = y.chunk(2, dim=-1)
    return nn.functional.silu(a) * b


class _P64:
    """64-bit leaves for a module's parameters, by name."""

    def __init__(self, module):
        self.by_param = {id(p): p.detach().double().requires_grad_() for p in module.parameters()}
        self.by_name = {n: self.by_param[id(p)] for n, p in module.named_parameters()}

    def at(self, prefix):
        return {n[len(prefix) + 1:]: t for n, t in self.by_name.items() if n.startswith(prefix + ".")}

    def grads(self, params):
        return [self.by_param[id(p)].grad for p in params]


def _attn64(x, w, prefix, spec):
    n = w.at(prefix + "input_layernorm")
    qkv = _linear64(_norm64(x, n["weight"], n.get("bias"), spec), w.at(prefix + "attention.linear_qkv"))
    return _linear64(_attention64(qkv, spec, spec.pos == "rope"), w.at(prefix + "attention.linear_proj"))


def _mlp64(a, x, w, prefix, spec):
    n = w.at(prefix + "post_attention_layernorm")
    h = a + x
    y = _act64(_linear64(_norm64(h, n["weight"], n.get("bias"), spec), w.at(prefix + "mlp.linear_fc1")), spec)
    return h + _linear64(y, w.at(prefix + "mlp.linear_fc2"))


def _stack64(model, tokens):
    """Logits [S, B, V] of a dense stack and its 64-bit parameters."""
    w = _P64(model.model)
    spec = model.spec
    names = [n for n, _ in model.model.named_parameters()]
    emb = next(n for n in names if n.endswith("embed_tokens.weight"))
    head = next(n for n in names if n.endswith("lm_head.weight"))
    x = w.by_name[emb][tokens.t()]
    for n in names:
        if n.endswith("attn.input_layernorm.weight"):
            unit = n[:-len("attn.input_layernorm.weight")]
            x = checkpoint(lambda t, u=unit: _mlp64(_attn64(t, w, u + "attn.", spec), t, w, u + "ffn.", spec), x,
                           use_reentrant=False)
        elif n.endswith(".norm.weight"):
            final = w.by_name[n]
    return nn.functional.linear(_norm64(x, final, None, spec), w.by_name[head]), w


def exact(case, seed):
    kind, st = case["kind"], prepare(case, seed)
    if kind == "generate":
        with torch.no_grad():
            return _stack64(st["model"], st["ids"])[0][case["past"]:].contiguous()
    if kind == "train_step":
        model = st["model"]
        logits, w = _stack64(model, st["tok"])
        loss = nn.functional.cross_entropy(logits.transpose(0, 1).reshape(-1, logits.shape[-1]), st["labels"].reshape(-1))
        loss.backward()
        grads = w.grads([p for u in model.sharded_units for p in u.params])
        return {"loss": loss.detach(), "grads": grads, "weights": [None] * len(model.sharded_units)}
    if kind == "optimizer":
        u = st["unit"]
        g, m, v, p = (t.double() for t in (u.main_grad, u.exp_avg, u.exp_avg_sq, u.master))
        g = g * min(1.0, 1.0 / (float(g.norm()) + 1e-6))
        m, v = 0.9 * m + 0.1 * g, 0.95 * v + 0.05 * g * g
        t = u.step_count + 1
        p = p * (1 - 3e-4 * 0.1) - 3e-4 / (1 - 0.9 ** t) * m / (v.sqrt() / math.sqrt(1 - 0.95 ** t) + 1e-8)
        return [p, p, m, v]

    spec = st["spec"]
    if kind == "attention":
        qkv = st["qkv"].detach().double().requires_grad_()
        out = _attention64(qkv.view(case["seq"], case["batch"], -1), spec, False).view(st["dout"].shape)
        return [out.detach(), torch.autograd.grad(out, qkv, st["dout"].double())[0]]
    unit, w = st["unit"], _P64(st["unit"].module)
    if kind == "attn_block":
        x = st["x"].detach().double().requires_grad_()
        out = _attn64(x, w, "", spec)
        out.backward(st["dout"].double())
        return [out.detach(), x.grad, w.grads(unit.params)]
    if kind == "mlp_block":
        a, x = (st[n].detach().double().requires_grad_() for n in ("attn", "x"))
        out = _mlp64(a, x, w, "", spec)
        out.backward(st["dout"].double())
        return [out.detach(), a.grad, x.grad, w.grads(unit.params)]
    if kind == "head":
        x = st["x"].detach().double().requires_grad_()
        n, lm = w.at("prenorm.norm"), w.at("head.lm_head")
        logits = nn.functional.linear(_norm64(x, n["weight"], n.get("bias"), spec), lm["weight"])
        loss = nn.functional.cross_entropy(logits.view(-1, spec.vocab), st["labels"].t().reshape(-1), reduction="none")
        loss = loss.view(case["seq"], case["batch"]).t().contiguous()
        loss.mean().backward()
        return [loss.detach(), x.grad, w.grads(unit.params)]
    if kind == "embedding":
        ids = st["tok"].t()
        table = w.by_name["embed_tokens.weight"]
        dw = torch.zeros_like(table.detach())
        dw.index_add_(0, ids.reshape(-1), st["dout"].double().view(-1, spec.hidden))
        return [table.detach()[ids], [dw]]
    x, probs = (st[n].detach().double().requires_grad_() for n in ("x", "probs"))   # moe
    w1, w2 = w.by_name["experts.linear_fc1.weight"], w.by_name["experts.linear_fc2.weight"]
    out = torch.zeros_like(x)
    for e in range(spec.experts):
        tok, slot = (st["idx"] == e).nonzero(as_tuple=True)
        y = nn.functional.linear(_act64(nn.functional.linear(x[tok], w1[e]), spec), w2[e])
        out = out.index_add(0, tok, y * probs[tok, slot][:, None])
    out.backward(st["dout"].double())
    return [out.detach(), x.grad, probs.grad, w.grads(unit.params)]
