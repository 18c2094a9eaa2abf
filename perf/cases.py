"""The calls that a user of this framework has it do, as cases that can be timed and checked: one forward of a shard of
transformer blocks (one token, a batch of tokens, a prompt, a further portion of a prompt), the output head, the samplers, a whole
generation, and the blocks of two designs with a floating-point stream (Nigenex, Setodra).  Every case goes through the public entry points (``cake_b200.model``,
the C ABI of ``include/cake_b200.h``).

A case is a dict of plain values.  ``prepare`` keeps one model per process, as a serving program does, and makes the request's own
inputs and cache from the seed; ``run`` is one call of such a program.  Steps and portions on a cached context run on one session
that grows from call to call, and begin a new session when its cache is full.  ``exact`` restates every path in plain torch, 64 bits."""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from cake_b200 import capi
from cake_b200.capi import byref, c_uint32, check, lib, ptr
from cake_b200.config import Config, LayerSpec, MixerSpec, MoeSpec, RotarySpec, llama3_8b, qwen3_0_6b
from cake_b200.model import BLOCK_CLASSES, B200Transformer, Cache, Context, TextModelBase, sampling_from_args

DEV = "cuda:0"
DT = {"bf16": torch.bfloat16, "f16": torch.float16}
DENSE = {"llama3-8b": llama3_8b, "qwen3-0.6b": qwen3_0_6b}
NIGENEX = {  # widths that the benchmark's Nigenex workload runs
    "2k": dict(width=2048, heads=16, kv_heads=4, head_dim=128, ff=8192, window=1024),
    "4k": dict(width=4096, heads=32, kv_heads=8, head_dim=128, ff=14336, window=1024)}
SETODRA = {  # widths that the benchmark's Setodra workload runs
    "1k": dict(width=1024, ret=dict(heads=8, dim=128, vdim=128), ssd=dict(heads=32, vdim=64, state=128, groups=4, conv=4, norm_groups=4),
               lat=dict(heads=8, dim=128, rot_dim=64, vdim=128, kv_rank=512), moe=dict(experts=32, identity=2, top=4, ff=704, shared_ff=1408)),
    "2k": dict(width=2048, ret=dict(heads=16, dim=128, vdim=128), ssd=dict(heads=64, vdim=64, state=128, groups=8, conv=4, norm_groups=8),
               lat=dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512), moe=dict(experts=64, identity=2, top=6, ff=1408, shared_ff=2816))}
MODEL_SEED = 20240611


def listed():
    return [
        # one token of one conversation through two blocks of the benchmark's model: the decode loop's unit
        dict(name="step 8b", kind="block", model="llama3-8b", dtype="bf16", layers=2, batch=1, seq=1, ctx=2048),
        # one token each of sixteen conversations: batched serving
        dict(name="step 8b batch 16", kind="block", model="llama3-8b", dtype="bf16", layers=1, batch=16, seq=1, ctx=1000),
        # a short question to a small model: the call where launches and latency count most
        dict(name="prompt 0.6b 37", kind="block", model="qwen3-0.6b", dtype="f16", layers=8, batch=1, seq=37, ctx=0),
        # an ordinary prompt
        dict(name="prompt 8b 512", kind="block", model="llama3-8b", dtype="bf16", layers=1, batch=1, seq=512, ctx=0),
        # the next message of a long conversation
        dict(name="portion 8b 200 at 3000", kind="block", model="llama3-8b", dtype="bf16", layers=1, batch=1, seq=200, ctx=3000),
        # a batch of long prompts, the shape of the prefill benchmark
        dict(name="prompts 8b 8x4096", kind="block", model="llama3-8b", dtype="bf16", layers=1, batch=8, seq=4096, ctx=0),
        # final norm and output projection of a batch of conversations
        dict(name="head 8b batch 16", kind="head", model="llama3-8b", dtype="bf16", batch=16),
        # the draw of one token: repeat penalty, temperature, nucleus
        dict(name="sample top-p", kind="sample", vocab=128256, dtype="bf16", temperature=0.8, top_k=0, top_p=0.95, penalty=1.1, recent=100),
        # a whole request to a small model: prompt, then token by token with a repeat penalty
        dict(name="generate 0.6b", kind="generate", model="qwen3-0.6b", dtype="f16", prompt=24, tokens=24),
        # one token through blocks with a floating-point stream and windowed attention
        dict(name="step nigenex", kind="nigenex", size="2k", dtype="bf16", layers=4, batch=1, seq=1, ctx=1500),
        # one token through a retention, a state-space and a latent-attention block, each with a routed feed-forward
        dict(name="step setodra", kind="setodra", size="2k", dtype="bf16", batch=1, seq=1, ctx=300),
        # a prompt through the same blocks
        dict(name="prompt setodra 1000", kind="setodra", size="2k", dtype="bf16", batch=1, seq=1000, ctx=0),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["block"] * 6 + ["head", "sample", "sample", "generate", "nigenex", "setodra"])
    dtype = rng.choice(["bf16", "f16"])
    if kind == "block":
        model = rng.choice(sorted(DENSE))
        layers = rng.randint(1, 2) if model == "llama3-8b" else rng.randint(4, 10)
        what = rng.choice(["step", "steps", "prompt", "portion"])
        batch = {"step": 1, "steps": _log(rng, 2, 64), "prompt": rng.choice([1, 1, 1, 2, 3, 5]), "portion": rng.choice([1, 1, 2, 4])}[what]
        seq = {"step": 1, "steps": 1, "prompt": _log(rng, 2, 4096), "portion": _log(rng, 2, 1024)}[what]
        ctx = {"step": _log(rng, 10, 6000), "steps": _log(rng, 10, 3000), "prompt": 0, "portion": _log(rng, 60, 4000)}[what]
        if model == "llama3-8b":
            seq = min(seq, 16384 // (batch * layers))
        return dict(kind=kind, model=model, dtype=dtype, layers=layers, batch=batch, seq=seq, ctx=ctx)
    if kind == "head":
        return dict(kind=kind, model=rng.choice(sorted(DENSE)), dtype=dtype, batch=_log(rng, 1, 64))
    if kind == "sample":
        k, p = rng.choice([(0, 0.0), (rng.randint(5, 200), 0.0), (0, rng.uniform(0.5, 0.98)), (rng.randint(5, 200), rng.uniform(0.5, 0.98))])
        return dict(kind=kind, vocab=rng.choice([32768, 128256, 151936]), dtype=dtype, temperature=round(rng.uniform(0.3, 1.3), 3), top_k=k,
                    top_p=round(p, 3), penalty=rng.choice([1.0, 1.1]), recent=rng.randint(1, 128))
    if kind == "generate":
        return dict(kind=kind, model="qwen3-0.6b", dtype=dtype, prompt=_log(rng, 3, 150), tokens=rng.randint(3, 24))
    step = rng.random() < 0.5
    size = rng.choice(["2k", "4k"]) if kind == "nigenex" else rng.choice(["1k", "2k"])
    batch, seq, ctx = rng.choice([1, 1, 2, 4]), 1 if step else _log(rng, 2, 1500), _log(rng, 20, 600) if step else 0
    case = dict(kind=kind, size=size, dtype=dtype, batch=batch, seq=seq, ctx=ctx)
    if kind == "nigenex":
        case["layers"] = rng.randint(2, 4)
    return case


# ---------------------------------------------------------------------------------------------- models (one per process, kept)
def _weights(shapes, dtype, seed):
    """name -> tensor for a list of (name, shape, scale, offset)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return {n: (torch.randn(s, generator=g, device=DEV, dtype=torch.float32) * a + b).to(dtype) for n, s, a, b in shapes}


def _dense_layer(cfg, i, dtype):
    H, I, q, kv, p = cfg.hidden_size, cfg.intermediate_size, cfg.size_q, cfg.size_kv, cfg.layer_name(i) + "."
    s = [(p + "self_attn.q_proj.weight", (q, H), 0.02, 0), (p + "self_attn.k_proj.weight", (kv, H), 0.02, 0), (p + "self_attn.v_proj.weight", (kv, H), 0.02, 0),
         (p + "self_attn.o_proj.weight", (H, q), 0.02, 0), (p + "mlp.gate_proj.weight", (I, H), 0.02, 0), (p + "mlp.up_proj.weight", (I, H), 0.02, 0),
         (p + "mlp.down_proj.weight", (H, I), 0.02, 0), (p + "input_layernorm.weight", (H,), 0.02, 1), (p + "post_attention_layernorm.weight", (H,), 0.02, 1)]
    if cfg.use_qk_norm:
        s += [(p + "self_attn.q_norm.weight", (cfg.hd,), 0.02, 1), (p + "self_attn.k_norm.weight", (cfg.hd,), 0.02, 1)]
    return _weights(s, dtype, MODEL_SEED + i)


def _dense_head(cfg, dtype):
    p, V, H = cfg.model_prefix, cfg.vocab_size, cfg.hidden_size
    s = [(p + ".embed_tokens.weight", (V, H), 1.0, 0), (p + ".norm.weight", (H,), 0.02, 1)]  # token vectors of unit size: the largest logit stands clear of the rest
    if not cfg.tie_word_embeddings:
        s.append(("lm_head.weight", (V, H), 0.02, 0))
    return _weights(s, dtype, MODEL_SEED - 1)


def _nigenex_cfg(case):
    z = NIGENEX[case["size"]]
    sp = LayerSpec(heads=z["heads"], kv_heads=z["kv_heads"], head_dim=z["head_dim"], window=z["window"], scale=z["head_dim"] ** -0.5, softcap=30.0, ff=z["ff"])
    return Config(z["width"], z["ff"], 256, case["layers"], z["heads"], z["kv_heads"], rms_norm_eps=1e-5, head_dim=z["head_dim"], max_seq_len=4096,
                  block_kind="nigenex", layers=[sp] * case["layers"], logit_softcap=30.0, model_prefix="")


def _nigenex_weights(cfg, dtype):
    s, W = [], cfg.hidden_size
    for i, sp in enumerate(cfg.layers):
        p, q, kv = cfg.layer_name(i) + ".", sp.heads * sp.head_dim, sp.kv_heads * sp.head_dim
        s += [(p + "norm1", (), 0.05, 1), (p + "shift", (W,), 0.1, 0.5), (p + "mix.q", (q, W), 0.02, 0), (p + "mix.k", (kv, W), 0.02, 0), (p + "mix.r1", (sp.heads,), 0.1, 0.5),
              (p + "mix.r2", (sp.heads,), 0.1, 1), (p + "mix.g", (sp.heads, W), 0.02, 0), (p + "mix.o", (W, q), 0.02, 0),
              (p + "mlp.gate", (sp.ff, W), 0.02, 0), (p + "mlp.up", (sp.ff, W), 0.02, 0), (p + "mlp.down", (W, sp.ff), 0.02, 0)]
    return _weights(s, dtype, MODEL_SEED)


def _setodra_cfg(case):
    z = SETODRA[case["size"]]
    mo = MoeSpec(scale=2.5, **z["moe"])
    rot = RotarySpec(dims=z["lat"]["rot_dim"], base=10000.0, factor=8.0, fast=32.0, slow=1.0, original=2048)
    layers = [MixerSpec(type="retention", decay=[1 - 2.0 ** (-5 - i % 4) for i in range(z["ret"]["heads"])], rot=RotarySpec(dims=z["ret"]["dim"], base=10000.0),
                        moe=mo, **z["ret"]),
              MixerSpec(type="mamba2", moe=mo, **z["ssd"]),
              MixerSpec(type="latent_attention", scale=(z["lat"]["dim"] + z["lat"]["rot_dim"]) ** -0.5, rot=rot, moe=mo, **z["lat"])]
    return Config(z["width"], 0, 256, len(layers), layers[0].heads, layers[0].heads, rms_norm_eps=1e-6, head_dim=128, max_seq_len=4096,
                  block_kind="setodra", layers=layers, model_prefix="")


def _setodra_weights(cfg, dtype):
    s, W = [], cfg.hidden_size
    for i, sp in enumerate(cfg.layers):
        p, a = cfg.layer_name(i) + ".", 0.02
        s += [(p + "norm1", (W,), 0.05, 1), (p + "norm2", (W,), 0.05, 1), (p + "mix.o", (W, sp.inner), a, 0)]
        if sp.type == "retention":
            s += [(p + "mix." + n, (r, W), a, 0) for n, r in (("q", sp.heads * sp.dim), ("k", sp.heads * sp.dim), ("v", sp.inner), ("g", sp.inner))]
        elif sp.type == "mamba2":
            ch = sp.inner + 2 * sp.groups * sp.state
            s += [(p + "mix.in", (sp.inner + ch + sp.heads, W), a, 0), (p + "mix.conv", (ch, sp.conv), 0.4, 0), (p + "mix.conv.b", (ch,), 0.1, 0),
                  (p + "mix.dt_bias", (sp.heads,), 0.7, -1), (p + "mix.A_log", (sp.heads,), 0.7, -0.5), (p + "mix.D", (sp.heads,), 0.2, 1), (p + "mix.norm", (sp.inner,), 0.05, 1)]
        else:
            s += [(p + "mix.q", (sp.heads * (sp.dim + sp.rot_dim), W), a, 0), (p + "mix.dkv", (sp.kv_rank + sp.rot_dim, W), a, 0), (p + "mix.dkv.norm", (sp.kv_rank,), 0.05, 1),
                  (p + "mix.uk", (sp.heads * sp.dim, sp.kv_rank), a, 0), (p + "mix.uv", (sp.inner, sp.kv_rank), a, 0)]
        mo = sp.moe
        s += [(p + "mlp.router", (mo.experts + mo.identity, W), 0.1, 0), (p + "mlp.correction", (mo.experts + mo.identity,), 0.02, 0)]
        for e in ["e%d" % j for j in range(mo.experts)] + ["shared"]:
            f = mo.shared_ff if e == "shared" else mo.ff
            s += [("%smlp.%s.gate" % (p, e), (f, W), a, 0), ("%smlp.%s.up" % (p, e), (f, W), a, 0), ("%smlp.%s.down" % (p, e), (W, f), a, 0)]
        s.append((p + "mlp.shared.sg", (1, W), a, 0))
    return _weights(s, dtype, MODEL_SEED)


class _Model:
    def __init__(self, ctx, blocks, text=None):
        self.ctx, self.blocks, self.text = ctx, blocks, text


_kept = {}


def _model(case):
    """The process's model: one context with its weights; another one takes its place when a case asks for it."""
    kind = case["kind"]
    key = (kind, case["dtype"], case.get("model"), case.get("size"), case.get("layers"), case.get("vocab"))
    if key in _kept:
        return _kept[key]
    for m in _kept.values():
        m.ctx.close()
    _kept.clear()
    dt = DT[case["dtype"]]
    if kind in ("block", "head", "generate"):
        cfg = DENSE[case["model"]](max_seq=8192)
        if kind == "block":
            ctx = Context(cfg, {}, dtype=case["dtype"])
            blocks = []
            for i in range(case["layers"]):
                ctx.var_builder = _dense_layer(cfg, i, dt)
                blocks.append(B200Transformer.load(cfg.layer_name(i), ctx))
            m = _Model(ctx, blocks)
        elif kind == "head":
            sd = _dense_head(cfg, dt)
            ctx = Context(cfg, {}, dtype=case["dtype"])
            p = cfg.model_prefix
            emb, norm, head = sd[p + ".embed_tokens.weight"], sd[p + ".norm.weight"], sd.get("lm_head.weight")
            check(lib().cake_b200_head_load(ctx.h, ptr(emb), ptr(norm), ptr(head)))
            m = _Model(ctx, [])
        else:
            sd = _dense_head(cfg, dt)
            for i in range(cfg.num_hidden_layers):
                sd.update(_dense_layer(cfg, i, dt))
            ctx = Context(cfg, sd, dtype=case["dtype"])
            m = _Model(ctx, [], TextModelBase.load(ctx, repeat_penalty=1.1))
    elif kind == "sample":
        m = _Model(Context(Config(64, 128, case["vocab"], 1, 4, 2, max_seq_len=64), {}, dtype=case["dtype"]), [])
    else:
        cfg = _nigenex_cfg(case) if kind == "nigenex" else _setodra_cfg(case)
        sd = _nigenex_weights(cfg, dt) if kind == "nigenex" else _setodra_weights(cfg, dt)
        ctx = Context(cfg, sd, dtype=case["dtype"])
        m = _Model(ctx, [BLOCK_CLASSES[cfg.block_kind].load(cfg.layer_name(i), ctx) for i in range(len(cfg.layers))])
    m.ctx.sync()
    m.ctx.var_builder = {}
    _kept[key] = m
    return m


# ---------------------------------------------------------------------------------------------- requests
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + 17)
    return g


def _rows(case, seed, width, dtype):
    """The hidden states that the call is given, and (designs without a synthetic cache) those of the context in front of them."""
    g = _rng(seed)
    x = torch.randn((case["batch"], case["seq"], width), generator=g, device=DEV).to(dtype)
    pre = torch.randn((case["batch"], case["ctx"], width), generator=g, device=DEV).to(dtype) if case["ctx"] and case["kind"] != "block" else None
    return x, pre


def _calls_per_session(case):
    return 1 if not case["ctx"] else 256 if case["seq"] == 1 else 4


def _penalised(case, seed):
    g = _rng(seed)
    return torch.randint(0, case["vocab"], (case["recent"],), generator=g, device=DEV).cpu().tolist()


def _raw_logits(case, seed):
    """Logits as a trained model has them: a broad body and a few dozen candidates that stand out."""
    g = _rng(seed + 1)
    V = case["vocab"]
    x = torch.randn((V,), generator=g, device=DEV) * 2.0
    at = torch.randperm(V, generator=g, device=DEV)[:40]
    x[at] += torch.linspace(4.0, 12.0, 40, device=DEV)
    return x.to(DT[case["dtype"]])


def _prompt_ids(case, seed):
    g = _rng(seed)
    return torch.randint(0, DENSE[case["model"]]().vocab_size, (case["prompt"],), generator=g, device=DEV).cpu().tolist()


def prepare(case, seed):
    m = _model(case)
    st = dict(case=case, m=m, seed=seed)
    kind = case["kind"]
    with torch.cuda.stream(m.ctx.torch_stream):
        if kind == "head":
            st["x"] = torch.randn((case["batch"], 1, m.ctx.config.hidden_size), generator=_rng(seed), device=DEV).to(DT[case["dtype"]])
        elif kind == "sample":
            st["logits"], st["ids"] = _raw_logits(case, seed), (c_uint32 * case["recent"])(*_penalised(case, seed))
            st["sampling"] = sampling_from_args(case["temperature"], case["top_k"] or None, case["top_p"] or None, seed)
        elif kind == "generate":
            st["ids"] = _prompt_ids(case, seed)
            st["cache"] = Cache(m.ctx, 1, case["prompt"] + case["tokens"])
        else:
            st["x"], st["pre"] = _rows(case, seed, m.ctx.config.hidden_size, m.ctx.stream_dtype)
            st["cache"] = Cache(m.ctx, case["batch"], case["ctx"] + case["seq"] * _calls_per_session(case))
            st["calls"] = 0
    m.ctx.sync()
    return st


def _forward(st, x, pos):
    m = st["m"]
    m.ctx.cache = st["cache"]
    names = [(b.layer_name(), pos, i) for i, b in enumerate(m.blocks)]
    return m.blocks[0].forward_batch(x, names, m.ctx, blocks=m.blocks)


def run(st):
    case, m = st["case"], st["m"]
    ctx, kind = m.ctx, case["kind"]
    if kind == "head":
        logits = ctx.empty(case["batch"], ctx.config.vocab_size, dtype=ctx.logits_dtype)
        check(lib().cake_b200_logits(ctx.h, ptr(st["x"]), case["batch"], 1, ptr(logits), None))
        return logits
    if kind == "sample":
        with torch.cuda.stream(ctx.torch_stream):
            logits = st["logits"].clone()   # the step's logits; the penalty is applied to them in place
        tok = c_uint32()
        check(lib().cake_b200_sample(ctx.h, ptr(logits), byref(st["sampling"]), case["penalty"], st["ids"], case["recent"], 3, None, byref(tok)))
        return {"logits": logits, "token": int(tok.value)}
    if kind == "generate":
        t = m.text
        ctx.cache = st["cache"]
        t.prepare_prompt(st["ids"])
        t.generated = 0
        logits, tokens = [], []
        for i in range(case["tokens"]):
            tokens.append(t.next_token(i).id)
            logits.append(t.last_logits)
        return {"logits": logits, "tokens": np.array(tokens)}
    cache, n = st["cache"], st["calls"] % _calls_per_session(case)
    st["calls"] += 1
    if n == 0:  # a new session
        cache.clear()
        if case["ctx"] and kind == "block":
            cache.fill_synthetic(range(len(m.blocks)), case["ctx"], st["seed"] & 0xffffff)
        elif case["ctx"]:
            _forward(st, st["pre"], 0)
    return _forward(st, st["x"], case["ctx"] + n * case["seq"])


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _pairs(case, window=0):
    """(query, key) pairs of one sequence."""
    n, c = case["seq"], case["ctx"]
    if not window:
        return n * c + n * (n + 1) // 2
    return sum(min(window, c + i + 1) for i in range(n))


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return dict(bytes=2.0 * case["vocab"] * 3, flops=4.0 * case["vocab"])
    if kind in ("block", "head", "generate"):
        cfg = DENSE[case["model"]]()
        H, I, V, q, kv = cfg.hidden_size, cfg.intermediate_size, cfg.vocab_size, cfg.size_q, cfg.size_kv
        per = H * (q + 2 * kv) + q * H + 3 * H * I
        if kind == "head":
            B = case["batch"]
            return dict(bytes=2.0 * (V * H + B * (V + H)), flops=2.0 * B * V * H)
        if kind == "generate":
            n, L = case["tokens"], cfg.num_hidden_layers
            rows = case["prompt"] + n - 1
            return dict(bytes=2.0 * n * (L * per + V * H), flops=2.0 * (rows * L * per + n * V * H) + 4.0 * q * L * rows * (rows + 1) / 2)
        B, S, C, L = case["batch"], case["seq"], case["ctx"], case["layers"]
        return dict(bytes=2.0 * (L * per + L * B * 2 * kv * (C + S) + 2 * B * S * H), flops=2.0 * B * S * L * per + 4.0 * q * L * B * _pairs(case))
    B, S, C = case["batch"], case["seq"], case["ctx"]
    if kind == "nigenex":
        z, L = NIGENEX[case["size"]], case["layers"]
        W, q, kv = z["width"], z["heads"] * z["head_dim"], z["kv_heads"] * z["head_dim"]
        per = W * (2 * q + kv + z["heads"] + 3 * z["ff"])
        keys = min(C + S, z["window"] + S - 1)
        return dict(bytes=2.0 * L * (per + B * kv * keys) + 8.0 * B * S * W, flops=2.0 * B * S * L * per + 4.0 * q * L * B * _pairs(case, z["window"]))
    z, W = SETODRA[case["size"]], SETODRA[case["size"]]["width"]
    r, s, la, mo = z["ret"], z["ssd"], z["lat"], z["moe"]
    ri, si, li = r["heads"] * r["vdim"], s["heads"] * s["vdim"], la["heads"] * la["vdim"]
    mix = W * (2 * r["heads"] * r["dim"] + 3 * ri) + W * (3 * si + 2 * s["groups"] * s["state"] + s["heads"]) \
        + W * (la["heads"] * (la["dim"] + la["rot_dim"]) + la["kv_rank"] + la["rot_dim"] + li) + la["kv_rank"] * (la["heads"] * la["dim"] + li)
    M = B * S
    touched = min(mo["experts"], M * mo["top"])
    ff = 3 * (W * (3 * touched * mo["ff"] + 3 * mo["shared_ff"] + mo["experts"] + mo["identity"]))
    ff_flops = 2.0 * M * 3 * W * (3 * mo["top"] * mo["ff"] + 3 * mo["shared_ff"] + mo["experts"])
    state = B * (ri * r["dim"] + si * s["state"]) * 4.0 * (2 if C else 1)
    return dict(bytes=2.0 * (mix + ff) + state + 2.0 * B * (C + S) * (la["kv_rank"] + la["rot_dim"]) + 8.0 * M * W,
                flops=2.0 * M * mix + ff_flops + 4.0 * M * (ri * r["dim"] + si * s["state"]) + 4.0 * la["heads"] * (la["kv_rank"] + la["rot_dim"]) * B * _pairs(case))


# About four times the error against 64 bits that the paths showed when this was written, per kind: bf16, f16 (block 0.0074 and 0.0011, head
# 0.0023 and 0.0003, generate 0.016 and 0.002, Nigenex 0.0062 and 0.0008; Setodra 0.022, where a token between two experts goes to the other one).
_REL = dict(block=(0.03, 0.0045), head=(0.009, 0.0012), generate=(0.064, 0.008), nigenex=(0.025, 0.0035), setodra=(0.08, 0.03))


def tolerance(case):
    if case["kind"] == "sample":   # the penalty is one rounded product, and the draw is a whole number
        return "exact"
    return {"rel": _REL[case["kind"]][case["dtype"] == "f16"]}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _d(sd):
    return {k: v.double() for k, v in sd.items()}


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _silu(z):
    return z * torch.sigmoid(z)


def _angles(pos, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=torch.float64) / dims)
    return pos.double()[:, None] * f[None, :]


def _turn(v, cos, sin):
    """v (..., S, D) with D / 2 pairs (i, i + D / 2); cos, sin (S, D / 2)."""
    h = v.shape[-1] // 2
    a, b = v[..., :h], v[..., h:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _softmax_pv(q, k, v, scale, pos0, window=0, score=None):
    """q (h, S, D) at positions pos0.., k and v (h, T, D): causal attention, a block of queries at a time."""
    out = torch.empty(q.shape[0], q.shape[1], v.shape[-1], device=DEV, dtype=torch.float64)
    step = max(1, (1 << 27) // (q.shape[0] * k.shape[1]))
    j = torch.arange(k.shape[1], device=DEV)
    for a in range(0, q.shape[1], step):
        b = min(q.shape[1], a + step)
        i = torch.arange(a, b, device=DEV) + pos0
        s = torch.einsum("hid,hjd->hij", q[:, a:b], k) * scale
        n = i[:, None] - j[None, :]
        if score is not None:
            s = score(s, n.clamp(min=0).double())
        hide = n < 0
        if window:
            hide = hide | (n >= window)
        out[:, a:b] = torch.einsum("hij,hjd->hid", torch.softmax(s.masked_fill(hide, -math.inf), -1), v)
    return out


def _synthetic(case, cfg, layer, seed, which):
    """The cached rows that a synthetic fill leaves: a hash of the element's place, uniform in [-1, 1)."""
    B, kv, hd, cap = case["batch"], cfg.num_key_value_heads, cfg.hd, case["ctx"] + case["seq"] * _calls_per_session(case)
    m32 = 0xffffffff
    h = (torch.arange(B * kv * cap * hd, device=DEV, dtype=torch.int64) * 2654435761 & m32) ^ ((seed & 0xffffff) + 2 * layer + which)
    h = h ^ (h >> 16)
    h = h * 0x85ebca6b & m32
    h = h ^ (h >> 13)
    h = h * 0xc2b2ae35 & m32
    h = h ^ (h >> 16)
    x = ((h & 0xffff).float() / 32768.0 - 1.0).to(DT[case["dtype"]])
    return x.view(B, kv, cap, hd)[:, :, :case["ctx"]].double()


def _dense_block(cfg, sd, i, x, pos0, past):
    """x (B, S, H) -> (y, K, V); past: cached K and V (B, kv, pos0, hd) or None."""
    p = cfg.layer_name(i) + "."
    B, S, H = x.shape
    nh, nk, hd = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.hd
    h = _rms(x, sd[p + "input_layernorm.weight"], cfg.rms_norm_eps)
    q, k, v = ((h @ sd[p + "self_attn.%s_proj.weight" % n].t()).view(B, S, -1, hd).transpose(1, 2) for n in "qkv")
    if cfg.use_qk_norm:
        q, k = _rms(q, sd[p + "self_attn.q_norm.weight"], cfg.rms_norm_eps), _rms(k, sd[p + "self_attn.k_norm.weight"], cfg.rms_norm_eps)
    a = _angles(torch.arange(pos0, pos0 + S, device=DEV), hd, cfg.rope_theta)
    q, k = _turn(q, a.cos(), a.sin()), _turn(k, a.cos(), a.sin())
    if past is not None:
        k, v = torch.cat([past[0], k], 2), torch.cat([past[1], v], 2)
    o = torch.empty(B, S, nh, hd, device=DEV, dtype=torch.float64)
    for b in range(B):
        o[b] = _softmax_pv(q[b], k[b].repeat_interleave(nh // nk, 0), v[b].repeat_interleave(nh // nk, 0), hd ** -0.5, pos0).transpose(0, 1)
    x = x + o.view(B, S, nh * hd) @ sd[p + "self_attn.o_proj.weight"].t()
    h = _rms(x, sd[p + "post_attention_layernorm.weight"], cfg.rms_norm_eps)
    for b in range(B):   # a batch row at a time: the wide intermediate of all rows at once would not fit beside the weights
        x[b] += (_silu(h[b] @ sd[p + "mlp.gate_proj.weight"].t()) * (h[b] @ sd[p + "mlp.up_proj.weight"].t())) @ sd[p + "mlp.down_proj.weight"].t()
    return x, k, v


def _nigenex_layer(cfg, sd, i, x):
    sp, p = cfg.layers[i], cfg.layer_name(i) + "."
    B, S, W = x.shape
    H, G, D = sp.heads, sp.kv_heads, sp.head_dim
    h = _rms(x, sd[p + "norm1"], cfg.rms_norm_eps)
    hs = h + (torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1) - h) * sd[p + "shift"]
    q = (hs @ sd[p + "mix.q"].t()).view(B, S, H, D).transpose(1, 2)
    k = (hs @ sd[p + "mix.k"].t()).view(B, S, G, D).transpose(1, 2).repeat_interleave(H // G, 1)
    r1, r2 = sd[p + "mix.r1"][:, None, None], sd[p + "mix.r2"][:, None, None]
    score = lambda s, n: sp.softcap * torch.tanh(s / sp.softcap) - r1 * torch.log(1 + r2 * n)  # noqa: E731
    o = torch.stack([_softmax_pv(q[b], k[b], k[b], sp.scale, 0, sp.window, score) for b in range(B)]).transpose(1, 2)
    o = o * torch.sigmoid(hs @ sd[p + "mix.g"].t())[..., None]
    u = torch.nn.functional.gelu(h @ sd[p + "mlp.gate"].t(), approximate="tanh") * (h @ sd[p + "mlp.up"].t())
    return x + o.reshape(B, S, H * D) @ sd[p + "mix.o"].t() + u @ sd[p + "mlp.down"].t()


def _scan(decay, k, v, q):
    """S <- decay S + k v^T, o = S^T q over time: decay (T, H), k and q (T, H, D), v (T, H, V)."""
    S = torch.zeros(k.shape[1], k.shape[2], v.shape[2], device=DEV, dtype=torch.float64)
    o = torch.empty_like(v)
    for t in range(k.shape[0]):
        S = torch.baddbmm(S * decay[t][:, None, None], k[t][:, :, None], v[t][:, None, :])
        o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
    return o


def _setodra_mixer(cfg, sd, i, h):
    """h (T, W): one sequence."""
    sp, p, T = cfg.layers[i], cfg.layer_name(i) + ".mix.", h.shape[0]
    pos = torch.arange(T, device=DEV)
    if sp.type == "retention":
        H, D = sp.heads, sp.dim
        a = _angles(pos, D, sp.rot.base)
        q, k = (_turn((h @ sd[p + n].t()).view(T, H, D).transpose(0, 1), a.cos(), a.sin()).transpose(0, 1) for n in "qk")
        o = _scan(torch.tensor(sp.decay, device=DEV, dtype=torch.float64).expand(T, H), k * D ** -0.5, (h @ sd[p + "v"].t()).view(T, H, sp.vdim), q)
        return (_rms(o, None, cfg.rms_norm_eps).reshape(T, sp.inner) * _silu(h @ sd[p + "g"].t())) @ sd[p + "o"].t()
    if sp.type == "mamba2":
        H, N, G, I = sp.heads, sp.state, sp.groups, sp.inner
        u = h @ sd[p + "in"].t()
        z, c, dt = u[:, :I], u[:, I:2 * I + 2 * G * N], u[:, 2 * I + 2 * G * N:]
        pad = torch.cat([torch.zeros(sp.conv - 1, c.shape[1], device=DEV, dtype=torch.float64), c])
        c = _silu(sum(pad[j:j + T] * sd[p + "conv"][:, j] for j in range(sp.conv)) + sd[p + "conv.b"])
        x = c[:, :I].view(T, H, sp.vdim)
        Bm, Cm = (c[:, I + j * G * N:I + (j + 1) * G * N].view(T, G, N).repeat_interleave(H // G, 1) for j in (0, 1))
        dt = torch.nn.functional.softplus(dt + sd[p + "dt_bias"])
        o = _scan(torch.exp(-torch.exp(sd[p + "A_log"]) * dt), Bm * dt[..., None], x, Cm) + sd[p + "D"][:, None] * x
        y = o.reshape(T, I) * _silu(z)
        return (_rms(y.view(T, sp.norm_groups, -1), None, cfg.rms_norm_eps).reshape(T, I) * sd[p + "norm"]) @ sd[p + "o"].t()
    H, D, R, C, r = sp.heads, sp.dim, sp.rot_dim, sp.kv_rank, sp.rot
    i2 = torch.arange(R // 2, device=DEV, dtype=torch.float64)
    pair = lambda turns: R * math.log(r.original / (2 * math.pi * turns)) / (2 * math.log(r.base))  # noqa: E731
    lo, hi = max(math.floor(pair(r.fast)), 0), min(math.ceil(pair(r.slow)), R - 1)
    ramp = ((i2 - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f = r.base ** (-2.0 * i2 / R)
    a = pos.double()[:, None] * (f / r.factor * ramp + f * (1 - ramp))[None]
    amp = 0.1 * math.log(r.factor) + 1.0
    q = (h @ sd[p + "q"].t()).view(T, H, D + R).transpose(0, 1)
    kv = h @ sd[p + "dkv"].t()
    c = _rms(kv[:, :C], sd[p + "dkv.norm"], cfg.rms_norm_eps)
    kr = _turn(kv[:, C:], a.cos() * amp, a.sin() * amp)
    q = torch.cat([q[..., :D], _turn(q[..., D:], a.cos() * amp, a.sin() * amp)], -1)
    k = torch.cat([(c @ sd[p + "uk"].t()).view(T, H, D).transpose(0, 1), kr[None].expand(H, T, R)], -1)
    v = (c @ sd[p + "uv"].t()).view(T, H, sp.vdim).transpose(0, 1)
    return _softmax_pv(q, k, v, sp.scale, 0).transpose(0, 1).reshape(T, sp.inner) @ sd[p + "o"].t()


def _routed(cfg, sd, i, h):
    mo, p = cfg.layers[i].moe, cfg.layer_name(i) + ".mlp."
    ff = lambda x, e: (_silu(x @ sd[p + e + ".gate"].t()) * (x @ sd[p + e + ".up"].t())) @ sd[p + e + ".down"].t()  # noqa: E731
    s = torch.softmax(h @ sd[p + "router"].t(), -1)
    chosen = torch.topk(s + sd[p + "correction"], mo.top, dim=-1).indices
    w = torch.gather(s, 1, chosen)
    w = w / (w.sum(-1, keepdim=True) + 1e-20) * mo.scale
    out = torch.sigmoid(h @ sd[p + "shared.sg"].t()) * ff(h, "shared")
    for e in range(mo.experts + mo.identity):
        row, col = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            x = h[row]
            out[row] += w[row, col][:, None] * (x if e >= mo.experts else ff(x, "e%d" % e))
    return out


def exact(case, seed):
    kind, dt = case["kind"], DT.get(case["dtype"])
    if kind == "sample":
        x, p = _raw_logits(case, seed).double(), case["penalty"]
        at = torch.tensor(sorted(set(_penalised(case, seed))), device=DEV)
        x[at] = torch.where(x[at] >= 0, x[at] / p, x[at] * p)
        return {"logits": x, "token": None}   # the draw depends on the framework's own random numbers
    if kind == "head":
        cfg = DENSE[case["model"]]()
        sd, p = _dense_head(cfg, dt), cfg.model_prefix
        x = torch.randn((case["batch"], 1, cfg.hidden_size), generator=_rng(seed), device=DEV).to(dt).double()[:, 0]
        w = sd.get("lm_head.weight", sd[p + ".embed_tokens.weight"])
        h = _rms(x, sd[p + ".norm.weight"].double(), cfg.rms_norm_eps)
        return torch.cat([h @ w[a:a + 16384].double().t() for a in range(0, cfg.vocab_size, 16384)], 1)
    if kind == "block":
        cfg = DENSE[case["model"]]()
        x = _rows(case, seed, cfg.hidden_size, dt)[0].double()
        for i in range(case["layers"]):
            past = [_synthetic(case, cfg, i, seed, w) for w in (0, 1)] if case["ctx"] else None
            x = _dense_block(cfg, _d(_dense_layer(cfg, i, dt)), i, x, case["ctx"], past)[0]
        return x
    if kind == "generate":
        cfg = DENSE[case["model"]]()
        sd = _d(_dense_head(cfg, dt))
        for i in range(cfg.num_hidden_layers):
            sd.update(_d(_dense_layer(cfg, i, dt)))
        p, ids, past = cfg.model_prefix, _prompt_ids(case, seed), {}
        feed, pos, tokens, logits = ids, 0, [], []
        for _ in range(case["tokens"]):
            x = sd[p + ".embed_tokens.weight"][torch.tensor(feed, device=DEV)][None]
            for i in range(cfg.num_hidden_layers):
                x, k, v = _dense_block(cfg, sd, i, x, pos, past.get(i))
                past[i] = (k, v)
            pos += len(feed)
            lg = _rms(x[0, -1], sd[p + ".norm.weight"], cfg.rms_norm_eps) @ sd[p + ".embed_tokens.weight"].t()
            if tokens:
                at = torch.tensor(sorted(set(tokens)), device=DEV)
                lg[at] = torch.where(lg[at] >= 0, lg[at] / 1.1, lg[at] * 1.1)
            logits.append(lg)
            tokens.append(int(lg.argmax()))
            feed = tokens[-1:]
        return {"logits": logits, "tokens": np.array(tokens)}
    cfg = _nigenex_cfg(case) if kind == "nigenex" else _setodra_cfg(case)
    sd = _d(_nigenex_weights(cfg, dt) if kind == "nigenex" else _setodra_weights(cfg, dt))
    x, pre = _rows(case, seed, cfg.hidden_size, torch.float32)
    x = (x if pre is None else torch.cat([pre, x], 1)).double()
    for i in range(len(cfg.layers)):
        if kind == "nigenex":
            x = _nigenex_layer(cfg, sd, i, x)
        else:
            y = []
            for b in range(x.shape[0]):
                z = x[b] + _setodra_mixer(cfg, sd, i, _rms(x[b], sd[cfg.layer_name(i) + ".norm1"], cfg.rms_norm_eps))
                y.append(z + _routed(cfg, sd, i, _rms(z, sd[cfg.layer_name(i) + ".norm2"], cfg.rms_norm_eps)))
            x = torch.stack(y)
    return x[:, case["ctx"]:].contiguous()
