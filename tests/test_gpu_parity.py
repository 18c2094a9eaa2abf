"""GPU parity tests proper: the CUDA path, called through the C ABI, against the CPU oracle on the
same seeded inputs.  Scenarios follow the reference's own block/attention/cache tests
(tests/unit_tests/test_blocks.rs:877-933, test_attention.rs:12-143, test_cache.rs:77-96) — which assert
shapes/determinism only — plus the numeric comparison the reference never had.

Tolerance: floating point, dtype D in {bf16, f16}.  GPU and oracle
round at the same points but accumulate fp32 sums in different orders, so a value that lands near a
rounding boundary can differ by 1 ulp of D and the flip propagates.  Bars:
  one block:            max |err| <= 3 ulp of D at the tensor's scale (tests/util.py ulp_at_scale), i.e.
                        bf16: 3 * 2^-7 * 2^floor(log2 max|ref|), f16: 3 * 2^-10 * ...; mean |err| <= 0.25 ulp
  final logits (<=4 layers): <= 4 ulp;  greedy token ids: bit-exact whenever the oracle's top-1/top-2
  margin exceeds the logit tolerance (margins are printed; flips inside the margin are reported).
"""
import numpy as np
import pytest
import torch

from cake_b200.config import reference_test_config
from oracle import oracle as O
from tests.util import checkpoint, max_ulp_err, mean_ulp_err, medium_config, rand_x, to_np

pytestmark = pytest.mark.gpu

BLOCK_TOL_ULP = 3.0   # measured on hardware: 1-2 ulp
LOGIT_TOL_ULP = 4.0   # <= 4 layers; measured <= 3 (the 32-layer bar is derived from the order sensitivity, test_gpu_l8_full.py)


def _ctx(cfg, sd, dtype, max_seq=None):
    from cake_b200.model import Context
    return Context(cfg, sd, dtype, device=0, max_seq=max_seq)


def _llama31_scaling():
    from cake_b200.config import RopeScaling
    # Llama-3.1 style scaling (cache.rs:49-80) with a short original context so that all three frequency bands
    # (kept / interpolated / divided by the factor) occur within head_dim 64
    return RopeScaling(factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0, original_max_position_embeddings=64, rope_type="llama3")


CONFIGS = {
    # an active sliding window (cache.rs:173-205; bites from the second decode step on), the GELU MLP
    "medium_window": lambda: medium_config(sliding_window=5),
    "medium_gelu": lambda: medium_config(use_gelu_mlp=True),
    "medium_rope_llama3": lambda: medium_config(rope_scaling=_llama31_scaling(), rope_theta=10000.0),
    "ref_tiny": lambda: reference_test_config(),                       # helpers.rs:8-44 (hd=16, GQA 4:2)
    "ref_tiny_qknorm": lambda: reference_test_config(use_qk_norm=True),  # test_blocks.rs:920-933
    "ref_tiny_bias": lambda: reference_test_config(use_qkv_bias=True),   # test_attention.rs bias case
    "medium": lambda: medium_config(),
    "medium_qwen": lambda: medium_config(use_qk_norm=True, tie_word_embeddings=True, rope_theta=1e6, rms_norm_eps=1e-6),
}


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("name", list(CONFIGS))
def test_block_prefill_then_decode_matches_oracle(name, dtype):
    """test_blocks.rs:877-918 scenarios: prefill (1,4,H) @0, then generation (1,1,H) @4, @5, ..."""
    from cake_b200.model import B200Transformer
    cfg = CONFIGS[name]()
    sd = checkpoint(cfg, dtype, seed=21)
    om = O.OracleModel(cfg, sd, dtype)
    oc = om.new_cache()
    ctx = _ctx(cfg, sd, dtype)
    blk = B200Transformer.load(cfg.layer_name(1), ctx)
    x = rand_x((1, 7, cfg.hidden_size), dtype, seed=5)
    # prefill 4
    y_ref = om.block_forward(1, x[0, :4].float().numpy(), 0, oc)
    y = blk.forward(ctx.to_device(x[:, :4]), 0, 1, ctx)
    ctx.sync()
    assert y.shape == (1, 4, cfg.hidden_size)
    e = max_ulp_err(to_np(y[0]), y_ref, dtype)
    assert e <= BLOCK_TOL_ULP, f"prefill: {e} ulp"
    assert mean_ulp_err(to_np(y[0]), y_ref, dtype) <= 0.25
    # decode 3 single tokens at positions 4,5,6 (exercises the decode kernels + in-place KV append)
    for t in range(4, 7):
        y_ref = om.block_forward(1, x[0, t:t + 1].float().numpy(), t, oc)
        y = blk.forward_mut(ctx.to_device(x[:, t:t + 1]), t, 1, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, dtype)
        assert e <= BLOCK_TOL_ULP, f"decode @{t}: {e} ulp"
        assert mean_ulp_err(to_np(y[0]), y_ref, dtype) <= 0.25
    # cache growth (test_cache.rs:77-96) and contents
    assert ctx.cache.len(1) == 7 and ctx.cache.len(0) == 0
    k, v = ctx.cache.kv(1)
    ko, vo = oc.kv(1)
    assert max_ulp_err(to_np(k[0]), ko[:, :7], dtype) <= 2.0
    assert max_ulp_err(to_np(v[0]), vo[:, :7], dtype) <= 2.0
    ctx.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_decode_from_empty_cache(dtype):
    """test_blocks.rs:891-903: generation step at position 0 on an empty cache."""
    from cake_b200.model import B200Transformer
    cfg = medium_config()
    sd = checkpoint(cfg, dtype, seed=3)
    om, ctx = O.OracleModel(cfg, sd, dtype), _ctx(cfg, sd, dtype)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = rand_x((1, 1, cfg.hidden_size), dtype, seed=9)
    y_ref = om.block_forward(0, x[0].float().numpy(), 0, om.new_cache())
    y = blk.forward(ctx.to_device(x), 0, 0, ctx)
    ctx.sync()
    assert max_ulp_err(to_np(y[0]), y_ref, dtype) <= BLOCK_TOL_ULP
    ctx.close()


def test_long_decode_many_attention_splits():
    """Decode at depth: 300 cached positions so every flash-decoding split and a multi-pass tile are used."""
    from cake_b200.model import B200Transformer
    dtype = "bf16"
    cfg = medium_config()
    sd = checkpoint(cfg, dtype, seed=8)
    om, ctx = O.OracleModel(cfg, sd, dtype), _ctx(cfg, sd, dtype)
    oc = om.new_cache()
    blk = B200Transformer.load(cfg.layer_name(2), ctx)
    x = rand_x((1, 304, cfg.hidden_size), dtype, seed=10)
    om.block_forward(2, x[0, :300].float().numpy(), 0, oc)
    blk.forward(ctx.to_device(x[:, :300]), 0, 2, ctx)
    for t in range(300, 304):
        y_ref = om.block_forward(2, x[0, t:t + 1].float().numpy(), t, oc)
        y = blk.forward(ctx.to_device(x[:, t:t + 1]), t, 2, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, dtype)
        assert e <= BLOCK_TOL_ULP, f"decode @{t}: {e} ulp"
    ctx.close()


def test_determinism_bit_equal_across_loads():
    """test_attention.rs determinism: two independent loads give bit-identical outputs."""
    from cake_b200.model import B200Transformer
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=4)
    x = rand_x((1, 6, cfg.hidden_size), "bf16", seed=2)
    outs = []
    for _ in range(2):
        ctx = _ctx(cfg, sd, "bf16")
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        a = blk.forward(ctx.to_device(x[:, :5]), 0, 0, ctx)
        b = blk.forward(ctx.to_device(x[:, 5:6]), 5, 0, ctx)
        ctx.sync()
        outs.append((a.cpu(), b.cpu()))
        ctx.close()
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


def test_forward_batch_equals_per_block_calls():
    """text_model.rs:298-321: a contiguous run through forward_batch == block-by-block forward."""
    from cake_b200.model import B200Transformer
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=6)
    x = rand_x((1, 5, cfg.hidden_size), "bf16", seed=1)
    ctx = _ctx(cfg, sd, "bf16")
    blks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(3)]
    xd = ctx.to_device(x)
    ya = blks[0].forward_batch(xd, [(b.layer_name(), 0, i) for i, b in enumerate(blks)], ctx, blocks=blks)
    ctx.sync()
    ctx.cache.clear()
    yb = xd
    for i, b in enumerate(blks):
        yb = b.forward(yb, 0, i, ctx)
    ctx.sync()
    assert torch.equal(ya, yb)
    ctx.close()


def test_error_behaviour_position_mismatch_and_recovery():
    """Errors are returned, not fatal (worker.rs:490-503 keeps the connection): a forward at the wrong
    position fails with a message; after cache.clear() the block works again."""
    from cake_b200.capi import CakeB200Error
    from cake_b200.model import B200Transformer
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=6)
    ctx = _ctx(cfg, sd, "bf16")
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = ctx.to_device(rand_x((1, 1, cfg.hidden_size), "bf16", seed=1))
    with pytest.raises(CakeB200Error, match="cache length"):
        blk.forward(x, 3, 0, ctx)
    blk.forward(x, 0, 0, ctx)
    ctx.cache.clear()
    blk.forward(x, 0, 0, ctx)
    ctx.sync()
    with pytest.raises(KeyError):
        B200Transformer.load("model.layers.99", ctx)
    ctx.close()


@pytest.mark.parametrize("name,dtype", [("medium", "bf16"), ("medium_qwen", "bf16"), ("ref_tiny", "f16")])
def test_model_logits_and_greedy_tokens_match_oracle(name, dtype):
    """TextModelBase::forward (text_model.rs:266-368) vs the oracle, teacher-forced on the oracle's greedy
    sequence so that one near-tie flip cannot hide or fake later errors: per-step logits within
    LOGIT_TOL_ULP; the greedy token (text_model.rs:104-105) must equal the oracle's whenever the oracle's
    top-1/top-2 margin exceeds twice the logit tolerance — flips inside the margin are reported."""
    from cake_b200.model import TextModelBase
    from tests.util import ulp_at_scale
    cfg = CONFIGS[name]()
    sd = checkpoint(cfg, dtype, seed=33, peaked=True)
    om = O.OracleModel(cfg, sd, dtype)
    prompt = np.random.default_rng(7).integers(0, cfg.vocab_size, 9).tolist()
    ref_toks, ref_logits = om.generate(prompt, 12)
    ctx = _ctx(cfg, sd, dtype)
    model = TextModelBase.load(ctx)
    feeds = [prompt] + [[t] for t in ref_toks[:-1]]
    pos, worst, flips = 0, 0.0, []
    for step, ids in enumerate(feeds):
        lg_d = model.forward([ids], pos)
        ctx.sync()
        lg = to_np(lg_d[0])
        pos += len(ids)
        e = max_ulp_err(lg, ref_logits[step], dtype)
        worst = max(worst, e)
        srt = np.sort(ref_logits[step])
        margin = float(srt[-1] - srt[-2])
        tol_abs = LOGIT_TOL_ULP * ulp_at_scale(ref_logits[step], dtype)
        tok = O.argmax(lg)  # same first-max-wins rule applied to the GPU logits
        if tok != ref_toks[step]:
            flips.append((step, margin))
            assert margin <= 2 * tol_abs, f"step {step}: token {tok} != {ref_toks[step]} with margin {margin}"
    print(f"{name}/{dtype}: worst logits err {worst:.2f} ulp over {len(feeds)} steps; flips inside margin: {flips}")
    assert worst <= LOGIT_TOL_ULP
    ctx.close()


def test_greedy_generation_token_ids_bit_exact():
    """Master::generate_text greedy loop (master.rs:131-155): with a peaked head (large margins) the token
    ids must be bit-exact against the oracle's loop, including the device-side argmax."""
    from cake_b200.model import Master, TextModelBase
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=33, peaked=True)
    prompt = np.random.default_rng(7).integers(0, cfg.vocab_size, 9).tolist()
    ref_toks, ref_logits = O.OracleModel(cfg, sd, "bf16").generate(prompt, 16)
    margins = [float(np.sort(l)[-1] - np.sort(l)[-2]) for l in ref_logits]
    ctx = _ctx(cfg, sd, "bf16")
    out = Master(TextModelBase.load(ctx)).generate_text(prompt, 16)
    print("min oracle margin", min(margins))
    assert out["tokens"] == ref_toks
    assert out["generated"] == 16 and out["tok_s"] > 0
    ctx.close()


def test_graph_decode_loop_equals_stepwise_api():
    """The CUDA-graph decode loop (device-resident position/token) must produce exactly the tokens and
    logits of the per-call Forwarder API."""
    from cake_b200.model import TextModelBase
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=12, peaked=True)
    prompt = np.random.default_rng(3).integers(0, cfg.vocab_size, 17).tolist()
    ctx = _ctx(cfg, sd, "bf16")
    model = TextModelBase.load(ctx)
    model.prepare_prompt(prompt)
    step_toks = [model.next_token(i).id for i in range(10)]
    step_logits = model.last_logits.cpu()
    # same thing: prefill through next_token(0), then 9 graph steps
    model.prepare_prompt(prompt)
    t0 = model.next_token(0).id
    model.decode_build()
    toks = [t0] + model.decode_greedy(t0, 9)
    assert toks == step_toks
    out = torch.empty(cfg.vocab_size, dtype=torch.bfloat16)
    from cake_b200.capi import check, lib, ptr
    check(lib().cake_b200_decode_logits(ctx.h, ptr(out), out.numel() * 2))
    assert torch.equal(out, step_logits)
    # host-driven single step (TextModelBase::next_token cadence) continues the same sequence
    from ctypes import byref, c_uint32
    nxt = c_uint32()
    check(lib().cake_b200_decode_step_host(ctx.h, toks[-1], byref(nxt)))
    model.prepare_prompt(prompt)
    ref = [model.next_token(i).id for i in range(11)]
    assert nxt.value == ref[-1]
    ctx.close()


def test_repeat_penalty_matches_oracle():
    """text_model.rs:60-99 on device vs the oracle's restatement."""
    from cake_b200.capi import check, lib, ptr
    from ctypes import byref, c_uint32
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=1)
    ctx = _ctx(cfg, sd, "bf16")
    lg = rand_x((cfg.vocab_size,), "bf16", seed=4, scale=3.0)
    toks = [5, 9, 5, 700, 1023]
    ref = O.repeat_penalty(lg.float().numpy(), 1.1, toks, "bf16")
    d = ctx.to_device(lg)
    out = c_uint32()
    arr = (c_uint32 * len(toks))(*toks)
    check(lib().cake_b200_repeat_penalty_argmax(ctx.h, ptr(d), 1.1, arr, len(toks), byref(out)))
    assert np.array_equal(to_np(d), ref)
    assert out.value == O.argmax(ref)
    ctx.close()


def test_megakernel_equals_per_op_kernels(monkeypatch):
    """The persistent decode megakernel (decode_mega.cuh) and the per-op kernel chain (gemv.cuh +
    attn_decode.cuh, CAKE_B200_PER_OP=1) implement the same arithmetic with the same rounding points; only
    the fp32 summation order inside a dot product differs (lanes and warps slice K differently), so
    outputs agree to <= 2 ulp of D and greedy tokens (peaked head) are identical."""
    from cake_b200.model import B200Transformer, TextModelBase
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=17, peaked=True)
    x = rand_x((1, 40, cfg.hidden_size), "bf16", seed=3)
    prompt = np.random.default_rng(5).integers(0, cfg.vocab_size, 11).tolist()
    res = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = _ctx(cfg, sd, "bf16")
        blks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(3)]
        batch = [(b.layer_name(), 0, i) for i, b in enumerate(blks)]
        blks[0].forward_batch(ctx.to_device(x[:, :33]), batch, ctx, blocks=blks)
        outs = []
        for t in range(33, 40):
            y = blks[0].forward_batch(ctx.to_device(x[:, t:t + 1]), [(n, t, i) for n, _, i in batch], ctx, blocks=blks)
            ctx.sync()
            outs.append(y.cpu())
        k, v = ctx.cache.kv(2)
        del blks
        ctx.cache.clear()
        model = TextModelBase.load(ctx)
        model.prepare_prompt(prompt)
        t0 = model.next_token(0).id
        model.decode_build()
        toks = [t0] + model.decode_greedy(t0, 8)
        res[mode] = (outs, k, v, toks)
        ctx.close()
    for a, b in zip(res["0"][0], res["1"][0]):
        assert max_ulp_err(to_np(a), to_np(b), "bf16") <= 2.0
    assert max_ulp_err(to_np(res["0"][1]), to_np(res["1"][1]), "bf16") <= 2.0
    assert max_ulp_err(to_np(res["0"][2]), to_np(res["1"][2]), "bf16") <= 2.0
    assert res["0"][3] == res["1"][3]


def test_sliding_window_chunked_prefill_and_long_decode_match_oracle():
    """cache.rs:173-205 through every kernel path: first call (6 tokens, stored and attended in full although the window
    is 5), a second multi-token chunk on the non-empty cache (all its queries see the same surviving old rows), then
    decode steps far past the window (several flash-decoding splits over the visible rows only)."""
    from cake_b200.model import B200Transformer
    dtype = "bf16"
    cfg = medium_config(sliding_window=5)
    sd = checkpoint(cfg, dtype, seed=12)
    om, ctx = O.OracleModel(cfg, sd, dtype), _ctx(cfg, sd, dtype)
    oc = om.new_cache()
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = rand_x((1, 40, cfg.hidden_size), dtype, seed=13)
    pos = 0
    for n in (6, 3, 1, 1, 2, 1) + (1,) * 26:
        y_ref = om.block_forward(0, x[0, pos:pos + n].float().numpy(), pos, oc)
        y = blk.forward(ctx.to_device(x[:, pos:pos + n]), pos, 0, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, dtype)
        assert e <= BLOCK_TOL_ULP, f"{n} token(s) @ {pos}: {e} ulp"
        pos += n
    # a chunk longer than the window on a non-empty cache is an error, not a silent mis-trim
    with pytest.raises(Exception, match="sliding window"):
        blk.forward(ctx.to_device(x[:, :7]), pos, 0, ctx)
    ctx.close()


def test_embed_scale_residual_norm_and_gelu_through_the_model():
    """text_model.rs:274-276 embed_scale, config.rs:155-173 residual RMS-norm weights ((1 + w) at load) and the GELU MLP
    through TextModelBase: host-stepped logits and the decode graph against the oracle."""
    from cake_b200.model import Context, TextModelBase
    cfg = medium_config(use_gelu_mlp=True, embed_scale=22.627416997969522, residual_rms_norm=True, use_qk_norm=True, num_hidden_layers=2)
    sd = checkpoint(cfg, "bf16", seed=77, peaked=True)
    for k in list(sd):   # residual checkpoints store norm weights as deltas around 0
        if k.endswith("norm.weight") or k.endswith("layernorm.weight"):
            sd[k] = (sd[k].float() - 1.0).to(sd[k].dtype)
    om = O.OracleModel(cfg, sd, "bf16", max_seq=64)
    prompt = [3, 700, 41, 9, 256]
    ref_toks, ref_logits = om.generate(prompt, 8)
    ctx = Context(cfg, sd, "bf16", device=0, max_seq=64)
    m = TextModelBase.load(ctx)
    m.prepare_prompt(prompt)
    t0 = m.next_token(0)
    assert max_ulp_err(to_np(m.last_logits), ref_logits[0], "bf16") <= LOGIT_TOL_ULP and t0.id == ref_toks[0]
    m.decode_build()
    assert [t0.id] + m.decode_greedy(t0.id, 7) == list(ref_toks)
    ctx.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_tcgen05_prefill_attention_head_dim_128_shapes(dtype):
    """attn_prefill_tc.cuh (head_dim 128 takes the tcgen05 path) against the oracle on the shapes that stress its tiling:
    a ragged query tile (200 = 128 + 72 rows: zero-filled Q rows, unwritten keys past the visible length), batch 2 with
    GQA 4:2, a second chunk on a non-empty cache (pos0 > 0, diagonal tiles not aligned to the 64-key tiles), and a
    sliding window that moves the K/V base of the chunk (cache.rs:173-205)."""
    from cake_b200.model import B200Transformer
    for window, chunks in ((None, (200, 77, 130)), (96, (200, 50, 90))):
        kw = dict(head_dim=128, num_attention_heads=4, num_key_value_heads=2)
        if window:
            kw["sliding_window"] = window
        cfg = medium_config(**kw)
        sd = checkpoint(cfg, dtype, seed=31)
        om, ctx = O.OracleModel(cfg, sd, dtype), _ctx(cfg, sd, dtype)
        from cake_b200.model import Cache
        ctx.cache = Cache(ctx, 2, cfg.max_seq_len)
        ocs = [om.new_cache(), om.new_cache()]
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        x = rand_x((2, sum(chunks), cfg.hidden_size), dtype, seed=32)
        pos = 0
        for n in chunks:
            y = blk.forward(ctx.to_device(x[:, pos:pos + n]), pos, 0, ctx)
            ctx.sync()
            for b in range(2):
                y_ref = om.block_forward(0, x[b, pos:pos + n].float().numpy(), pos, ocs[b])
                e = max_ulp_err(to_np(y[b]), y_ref, dtype)
                assert e <= BLOCK_TOL_ULP, f"window {window}, batch row {b}, {n} tokens @ {pos}: {e} ulp"
            pos += n
        ctx.close()


SIBLINGS = {
    # models/olmo2/block.rs:62-90 + attention.rs:176-192: no pre-norms, post-norms, QK-norm over the whole projection
    "olmo2": dict(block_kind="olmo2", use_qk_norm=True, pre_reshape_qk_norm=True),
    # models/gemma3/block.rs:60-135: four norms with (1 + w) weights, gelu MLP, scaled embeddings, tied head; local layers
    # (0, 2): window 5, NO RoPE; global layers (1, 3): full context + RoPE
    "gemma3": dict(block_kind="gemma3", use_qk_norm=True, residual_rms_norm=True, use_gelu_mlp=True, tie_word_embeddings=True,
                   embed_scale=22.627416997969522, sliding_window=5, global_layers=[False, True, False, True]),
    # models/exaone4/block.rs:50-110: the standard pre-norm block; local layers: window 5 + RoPE, global: full context, NO RoPE
    "exaone4": dict(block_kind="exaone4", use_qk_norm=True, sliding_window=5, global_layers=[False, True, False, True]),
}


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("kind", list(SIBLINGS))
def test_sibling_block_structures_match_oracle(kind, dtype):
    """The OLMo2 / Gemma3 / EXAONE4 blocks (cake_b200_block_set_variant + pre-reshape QK-norm) through the model: a prompt
    that fits the local window, then host-stepped tokens far past it (single-token steps of these blocks go through the
    batched path), logits and greedy tokens against the oracle; then every block on a multi-token second chunk."""
    from cake_b200.model import B200Transformer, Context, TextModelBase
    from cake_b200.synth import residual_deltas
    from cake_b200.capi import CakeB200Error
    from tests.util import ulp_at_scale
    cfg = medium_config(num_hidden_layers=4, **SIBLINGS[kind])
    sd = checkpoint(cfg, dtype, seed=91, peaked=not cfg.tie_word_embeddings)
    if cfg.residual_rms_norm:
        sd = residual_deltas(sd)
    om = O.OracleModel(cfg, sd, dtype, max_seq=64)
    prompt = [3, 700, 41, 9, 256]
    ref_toks, ref_logits = om.generate(prompt, 14)
    ctx = Context(cfg, sd, dtype, device=0, max_seq=64)
    m = TextModelBase.load(ctx)
    with pytest.raises(CakeB200Error, match="sibling block structure"):
        m.decode_build()   # the decode graph covers the standard block only
    m.prepare_prompt(prompt)
    for i in range(14):    # teacher-forced on the oracle's greedy sequence
        t = m.next_token(i)
        e = max_ulp_err(to_np(m.last_logits), ref_logits[i], dtype)
        assert e <= LOGIT_TOL_ULP, f"{kind} step {i}: logits {e} ulp"
        top2 = np.sort(ref_logits[i])[-2:]
        if top2[1] - top2[0] > 2 * LOGIT_TOL_ULP * ulp_at_scale(ref_logits[i], dtype):
            assert t.id == ref_toks[i], f"{kind} step {i}: token {t.id} != {ref_toks[i]}"
        m.tokens[-1] = int(ref_toks[i])
    # block level: 4 tokens, then a 3-token chunk on the non-empty cache (<= the window), then single tokens
    x = rand_x((1, 12, cfg.hidden_size), dtype, seed=92)
    for layer in range(4):
        ctx.cache.clear()
        oc = om.new_cache()
        blk = m.blocks[layer]
        pos = 0
        for n in (4, 3, 1, 1, 2, 1):
            y_ref = om.block_forward(layer, x[0, pos:pos + n].float().numpy(), pos, oc)
            y = blk.forward(ctx.to_device(x[:, pos:pos + n]), pos, layer, ctx)
            ctx.sync()
            e = max_ulp_err(to_np(y[0]), y_ref, dtype)
            assert e <= BLOCK_TOL_ULP, f"{kind} layer {layer}: {n} token(s) @ {pos}: {e} ulp"
            pos += n
    ctx.close()
