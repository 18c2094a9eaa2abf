"""Parity at full layer dimensions (Llama-3-8B: H=4096, I=14336, 32/8 heads of 128), where every
kernel runs with its production geometry (32 KB TMA stages, 16-warp megakernel slices, 128x128 UMMA tiles, 64x64
flash tiles): one block against the oracle, plus size-independent properties at depth."""
import numpy as np
import pytest
import torch

from cake_b200.config import llama3_8b
from cake_b200.synth import make_layer
from oracle import oracle as O
from tests.util import max_ulp_err, mean_ulp_err, rand_x, to_np

pytestmark = pytest.mark.gpu


def _ctx(cfg, sd, max_seq):
    from cake_b200.model import Context
    return Context(cfg, sd, "bf16", device=0, max_seq=max_seq)


def test_llama3_8b_block_matches_oracle_prefill_and_decode():
    from cake_b200.model import B200Transformer
    cfg = llama3_8b(max_seq=256)
    cfg.num_hidden_layers = 1
    sd = make_layer(cfg, 0, "bf16", seed=77)
    om = O.OracleModel(cfg, sd, "bf16", max_seq=256)
    oc = om.new_cache(256)
    ctx = _ctx(cfg, sd, 256)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = rand_x((1, 52, cfg.hidden_size), "bf16", seed=6)
    y_ref = om.block_forward(0, x[0, :48].float().numpy(), 0, oc)      # prefill: tcgen05 GEMMs + flash attention
    y = blk.forward(ctx.to_device(x[:, :48]), 0, 0, ctx)
    ctx.sync()
    e = max_ulp_err(to_np(y[0]), y_ref, "bf16")
    print(f"L8 block prefill(48): max {e:.2f} ulp, mean {mean_ulp_err(to_np(y[0]), y_ref, 'bf16'):.3f} ulp")
    assert e <= 3.0 and mean_ulp_err(to_np(y[0]), y_ref, "bf16") <= 0.25
    for t in range(48, 52):                                             # decode: persistent megakernel
        y_ref = om.block_forward(0, x[0, t:t + 1].float().numpy(), t, oc)
        y = blk.forward(ctx.to_device(x[:, t:t + 1]), t, 0, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, "bf16")
        assert e <= 3.0, f"decode @{t}: {e} ulp"
    k, v = ctx.cache.kv(0)
    ko, vo = oc.kv(0)
    assert max_ulp_err(to_np(k[0]), ko[:, :52], "bf16") <= 2.0
    assert max_ulp_err(to_np(v[0]), vo[:, :52], "bf16") <= 2.0
    ctx.close()


def test_llama3_8b_decode_equals_prefill_at_depth():
    """Size-independent property: the hidden state of position t computed by token-by-token decode (megakernel,
    flash-decoding over 1200+ cached rows, several K/V tiles per split) equals the one computed by a one-shot
    causal prefill (tcgen05 GEMM + flash prefill) — two disjoint kernel paths, same arithmetic."""
    from cake_b200.model import B200Transformer
    cfg = llama3_8b(max_seq=1536)
    cfg.num_hidden_layers = 2
    sd = {}
    for i in range(2):
        sd.update(make_layer(cfg, i, "bf16", seed=5))
    ctx = _ctx(cfg, sd, 1536)
    blks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(2)]
    batch = lambda pos: [(b.layer_name(), pos, i) for i, b in enumerate(blks)]
    # 1280 rows = 10 m-tiles: every projection has >= 148 tiles of 128 x 256, so all three epilogues of the large-tile
    # tcgen05 GEMM (plain, +residual, silu*mul) are on this path; 632 rows (5 m-tiles) keep qkv / o / down on 128 x 128
    x = ctx.to_device(rand_x((1, 1280, cfg.hidden_size), "bf16", seed=9))
    full = blks[0].forward_batch(x, batch(0), ctx, blocks=blks)         # one-shot prefill of 1280
    ctx.sync()
    full = full.cpu()
    ctx.cache.clear()
    blks[0].forward_batch(x[:, :632], batch(0), ctx, blocks=blks)       # prefill 632 ...
    blks[0].forward_batch(x[:, 632:1272], batch(632), ctx, blocks=blks)  # ... a second chunk on the non-empty cache, then decode 8
    for t in range(1272, 1280):
        y = blks[0].forward_batch(x[:, t:t + 1], batch(t), ctx, blocks=blks)
        ctx.sync()
        e = max_ulp_err(to_np(y[0, 0]), to_np(full[0, t]), "bf16")
        assert e <= 3.0, f"position {t}: {e} ulp"
    # determinism of the whole path: a second identical run is bit-equal
    ctx.cache.clear()
    again = blks[0].forward_batch(x, batch(0), ctx, blocks=blks)
    ctx.sync()
    assert torch.equal(again.cpu(), full)
    ctx.close()


def test_qwen3_0_6b_config0_f16_greedy_against_oracle():
    """The smallest workload — "Qwen3-0.6B ... greedy decode 32 tokens from one prompt (reference runs this
    today)" — at the real widths (H=1024, I=3072, 16/8 heads of 128, per-head QK-norm, tied 151 936-row head, the
    reference's default dtype f16, cake/mod.rs:75) with 4 of the 28 layers so the oracle stays fast.  Teacher-forced
    on the oracle's greedy sequence: per-step logits within tolerance; the greedy token must match wherever the
    oracle's top-1/top-2 margin exceeds twice the tolerance."""
    from cake_b200.config import qwen3_0_6b
    from cake_b200.model import TextModelBase
    from cake_b200.synth import make_checkpoint
    from tests.util import ulp_at_scale
    cfg = qwen3_0_6b(max_seq=128)
    cfg.num_hidden_layers = 4
    sd = make_checkpoint(cfg, "f16", seed=2024, std=0.03)
    om = O.OracleModel(cfg, sd, "f16", max_seq=128)
    prompt = np.random.default_rng(1).integers(0, cfg.vocab_size, 6).tolist()
    ref_toks, ref_logits = om.generate(prompt, 32)
    ctx = _ctx_dtype(cfg, sd, "f16", 128)
    model = TextModelBase.load(ctx)
    feeds = [prompt] + [[t] for t in ref_toks[:-1]]
    pos, worst, flips = 0, 0.0, 0
    for step, ids in enumerate(feeds):
        lg = model.forward([ids], pos)
        ctx.sync()
        lg = to_np(lg[0])
        pos += len(ids)
        e = max_ulp_err(lg, ref_logits[step], "f16")
        worst = max(worst, e)
        srt = np.sort(ref_logits[step])
        margin = float(srt[-1] - srt[-2])
        if O.argmax(lg) != ref_toks[step]:
            flips += 1
            assert margin <= 2 * 4.0 * ulp_at_scale(ref_logits[step], "f16"), f"step {step}: token flip with margin {margin}"
    print(f"Qwen3-0.6B-shaped f16: worst logits err {worst:.2f} ulp over 32 greedy steps, in-margin flips {flips}")
    assert worst <= 4.0
    # and the whole greedy loop through the decode graph reproduces its own step-wise tokens
    model.prepare_prompt(prompt)
    a = [model.next_token(i).id for i in range(8)]
    model.prepare_prompt(prompt)
    t0 = model.next_token(0).id
    model.decode_build()
    assert [t0] + model.decode_greedy(t0, 7) == a
    ctx.close()


def _ctx_dtype(cfg, sd, dtype, max_seq):
    from cake_b200.model import Context
    return Context(cfg, sd, dtype, device=0, max_seq=max_seq)


def test_llama3_70b_layer_geometry_matches_oracle():
    """Llama-3-70B layer dimensions (H=8192, I=28672, 64/8 heads of 128 -> G=8): rows of 16 KB / 56 KB,
    i.e. the 2-row and the split-row (2 x 28 KB) stage geometries of the megakernel, and 8 query heads per kv head."""
    from cake_b200.config import llama3_70b
    from cake_b200.model import B200Transformer
    cfg = llama3_70b(max_seq=128)
    cfg.num_hidden_layers = 1
    sd = make_layer(cfg, 0, "bf16", seed=70)
    om = O.OracleModel(cfg, sd, "bf16", max_seq=128)
    oc = om.new_cache(128)
    ctx = _ctx(cfg, sd, 128)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = rand_x((1, 20, cfg.hidden_size), "bf16", seed=3)
    y_ref = om.block_forward(0, x[0, :17].float().numpy(), 0, oc)
    y = blk.forward(ctx.to_device(x[:, :17]), 0, 0, ctx)
    ctx.sync()
    assert max_ulp_err(to_np(y[0]), y_ref, "bf16") <= 3.0
    for t in range(17, 20):
        y_ref = om.block_forward(0, x[0, t:t + 1].float().numpy(), t, oc)
        y = blk.forward(ctx.to_device(x[:, t:t + 1]), t, 0, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, "bf16")
        assert e <= 3.0, f"decode @{t}: {e} ulp"
    ctx.close()


def test_llama3_8b_decode_at_2500_context_multi_tile_attention():
    """Decode at KV length 2500+ (beyond 18 splits x 128 rows): every flash-decoding split walks more than one K/V
    tile, the online-softmax rescaling between tiles is exercised, and the appended row lands in a later tile.  The
    cache is filled with the library's synthetic pattern, read back, and handed to the oracle."""
    from cake_b200.model import B200Transformer, Cache
    cfg = llama3_8b(max_seq=2600)
    cfg.num_hidden_layers = 1
    sd = make_layer(cfg, 0, "bf16", seed=31)
    ctx = _ctx(cfg, sd, 2600)
    ctx.cache = Cache(ctx, 1, 2600)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    L0 = 2500
    ctx.cache.fill_synthetic([0], L0, seed=11)
    ctx.sync()
    k, v = ctx.cache.kv(0)
    om = O.OracleModel(cfg, sd, "bf16", max_seq=2600)
    oc = om.new_cache(2600)
    ko, vo = oc.kv(0)
    ko[:, :L0] = k[0].float().numpy()
    vo[:, :L0] = v[0].float().numpy()
    oc.set_len(0, L0)
    x = rand_x((1, 3, cfg.hidden_size), "bf16", seed=8)
    for i in range(3):
        y_ref = om.block_forward(0, x[0, i:i + 1].float().numpy(), L0 + i, oc)
        y = blk.forward(ctx.to_device(x[:, i:i + 1]), L0 + i, 0, ctx)
        ctx.sync()
        e = max_ulp_err(to_np(y[0]), y_ref, "bf16")
        assert e <= 3.0, f"decode @{L0 + i}: {e} ulp"
    ctx.close()


def test_llama3_8b_block_batch_gt_1_matches_oracle_per_sequence():
    """The Forwarder's (b, s, H) contract with b > 1 at the Llama-3-8B layer widths — a
    (2, 144, H) prefill (tcgen05 GEMMs over 288 rows, flash attention per sequence) and two (2, 1, H) steps — every
    sequence against its own oracle run."""
    from cake_b200.model import B200Transformer, Cache
    cfg = llama3_8b(max_seq=256)
    cfg.num_hidden_layers = 1
    sd = make_layer(cfg, 0, "bf16", seed=41)
    ctx = _ctx(cfg, sd, 256)
    B, S = 2, 144
    ctx.cache = Cache(ctx, batch=B, max_seq=256)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    om = O.OracleModel(cfg, sd, "bf16", max_seq=256)
    caches = [om.new_cache(256) for _ in range(B)]
    x = rand_x((B, S + 2, cfg.hidden_size), "bf16", seed=12)
    y = blk.forward(ctx.to_device(x[:, :S].contiguous()), 0, 0, ctx)
    ctx.sync()
    for b in range(B):
        ref = om.block_forward(0, x[b, :S].float().numpy(), 0, caches[b])
        e = max_ulp_err(to_np(y[b]), ref, "bf16")
        assert e <= 3.0 and mean_ulp_err(to_np(y[b]), ref, "bf16") <= 0.25, f"prefill seq {b}: {e} ulp"
    for t in (S, S + 1):
        y = blk.forward(ctx.to_device(x[:, t:t + 1].contiguous()), t, 0, ctx)
        ctx.sync()
        for b in range(B):
            ref = om.block_forward(0, x[b, t:t + 1].float().numpy(), t, caches[b])
            e = max_ulp_err(to_np(y[b]), ref, "bf16")
            assert e <= 3.0, f"step @{t} seq {b}: {e} ulp"
    ctx.close()
