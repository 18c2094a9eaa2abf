"""Steps and prompts of a few rows: the sizes at which the products of a block change their kernel or their tiling, against the
oracle with the bars of test_gpu_parity.py (same rounding points, fp32 sums in another order)."""
import ctypes

import numpy as np
import pytest

from cake_b200.capi import check, lib, ptr
from cake_b200.model import B200Transformer, Cache, Context
from oracle import oracle as O
from tests.util import checkpoint, max_ulp_err, mean_ulp_err, medium_config, rand_x, to_np

pytestmark = pytest.mark.gpu

# K = 512 (8 k-blocks), 1088 (17: uneven cuts), N = 768, 512, 2176; head_dim 128 with four query heads per key head
CFG = dict(num_attention_heads=4, num_key_value_heads=1, head_dim=128, intermediate_size=1088)


def _check(y, ref, dtype, what):
    e = max_ulp_err(y, ref, dtype)
    assert e <= 3.0, f"{what}: {e} ulp"
    assert mean_ulp_err(y, ref, dtype) <= 0.25, what


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("rows", [2, 15, 16, 17, 40, 64, 65])
def test_rows_of_one_sequence_and_of_a_batch(rows, dtype):
    cfg = medium_config(**CFG)
    sd = checkpoint(cfg, dtype, seed=31)
    om, ctx = O.OracleModel(cfg, sd, dtype), Context(cfg, sd, dtype)
    blk = B200Transformer.load(cfg.layer_name(1), ctx)
    x = rand_x((1, rows, cfg.hidden_size), dtype, seed=rows)
    y = blk.forward(ctx.to_device(x), 0, 1, ctx)
    ctx.sync()
    _check(to_np(y[0]), om.block_forward(1, x[0].float().numpy(), 0, om.new_cache()), dtype, f"prompt of {rows}")
    ctx.cache = Cache(ctx, rows, 8)   # the same rows as one token each of `rows` sequences
    y = blk.forward(ctx.to_device(x.transpose(0, 1)), 0, 1, ctx)
    ctx.sync()
    y = to_np(y)
    for b in range(0, rows, max(1, rows // 4)):
        _check(y[b], om.block_forward(1, x[0, b:b + 1].float().numpy(), 0, om.new_cache()), dtype, f"row {b} of a batch of {rows}")
    ctx.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("heads,kv,batch,ctx,seq", [
    (4, 1, 1, 700, 33),    # 4 heads per tile row group, a tile of 32 tokens and one of 1, keys cut over a cluster
    (4, 1, 3, 300, 1),     # one token each
    (3, 1, 1, 260, 50),    # 3 heads: 126 of 128 rows of a tile
    (2, 2, 1, 0, 130),     # one head per key head: tiles of 128 tokens from an empty cache
    (8, 1, 1, 63, 2),      # 8 heads, the keys end just past a tile
])
def test_attention_of_a_portion_on_a_cached_context(heads, kv, batch, ctx, seq, dtype):
    cfg = medium_config(num_attention_heads=heads, num_key_value_heads=kv, head_dim=128, max_seq_len=1024)
    sd = checkpoint(cfg, dtype, seed=37)
    om, dev = O.OracleModel(cfg, sd, dtype), Context(cfg, sd, dtype)
    blk = B200Transformer.load(cfg.layer_name(0), dev)
    dev.cache = Cache(dev, batch, ctx + seq + 3)
    x = rand_x((batch, ctx + seq, cfg.hidden_size), dtype, seed=heads + seq)
    if ctx:
        blk.forward(dev.to_device(x[:, :ctx]), 0, 0, dev)
    y = blk.forward(dev.to_device(x[:, ctx:]), ctx, 0, dev)
    dev.sync()
    y = to_np(y)
    for b in range(batch):
        ref = om.block_forward(0, x[b].float().numpy(), 0, om.new_cache())[ctx:]
        _check(y[b], ref, dtype, f"row {b}")
    dev.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("batch,seq,vocab", [(2, 1, 1024), (17, 3, 1024), (64, 1, 1152), (3, 2, 1000)])   # 1000: no tiles, row by row
def test_head_of_a_batch(batch, seq, vocab, dtype):
    """Logits of every row's last position against the head of each row alone (another kernel, the same rounding points) and against the
    oracle's head; the tokens are the first maxima of these logits, with and without a logits buffer."""
    cfg = medium_config(vocab_size=vocab)
    sd = checkpoint(cfg, dtype, seed=41, peaked=True)
    ctx = Context(cfg, sd, dtype)
    p = cfg.model_prefix
    head = [sd[p + ".embed_tokens.weight"], sd[p + ".norm.weight"], sd["lm_head.weight"]]
    check(lib().cake_b200_head_load(ctx.h, *[ptr(t) for t in head]))
    x_host = rand_x((batch, seq, cfg.hidden_size), dtype, seed=batch)
    x = ctx.to_device(x_host)
    both, alone = ctx.empty(batch, vocab), ctx.empty(batch, vocab)
    tok, tok2 = (ctypes.c_uint32 * batch)(), (ctypes.c_uint32 * batch)()
    check(lib().cake_b200_logits(ctx.h, ptr(x), batch, seq, ptr(both), tok))
    check(lib().cake_b200_logits(ctx.h, ptr(x), batch, seq, None, tok2))
    for b in range(batch):
        check(lib().cake_b200_logits(ctx.h, ptr(x[b]), 1, seq, ptr(alone[b]), None))
    ctx.sync()
    _check(to_np(both), to_np(alone), dtype, "logits")
    om = O.OracleModel(cfg, sd, dtype)
    for b in range(0, batch, max(1, batch // 4)):
        _check(to_np(both[b]), om.logits(x_host[b].float().numpy()), dtype, f"logits of row {b} against the oracle")
    first = np.argmax(to_np(both), axis=1)   # numpy's argmax is the first maximum
    assert list(tok) == list(first) == list(tok2)
    ctx.close()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("rows", [129, 200, 257, 300])   # a second row tile with one row, a ragged one, a third with one row, a ragged third
def test_products_of_wide_tiles(rows, dtype):
    # gate / up: 16384 columns, two rounds of small tiles or one of wide ones (pairs of SMs: test_products.py)
    cfg = medium_config(num_attention_heads=4, num_key_value_heads=1, head_dim=128, intermediate_size=8192)
    sd = checkpoint(cfg, dtype, seed=43, std=0.03)
    om, ctx = O.OracleModel(cfg, sd, dtype), Context(cfg, sd, dtype)
    blk = B200Transformer.load(cfg.layer_name(0), ctx)
    x = rand_x((1, rows, cfg.hidden_size), dtype, seed=rows)
    y = blk.forward(ctx.to_device(x), 0, 0, ctx)
    ctx.sync()
    _check(to_np(y[0]), om.block_forward(0, x[0].float().numpy(), 0, om.new_cache()), dtype, f"{rows} rows")
    ctx.close()
