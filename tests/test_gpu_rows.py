"""Steps and prompts of a few rows: the sizes at which the products of a block change their kernel or their tiling, against the
oracle with the bars of test_gpu_parity.py (same rounding points, fp32 sums in another order)."""
import pytest

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
    _check(to_np(y[0]), om.block_forward(1, x[0].float().numpy(), 0, om.new_cache()), dtype, f"prompt of {rows}")
    ctx.cache = Cache(ctx, rows, 8)   # the same rows as one token each of `rows` sequences
    y = to_np(blk.forward(ctx.to_device(x.transpose(0, 1)), 0, 1, ctx))
    for b in range(0, rows, max(1, rows // 4)):
        _check(y[b], om.block_forward(1, x[0, b:b + 1].float().numpy(), 0, om.new_cache()), dtype, f"row {b} of a batch of {rows}")
    ctx.close()
