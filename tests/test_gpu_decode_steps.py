"""The decode kernel at the sizes where its plan changes, against the chain of one kernel per operation: rows per stage 16 .. 1 and rows of
several stages, phases dealt out evenly and with a pool, models too small for every CTA to own rows, one CTA or several per key head."""
import pytest
import torch

from cake_b200.config import Config
from cake_b200.model import B200Transformer, Cache, Context
from tests.util import checkpoint, max_ulp_err, rand_x, to_np

pytestmark = pytest.mark.gpu
LAYERS = 2
# positions around one CTA / several CTAs per key head (128) and their shares (64, multiples of 8), and around a tile of 128 rows
POSITIONS = (0, 1, 127, 128, 129, 700)
SHAPES = {  # hidden, inter, heads, kv heads, head size, dtype
    "too small for every CTA": (192, 448, 4, 2, 16, "bf16"),
    "16 rows a stage, an odd number of vectors": (576, 1600, 8, 2, 64, "f16"),
    "16 and 4 rows, even shares": (1024, 3072, 16, 8, 128, "f16"),
    "8 and 2 rows, pools": (2048, 8192, 16, 16, 128, "bf16"),
    "4 rows, rows of two stages": (2560, 17408, 32, 4, 128, "bf16"),
}


@pytest.mark.parametrize("shape", SHAPES)
def test_steps_equal_the_chain_of_kernels(shape, monkeypatch):
    hidden, inter, heads, kv, hd, dtype = SHAPES[shape]
    cfg = Config(hidden_size=hidden, intermediate_size=inter, vocab_size=384, num_hidden_layers=LAYERS, num_attention_heads=heads,
                 num_key_value_heads=kv, rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=1024, head_dim=hd)
    sd = checkpoint(cfg, dtype, seed=11, std=0.7 * hidden ** -0.5)
    outs = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = Context(cfg, sd, dtype)
        blocks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(LAYERS)]
        outs[mode] = []
        for pos in POSITIONS:
            ctx.cache = Cache(ctx, 1, pos + 3)
            ctx.cache.fill_synthetic(range(LAYERS), pos, 5)
            for t in range(3):   # the second and third step read the rows that the first ones appended
                x = ctx.to_device(rand_x((1, 1, hidden), dtype, seed=7 * pos + t))
                y = blocks[0].forward_batch(x, [(b.layer_name(), pos + t, i) for i, b in enumerate(blocks)], ctx, blocks=blocks)
                ctx.sync()
                outs[mode].append(y.cpu())
        ctx.close()
    # the same roundings, sums in another order: two layers of them differ by a rounding here and there (2 ulp, as for the whole model)
    for a, b in zip(outs["0"], outs["1"]):
        assert torch.isfinite(a.float()).all()
        assert max_ulp_err(to_np(a), to_np(b), dtype) <= 2.0


@pytest.mark.parametrize("hidden,heads,kv,hd,dtype", [(1024, 16, 2, 128, "bf16"), (4096, 32, 4, 128, "f16"), (512, 8, 2, 64, "f16"), (192, 4, 2, 16, "bf16")])
def test_attention_cut_over_many_ctas_repeats_itself(hidden, heads, kv, hd, dtype, monkeypatch):
    """2, 16 to 17 and 32 CTAs per key head (the most): a few threads of a CTA merge the parts while the others gather the next product's input, so every
    run has the same bits, and they are those of the chain of kernels up to the order of sums."""
    cfg = Config(hidden_size=hidden, intermediate_size=1024, vocab_size=384, num_hidden_layers=LAYERS, num_attention_heads=heads,
                 num_key_value_heads=kv, rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=4096, head_dim=hd)
    sd = checkpoint(cfg, dtype, seed=12, std=0.7 * hidden ** -0.5)
    outs = {}
    for mode, runs in (("1", 1), ("0", 25)):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = Context(cfg, sd, dtype)
        blocks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(LAYERS)]
        outs[mode] = []
        for pos in (129, 1030, 2047, 2300):
            ctx.cache = Cache(ctx, 1, pos + 1)
            ctx.cache.fill_synthetic(range(LAYERS), pos, 5)
            x = ctx.to_device(rand_x((1, 1, hidden), dtype, seed=pos))
            ys = []
            for _ in range(runs):   # (the step writes its own position's key and value: the same ones each time)
                ctx.cache.fill_synthetic(range(LAYERS), pos, 5)
                ys.append(blocks[0].forward_batch(x, [(b.layer_name(), pos, i) for i, b in enumerate(blocks)], ctx, blocks=blocks))
            ctx.sync()
            assert all(torch.equal(y, ys[0]) for y in ys[1:]), pos
            outs[mode].append(ys[0].cpu())
        ctx.close()
    for a, b in zip(outs["0"], outs["1"]):
        assert torch.isfinite(a.float()).all()
        assert max_ulp_err(to_np(a), to_np(b), dtype) <= 2.0
