"""The decode kernel at the sizes where its plan changes, against the chain of one kernel per operation: rows per stage 16 .. 1 and rows of
several stages, phases dealt out evenly and with a pool, models too small for every CTA to own rows, one CTA or several per key head."""
import ctypes

import pytest
import torch

from cake_b200.capi import check, lib, ptr
from cake_b200.config import Config, llama3_70b
from cake_b200.model import B200Transformer, Cache, Context, TextModelBase
from cake_b200.synth import make_layer
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
    "no room for the copy of the residual stream": (2560, 21504, 32, 4, 128, "bf16"),   # 5 stages without it, 4 with it
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


def _one_hot(n, k, column, scale, dtype):
    w = torch.zeros(n, k)
    w[torch.arange(n), column] = scale
    return w.to(dtype)


@pytest.mark.parametrize("part,act", [("norm and gate", "silu"), ("norm and gate", "gelu"), ("attention", "silu")])
def test_what_is_not_a_sum_is_rounded_as_in_the_chain(part, act, monkeypatch):
    """Weights with one entry per row and inputs whose squares add up without a rounding in any order: what is left are the divisions and square
    roots of the norm, the gate and the attention, and these are the correctly rounded ones in both forms.  Equal bits; a reciprocal or root
    that is an ulp off moves about one f16 value in ten thousand."""
    H, I, heads, kv, hd, steps = 2048, 8192, 16, 16, 128, 96
    cfg = Config(hidden_size=H, intermediate_size=I, vocab_size=384, num_hidden_layers=1, num_attention_heads=heads, num_key_value_heads=kv,
                 rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=256, head_dim=hd, use_gelu_mlp=act == "gelu")
    sd = checkpoint(cfg, "f16", seed=3)
    g, f16, p = torch.Generator().manual_seed(5), torch.float16, cfg.layer_name(0) + "."
    zero = lambda n, k: torch.zeros(n, k, dtype=f16)
    qkvo = {n: zero(H, H) for n in ("q", "k", "v", "o")}
    mlp = {"gate": zero(I, H), "up": zero(I, H), "down": zero(H, I)}
    i, h = torch.arange(I), torch.arange(H)
    if part == "attention":   # equal scores: value sums of whole 64ths over the number of positions
        qkvo["v"], qkvo["o"] = _one_hot(H, H, (3 * h + 1) % H, 1.0, f16), _one_hot(H, H, (5 * h + 2) % H, 1.0, f16)
        sd[p + "input_layernorm.weight"] = (torch.randint(-128, 129, (H,), generator=g) / 64).to(f16)
        xs = [(4 * torch.randint(0, 2, (1, 1, H), generator=g) - 2).to(f16) for _ in range(steps)]
    else:
        mlp = {"gate": _one_hot(I, H, (3 * i + 1) % H, 4.0, f16), "up": _one_hot(I, H, (7 * i + i // H) % H, 1.0, f16),
               "down": _one_hot(H, I, (5 * h + 3) % I, 1.0, f16)}
        xs = [(torch.randint(-64, 65, (1, 1, H), generator=g) / 16).to(f16) for _ in range(steps)]
    for n, w in qkvo.items():
        sd[p + f"self_attn.{n}_proj.weight"] = w
    for n, w in mlp.items():
        sd[p + f"mlp.{n}_proj.weight"] = w
    outs = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = Context(cfg, sd, "f16")
        block = B200Transformer.load(cfg.layer_name(0), ctx)
        ctx.cache = Cache(ctx, 1, steps)
        dev = [ctx.to_device(x) for x in xs]
        ys = [block.forward(x, t, 0, ctx) for t, x in enumerate(dev)]
        ctx.sync()
        outs[mode] = torch.cat([y.cpu() for y in ys])
        ctx.close()
    assert torch.isfinite(outs["0"].float()).all() and outs["0"].float().abs().max() > 1
    assert torch.equal(outs["0"], outs["1"]), int((outs["0"] != outs["1"]).sum())


EDGE_SHAPES = {  # hidden, inter, heads, kv heads, head size, dtype
    "a stage holds one row of gate or up": (12288, 1088, 8, 1, 128, "bf16"),
    "the longest row of one stage": (16384, 320, 8, 2, 64, "f16"),
    "gate and up rows of two stages": (20480, 704, 8, 2, 64, "bf16"),
    "no stage holds a row of down": (1024, 16448, 16, 8, 128, "bf16"),   # steps by the chain of kernels, the head by the decode kernel
    "vectors larger than the shared memory": (512, 73728, 8, 2, 64, "f16"),
}


@pytest.mark.parametrize("shape", EDGE_SHAPES)
def test_sizes_at_the_edge_of_the_plan_step_and_have_a_head(shape, monkeypatch):
    hidden, inter, heads, kv, hd, dtype = EDGE_SHAPES[shape]
    cfg = Config(hidden_size=hidden, intermediate_size=inter, vocab_size=1000, num_hidden_layers=1, num_attention_heads=heads,
                 num_key_value_heads=kv, rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=512, head_dim=hd)
    sd = checkpoint(cfg, dtype, seed=11, std=0.7 * hidden ** -0.5)
    outs, toks = {}, {}
    for mode in ("0", "1"):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = Context(cfg, sd, dtype, max_seq=512)
        model = TextModelBase.load(ctx)
        blk = model.blocks[0]
        outs[mode], toks[mode] = [], []
        for pos in (0, 200):
            ctx.cache = Cache(ctx, 1, pos + 4)
            ctx.cache.fill_synthetic(range(1), pos, 5)
            y = blk.forward(ctx.to_device(rand_x((1, 1, hidden), dtype, seed=pos)), pos, 0, ctx)
            lg, tok = ctx.to_device(torch.zeros(1, cfg.vocab_size)), (ctypes.c_uint32 * 1)()
            check(lib().cake_b200_logits(ctx.h, ptr(y), 1, 1, ptr(lg), tok))
            outs[mode] += [y.cpu(), lg.cpu()]
            assert tok[0] == int(torch.argmax(lg.float()))
        # the captured loop: the same kernels with the token and the position on the device
        model.decode_build()
        model.index_pos = 201
        toks[mode] = model.decode_greedy(7, 3)
        assert max(toks[mode]) < cfg.vocab_size
        ctx.close()
    for a, b in zip(outs["0"], outs["1"]):
        assert torch.isfinite(a.float()).all()
        assert max_ulp_err(to_np(a), to_np(b), dtype) <= 2.0


@pytest.mark.parametrize("hidden,vocab", [(1024, 20001), (4096, 3000), (192, 151)])   # 16 and 4 rows a stage with a pool; a vocabulary smaller than the grid's rows
def test_heads_of_a_row_behind_each_other(hidden, vocab):
    """Ten heads of different rows in flight at once, each placed while the one in front ends and with the claim counter that it leaves: the logits of each row
    against fp32 torch, and the same bits when a row comes again."""
    cfg = Config(hidden_size=hidden, intermediate_size=256, vocab_size=vocab, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2,
                 rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=64, head_dim=64)
    sd = checkpoint(cfg, "bf16", seed=13, std=hidden ** -0.5)
    ctx = Context(cfg, sd, "bf16")
    try:
        p = cfg.model_prefix
        norm, head = sd[p + ".norm.weight"], sd["lm_head.weight"]
        check(lib().cake_b200_head_load(ctx.h, ptr(sd[p + ".embed_tokens.weight"]), ptr(norm), ptr(head)))
        xs = [ctx.to_device(rand_x((1, 1, hidden), "bf16", seed=i % 5)) for i in range(10)]
        lgs = [ctx.to_device(torch.zeros(1, vocab)) for _ in xs]
        for x, lg in zip(xs, lgs):
            check(lib().cake_b200_logits(ctx.h, ptr(x), 1, 1, ptr(lg), None))
        tok = (ctypes.c_uint32 * 1)()
        check(lib().cake_b200_logits(ctx.h, ptr(xs[0]), 1, 1, ptr(lgs[0]), tok))
        for i, (x, lg) in enumerate(zip(xs, lgs)):
            f = x.float().cpu()[0]
            h = (f * (f.pow(2).mean() + 1e-5).rsqrt() * norm.float()).to(torch.bfloat16)
            assert max_ulp_err(to_np(lg), (h.float() @ head.float().T).to(torch.bfloat16).float().numpy(), "bf16") <= 2.0, i
            assert torch.equal(lg, lgs[i % 5])
        assert tok[0] == int(torch.argmax(lgs[0].float()))
    finally:
        ctx.close()


def test_eighty_layers_against_64_bits(monkeypatch):
    """The shard of the 70B model on one GPU: eighty layers, no copy of the residual stream beside four stages.  (The layers share one block's weights.)  A step's
    error against the same step in 64 bits is that of the chain of kernels: both round at the same 800 places, in bf16, to different sides where sums differ in order,
    so the two errors are two draws of one distribution; their 2-norms over 8192 values lie within a quarter of each other."""
    layers, pos = 80, 140
    cfg = llama3_70b(max_seq=256)
    sd = make_layer(cfg, 0, "bf16", device="cuda")
    H, heads, kv, hd = cfg.hidden_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.hd
    x = rand_x((1, 1, H), "bf16", seed=1)
    outs = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("CAKE_B200_PER_OP", mode)
        ctx = Context(cfg, sd, "bf16", max_seq=256)
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        ctx.cache = Cache(ctx, 1, pos + 1)
        ctx.cache.fill_synthetic(range(layers), pos, 5)
        if mode == "0":
            ctx.sync()
            kvs = [ctx.cache.kv(i) for i in range(layers)]
        y = blk.forward_batch(ctx.to_device(x), [(blk.layer_name(), pos, i) for i in range(layers)], ctx, blocks=[blk] * layers)
        ctx.sync()
        outs[mode] = y.cpu().double()[0, 0]
        ctx.close()
    w = {k.split(".", 3)[3]: v.double() for k, v in sd.items()}
    norm = lambda v, g: v / torch.sqrt((v * v).mean() + cfg.rms_norm_eps) * g
    angle = pos * cfg.rope_theta ** (-2.0 * torch.arange(hd // 2, dtype=torch.float64, device="cuda") / hd)
    cos, sin = angle.cos().bfloat16().double(), angle.sin().bfloat16().double()
    turn = lambda v: torch.cat([v[:, :hd // 2] * cos - v[:, hd // 2:] * sin, v[:, hd // 2:] * cos + v[:, :hd // 2] * sin], -1)
    h = x.double().cuda()[0, 0]
    for k0, v0 in kvs:
        n = norm(h, w["input_layernorm.weight"])
        q, k, v = (w[f"self_attn.{c}_proj.weight"] @ n for c in "qkv")
        keys = torch.cat([k0.double().cuda()[0], turn(k.view(kv, hd))[:, None]], 1)
        vals = torch.cat([v0.double().cuda()[0], v.view(kv, 1, hd)], 1)
        p = (torch.einsum("gmd,gtd->gmt", turn(q.view(heads, hd)).view(kv, heads // kv, hd), keys) * hd ** -0.5).softmax(-1)
        h = h + w["self_attn.o_proj.weight"] @ torch.einsum("gmt,gtd->gmd", p, vals).reshape(-1)
        n = norm(h, w["post_attention_layernorm.weight"])
        g = w["mlp.gate_proj.weight"] @ n
        h = h + w["mlp.down_proj.weight"] @ (g * torch.sigmoid(g) * (w["mlp.up_proj.weight"] @ n))
    want = h.cpu()
    err = {m: float((y - want).norm() / want.norm()) for m, y in outs.items()}
    print("80 layers, error against 64 bits: decode kernel %.5f, chain %.5f" % (err["0"], err["1"]))
    assert err["0"] <= 1.25 * err["1"] and err["1"] < 0.1
