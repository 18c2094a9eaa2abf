"""The bounded waits of the tensor-core kernels (mbar_wait_lim) and of the decode kernel (MkWait): a wait that nothing ends gives up after its limit, sets the error word that
the next synchronising call reports, and the thread's later waits return at once.  Nothing faults: the probe kernel waits on a
barrier (or packets, or a counter) of its own, returns, and the context stays usable."""
import ctypes

import numpy as np
import pytest
import torch

from cake_b200.capi import CakeB200Error, check, lib, ptr
from cake_b200.config import Config
from cake_b200.model import B200Transformer, Cache, Context, sampling_from_args
from tests.util import checkpoint, medium_config, rand_x, to_np

pytestmark = pytest.mark.gpu


def probe(ctx, arrivals, tries, ok, kcycles):
    fn = lib().cake_b200_debug_wait
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_uint32, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int)]
    check(fn(ctx.h, arrivals, tries, ok, kcycles))


def test_a_wait_that_runs_out_is_reported_and_the_thread_does_not_wait_again():
    cfg = medium_config()
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    ok, kcycles = (ctypes.c_int * 2)(), (ctypes.c_int * 2)()
    try:
        probe(ctx, 2, 256, ok, kcycles)      # both arrivals came: no error
        assert list(ok) == [1, 1]
        ctx.sync()
        probe(ctx, 1, 8192, ok, kcycles)     # one of two: the first wait takes all of its tries, the second one at most two
        print(f"8192 tries {kcycles[0]} kcycles, then {kcycles[1]}")
        assert list(ok) == [0, 0] and kcycles[0] < 2000000 and kcycles[1] < kcycles[0] / 100
        with pytest.raises(CakeB200Error, match="gave up a wait"):
            ctx.sync()
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        ctx.cache.clear()
        x = ctx.to_device(rand_x((1, 40, cfg.hidden_size), "bf16", seed=1))
        y = blk.forward(x, 0, 0, ctx)
        ctx.sync()
        assert np.isfinite(to_np(y)).all()
    finally:
        ctx.close()


def test_every_call_that_hands_results_to_the_host_reports_it_and_caches_in_use_are_refused():
    """The wait runs out while the call is under way (a probe kernel in front of it in the stream): the call itself reports it."""
    cfg = medium_config()
    sd = checkpoint(cfg, "bf16", seed=3, peaked=True)
    ctx = Context(cfg, sd, "bf16")
    h, L = ctx.h, lib()
    kcycles = (ctypes.c_int * 2)()
    try:
        p = cfg.model_prefix
        check(L.cake_b200_head_load(h, *[ptr(sd[k]) for k in (p + ".embed_tokens.weight", p + ".norm.weight", "lm_head.weight")]))
        blk = B200Transformer.load(cfg.layer_name(0), ctx)
        x = ctx.to_device(rand_x((3, 40, cfg.hidden_size), "bf16", seed=1))
        row, out = x[:1, :1].contiguous(), np.empty((1, 40, cfg.hidden_size), np.uint16)
        logits = ctx.to_device(rand_x((3, cfg.vocab_size), "bf16", seed=2))
        tok = (ctypes.c_uint32 * 3)()
        samp = sampling_from_args(0.8, None, 0.9, 5)
        kv = np.empty((1 << 20,), np.uint16)
        one = (ctypes.c_void_p * 1)(blk.h)
        zero = (ctypes.c_int * 1)(0)
        x_host = np.zeros((1, 40, cfg.hidden_size), np.uint16)
        calls = {
            "sync": lambda: ctx.sync(),
            "logits of a batch": lambda: check(L.cake_b200_logits(h, ptr(x), 3, 40, None, tok)),
            "logits of a row": lambda: check(L.cake_b200_logits(h, ptr(row), 1, 1, None, tok)),
            "penalty and argmax": lambda: check(L.cake_b200_repeat_penalty_argmax(h, ptr(logits), 1.1, tok, 1, tok)),
            "sample": lambda: check(L.cake_b200_sample(h, ptr(logits), ctypes.byref(samp), 1.0, tok, 0, 0, None, tok)),
            "cache_read": lambda: check(L.cake_b200_cache_read(ctx.cache.h, 0, 0, kv.ctypes.data, kv.nbytes)),
            "forward on host buffers": lambda: check(L.cake_b200_forward_batch_host(h, one, zero, 1, ctx.cache.h, x_host.ctypes.data, out.ctypes.data, 1, 40, 40)),
        }
        for name, call in calls.items():
            ctx.cache.clear()
            blk.forward(x[:1], 0, 0, ctx)
            ctx.sync()
            probe(ctx, 1, 1 << 14, None, kcycles)   # some 70 ms: the host is inside `call` when it runs out
            with pytest.raises(CakeB200Error, match="gave up a wait"):
                call()
            ctx.sync()                                          # reported once
            with pytest.raises(CakeB200Error, match="clear it"):
                blk.forward(row, 40, 0, ctx)
            with pytest.raises(CakeB200Error, match="clear it"):
                check(L.cake_b200_cache_read(ctx.cache.h, 0, 0, kv.ctypes.data, kv.nbytes))
            ctx.cache.clear()
            y = blk.forward(x[:1], 0, 0, ctx)
            ctx.sync()
            assert np.isfinite(to_np(y)).all(), name
    finally:
        ctx.close()


@pytest.mark.parametrize("what", ["a vector of packets", "the parts of attention", "the grid barrier", "the inbox"])
def test_a_wait_of_the_decode_kernel_that_runs_out(what):
    cfg = medium_config()
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    kind = ["a vector of packets", "the parts of attention", "the grid barrier", "the inbox"].index(what)
    ok, kcycles = (ctypes.c_int * 2)(), (ctypes.c_int * 2)()
    fn = lib().cake_b200_debug_packet_wait
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int)]
    try:
        check(fn(ctx.h, kind, 1, 4096, ok, kcycles))
        assert list(ok) == [1, 1]
        ctx.sync()
        check(fn(ctx.h, kind, 0, 4096, ok, kcycles))   # the first wait takes all of its polls, the second one none
        print(f"{what}: 4096 polls {kcycles[0]} kcycles, then {kcycles[1]}")
        assert list(ok) == [0, 0] and kcycles[0] < 100000 and kcycles[1] <= kcycles[0] / 50
        with pytest.raises(CakeB200Error, match="gave up a wait"):
            ctx.sync()
        ctx.sync()
    finally:
        ctx.close()


@pytest.mark.parametrize("hidden,inter,heads,kv,hd", [(192, 448, 4, 2, 16), (1024, 3072, 16, 8, 128), (2560, 17408, 32, 4, 128)])
def test_steps_after_one_whose_waits_ran_out(hidden, inter, heads, kv, hd):
    """Every wait of a step gives up at its second poll: the launch ends, the call that synchronises reports it, and the same session begun again on
    the same context has the bits that it had before (tags, the barrier's counter and its start went on)."""
    layers, first = 3, 140
    cfg = Config(hidden_size=hidden, intermediate_size=inter, vocab_size=384, num_hidden_layers=layers, num_attention_heads=heads,
                 num_key_value_heads=kv, rms_norm_eps=1e-5, rope_theta=10000.0, max_seq_len=512, head_dim=hd)
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3, std=0.7 * hidden ** -0.5), "bf16")
    polls = lib().cake_b200_debug_polls
    polls.argtypes = [ctypes.c_void_p, ctypes.c_int]
    try:
        blocks = [B200Transformer.load(cfg.layer_name(i), ctx) for i in range(layers)]
        ctx.cache = Cache(ctx, 1, first + 4)
        xs = [ctx.to_device(rand_x((1, 1, hidden), "bf16", seed=t)) for t in range(3)]

        def step(t):
            return blocks[0].forward_batch(xs[t], [(b.layer_name(), first + t, i) for i, b in enumerate(blocks)], ctx, blocks=blocks)

        def session():
            ctx.cache.clear()
            ctx.cache.fill_synthetic(range(layers), first, 5)
            ys = [step(t) for t in range(3)]
            ctx.sync()
            return [y.cpu() for y in ys]

        want = session()
        for _ in range(2):
            ctx.cache.clear()
            ctx.cache.fill_synthetic(range(layers), first, 5)
            check(polls(ctx.h, 1))
            step(0)
            check(polls(ctx.h, 0))
            with pytest.raises(CakeB200Error, match="gave up a wait"):
                ctx.sync()
            with pytest.raises(CakeB200Error, match="clear it"):
                step(1)
            assert all(torch.equal(a, b) for a, b in zip(session(), want))
    finally:
        ctx.close()


@pytest.mark.parametrize("M,N,K,split", [(16, 6144, 4096, 8), (37, 4096, 1024, 4), (225, 1024, 4096, 4), (250, 2048, 4096, 4)])
def test_sums_of_a_cluster_that_never_come(M, N, K, split):
    """The first CTA of every cluster gives up at its first wait and sends nothing, the others wait for its sums until their tries are spent: all of them let what
    is in flight end and leave, the call reports it, and the next product on the same context has the bits that it had before.  Sums received
    behind the ring, over it, and with a share kept in tensor memory."""
    from tests.test_products import SKINNY, plan
    cfg = medium_config()
    ctx = Context(cfg, checkpoint(cfg, "bf16", seed=3), "bf16")
    V, I = ctypes.c_void_p, ctypes.c_int
    fn, tries = lib().cake_b200_debug_product, lib().cake_b200_debug_tries
    fn.argtypes = [V, I, V, V, V, V, V, I, I, I, I, ctypes.c_float, V, I, I, V, I]
    tries.argtypes = [V, I]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms == 148:
        assert plan(M, N, K, sms=sms)[:2] == (SKINNY, split)
    g = torch.Generator(device="cuda:0").manual_seed(M)
    a, w = (torch.randn(n, K, device="cuda:0", generator=g).bfloat16() for n in (M, N))

    def product():
        c = torch.zeros(M, N, device="cuda:0", dtype=torch.bfloat16)
        torch.cuda.synchronize()
        check(fn(ctx.h, 0, ptr(a), ptr(w), None, None, ptr(c), M, N, K, 0, 0.0, None, 0, 0, None, 1))
        return c
    try:
        want = product()
        for n in (1, 1024):
            check(tries(ctx.h, n))
            with pytest.raises(CakeB200Error, match="gave up a wait"):
                product()
            check(tries(ctx.h, 0))
            for _ in range(3):
                assert torch.equal(product(), want)
    finally:
        ctx.close()
