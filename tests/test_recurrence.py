"""The gated linear recurrence on given buffers: token by token and in chunks of 64, against a scan in 64 bits."""
import ctypes

import pytest
import torch

from cake_b200.capi import check, lib
from cake_b200.config import Config, MixerSpec
from cake_b200.model import Context

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
CHUNK_MIN = 256   # tokens from which a call is taken in chunks


@pytest.fixture(params=list(DTYPES))
def ctx(request):
    layer = MixerSpec(type="retention", heads=2, dim=64, vdim=64, decay=[0.9, 0.95])
    c = Context(Config(128, 0, 256, 1, 2, 2, head_dim=64, max_seq_len=64, block_kind="setodra", layers=[layer]), {}, dtype=request.param)
    c.D = DTYPES[request.param]
    yield c
    c.close()


def inputs(ctx, form, B, S, H, dk, dv, group, pos0, seed=0):
    """What the three designs hand over: retention (fixed decays, rotation), a state-space layer (input-dependent decays, groups of heads that
    share q and k, a skip; "forgetful": now and then a step so large that nothing of the tokens in front is left), a matrix memory (factors per token)."""
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda:0")  # noqa: E731
    q, k, v = rnd(B * S, H // group * dk).to(ctx.D), rnd(B * S, H // group * dk).to(ctx.D), rnd(B * S, H * dv).to(ctx.D)
    d = dict(q=q, k=k, v=v, state=rnd(B, H, dk, dv))
    if form == "retention":
        d["decay"] = torch.tensor([1 - 2.0 ** (-5 - i % 4) for i in range(H)], device="cuda:0")
        f = 10000.0 ** (-torch.arange(dk // 2, device="cuda:0", dtype=torch.float64) * 2 / dk)
        a = torch.arange(pos0 + S, device="cuda:0", dtype=torch.float64)[:, None] * f
        d["cos"], d["sin"] = a.cos().float(), a.sin().float()
    elif form in ("ssd", "forgetful"):
        d["dt"], d["dt_bias"], d["a_log"], d["skip"] = rnd(B * S, H).to(ctx.D), (rnd(H) * 0.7 - 1).to(ctx.D), (rnd(H) * 0.7 - 0.5).to(ctx.D), (rnd(H) * 0.2 + 1).to(ctx.D)
        if form == "forgetful":
            d["a_log"].clamp_(min=1.0)
            d["dt"][::7] = 50.0   # a decay of exp(-50 e): 0 in fp32
    else:
        a = torch.rand(B * S, H, generator=g, device="cuda:0")
        a[::7] = 0.0   # a token that forgets everything in front of it
        d["a_tok"], d["b_tok"] = a, rnd(B * S, H)
    return d


def call(ctx, d, B, S, H, dk, dv, group, pos0, kscale, chunks):
    state, o = d["state"].clone(), torch.full((B * S, H * dv), float("nan"), device="cuda:0")
    names = ["q", "k", "v", "dt", "dt_bias", "a_log", "skip", "decay", "cos", "sin"]
    t = [d.get(n) for n in names] + [state, o, d.get("a_tok"), d.get("b_tok")]
    ptrs = (ctypes.c_void_p * 14)(*[x.data_ptr() if x is not None else None for x in t])
    dims = (ctypes.c_int * 12)(d["q"].shape[1], d["k"].shape[1], d["v"].shape[1], group, H, dk if "cos" in d else 0, B, S, H, dk, dv, pos0)
    n = ctypes.c_int()
    fn = lib().cake_b200_debug_recurrence
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_float, ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    torch.cuda.synchronize()
    check(fn(ctx.h, ptrs, dims, kscale, chunks, ctypes.byref(n)))
    return o, state, n.value


def scan(d, B, S, H, dk, dv, group, pos0, kscale):
    q, k = (d[n].double().view(B, S, H // group, dk).repeat_interleave(group, 2) for n in "qk")
    v = d["v"].double().view(B, S, H, dv)
    if "cos" in d:
        c, s = (d[n].double()[pos0:pos0 + S][None, :, None] for n in ("cos", "sin"))
        turn = lambda x: torch.cat([x[..., :dk // 2] * c - x[..., dk // 2:] * s, x[..., dk // 2:] * c + x[..., :dk // 2] * s], -1)  # noqa: E731
        q, k = turn(q), turn(k)
    if "dt" in d:
        b = torch.nn.functional.softplus(d["dt"].double().view(B, S, H) + d["dt_bias"].double())
        a = torch.exp(-torch.exp(d["a_log"].double()) * b)
    elif "a_tok" in d:
        a, b = d["a_tok"].double().view(B, S, H), d["b_tok"].double().view(B, S, H)
    else:
        a, b = d["decay"].double().expand(B, S, H), torch.full((B, S, H), kscale, device="cuda:0", dtype=torch.float64)
    st = d["state"].double() if pos0 else torch.zeros(B, H, dk, dv, device="cuda:0", dtype=torch.float64)
    o = torch.empty(B, S, H, dv, device="cuda:0", dtype=torch.float64)
    for t in range(S):
        st = st * a[:, t, :, None, None] + b[:, t, :, None, None] * k[:, t, :, :, None] * v[:, t, :, None, :]
        o[:, t] = torch.einsum("bhd,bhdn->bhn", q[:, t], st)
    if "skip" in d:
        o = o + d["skip"].double()[:, None] * v
    return o.reshape(B * S, H * dv), st


def rel(x, y):
    return ((x.double() - y).norm() / y.norm()).item()


@pytest.mark.gpu
@pytest.mark.parametrize("form,group,dk,dv", [("retention", 1, 128, 128), ("ssd", 4, 128, 64), ("forgetful", 1, 64, 64), ("ssd", 2, 64, 192)])
@pytest.mark.parametrize("B,S,pos0", [(1, CHUNK_MIN, 0), (2, CHUNK_MIN + 1, 5), (1, 319, 0), (2, 320, 64), (1, 1000, 17)])
def test_chunks_against_a_scan(ctx, form, group, dk, dv, B, S, pos0):
    H = 8
    d = inputs(ctx, form, B, S, H, dk, dv, group, pos0, seed=S)
    want, want_state = scan(d, B, S, H, dk, dv, group, pos0, dk ** -0.5)
    o1, s1, n1 = call(ctx, d, B, S, H, dk, dv, group, pos0, dk ** -0.5, 0)
    o2, s2, n2 = call(ctx, d, B, S, H, dk, dv, group, pos0, dk ** -0.5, 1)
    assert n1 == 1 and n2 == 3
    # fp32 sums of at most S dk terms in any order; and about as far from 64 bits as token by token
    bound = 2.0 ** -24 * 8 * (S * dk) ** 0.5
    assert rel(o2, want) <= bound and rel(s2, want_state) <= bound
    assert rel(o2, want) <= 1.25 * rel(o1, want) + 2.0 ** -24 and rel(s2, want_state) <= 1.25 * rel(s1, want_state) + 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("B,launches", [(8, 6), (24, 1)])
def test_states_held_at_once_are_bounded(ctx, B, launches):
    """A batch whose states don't all fit goes through the tokens in several passes (8 of 11 chunks, then 3), a large one walks them."""
    S, H, dk, dv = 700, 16, 128, 128
    d = inputs(ctx, "ssd", B, S, H, dk, dv, 1, 3, seed=1)
    o1, s1, n1 = call(ctx, d, B, S, H, dk, dv, 1, 3, 1.0, 0)
    o2, s2, n2 = call(ctx, d, B, S, H, dk, dv, 1, 3, 1.0, 1)
    assert n1 == 1 and n2 == launches
    assert rel(o2, o1.double()) < 1e-5 and rel(s2, s1.double()) < 1e-5


@pytest.mark.gpu
def test_an_infinity_reaches_no_token_in_front_of_it(ctx):
    S, H, dk, dv = 300, 4, 64, 64
    d = inputs(ctx, "ssd", 1, S, H, dk, dv, 1, 0, seed=2)
    d["dt"].clamp_(max=1.0)
    d["a_log"].clamp_(max=0.0)   # no decay below exp(-1.3): what follows keeps something of it
    o0, _, _ = call(ctx, d, 1, S, H, dk, dv, 1, 0, 1.0, 1)
    d["v"][133] = float("inf")
    o1, _, n = call(ctx, d, 1, S, H, dk, dv, 1, 0, 1.0, 1)
    assert n == 3 and torch.equal(o0[:133], o1[:133]) and not torch.isfinite(o1[133:]).any()


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["few tokens", "key size", "value size", "row stride", "factors"])
def test_what_chunks_do_not_cover_walks_the_tokens(ctx, what):
    S, H, dk, dv = 300, 4, 64, 64
    if what == "few tokens":
        S = CHUNK_MIN - 1
    if what == "key size":
        dk = 96
    if what == "value size":
        dv = 32
    d = inputs(ctx, "factors" if what == "factors" else "ssd", 1, S, H, dk, dv, 1, 0, seed=3)
    if what == "row stride":
        d["v"] = torch.cat([d["v"], d["v"][:, :1]], 1)
    want, want_state = scan(dict(d, v=d["v"][:, :H * dv]), 1, S, H, dk, dv, 1, 0, 1.0)
    o, s, n = call(ctx, d, 1, S, H, dk, dv, 1, 0, 1.0, 1)
    assert n == 1 and rel(o, want) < 1e-5 and rel(s, want_state) < 1e-5
