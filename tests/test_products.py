"""The product kernels one by one: which of them a shape takes (no GPU needed), and what each gives with every epilogue, against plain torch
in fp32 on the same 16-bit operands."""
import ctypes

import pytest
import torch

from cake_b200.capi import CakeB200Error, check, lib, ptr
from cake_b200.model import Context
from tests.util import checkpoint, medium_config

SMALL, WIDE, PAIR, SKINNY = range(4)
PLAIN, RESIDUAL, SWIGLU, RESIDUAL_F32, SOFTCAP_F32, ACT = range(6)
SMS = 148


def plan(M, N, K, group_rows=0, batch=1, sms=SMS):
    fn, out = lib().cake_b200_debug_plan, (ctypes.c_int * 4)()
    check(fn(sms, M, N, K, group_rows, batch, out))
    return tuple(out)


def test_plans_stay_within_the_kernels_limits():
    for sms in (132, 148):
        for N in (128, 256, 384, 1024, 3072, 6144, 28672):
            for K in (64, 128, 448, 1024, 4096, 14336):
                for M in (1, 16, 17, 33, 64, 65, 96, 127, 128, 129, 240, 241, 256, 257, 1000, 4096):
                    kind, split, stages, smem = plan(M, N, K, sms=sms)
                    if kind == SKINNY:
                        nt = (M + 15) // 16 * 16
                        assert M <= 256 and split in (1, 2, 4, 8) and 3 <= stages <= 8 and smem <= 220 * 1024
                        assert split == 1 or K // 64 >= 2 * split          # every CTA has at least two k-blocks
                        assert nt % split == 0 and (nt // split) % 2 == 0  # a share is a number of row pairs
                        assert smem >= stages * (16384 + nt * 128) + 1280 and (split == 1 or smem >= nt * 512 + 1280)
                    else:
                        assert M > 64 and (kind == SMALL or N % 256 == 0) and (kind != PAIR or M > 128)
        for rows in (1, 64):
            assert plan(384, 512, 2048, group_rows=rows, sms=sms)[0] == SKINNY
        assert plan(384, 512, 2048, group_rows=65, sms=sms)[0] in (SMALL, WIDE)   # blocks of a grouped product never pair
        assert plan(300, 128, 128, batch=3, sms=sms)[0] == SMALL and plan(33, 256, 128, batch=3, sms=sms)[0] != SKINNY


# (M, N, K) and the kernel it is there for: even and odd numbers of row tiles, the last one with one row or full
SHAPES = [
    (300, 512, 512, SMALL), (1000, 4096, 1024, WIDE), (512, 8192, 512, WIDE),
    (257, 8192, 3072, PAIR), (512, 8192, 3072, PAIR), (700, 6144, 3072, PAIR),
    (1, 512, 2048, SKINNY), (63, 640, 1088, SKINNY), (127, 2048, 2048, SKINNY), (241, 2048, 4096, SKINNY), (256, 2048, 4096, SKINNY),
]


def reference(epi, a, w, bias, res, act, cap, dtype, row_scale):
    """(value, bound on the distance): bound = roundings of the 16-bit steps on the way + K fp32 sums of the product."""
    eps = 2.0 ** -8 if dtype is torch.bfloat16 else 2.0 ** -11   # half an ulp, relative
    z = a.float() @ w.float().T
    s = (a.float().abs() @ w.float().abs().T) * (a.shape[1] * 2.0 ** -24)   # any order of the sums
    r = lambda t: t.to(dtype).float()
    if epi == SOFTCAP_F32:
        y = cap * torch.tanh(z / cap) if cap > 0 else z
        return y, s + 1e-5 * y.abs()
    if epi == RESIDUAL_F32:
        sc = row_scale[:, None] if row_scale is not None else 1.0
        y = res + sc * z
        return y, s * (sc.abs() if row_scale is not None else 1.0) + 1e-6 * y.abs() + 1e-6
    if epi == ACT:
        t = 1.5957691216057308 * z * (1 + 0.044715 * z * z) if act == 1 else z
        y = z.clamp(min=0) if act == 3 else z * torch.sigmoid(t)
        return y, 1.2 * s + 1.01 * eps * y.abs() + 1e-5
    if epi == SWIGLU:
        g, u = r(z[:, 0::2]), r(z[:, 1::2])
        h = r(g * torch.sigmoid(g))
        y = h * u
        sg, su = s[:, 0::2] + 2 * eps * g.abs(), s[:, 1::2] + 2 * eps * u.abs()   # a sum next to a rounding line goes to the other side
        return y, 1.2 * sg * u.abs() + 2 * eps * h.abs() * u.abs() + su * h.abs() + 1.01 * eps * y.abs() + 1e-5
    y = r(z)
    b = s + 2 * eps * z.abs()
    if epi == PLAIN and bias is not None:
        y = r(y + bias.float())
        b = b + 2 * eps * y.abs()
    if epi == RESIDUAL:
        y = y + res.float()
    return y, b + 1.01 * eps * y.abs() + 1e-6


def product(ctx, epi, a, w, M, N, K, bias=None, res=None, act=0, cap=0.0, group=None, n_groups=0, group_rows=0, row_scale=None, batch=1):
    f32 = epi in (RESIDUAL_F32, SOFTCAP_F32)
    cols = N // 2 if epi == SWIGLU else N * batch
    c = torch.full((M, cols), float("nan"), device=a.device, dtype=torch.float32 if f32 else a.dtype)
    fn = lib().cake_b200_debug_product
    V, I = ctypes.c_void_p, ctypes.c_int
    fn.argtypes = [V, I, V, V, V, V, V, I, I, I, I, ctypes.c_float, V, I, I, V, I]
    torch.cuda.synchronize()
    opt = lambda t: ptr(t) if t is not None else None
    check(fn(ctx.h, epi, ptr(a), ptr(w), opt(bias), opt(res), ptr(c), M, N, K, act, cap, opt(group), n_groups, group_rows, opt(row_scale), batch))
    return c


def near(got, want, bound, what):
    worst = ((got.float() - want).abs() - bound).max().item()
    assert worst <= 0, (what, worst)   # a NaN fails too


@pytest.fixture(params=["bf16", "f16"])
def ctx(request):
    torch.backends.cuda.matmul.allow_tf32 = False
    cfg = medium_config()
    c = Context(cfg, checkpoint(cfg, request.param, seed=3), request.param)
    c.D = torch.bfloat16 if request.param == "bf16" else torch.float16
    yield c
    c.close()


def operands(ctx, M, N, K, seed, n_w=1):
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    a = torch.randn(M, K, device="cuda:0", generator=g).to(ctx.D)
    w = (torch.randn(n_w * N, K, device="cuda:0", generator=g) * K ** -0.5).to(ctx.D)
    return a, w, g


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,kind", SHAPES)
def test_products_with_every_epilogue(ctx, M, N, K, kind):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert plan(M, N, K, sms=sms)[0] == kind
    a, w, g = operands(ctx, M, N, K, M + N)
    bias = torch.randn(N, device=a.device, generator=g).to(ctx.D)
    res = torch.randn(M, N, device=a.device, generator=g).to(ctx.D)
    scale = torch.rand(M, device=a.device, generator=g) + 0.5
    for epi, act, cap, b, r, rs in [(PLAIN, 0, 0.0, None, None, None), (PLAIN, 0, 0.0, bias, None, None), (RESIDUAL, 0, 0.0, None, res, None), (SWIGLU, 0, 0.0, None, None, None),
                                    (RESIDUAL_F32, 0, 0.0, None, res.float(), None), (RESIDUAL_F32, 0, 0.0, None, res.float(), scale), (SOFTCAP_F32, 0, 1.5, None, None, None),
                                    (SOFTCAP_F32, 0, 0.0, None, None, None), (ACT, 0, 0.0, None, None, None), (ACT, 1, 0.0, None, None, None), (ACT, 3, 0.0, None, None, None)]:
        want, bound = reference(epi, a, w, b, r, act, cap, ctx.D, rs)
        near(product(ctx, epi, a, w, M, N, K, b, r, act, cap, row_scale=rs), want, bound, (epi, act, cap))


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 31, 33, 129, 300])
@pytest.mark.parametrize("N,K,batch,kind", [(128, 128, 3, SMALL), (256, 128, 3, SMALL), (512, 128, 16, None), (256, 1024, 32, None)])   # None: small, wide or pairs by M
def test_products_side_by_side(ctx, M, N, K, batch, kind):
    got_kind = plan(M, N, K, batch=batch)[0]
    assert got_kind != SKINNY and (kind is None or got_kind == kind)
    a, w, _ = operands(ctx, M, N, K * batch, M, 1)
    w = (torch.randn(batch * N, K, device=a.device) * K ** -0.5).to(ctx.D)
    c = product(ctx, PLAIN, a, w, M, N, K, batch=batch)
    for h in range(batch):
        want, bound = reference(PLAIN, a[:, h * K:(h + 1) * K], w[h * N:(h + 1) * N], None, None, 0, 0.0, ctx.D, None)
        near(c[:, h * N:(h + 1) * N], want, bound, h)


def test_side_by_side_shapes_reach_every_tile():
    assert {plan(M, N, K, batch=b)[0] for M in (1, 31, 33, 129, 300) for N, K, b in [(128, 128, 3), (256, 128, 3), (512, 128, 16), (256, 1024, 32), (512, 3072, 16)]} >= {SMALL, WIDE}


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 2, 17, 64, 65])
@pytest.mark.parametrize("N,K", [(512, 2048), (1024, 512)])
def test_grouped_products(ctx, rows, N, K):
    """Row blocks of 128 that belong to experts 2, 0, none and 2; only the first `rows` of a block are used.  K is cut over a cluster."""
    kind, split, _, _ = plan(512, N, K, group_rows=rows)
    assert (kind == SKINNY and split > 1) if rows <= 64 else kind in (SMALL, WIDE)
    groups = [2, 0, -1, 2]
    a, w, g = operands(ctx, 512, N, K, rows, 3)
    group = torch.tensor(groups, dtype=torch.int32, device=a.device)
    res = torch.randn(512, N, device=a.device, generator=g)
    for epi in (SWIGLU, SOFTCAP_F32, RESIDUAL_F32, PLAIN):
        c = product(ctx, epi, a, w, 512, N, K, None, res if epi == RESIDUAL_F32 else None, group=group, n_groups=3, group_rows=rows)
        for i, e in enumerate(groups):
            if e < 0:
                continue
            sl = slice(i * 128, i * 128 + rows)
            want, bound = reference(epi, a[sl], w[e * N:(e + 1) * N], None, res[sl], 0, 0.0, ctx.D, None)
            near(c[sl], want, bound, (epi, i))


# sums that meet over a cluster: (M, N, K), CTAs of a slice; received behind the ring or over it, shares of 2 .. 128 rows, a share that is half empty
EXCHANGES = [(1, 1024, 1024, 8), (16, 6144, 4096, 8), (37, 4096, 1024, 4), (49, 1024, 2048, 8), (64, 2048, 4096, 8), (97, 4096, 1024, 4), (112, 2048, 2048, 8),
             (193, 2048, 2048, 4), (209, 1024, 4096, 8), (225, 1024, 4096, 4), (250, 2048, 4096, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,split", EXCHANGES)
def test_sums_of_a_cluster(ctx, M, N, K, split):
    """Every cut along K gives the same as a plain product, for C and residual that take wide accesses and, two bytes off, for those that don't."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    kind, got_split = plan(M, N, K, sms=sms)[:2]
    if sms == SMS:
        assert (kind, got_split) == (SKINNY, split)
    a, w, g = operands(ctx, M, N, K, M + N)
    res = torch.randn(M, N, device=a.device, generator=g)
    for epi in (RESIDUAL, RESIDUAL_F32, SWIGLU, PLAIN):
        r = res.to(ctx.D) if epi == RESIDUAL else res if epi == RESIDUAL_F32 else None
        want, bound = reference(epi, a, w, None, r, 0, 0.0, ctx.D, None)
        near(product(ctx, epi, a, w, M, N, K, None, r), want, bound, epi)
        if kind != SKINNY:
            continue
        c = torch.full((want.numel() + 1,), float("nan"), device=a.device, dtype=torch.float32 if epi == RESIDUAL_F32 else ctx.D)[1:]
        off = torch.cat([r.flatten()[:1], r.flatten()])[1:] if r is not None else None
        torch.cuda.synchronize()
        check(lib().cake_b200_debug_product(ctx.h, epi, ptr(a), ptr(w), None, ptr(off) if off is not None else None, ptr(c), M, N, K, 0, 0.0, None, 0, 0, None, 1))
        near(c.view(want.shape), want, bound, (epi, "two bytes off"))


# shapes of 65 .. 256 rows that the estimates give to gemm_tc_kernel, whose accesses are 16 bytes wide, and one with more rows than gemm_skinny_kernel has
@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(227, 256, 2048), (254, 128, 2048), (215, 6144, 14336), (257, 256, 2048)])
def test_outputs_on_any_address(ctx, M, N, K):
    """A caller's output two bytes off a 16-byte address: as many rows as the kernel for any address has go there, more are refused before a launch."""
    a, w, g = operands(ctx, M, N, K, M + N)
    res = torch.randn(M, N, device=a.device, generator=g).to(ctx.D)
    for epi, r in ((PLAIN, None), (RESIDUAL, res)):
        want, bound = reference(epi, a, w, None, r, 0, 0.0, ctx.D, None)
        near(product(ctx, epi, a, w, M, N, K, None, r), want, bound, epi)
        c = torch.full((want.numel() + 1,), float("nan"), device=a.device, dtype=ctx.D)[1:]
        torch.cuda.synchronize()
        call = lambda: check(lib().cake_b200_debug_product(ctx.h, epi, ptr(a), ptr(w), None, ptr(r) if r is not None else None, ptr(c), M, N, K, 0, 0.0, None, 0, 0, None, 1))  # noqa: E731
        if M > 256:
            with pytest.raises(CakeB200Error, match="multiple of 16"):
                call()
            continue
        call()
        near(c.view(want.shape), want, bound, (epi, "two bytes off"))
