"""The prompt attention on tcgen05 for heads of 128 (csrc/attention_tcgen05.cu: attn_prefill_wide_kernel and its kinds)
against the plain kernels, which work in float32 from the same bfloat16 q and pages: softmax with a window, a distance
table, a sink, a factor, a gate and rows that are key and value; attention without softmax.

Tolerance: both sides round the result to bfloat16 (half a unit, 2^-8 of it at most, each) and the tensor cores take the weights
as bfloat16 (2^-8 of each at most; a row's weighted mean of values moves by at most that times the largest value): 3 * 2^-8
of the largest value.  Without softmax a row's weights do not sum to one: n weights rounded one by one move the sum of n
values by about sqrt(n) 2^-9 of the largest weight and value, few of up to 2,048 keys weigh much; 3 * 2^-8 of the larger of the
largest result and the largest value."""
from types import SimpleNamespace

import pytest
import torch

from test_pirerax import batch_ctx, scrambled_table

gpu = pytest.mark.gpu

# heads, kv heads, page, window, tail, table rows, sink, gate, out_scale, spans (first position, end) of the requests
CASES = [
    (1, 1, 16, 0, -1, 0, False, False, 1.0, [(0, 193)]),
    (2, 1, 16, 0, -1, 0, True, False, 0.7, [(0, 128), (3, 67)]),
    (4, 2, 32, 0, -1, 0, True, True, 1.0, [(0, 129), (500, 501), (77, 205)]),
    (3, 1, 16, 100, -1, 0, False, True, 1.0, [(130, 500)]),
    (6, 1, 64, 1, -1, 0, False, False, 1.0, [(0, 200)]),
    (16, 1, 16, 0, -1, 0, True, False, 1.0, [(1000, 1255)]),
    (16, 8, 16, 1024, -1, 0, False, False, 1.0, [(0, 2048)]),
    (2, 2, 16, 0, -1, 40, True, False, 1.3, [(0, 300), (5, 6)]),
    (16, 8, 16, 0, -1, 700, True, False, 1.0, [(0, 1027), (0, 2), (900, 1300)]),
    (12, 1, 32, 0, -1, 5, False, False, 1.0, [(250, 449)]),
    (5, 1, 16, 333, -1, 1, True, True, 1.0, [(0, 700)]),
    (4, 2, 16, 90, 64, 0, True, False, 1.0, [(0, 257), (40, 140)]),
    (3, 3, 16, 0, 8, 0, False, False, 1.0, [(10, 211)]),
]
SIGMOID_CASES = [(1, 1, 16, 0, True, True, [(0, 193)]), (2, 1, 32, 0, True, False, [(0, 128), (3, 67), (9, 10)]), (16, 8, 16, 0, True, True, [(0, 2048)]),
                 (12, 1, 16, 200, False, True, [(250, 449)]), (3, 1, 64, 1, True, True, [(5, 300)]), (4, 2, 16, 0, False, False, [(0, 255), (1, 300)])]


def made(nh, nkv, page, tail, spans, seed):
    g = torch.Generator().manual_seed(seed)
    bt, num_pages = scrambled_table([e for _, e in spans], page, g)
    width = 128 + tail if tail >= 0 else 256
    pool = (0.8 * torch.randn(num_pages, nkv * page * width, generator=g)).to("cuda", torch.bfloat16)
    ctx = batch_ctx(spans)
    T = ctx.num_tokens
    q = torch.randn(T, nh * 128, generator=g).to("cuda", torch.bfloat16)
    return g, SimpleNamespace(pool=pool, block_table=bt, page_size=page, shared=False), ctx, q


def run_both(ctx, q, nh, tc, plain):
    got = torch.full((q.shape[0], nh * 128 + 16), 7.0, device="cuda", dtype=torch.bfloat16)
    want = torch.zeros(q.shape[0], nh * 128, device="cuda", dtype=torch.bfloat16)
    assert tc(got[:, 8:8 + nh * 128])
    plain(want)
    assert int(ctx.err.item()) == 0
    assert bool((got[:, :8] == 7.0).all()) and bool((got[:, 8 + nh * 128:] == 7.0).all())
    lens = [n for n in ctx.query_lens for _ in range(n)]
    rows = torch.tensor([n > 1 for n in lens], device="cuda")
    assert bool((got[~rows][:, 8:8 + nh * 128] == 7.0).all())          # single tokens are another kernel's
    return got[rows][:, 8:8 + nh * 128].float(), want[rows].float()


def absolute(ctx, q, cache, nh, nkv, plain):
    """What the weights give of the values' absolute values.  Rounding a weight and the two results to bfloat16 (2^-9 each) moves an
    element by three of 2^-9 of that; 2^-7 leaves a quarter for the float32 sums and exponentials."""
    pages = cache.pool.view(cache.pool.shape[0], 2, -1).clone()
    pages[:, 1] = pages[:, 1].abs()
    out = torch.zeros(q.shape[0], nh * 128, device="cuda", dtype=torch.bfloat16)
    plain(out, SimpleNamespace(pool=pages.view_as(cache.pool), block_table=cache.block_table, page_size=cache.page_size, shared=False))
    rows = torch.tensor([n > 1 for n in ctx.query_lens for _ in range(n)], device="cuda")
    return out[rows].float()


@gpu
@pytest.mark.parametrize("nh,nkv,page,window,tail,rows,sink,gated,scale,spans", CASES)
def test_softmax_kinds(nh, nkv, page, window, tail, rows, sink, gated, scale, spans):
    from airun_b200.kernels import fast, ops
    g, cache, ctx, q = made(nh, nkv, page, tail, spans, nh * 100 + len(spans) + window)
    T = q.shape[0]
    part = SimpleNamespace(D=128, Dv=128, nh=nh, nkv=nkv, scale=0.13, window=window, out_scale=scale, tail=tail,
                           table=(2.0 * torch.randn(nh, rows, generator=g)).cuda() if rows else None,
                           sink=(2.0 * torch.randn(nh, generator=g)).cuda() if sink else None)
    gate = torch.randn(T, nh * 128 + 4, generator=g).cuda()[:, 4:] if gated else None
    got, want = run_both(
        ctx, q, nh,
        lambda o: fast.attn_prompt_kind(ctx, "table" if rows else "options", q, o, cache, part, tail=tail, gate=gate,
                                        gate_stride=ops.attention_gate(gate, T, nh * 128)),
        lambda o: ops.softmax_attention(q, o, cache, ctx, nh, nkv, 128, 128, 0.13, part.table, part.sink, window, scale, tail=tail, gate=gate))
    assert float((got - want).abs().max()) < 3 * 2.0 ** -8 * scale * float(cache.pool.abs().max())
    if tail < 0:                                             # and each element by the weights' sum of its absolute values
        most = absolute(ctx, q, cache, nh, nkv, lambda o, c: ops.softmax_attention(q, o, c, ctx, nh, nkv, 128, 128, 0.13, part.table, part.sink, window, scale, gate=gate))
        assert bool(((got - want).abs() <= 2.0 ** -7 * most + 1e-6).all())


@gpu
@pytest.mark.parametrize("nh,nkv,page,window,dist,offset,spans", SIGMOID_CASES)
def test_attention_without_softmax(nh, nkv, page, window, dist, offset, spans):
    from airun_b200.kernels import fast, ops
    g, cache, ctx, q = made(nh, nkv, page, -1, spans, nh * 7 + len(spans))
    a, b, c = ((0.2 + torch.rand(nh, generator=g)).cuda(), (0.1 + torch.rand(nh, generator=g)).cuda(), (-2.0 + torch.randn(nh, generator=g)).cuda())
    part = SimpleNamespace(D=128, Dv=128, nh=nh, nkv=nkv, scale=0.13, window=window, dist_a=a if dist else None, dist_b=b if dist else None,
                           head_c=c if offset else None)
    got, want = run_both(
        ctx, q, nh, lambda o: fast.attn_prompt_kind(ctx, "sigmoid", q, o, cache, part),
        lambda o: ops.sigmoid_attention(q, o, cache, ctx, nh, nkv, 128, 128, 0.13, part.dist_a, part.dist_b, part.head_c, window))
    assert float((got - want).abs().max()) < 3 * 2.0 ** -8 * max(float(want.abs().max()), float(cache.pool.abs().max()))
    most = absolute(ctx, q, cache, nh, nkv, lambda o, c: ops.sigmoid_attention(q, o, c, ctx, nh, nkv, 128, 128, 0.13, part.dist_a, part.dist_b, part.head_c, window))
    assert bool(((got - want).abs() <= 2.0 ** -7 * most + 1e-6).all())


@gpu
@pytest.mark.parametrize("nh,nkv,page,window,spans,halves", [
    (16, 8, 16, 0, [(0, 2048)], True), (16, 8, 16, 0, [(512, 2612)], True), (16, 8, 32, 1100, [(300, 2360)], True), (16, 4, 16, 0, [(0, 2290)], True),
    (16, 4, 32, 0, [(100, 2148), (3, 4)], True), (16, 4, 16, 1200, [(77, 2300)], True), (16, 8, 16, 1024, [(0, 2048)], False),
    (16, 8, 16, 0, [(0, 2176)], False), (2, 1, 16, 0, [(900, 1143)], False)])
def test_attention_without_softmax_in_halves(nh, nkv, page, window, spans, halves):
    """Tiles whose keys two CTAs take, and that it is so: whole tiles of few keys beside them, a last tile of few rows and of one query tile, windows that cut
    the first half's keys, tokens in front; and the borders of the rule."""
    from airun_b200.kernels import fast
    from ctypes import c_int
    ctx, T, G = batch_ctx(spans), sum(e - s for s, e in spans), nh // nkv
    rows = fast._prompt_tile_rows(T, G, nkv, torch.device("cuda"))
    n = fast._prompt_tiles(ctx, G, rows, T)[1]
    if fast.machine().sms == fast.B200_SMS:
        f = fast._fn("attention_tcgen05", "airun_attn_prefill_in_halves", [c_int] * 5, {"HD": 128})
        assert bool(f(fast.PROMPT_KINDS["sigmoid"], n, nkv, rows, window)) == halves
    test_attention_without_softmax(nh, nkv, page, window, True, True, spans)


SPLIT_CASES = [  # head size, heads, kv heads, page, window, spans: key tiles a query tile has, 1 to 17
    (128, 16, 8, 16, 0, [(900, 1143), (872, 1107)]), (128, 2, 1, 16, 0, [(0, 193)]), (128, 4, 1, 16, 0, [(300, 364)]), (64, 1, 1, 16, 0, [(0, 128)]),
    (128, 2, 2, 32, 0, [(500, 600), (3, 4), (380, 390)]), (64, 8, 2, 32, 0, [(1000, 1100)]), (128, 3, 1, 16, 200, [(700, 900)]),
    (128, 2, 2, 64, 0, [(2000, 2070), (5, 300)]), (64, 20, 4, 16, 0, [(1024, 1100)]), (128, 8, 8, 16, 129, [(0, 700)])]


@gpu
@pytest.mark.parametrize("hd,nh,nkv,page,window,spans", SPLIT_CASES)
def test_few_tiles_whose_keys_are_cut(hd, nh, nkv, page, window, spans):
    """attn_prefill_tc_kernel with the keys of a tile in slices that meet in a cluster: slices of two key tiles and of more, last
    slices that are shorter or empty, tiles too short to be cut beside others that are not."""
    from airun_b200.kernels import fast, ops
    g = torch.Generator().manual_seed(hd + nh + window)
    bt, num_pages = scrambled_table([e for _, e in spans], page, g)
    pool = (0.8 * torch.randn(num_pages, 2, nkv, page, hd, generator=g)).to("cuda", torch.bfloat16)
    ctx = batch_ctx(spans)
    ctx.token_ids = ctx.positions
    q = (2.0 * torch.randn(ctx.num_tokens, nh * hd, generator=g)).to("cuda", torch.bfloat16)
    got, want = torch.full_like(q, 7.0), torch.zeros_like(q)
    plan = fast._attention_plan(ctx, nh // nkv, fast.PREFILL_ROWS)
    fast.attn_prefill_tc(ctx, q, got, SimpleNamespace(pool=pool, block_table=bt, page_size=page), nh, nkv, hd, 0.13, window, plan["tiles"], plan["n_tiles"])
    ops.softmax_attention(q, want, SimpleNamespace(pool=pool.view(num_pages, -1), block_table=bt, page_size=page, shared=False), ctx, nh, nkv, hd, hd,
                          0.13, None, None, window, 1.0)
    rows = torch.tensor([n > 1 for n in ctx.query_lens for _ in range(n)], device="cuda")
    assert int(ctx.err.item()) == 0 and bool((got[~rows] == 7.0).all())
    assert float((got[rows].float() - want[rows].float()).abs().max()) < 3 * 2.0 ** -8 * float(pool.abs().max())


DIFF_CASES = [(1, 1, 16, 0, 0, [(0, 193)]), (4, 2, 32, 64, 0, [(0, 129), (500, 501), (77, 205)]), (3, 1, 16, 37, 0, [(130, 500)]),
              (16, 8, 16, 2048, 0, [(0, 2100)]), (16, 1, 16, 0, 50, [(1000, 1255)]), (6, 3, 64, 300, 90, [(250, 700), (0, 2)])]


@gpu
@pytest.mark.parametrize("nh,nkv,page,chunk,window,spans", DIFF_CASES)
def test_differential(nh, nkv, page, chunk, window, spans):
    """Two maps, a soft cap and the difference's norm, against the plain kernel.  A result is a difference over its root mean
    square: the two means are rounded in their weights alone here (2^-9 of a mean of absolute values, 0.64, at the most, less by
    the root of the keys that matter), over the difference's root mean square, which falls to about 0.04 for rows of a
    thousand keys, times the factor 0.8: 0.03; a mean over the rows of a tenth of that, and the results' own 2^-9."""
    from airun_b200.kernels import fast, ops
    g, cache, ctx, q = made(nh, nkv, page, -1, spans, nh * 31 + chunk)
    part = SimpleNamespace(D=64, Dv=128, nh=nh, nkv=nkv, scale=0.3, cap=20.0, chunk=chunk, window=window, lam=0.45, eps=1e-5, lambda_init=0.2)

    def plain(o):
        ops.diff_attention(q, o, cache.pool, cache.block_table, ctx.positions, ctx.req_of_token, ctx.num_reqs, page, nh, nkv, 64, 128, 0.3, 20.0,
                           chunk, window, 0.45, 1e-5, 0.8, ctx.err)

    got, want = run_both(ctx, q, nh, lambda o: fast.diff_prefill_tc(ctx, q, o, cache, part), plain)
    err = (got - want).view(-1, nh, 128).square().mean(-1).sqrt()
    assert float(err.max()) < 0.03 and float(err.mean()) < 0.004


LATENT_CASES = [  # heads, R, rd, page, window, sink, gate, spans
    (16, 512, 64, 16, 0, True, True, [(0, 300)]), (16, 512, 64, 32, 0, True, False, [(0, 129), (400, 401), (63, 193)]),
    (1, 64, 0, 16, 0, False, False, [(0, 257)]), (33, 320, 64, 16, 100, True, True, [(70, 171)]), (128, 512, 64, 16, 0, False, False, [(190, 260)]),
    (2, 256, 64, 64, 1, False, True, [(0, 65), (3, 5)]), (20, 448, 128, 16, 0, True, True, [(1000, 1064)]), (3, 128, 0, 16, 0, True, False, [(0, 64)]),
    (16, 512, 64, 16, 2048, True, False, [(0, 1100)])]


@gpu
@pytest.mark.parametrize("H,R,rd,page,window,sink,gated,spans", LATENT_CASES)
def test_latent(H, R, rd, page, window, sink, gated, spans):
    """The attention over a cached latent (csrc/latent_attention_tcgen05.cu) against its plain twin."""
    from airun_b200.kernels import fast, ops
    g = torch.Generator().manual_seed(H + R)
    bt, num_pages = scrambled_table([e for _, e in spans], page, g)
    pool = (0.8 * torch.randn(num_pages, page * (R + rd), generator=g)).to("cuda", torch.bfloat16)
    cache = SimpleNamespace(pool=pool, block_table=bt, page_size=page, shared=False)
    ctx = batch_ctx(spans)
    T = ctx.num_tokens
    q = torch.randn(T, H * (R + rd), generator=g).to("cuda", torch.bfloat16)
    sd = (2.0 * torch.randn(H, generator=g)).cuda() if sink else None
    gate = torch.randn(T, H + 3, generator=g).cuda()[:, 3:] if gated else None
    part = SimpleNamespace(nh=H, R=R, rd=rd, scale=1.2 * (R + rd) ** -0.5, window=window, sink=sd)
    got = torch.full((T, H * R), 7.0, device="cuda", dtype=torch.bfloat16)
    want = torch.zeros_like(got)
    assert fast.latent_prefill_tc(ctx, q, got, cache, part, gate)
    ops.latent_attention(q, want, cache, ctx, H, R, rd, part.scale, window, sd, gate)
    assert int(ctx.err.item()) == 0
    rows = torch.tensor([n > 1 for n in ctx.query_lens for _ in range(n)], device="cuda")
    assert bool((got[~rows] == 7.0).all())
    assert float((got[rows].float() - want[rows].float()).abs().max()) < 3 * 2.0 ** -8 * float(pool.abs().max())


# heads, kv heads, page, window, tail, table rows, sink, gate, spans
SINGLE_CASES = [(1, 1, 16, 0, -1, 0, False, False, [(0, 1)]), (2, 1, 16, 0, -1, 0, True, True, [(1499, 1500), (14, 15), (15, 16), (699, 700)]),
                (16, 8, 32, 100, -1, 0, True, False, [(99, 100), (100, 101), (2000, 2001)]), (3, 1, 16, 0, -1, 90, True, True, [(128, 129), (899, 900)]),
                (16, 1, 64, 1, -1, 5, False, False, [(300, 301), (0, 1)]), (4, 2, 16, 0, 64, 0, True, False, [(1023, 1024), (31, 32)]),
                (6, 2, 16, 333, 8, 0, False, True, [(1200, 1201), (17, 18), (0, 1)])]


@gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("nh,nkv,page,window,tail,rows,sink,gated,spans", SINGLE_CASES)
def test_single_tokens(nh, nkv, page, window, tail, rows, sink, gated, spans, mixed):
    """Single tokens alone and beside a portion (csrc/attention_mma.cu: attn_decode_kernel and its kinds), softmax with its options
    and without softmax, against the plain kernels."""
    from airun_b200.kernels import fast, ops
    if mixed:
        spans = spans[:1] + [(3, 30)] + spans[1:]
    g, cache, ctx, q = made(nh, nkv, page, tail, spans, nh + window)
    T = q.shape[0]
    one = torch.tensor([n == 1 for n in ctx.query_lens for _ in range(n)], device="cuda")
    part = SimpleNamespace(D=128, Dv=128, nh=nh, nkv=nkv, scale=0.13, window=window, out_scale=1.3, tail=tail,
                           table=(2.0 * torch.randn(nh, rows, generator=g)).cuda() if rows else None,
                           sink=(2.0 * torch.randn(nh, generator=g)).cuda() if sink else None)
    gate = torch.randn(T, nh * 128 + 4, generator=g).cuda()[:, 4:] if gated else None
    stride = ops.attention_gate(gate, T, nh * 128)
    got = torch.full((T, nh * 128 + 16), 7.0, device="cuda", dtype=torch.bfloat16)
    want = torch.zeros(T, nh * 128, device="cuda", dtype=torch.bfloat16)
    assert fast.attn_single_kind(ctx, "options", q, got[:, 8:8 + nh * 128], cache, part, not mixed, tail=tail, gate=gate, gate_stride=stride)
    ops.softmax_attention(q, want, cache, ctx, nh, nkv, 128, 128, 0.13, part.table, part.sink, window, 1.3, tail=tail, gate=gate)
    assert int(ctx.err.item()) == 0 and bool((got[~one][:, 8:8 + nh * 128] == 7.0).all()) and bool((got[:, :8] == 7.0).all())
    assert float((got[one][:, 8:8 + nh * 128].float() - want[one].float()).abs().max()) < 3 * 2.0 ** -8 * 1.3 * float(cache.pool.abs().max())
    if tail >= 0:
        return
    part.dist_a, part.dist_b, part.head_c = (0.2 + torch.rand(nh, generator=g)).cuda(), (0.1 + torch.rand(nh, generator=g)).cuda(), None
    assert fast.attn_single_kind(ctx, "sigmoid", q, got[:, 8:8 + nh * 128], cache, part, not mixed)
    ops.sigmoid_attention(q, want, cache, ctx, nh, nkv, 128, 128, 0.13, part.dist_a, part.dist_b, None, window)
    assert int(ctx.err.item()) == 0
    most = max(float(want[one].abs().max()), float(cache.pool.abs().max()))
    assert float((got[one][:, 8:8 + nh * 128].float() - want[one].float()).abs().max()) < 3 * 2.0 ** -8 * most


@gpu
def test_what_the_kernel_does_not_take_stays_with_the_other():
    """Small batches, other head sizes, pages of 24, wide groups and unaligned rows are refused, not run."""
    from airun_b200.kernels import fast
    for nh, nkv, page, D, T, off in ((2, 1, 16, 128, 100, 8), (2, 1, 24, 128, 300, 8), (2, 1, 16, 64, 300, 8), (17, 1, 16, 128, 300, 8), (2, 1, 16, 128, 300, 4)):
        bt, pages = scrambled_table([T], page, torch.Generator().manual_seed(1))
        cache = SimpleNamespace(pool=torch.zeros(pages, nkv * page * 2 * D, device="cuda", dtype=torch.bfloat16), block_table=bt, page_size=page)
        part = SimpleNamespace(D=D, Dv=D, nh=nh, nkv=nkv, scale=1.0, window=0, out_scale=1.0, tail=-1, table=None, sink=None)
        q = torch.zeros(T, nh * D, device="cuda", dtype=torch.bfloat16)
        out = torch.zeros(T, nh * D + 8, device="cuda", dtype=torch.bfloat16)[:, off:off + nh * D]
        assert not fast.attn_prompt_kind(batch_ctx([(0, T)]), "options", q, out, cache, part)


@gpu
@pytest.mark.parametrize("scale", [-0.11, 0.0, 1e-32])
def test_latent_with_a_scale_that_is_not_positive(scale):
    """The kernel takes a row's largest score before it scales: a scale of 0 or less goes to the other kernel, and hidden keys stay
    hidden under the smallest ones (the result is the plain kernel's, tolerance as above)."""
    from airun_b200.kernels import fast, ops
    H, R, rd, spans = 4, 128, 64, [(0, 200), (70, 130)]
    g = torch.Generator().manual_seed(5)
    bt, num_pages = scrambled_table([e for _, e in spans], 16, g)
    cache = SimpleNamespace(pool=(0.8 * torch.randn(num_pages, 16 * (R + rd), generator=g)).to("cuda", torch.bfloat16), block_table=bt, page_size=16,
                            shared=False)
    ctx = batch_ctx(spans)
    q = torch.randn(ctx.num_tokens, H * (R + rd), generator=g).to("cuda", torch.bfloat16)
    part = SimpleNamespace(nh=H, R=R, rd=rd, scale=scale, window=0, sink=None)
    got, want = (torch.zeros(ctx.num_tokens, H * R, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    assert fast.latent_attention_bf16(ctx, q, got, cache, part)
    ops.latent_attention(q, want, cache, ctx, H, R, rd, scale, 0, None)
    assert int(ctx.err.item()) == 0 and bool(torch.isfinite(got).all())
    assert float((got.float() - want.float()).abs().max()) < 3 * 2.0 ** -8 * float(cache.pool.abs().max())
