"""What is not a number, not finite or near the ends of float32 in the attentions.  Rows of a page that no token of the batch may see hold anything: what an
earlier request left there, or another request's rows where a tile reads past a request's last page.  They must not reach a
result, so every kernel gives the same bits over pages whose unseen rows are zeros and over pages where these are NaN or
infinite.  A visible key that is NaN reaches exactly the rows that see it."""
from types import SimpleNamespace

import pytest
import torch

from test_pirerax import batch_ctx, scrambled_table

gpu = pytest.mark.gpu
PROMPTS = [(130, 333), (5, 41), (700, 701)]              # (first position, end) of the requests
SINGLES = [(0, 1), (14, 15), (299, 300), (1000, 1001), (1023, 1024)]
KINDS = {  # window, chunk
    "options": (0, 0), "window": (100, 0), "table": (0, 0), "table window": (77, 0), "one row": (0, 0), "sigmoid": (0, 0), "sigmoid window": (33, 0),
    "differential": (0, 64), "differential window": (50, 0), "latent": (0, 0), "latent window": (70, 0)}


def made(kind, spans, seed, page=16):
    """(run, plain, pages, rows of a page that some token sees, context): ``run(pages)`` and ``plain(pages)`` are the kernel
    for this kind on the tensor cores and its plain twin, or run gives None where the kernel does not take single tokens."""
    from airun_b200.kernels import fast, ops
    window, chunk = KINDS[kind]
    kind = kind.split()[0]
    g = torch.Generator().manual_seed(seed)
    bt, num_pages = scrambled_table([e for _, e in spans], page, g)
    nh, nkv, R, rd = 4, 2, 192, 64
    seen = torch.zeros(num_pages, page, dtype=torch.bool)
    for r, (a, b) in enumerate(spans):
        lo = max(0, a - window + 1) if window else 0
        if chunk:
            lo = max(lo, a // chunk * chunk)
        for j in range(lo, b):
            seen[int(bt[r, j // page]), j % page] = True
    ctx = batch_ctx(spans)
    T, single = ctx.num_tokens, ctx.decode_only
    if kind == "latent":
        width, shape, qw, ow = R + rd, (num_pages, 1, page, R + rd), nh * (R + rd), nh * R
    else:
        width = 192 if kind == "one" else 256
        shape, qw, ow = ((num_pages, nkv, page, 192) if kind == "one" else (num_pages, 2 * nkv, page, 128)), nh * 128, nh * 128
    pages = (0.8 * torch.randn(shape, generator=g)).to("cuda", torch.bfloat16)
    q = torch.randn(T, qw, generator=g).to("cuda", torch.bfloat16)
    part = SimpleNamespace(D=128, Dv=128, nh=nh, nkv=nkv, scale=0.13, window=window, out_scale=1.0, tail=64 if kind == "one" else -1,
                           table=torch.randn(nh, 400, generator=g).cuda() if kind == "table" else None, sink=torch.zeros(nh, device="cuda"),
                           dist_a=torch.full((nh,), 0.4, device="cuda"), dist_b=torch.full((nh,), 0.2, device="cuda"), head_c=None, R=R, rd=rd,
                           chunk=chunk, cap=20.0, lam=0.45, eps=1e-5, lambda_init=0.2, gate=None, q=q)
    if kind == "differential":
        part.D = 64

    def cache(p):
        return SimpleNamespace(pool=p.reshape(num_pages, -1), block_table=bt, page_size=page, shared=False)

    def run(p):
        out = torch.full((T, ow), 7.0, device="cuda", dtype=torch.bfloat16)
        if kind == "latent":
            took = not single and fast.latent_prefill_tc(ctx, part.q, out, cache(p), part, part.gate)
        elif kind == "differential":
            took = not single and fast.diff_prefill_tc(ctx, part.q, out, cache(p), part)
        else:
            name = "options" if kind in ("one", "window") else kind
            more = {} if kind == "sigmoid" else dict(gate=part.gate, gate_stride=ops.attention_gate(part.gate, T, ow))
            if single:
                took = fast.attn_single_kind(ctx, name if name == "sigmoid" else "options", part.q, out, cache(p), part, True, tail=part.tail, **more)
            else:
                took = fast.attn_prompt_kind(ctx, name, part.q, out, cache(p), part, tail=part.tail, **more)
        assert int(ctx.err.item()) == 0
        return out if took else None

    def plain(p):
        out = torch.zeros(T, ow, device="cuda", dtype=torch.bfloat16)
        if kind == "latent":
            ops.latent_attention(part.q, out, cache(p), ctx, nh, R, rd, 0.13, window, part.sink, part.gate)
        elif kind == "differential":
            ops.diff_attention(part.q, out, cache(p).pool, bt, ctx.positions, ctx.req_of_token, ctx.num_reqs, page, nh, nkv, 64, 128, 0.13, 20.0, chunk,
                               window, 0.45, 1e-5, 0.8, ctx.err)
        elif kind == "sigmoid":
            ops.sigmoid_attention(part.q, out, cache(p), ctx, nh, nkv, 128, 128, 0.13, part.dist_a, part.dist_b, part.head_c, window)
        else:
            ops.softmax_attention(part.q, out, cache(p), ctx, nh, nkv, 128, 128, 0.13, part.table, part.sink, window, 1.0, tail=part.tail, gate=part.gate)
        return out

    rows = torch.tensor([single or n > 1 for n in ctx.query_lens for _ in range(n)], device="cuda")
    return run, plain, pages, seen.cuda(), rows, ctx, part, bt


def spoil(kind, pages, page, row):
    """The key of the first KV head; of a row that is key and value the part that is no value (a weight of zero times a value that
    is NaN is NaN in a matrix product: a NaN VALUE reaches the tokens of its own request beside it, as it always did)."""
    part = slice(0, 64) if kind == "one row" else slice(192, 256) if kind.startswith("latent") else slice(None)
    pages[page, 0, row, part] = float("nan")


@gpu
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3.0e38])
@pytest.mark.parametrize("spans", [PROMPTS, SINGLES], ids=["prompts", "singles"])
@pytest.mark.parametrize("kind", list(KINDS))
def test_rows_that_no_token_sees(kind, spans, bad):
    run, _, pages, seen, rows, _, _, _ = made(kind, spans, len(kind))
    unseen = ~seen[:, None, :, None].expand_as(pages)
    zeros = run(pages.masked_fill(unseen, 0.0))
    if zeros is None:
        pytest.skip("single tokens of this kind have a kernel of their own")
    anything = run(pages.masked_fill(unseen, bad))
    assert bool(torch.isfinite(zeros[rows]).all()) and torch.equal(zeros[rows], anything[rows])


@gpu
@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("nh,nkv", [(1, 1), (4, 2), (8, 2)])
def test_unseen_rows_and_nan_keys_in_float32(hd, nh, nkv):
    """The attention of the true 32-bit path: as above, and a NaN score makes its row NaN as it does in plain torch."""
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(hd + nh)
    spans = [(3, 40), (0, 1), (70, 71), (98, 99)]
    bt, num_pages = scrambled_table([e for _, e in spans], 16, g)
    ctx = batch_ctx(spans)
    seen = torch.zeros(num_pages, 16, dtype=torch.bool)
    for r, (_, b) in enumerate(spans):
        for j in range(b):
            seen[int(bt[r, j // 16]), j % 16] = True
    pages = torch.randn(num_pages, 2, nkv, 16, hd, generator=g)
    q = torch.randn(ctx.num_tokens, nh * hd, generator=g).cuda()

    def run(p):
        out = torch.empty_like(q)
        ops.attention_generic(q, out, p.cuda(), bt, ctx.positions, ctx.req_of_token, ctx.num_reqs, nh, nkv, hd, hd ** -0.5, 0, ctx.err)
        assert int(ctx.err.item()) == 0
        return out

    unseen = ~seen[:, None, None, :, None].expand_as(pages)
    clean = run(pages.masked_fill(unseen, 0.0))
    assert bool(torch.isfinite(clean).all())
    for bad in (float("nan"), float("inf")):
        assert torch.equal(clean, run(pages.masked_fill(unseen, bad)))
    for bad in (float("nan"), float("inf")):
        sick = pages.masked_fill(unseen, 0.0)
        sick[int(bt[0, 1]), 0, 0, 4] = bad               # key 20 of request 0, first KV head
        got = run(sick).view(-1, nh, hd)
        hit = ((ctx.req_of_token == 0) & (ctx.positions >= 20))[:, None] & (torch.arange(nh, device="cuda") < nh // nkv)[None]
        # (an infinite key gives an infinite score or, where signs differ, a NaN: neither leaves a finite row)
        assert bool(torch.isnan(got[hit]).all()) and torch.equal(got[~hit], clean.view(-1, nh, hd)[~hit])


@gpu
@pytest.mark.parametrize("key", [140, 141, 255, 256, 332])
@pytest.mark.parametrize("kind", list(KINDS))
def test_a_nan_key_of_a_prompt_reaches_the_rows_that_see_it(kind, key):
    run, plain, pages, seen, rows, ctx, part, bt = made(kind, PROMPTS, len(kind) + key)
    clean = run(pages)
    sick = pages.clone()
    spoil(kind, sick, int(bt[0, key // 16]), key % 16)
    got = run(sick)
    want = torch.isnan(plain(sick))
    hit = (ctx.req_of_token == 0) & (ctx.positions >= key) & rows
    assert bool(want[hit].any()) and torch.equal(torch.isnan(got[rows]), want[rows])
    fine = ~want[rows].view(rows.sum(), part.nh, -1).any(-1)
    assert torch.equal(got[rows].view(fine.shape[0], part.nh, -1)[fine], clean[rows].view(fine.shape[0], part.nh, -1)[fine])


@gpu
@pytest.mark.parametrize("key", [0, 13, 14, 290, 299])
@pytest.mark.parametrize("kind", [k for k in KINDS if not k.startswith(("diff", "latent"))])
def test_a_nan_key_of_a_single_token(kind, key):
    run, plain, pages, seen, rows, ctx, part, bt = made(kind, SINGLES, len(kind) + key)
    clean = run(pages)
    sick = pages.clone()
    spoil(kind, sick, int(bt[2, key // 16]), key % 16)
    got, want = run(sick), torch.isnan(plain(sick))
    assert torch.equal(torch.isnan(got), want) and torch.equal(got[~want], clean[~want])
    if not part.window or 299 - key < part.window:
        assert bool(want[2].any())


@gpu
@pytest.mark.parametrize("spans", [PROMPTS, SINGLES], ids=["prompts", "singles"])
def test_distance_terms_near_the_lowest_number(spans):
    """Every distance of the second head costs 1e32: a row's weights go by the differences, and no row may come out empty."""
    run, plain, pages, seen, rows, ctx, part, bt = made("table", spans, 3)
    part.table[1] = -1.0e32
    part.sink = None
    got, want = run(pages)[rows].float(), plain(pages)[rows].float()
    assert bool(torch.isfinite(want).all()) and bool((want.view(-1, 4, 128)[:, 1].abs().amax(-1) > 0).all())
    # both work in float32 at 1e32, where the scores vanish: the mean of the visible values, rounded (see test_prompt_attention)
    assert float((got - want).abs().max()) < 3 * 2.0 ** -8 * float(pages.abs().max())


@gpu
@pytest.mark.parametrize("spans", [PROMPTS, SINGLES], ids=["prompts", "singles"])
def test_sigmoid_weights_far_below_one(spans):
    """A score offset of -60: weights of e^-60 times values of up to 1e25.  bfloat16 weights and results: 3 * 2^-8 of the
    largest result, as in test_prompt_attention."""
    run, plain, pages, seen, rows, ctx, part, bt = made("sigmoid", spans, 4)
    part.head_c = torch.full((4,), -60.0, device="cuda")
    pages[:, 2:] *= 1.0e25
    got, want = run(pages)[rows].float(), plain(pages)[rows].float()
    assert bool(torch.isfinite(got).all()) and float((got - want).abs().max()) < 3 * 2.0 ** -8 * float(want.abs().max())


@gpu
@pytest.mark.parametrize("spans", [PROMPTS, SINGLES], ids=["prompts", "singles"])
@pytest.mark.parametrize("kind", ["options", "table", "one row", "latent"])
def test_gates_far_below_zero(kind, spans):
    """sigmoid(-88) is 6e-39 times values of 1e30: a quotient whose divisor is beyond 2^126 must not become zero."""
    run, plain, pages, seen, rows, ctx, part, bt = made(kind, spans, 6)
    if kind in ("options", "table"):
        pages[:, 2:] *= 1.0e30
    else:
        pages *= 1.0e30                                      # key and value at once: the queries make up for it
        part.q = (part.q * 1.0e-30).contiguous()
    part.gate = torch.full((ctx.num_tokens, 4 if kind == "latent" else 512), -88.0, device="cuda")
    got = run(pages)
    if got is None:
        pytest.skip("single tokens of this kind have a kernel of their own")
    got, want = got[rows].float(), plain(pages)[rows].float()
    assert float(want.abs().max()) > 1e-10 and float((got - want).abs().max()) < 3 * 2.0 ** -8 * float(want.abs().max())
