"""One key that outweighs all others, at every place where a kernel's tiles, slices, windows or pages begin or end: the rows that see
it have its value's direction, the others do not.  A key that is lost, counted for a hidden row or read from another place
turns some row round; mean values of a thousand keys would hardly move."""
from types import SimpleNamespace

import pytest
import torch

from test_not_finite import KINDS, made
from test_pirerax import batch_ctx, scrambled_table

gpu = pytest.mark.gpu
KEYS = [0, 15, 16, 63, 64, 127, 128, 129, 255, 256, 383, 384, 511, 512, 640, 699]


def planted(kind, spans, seed):
    run, _, pages, _, rows, ctx, part, bt = made(kind, spans, seed)
    g = torch.Generator().manual_seed(seed)
    width = part.q.shape[1] // part.nh
    u = torch.where(torch.rand(width, generator=g) < 0.5, -0.5, 0.5)
    part.q = u.repeat(part.nh).expand_as(part.q).to("cuda", torch.bfloat16).contiguous()
    pages *= 0.05                                            # every other score lies near zero
    row = (8.0 * u).to("cuda", torch.bfloat16)               # a score of 33 and more above them
    return run, pages, rows, ctx, part, bt, row, torch.randn(512, generator=g).to("cuda", torch.bfloat16)


def plant(kind, pages, part, page, at, row, value):
    """The key in every head; the direction of its value per head [width]."""
    kind = kind.split()[0]
    if kind == "latent":
        pages[page, 0, at] = row
        return row[:part.R].float()
    if kind == "one":
        pages[page, :, at, :128], pages[page, :, at, 128:] = row, value[:64]
        return pages[page, 0, at, 64:].float()
    pages[page, :part.nkv, at] = row
    pages[page, part.nkv:, at] = value[:128]
    return value[:128].float()


def like(out, direction, heads):
    o = out.float().view(out.shape[0], heads, -1)
    return torch.nn.functional.cosine_similarity(o, direction.expand_as(o), dim=-1)


@gpu
@pytest.mark.parametrize("kind", list(KINDS))
def test_prompts(kind):
    spans = [(130, 700), (0, 40)]
    window, chunk = KINDS[kind]
    run, pages, rows, ctx, part, bt, row, value = planted(kind, spans, 5)
    pos, mine = ctx.positions, ctx.req_of_token == 0
    for j in KEYS:
        p = pages.clone()
        d = plant(kind, p, part, int(bt[0, j // 16]), j % 16, row, value)
        sees = mine & (pos >= j)
        if window:
            sees &= pos - j < window
        if chunk:
            sees &= pos // chunk == j // chunk
        got = like(run(p), d, part.nh)
        assert bool((got[sees] > 0.9).all()) and bool((got[rows & ~sees].abs() < 0.7).all()), (j, got[sees].min() if sees.any() else None)


@gpu
@pytest.mark.parametrize("kind", [k for k in KINDS if not k.startswith(("diff", "latent"))])
def test_single_tokens(kind):
    spans = [(1023, 1024), (699, 700), (99, 100), (15, 16), (300, 301)]
    window, _ = KINDS[kind]
    run, pages, rows, ctx, part, bt, row, value = planted(kind, spans, 6)
    for r, (first, _) in enumerate(spans):
        for j in sorted({0, first} | {k for k in KEYS + [1007, 1008] if k < first} | ({first - window, first - window + 1} if window and first >= window else set())):
            p = pages.clone()
            d = plant(kind, p, part, int(bt[r, j // 16]), j % 16, row, value)
            got = like(run(p), d, part.nh)
            sees = not window or first - j < window
            assert bool((got[r] > 0.9).all()) == sees, (r, j, got[r])
            assert bool((got[torch.arange(len(spans)) != r].abs() < 0.7).all())


@gpu
@pytest.mark.parametrize("hd,nh,nkv,window,spans", [(128, 4, 2, 0, [(900, 1143)]), (128, 2, 1, 300, [(700, 900), (0, 130)]), (64, 4, 1, 0, [(640, 700)])])
def test_prompts_of_few_tiles_whose_keys_are_cut(hd, nh, nkv, window, spans):
    """The plain prompt attention with a tile's keys in slices that meet in a cluster (csrc/attention_tcgen05.cu)."""
    from airun_b200.kernels import fast
    g = torch.Generator().manual_seed(hd)
    bt, num_pages = scrambled_table([e for _, e in spans], 16, g)
    pool = (0.04 * torch.randn(num_pages, 2, nkv, 16, hd, generator=g)).to("cuda", torch.bfloat16)
    ctx = batch_ctx(spans)
    ctx.token_ids = ctx.positions
    u = torch.where(torch.rand(hd, generator=g) < 0.5, -0.5, 0.5)
    q = u.repeat(nh).expand(ctx.num_tokens, nh * hd).to("cuda", torch.bfloat16).contiguous()
    value = torch.randn(hd, generator=g).to("cuda", torch.bfloat16)
    plan = fast._attention_plan(ctx, nh // nkv, fast.PREFILL_ROWS)
    pos, mine = ctx.positions, ctx.req_of_token == 0
    for j in [k for k in KEYS + [767, 768, 895, 896, 1023, 1024, 1142] if k < spans[0][1]]:
        p = pool.clone()
        p[int(bt[0, j // 16]), 0, :, j % 16], p[int(bt[0, j // 16]), 1, :, j % 16] = (16.0 * u).to("cuda", torch.bfloat16), value
        out = torch.zeros_like(q)
        fast.attn_prefill_tc(ctx, q, out, SimpleNamespace(pool=p, block_table=bt, page_size=16), nh, nkv, hd, 0.13, window, plan["tiles"], plan["n_tiles"])
        sees = mine & (pos >= j)
        if window:
            sees &= pos - j < window
        got = like(out, value.float(), nh)
        assert bool((got[sees] > 0.9).all()) and bool((got[~sees].abs() < 0.7).all()), j
    assert int(ctx.err.item()) == 0
