"""What is not a number or not finite in the attentions.  Rows of a page that no token of the batch may see hold anything: what an
earlier request left there, or another request's rows where a tile reads past a request's last page.  They must not reach a
result, so every kernel gives the same bits over pages whose unseen rows are zeros and over pages where these are NaN or
infinite.  A visible key that is NaN reaches exactly the rows that see it."""
import pytest
import torch

from test_pirerax import batch_ctx, scrambled_table

gpu = pytest.mark.gpu


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
