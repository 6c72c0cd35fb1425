"""The kernels between the products at the sizes where their forms change: the router's single block and its many, norms whose
rows, weights and results do or do not allow 16-byte accesses, copies of pages that one block or several take, and the
epilogue of the products for up to 128 tokens."""
import pytest
import torch

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("T,E,top", [(1, 16, 4), (31, 16, 16), (32, 40, 3), (33, 40, 3), (70, 16, 1), (7, 64, 40), (40, 64, 33), (32, 700, 8), (2, 1024, 8)])
def test_router_of_one_block_and_of_many(T, E, top, grouped):
    """Scores in float32 differ from float64 by a few units of their last place (expf: 2) and by the sum over E of them;
    8 + E / 16 units of 2^-24 of the score hold."""
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(T + E)
    z = torch.randn(T, E, generator=g)
    off = torch.randn(E, generator=g) * 0.1
    req = torch.zeros(T, dtype=torch.int32)
    if T > 2:
        req[[1, T - 1]] = -1
    live = req >= 0
    ids, rank = (torch.full((T, top), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    wts = torch.zeros(T, top, device="cuda")
    real = E - 3 if grouped else E
    counts, seg = torch.zeros(real, dtype=torch.int32, device="cuda"), torch.full((real + 1,), -1, dtype=torch.int32, device="cuda")
    if grouped:
        s = torch.softmax(z.double(), -1)
        choice = s + off.double()
        ops.moe_route_grouped(z.cuda(), real, top, 1, 1, 1.5, off.cuda(), req.cuda(), ids, wts, rank, counts, seg)
    else:
        s = torch.sigmoid(z.double() + off.double())
        choice = z.double() + off.double()
        ops.moe_route(z.cuda(), top, False, True, req.cuda(), ids, wts, rank, counts, seg, bias=off.cuda())
    got, r, c, sg = ids.cpu().long(), rank.cpu().long(), counts.cpu().long(), seg.cpu().long()
    assert (got[~live] == -1).all()
    # the order of the choice, up to float32's doubt about two scores
    order = choice.gather(1, got.clamp(min=0))[live]
    doubt = 1e-6
    assert bool((order[:, 1:] <= order[:, :-1] + doubt).all())
    assert bool((order[:, -1] >= torch.topk(choice[live], top, -1).values[:, -1] - doubt).all())
    assert all(len(set(row.tolist())) == top for row in got[live])
    chosen = s.gather(1, got.clamp(min=0))[live]
    want = chosen / chosen.sum(-1, keepdim=True) * (1.5 if grouped else 1.0)
    assert bool(((wts.cpu().double()[live] - want).abs() <= (8 + E / 16 + top) * 2.0 ** -24 * want).all())
    flat, fr = got[live].reshape(-1), r[live].reshape(-1)
    here = flat < real
    assert torch.equal(c, torch.bincount(flat[here], minlength=real))
    assert torch.equal(sg, torch.cat([torch.zeros(1, dtype=torch.long), torch.cumsum(c, 0)]))
    rows = sg[flat[here]] + fr[here]
    assert sorted(rows.tolist()) == list(range(int(here.sum())))                    # every row of the segments is used once


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n", [(1, 4), (3, 130), (1, 4096), (64, 1024), (65, 4096), (200, 8200), (2, 9000), (300, 512), (5, 33)])
@pytest.mark.parametrize("off", [0, 1])
def test_norms_on_and_off_their_alignment(rows, n, off, dtype):
    """float32: a sum of n squares in chains of at most n / 32 and six levels of adds, halved by the root, and three
    products: (n / 64 + 8) units of 2^-24 of the value; bfloat16 rounds once more, to half a unit: 2^-8 of the value at most."""
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(rows + n)

    def shifted(t):                                      # the same numbers, `off` elements into their storage
        store = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
        store[off:off + t.numel()] = t.reshape(-1).cuda()
        return store[off:off + t.numel()].view(t.shape)

    x, d = torch.randn(rows, n, generator=g), torch.randn(rows, n, generator=g)
    w, w2 = torch.randn(n, generator=g), torch.randn(n, generator=g)
    tol = (n / 64 + 8) * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    norm = lambda v, weight: v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * weight
    ok = lambda got, want: bool(((got.cpu().double() - want).abs() <= tol * want.abs() + 1e-30).all())
    X, out, out2 = shifted(x), shifted(torch.zeros(rows, n, dtype=dtype)), shifted(torch.zeros(rows, n, dtype=dtype))
    ops.rmsnorm_pair(X, shifted(w), out, shifted(w2), out2, 1e-5, delta=shifted(d))
    s = (x + d).double()
    assert torch.equal(X.cpu(), x + d) and ok(out, norm(s, w.double())) and ok(out2, norm(s, w2.double()))
    pick = torch.tensor([rows - 1, 0], dtype=torch.int32, device="cuda")
    gathered = shifted(torch.zeros(2, n, dtype=dtype))
    ops.rmsnorm(X, shifted(w), 1e-5, gathered, rows=pick)
    assert ok(gathered, norm(s, w.double())[[rows - 1, 0]]) and torch.equal(X.cpu(), x + d)
    Y, cast = shifted(x), shifted(torch.zeros(rows, n, dtype=dtype))
    ops.postnorm_add(Y, shifted(d), shifted(w), 1e-5, 0.7, cast=cast)
    part = 0.7 * norm(d.double(), w.double())
    want, size = x.double() + part, x.abs().double() + part.abs()
    assert bool(((Y.cpu().double() - want).abs() <= (n / 64 + 8) * 2.0 ** -24 * size).all())
    assert torch.equal(cast.cpu(), Y.cpu().to(dtype))


@gpu
@pytest.mark.parametrize("words", [1, 1023, 1024, 1025, 70000])
def test_pages_of_one_block_and_of_several(words):
    from airun_b200.kernels import ops
    pool = torch.randint(-2 ** 31, 2 ** 31 - 1, (3, 6, 4 * words), dtype=torch.int32, device="cuda")
    want = pool.clone()
    want[:, 5], want[:, 0] = pool[:, 1], pool[:, 4]
    ops.copy_pages(pool, torch.tensor([[1, 5], [4, 0]], dtype=torch.int32, device="cuda"))
    assert torch.equal(pool, want)


@gpu
@pytest.mark.parametrize("ksplit", [1, 3, 10])           # one slice, a cluster, slices through the scratch
@pytest.mark.parametrize("epi", [0, 1, 2])
@pytest.mark.parametrize("M,bn", [(1, 32), (8, 32), (9, 32), (16, 32), (17, 32), (31, 32), (33, 64), (40, 64), (48, 64), (49, 64), (64, 64),
                                  (65, 128), (80, 128), (97, 128), (127, 128), (128, 128), (70, 64), (200, 128)])
def test_products_with_the_tokens_as_columns(M, bn, epi, ksplit):
    """The epilogue of the swapped product takes the tile's tokens 32, 16 and 8 at a time.  Rows behind the last token stay as
    they are.  float32: sums of K products in the tensor core, 2^-14 of the largest possible sum; bfloat16 results round
    to half a unit more; the gated unit g sigmoid(g) u has slopes of at most 1.1 |u| and |g|."""
    from airun_b200.kernels import fast
    N, K = 288, 712
    g = torch.Generator().manual_seed(M + epi)
    x, w = torch.randn(M, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) * K ** -0.5).bfloat16()
    out = torch.full((M + 3, N // 2 if epi == 2 else N), 7.0, dtype=torch.float32 if epi == 0 else torch.bfloat16, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):
        fast.gemm_tcgen05(x.cuda(), w.cuda(), out[:M], epi, True, bn, ksplit, err)
    want = x.double() @ w.double().T
    e = 2.0 ** -14 * (x.double().abs() @ w.double().abs().T)
    if epi == 2:
        a, b = (t.view(M, N // 32, 2, 16) for t in (want, e))
        (gate, up), (eg, eu) = ((t[:, :, 0].reshape(M, -1), t[:, :, 1].reshape(M, -1)) for t in (a, b))
        want = gate * torch.sigmoid(gate) * up
        e = 1.1 * up.abs() * eg + gate.abs() * eu
    if epi:
        e = e + 2.0 ** -8 * want.abs()
    assert int(err.item()) == 0 and bool(((out[:M].cpu().double() - want).abs() <= e + 1e-30).all())
    assert bool((out[M:] == 7.0).all())


@gpu
@pytest.mark.parametrize("how", ["rows", "rows grouped", "columns", "columns cluster", "persistent", "pairs", "pairs grouped"])
@pytest.mark.parametrize("limit", [0.0, 7.0])
def test_gated_units_of_gates_far_below_zero(how, limit):
    """silu(-88) is -5e-37 and is multiplied by up to 1e30: the quotient's divisor, e^88, lies beyond 2^126, where the fast
    division gives zero.  e^x is right to 2 + 1.2 |x| units of 2^-24; bfloat16 results round to 2^-8."""
    from types import SimpleNamespace

    from airun_b200.kernels import fast
    M, N, K = (5 if how.startswith("rows") else 40 if how.startswith("columns") else 300), 512, 64
    g = torch.Generator().manual_seed(M)
    gate, up = -80.0 - 8.4 * torch.rand(N // 2, generator=g), 1.0e30 * torch.randn(N // 2, generator=g)
    w = torch.zeros(N // 32, 2, 16, K)
    w[:, 0, :, 0], w[:, 1, :, 1] = gate.view(-1, 16), up.view(-1, 16)
    w = w.view(N, K).bfloat16()
    x = torch.zeros(M, K).bfloat16()
    x[:, 0] = 1.0
    x[:, 1] = torch.randn(M, generator=g).bfloat16()
    z = (x.double() @ w.double().T).view(M, N // 32, 2, 16)
    a, b = z[:, :, 0].reshape(M, -1), z[:, :, 1].reshape(M, -1)
    if limit:
        want = a * torch.sigmoid(a) * (b.clamp(-limit, limit) + 1)
    else:
        want = a * torch.sigmoid(a) * b
    out = torch.full((M, N // 2), 7.0, dtype=torch.bfloat16, device="cuda")
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    xd, wd, glu = x.cuda(), w.cuda(), (limit, 1.0 if limit else 0.0)
    if "grouped" in how:
        seg = torch.tensor([0, M], dtype=torch.int32, device="cuda")
        old, fast.GROUPED_ROWS_MAX = fast.GROUPED_ROWS_MAX, 64 if how.startswith("rows") else 0
        try:
            assert fast.grouped_linear_bf16(ctx, xd, wd[None].contiguous(), out, seg, swiglu_group=16, **(dict(glu=glu) if limit else {}))
        finally:
            fast.GROUPED_ROWS_MAX = old
    elif how == "pairs":
        fast.gemm_pair(xd, wd, out, fast.EPI_SWIGLU, ctx.err, glu=glu, in_parts=limit > 0)
    elif limit:
        assert fast.linear_glu_clamped_bf16(ctx, xd, wd, out, 16, limit, 1.0)
    elif how == "rows":
        fast.gemm_rows(xd, wd, out, fast.EPI_SWIGLU, glu=glu)
    else:
        swap = how.startswith("columns")
        fast.gemm_tcgen05(xd, wd, out, fast.EPI_SWIGLU, swap, 64 if swap else 256, 1, ctx.err)
    assert int(ctx.err.item()) == 0 and float(want.abs().min()) > 0
    assert bool(((out.cpu().double() - want).abs() <= (2.0 ** -8 + 2e-5) * want.abs() + 1.2e-38).all())


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M", [5, 40, 300])
def test_silu_far_below_zero(M, dtype):
    """z sigmoid(z) as an epilogue where e^-z lies beyond 2^126 (see above)."""
    from types import SimpleNamespace

    from airun_b200.kernels import fast, ops
    N, K = 512, 64
    w = torch.zeros(N, K)
    w[:, 0] = -80.0 - 8.4 * torch.rand(N, generator=torch.Generator().manual_seed(M))
    w, x = w.bfloat16(), torch.zeros(M, K).bfloat16()
    x[:, 0] = 1.0
    z = x.double() @ w.double().T
    want = z * torch.sigmoid(z)
    out, err = torch.full((M, N), 7.0, dtype=dtype, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    epi, silu = (fast.EPI_F32 if dtype == torch.float32 else fast.EPI_BF16), ops.ACTIVATIONS["silu"]
    if M == 5:
        fast.gemm_rows(x.cuda(), w.cuda(), out, epi, act=silu)
    else:
        fast.gemm_tcgen05(x.cuda(), w.cuda(), out, epi, M == 40, 64 if M == 40 else 256, 1, err, act=silu)
    assert int(err.item()) == 0
    assert bool(((out.cpu().double() - want).abs() <= ((2.0 ** -8 if dtype == torch.bfloat16 else 0) + 2e-5) * want.abs() + 1.2e-38).all())


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,top,W", [(5, 2, 64), (3, 1, 10)])
def test_rows_of_experts_that_have_no_place(T, top, W, dtype):
    """Ranks and segments that place a row outside the buffer (an older list, say): the row is left out, the error word says so, and
    what lies around the buffer stays."""
    from airun_b200.kernels import ops
    store = torch.full((T * top + 4, W), 7.0, dtype=dtype, device="cuda")
    xs, err = store[2:-2], torch.zeros(1, dtype=torch.int32, device="cuda")
    h = torch.randn(T, W, dtype=torch.float32).to("cuda", dtype)
    ids, rank = torch.zeros(T, top, dtype=torch.int32), torch.arange(T * top, dtype=torch.int32).view(T, top)
    rank[0, 0], rank[T - 1, top - 1] = -1, T * top
    seg = torch.tensor([0, T * top], dtype=torch.int32, device="cuda")
    row_of, wts = torch.full((T, top), -9, dtype=torch.int32, device="cuda"), torch.ones(T, top, device="cuda")
    ids, rank = ids.cuda(), rank.cuda()
    ops.moe_scatter(h, top, ids, wts, rank, seg, False, xs, row_of, num_real=1, err=err)
    assert int(err.item()) == 16 and "row" in ops.describe_device_error(16)
    assert row_of[0, 0] == -1 and row_of[T - 1, top - 1] == -1 and bool((store[:2] == 7).all()) and bool((store[-2:] == 7).all())
    assert bool((xs[0] == 7).all()) and bool((xs[T * top - 1] == 7).all())
    for r in range(1, T * top - 1):
        assert torch.equal(xs[r], h[r // top]) and int(row_of.view(-1)[r]) == r
    ys, out = torch.randn(T * top, W, device="cuda"), torch.empty(T, W, device="cuda")
    bad = row_of.clone()
    bad[bad < 0] = T * top + 1000                                    # and a row number from elsewhere is not read
    ops.moe_combine(ys, top, ids, wts, bad, False, out)
    want = torch.where((row_of >= 0)[..., None], ys.view(T, top, W), torch.zeros(1, device="cuda")).sum(1)
    assert torch.allclose(out, want, atol=1e-6)


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,n,rank", [(1, 5, 8), (8, 128, 16), (21, 300, 24), (9, 130, 32), (17, 64, 40), (10, 200, 12), (3, 33, 1), (16, 129, 1024)])
def test_low_rank_pairs_that_end_in_a_function(T, n, rank, dtype):
    """Rows of the second matrix in pieces of eight (up to 32 of them ahead, more in turn) and one number at a time, against 64 bits.  Tolerance: z is a sum
    of rank products in float32 (2^-24 * rank of the sum of absolute values), and no function is steeper than 4 where it is not saturated."""
    from airun_b200.kernels import ops
    g = torch.Generator().manual_seed(rank + n)
    low, w2, bias = torch.randn(T, rank + 4, generator=g)[:, :rank], (torch.randn(n, rank, generator=g) * rank ** -0.5).to(dtype), torch.randn(n, generator=g)
    req = torch.zeros(T, dtype=torch.int32)
    req[T // 2] = -1 if T > 4 else 0
    param = torch.randn(n, generator=g) * 0.5
    z = bias.double() + low.double() @ w2.double().T
    zt = low.double().tanh() @ w2.double().T
    err = 2.0 ** -24 * (rank + 8) * (bias.double().abs() + low.double().abs() @ w2.double().abs().T + 1)
    soft = torch.nn.functional.softplus
    out = torch.full((T, n), 7.0, device="cuda")
    for mode, want, kw in ((ops.LOWRANK_EXP_SOFTPLUS, torch.exp(-torch.exp(param.double()) * soft(z)), dict(group_param=param.cuda(), group=1)),
                           (ops.LOWRANK_SIGMOID, torch.sigmoid(z), {}), (ops.LOWRANK_EXP_NEG_EXP, torch.exp(-torch.exp(zt)), dict(in_tanh=True)),
                           (ops.LOWRANK_POW_SIGMOID, torch.sigmoid(z) ** (1 / 16.0), dict(tau=16.0))):
        out.fill_(7.0)
        ops.lowrank_act(low.cuda(), w2.cuda(), None if "in_tanh" in kw else bias.cuda(), out, req.cuda(), mode, **kw)
        got = out.cpu().double()
        live = req >= 0
        assert bool(((got - want).abs()[live] <= 4 * err[live] + 2e-6).all()) and bool((got[~live] == 7.0).all())
