"""Products on pairs of SMs (csrc/gemm_tcgen05.cu) against float64 products of the same bfloat16 operands.

Tolerance: sums of K products in float32 (2^-24 * K of the sum of absolute values at most; the tensor cores cut off, 2^-23 a step of 16), and for
bfloat16 results half a unit of theirs (2^-9, doubled for the gated unit's and the activation's own roundings)."""
import pytest
import torch

gpu = pytest.mark.gpu
# tokens, weight rows, K, tokens of a tile: one row, edges of tiles and of pairs, ragged rows and K, several rounds of the persistent pairs
SHAPES = [(1, 32, 8, 32), (33, 256, 64, 32), (64, 288, 520, 64), (129, 300, 1000, 96), (257, 4096, 128, 256), (600, 5120, 72, 32), (700, 544, 2048, 160),
          (2048, 6144, 256, 224)]


def operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K + 8, device="cuda", generator=g).bfloat16()[:, :K]
    return x, (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).bfloat16()


def check(got, want, most, K, dtype):
    tol = 2.0 ** -23 * (K / 16 + 8) * most + (2.0 ** -8 * want.abs() + 1e-6 if dtype == torch.bfloat16 else 1e-7)
    assert bool(((got.double() - want).abs() <= tol).all())


@gpu
@pytest.mark.parametrize("in_parts", [False, True])
@pytest.mark.parametrize("M,N,K,bn", SHAPES)
def test_plain_activation_and_gated(M, N, K, bn, in_parts):
    """``in_parts``: one part of a few K-steps to several with a short last one, over several tiles."""
    from airun_b200.kernels import fast, ops
    bn = min(bn, fast.PAIR_PARTS_BN) if in_parts else bn
    x, w = operands(M, N, K, M + N + K)
    want, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for dtype, epi in ((torch.float32, fast.EPI_F32), (torch.bfloat16, fast.EPI_BF16)):
        out = torch.full((M, N + 8), 3.0, device="cuda", dtype=dtype)
        fast.gemm_pair(x, w, out[:, :N], epi, err, bn=bn, in_parts=in_parts)
        check(out[:, :N], want, most, K, dtype)
        assert bool((out[:, N:] == 3.0).all())
        fast.gemm_pair(x, w, out[:, :N], epi, err, bn=bn, act=ops.ACT_SILU, in_parts=in_parts)
        check(out[:, :N], want * torch.sigmoid(want), 1.1 * most, K, dtype)
    if N % 32 == 0:
        g, u = want.view(M, N // 32, 2, 16).unbind(2)
        s = most.view(M, N // 32, 2, 16)
        for limit, slope in ((0.0, 0.0), (0.75, 1.702)):
            if limit:
                gc, uc = g.clamp(max=limit), u.clamp(-limit, limit)
                y = gc * torch.sigmoid(slope * gc) * (uc + 1.0)
            else:
                y = g * torch.sigmoid(g) * u
            out = torch.full((M, N // 2 + 8), 3.0, device="cuda", dtype=torch.bfloat16)
            fast.gemm_pair(x, w, out[:, :N // 2], fast.EPI_SWIGLU, err, bn=bn, glu=(limit, slope), in_parts=in_parts)
            size = (g.abs() + 1.0) * s[:, :, 1] + (u.abs() + 1.0) * s[:, :, 0] * 1.2
            check(out[:, :N // 2], y.reshape(M, -1), size.reshape(M, -1), K, torch.bfloat16)
            assert bool((out[:, N // 2:] == 3.0).all())
    assert err.item() == 0


@gpu
@pytest.mark.parametrize("cuts", [[0, 0, 1, 257, 257, 600], [0, 31, 64, 300, 556, 590], [0, 0, 0, 0, 0, 0], [0, 600, 600, 600, 600, 600]])
def test_segments(cuts):
    """Empty segments, single rows, edges of the widths, and rows behind the last segment, which stay as they are."""
    from airun_b200.kernels import fast
    E, M, N, K = 5, 600, 320, 200
    x, _ = operands(M, 1, K, 3)
    x = x.contiguous()
    w = (torch.randn(E, N, K, device="cuda") * K ** -0.5).bfloat16()
    from types import SimpleNamespace
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    out = torch.full((M, N), 7.0, device="cuda")
    assert fast.grouped_linear_bf16(ctx, x, w, out, torch.tensor(cuts, dtype=torch.int32, device="cuda"))
    for e in range(E):
        a = x[cuts[e]:cuts[e + 1]].double()
        check(out[cuts[e]:cuts[e + 1]], a @ w[e].double().T, a.abs() @ w[e].double().abs().T, K, torch.float32)
    assert bool((out[cuts[-1]:] == 7.0).all()) and ctx.err.item() == 0


@gpu
@pytest.mark.parametrize("one_sign", [False, True])
@pytest.mark.parametrize("M,N,K", [(65, 64, 1024), (100, 1024, 1024), (128, 5632, 1000), (129, 300, 2048), (200, 2048, 2048), (900, 512, 2048)])
def test_sums_are_no_less_exact_where_pairs_replace_slices(M, N, K, one_sign):
    """Float32 results of the two against 64 bits.  Both cut K where one long sum in tensor memory, whose cuts grow with it, would be further off."""
    from types import SimpleNamespace
    from airun_b200.kernels import fast
    x, w = operands(M, N, K, 12)
    if one_sign:
        x, w = x.abs(), w.abs()
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    sms, plan = fast.machine().sms, fast.plan_gemm(M, N, K)
    if sms == fast.B200_SMS:
        assert plan[2] > 1 and fast.pair_form(M, N, K) == fast.PAIRS_PARTS
    want, pairs, slices = x.double() @ w.double().T, torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    assert fast.linear_bf16(ctx, x, w, pairs)
    fast.gemm_tcgen05(x, w, slices, fast.EPI_F32, *plan, ctx.err)
    assert ctx.err.item() == 0 and (pairs.double() - want).norm() <= 1.02 * (slices.double() - want).norm()


@gpu
@pytest.mark.parametrize("K", [200, 1000])
def test_more_tiles_of_segments_than_pairs(K):
    """The stages and the two sums run on over tiles of different widths: K shorter and longer than the six stages."""
    from types import SimpleNamespace
    from airun_b200.kernels import fast
    E, N, cuts = 6, 4160, [0, 1, 34, 291, 891, 891, 1400]
    M = cuts[-1]
    x, _ = operands(M, 1, K, 13)
    x = x.contiguous()
    w = (torch.randn(E, N, K, device="cuda") * K ** -0.5).bfloat16()
    ctx, out = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda")), torch.empty(M, N, device="cuda")
    assert 17 * sum(-(-(b - a) // 256) for a, b in zip(cuts, cuts[1:])) > fast.machine().sms // 2
    assert fast.grouped_linear_bf16(ctx, x, w, out, torch.tensor(cuts, dtype=torch.int32, device="cuda"))
    for e in range(E):
        a = x[cuts[e]:cuts[e + 1]].double()
        check(out[cuts[e]:cuts[e + 1]], a @ w[e].double().T, a.abs() @ w[e].double().abs().T, K, torch.float32)
    assert ctx.err.item() == 0


@gpu
def test_as_many_rows_as_the_list_of_tiles_holds():
    """The largest number of rows for five matrices, and one more, which is another kernel's."""
    from types import SimpleNamespace
    from airun_b200.kernels import fast
    E, N, K = 5, 32, 64
    M = 256 * (fast.GROUPED_MAX_TILES - E)
    g = torch.Generator(device="cuda").manual_seed(14)
    x, w = torch.randn(M + 1, K, device="cuda", generator=g).bfloat16(), torch.randn(E, N, K, device="cuda", generator=g).bfloat16()
    cuts = [0, 1, M // 3, M // 3 + 1, M - 300, M]
    seg, ctx = torch.tensor(cuts, dtype=torch.int32, device="cuda"), SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    out = torch.full((M + 1, N), 7.0, device="cuda")
    assert not fast.grouped_linear_bf16(ctx, x, w, out, seg) and fast.grouped_linear_bf16(ctx, x[:M], w, out[:M], seg)
    for e in range(E):
        a = x[cuts[e]:cuts[e + 1]].double()
        check(out[cuts[e]:cuts[e + 1]], a @ w[e].double().T, a.abs() @ w[e].double().abs().T, K, torch.float32)
    assert bool((out[M] == 7.0).all()) and ctx.err.item() == 0


@gpu
@pytest.mark.parametrize("swiglu", [False, True])
def test_segments_that_end_behind_the_rows(swiglu):
    """A list that names more rows than there are: no row behind the last is stored, the others are as without it."""
    from types import SimpleNamespace
    from airun_b200.kernels import fast
    E, M, N, K = 3, 300, 320, 200
    x, _ = operands(M, 1, K, 4)
    x = x.contiguous()
    w = (torch.randn(E, N, K, device="cuda") * K ** -0.5).bfloat16()
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    outs = []
    for last in (M, M + 90):
        out = torch.full((M + 100, N // 2 if swiglu else N), 7.0, device="cuda", dtype=torch.bfloat16 if swiglu else torch.float32)
        cuts = torch.tensor([0, 40, 230, last], dtype=torch.int32, device="cuda")
        assert fast.grouped_linear_bf16(ctx, x, w, out[:M], cuts, swiglu_group=16 if swiglu else 0)
        assert bool((out[M:] == 7.0).all()) and ctx.err.item() == 0
        outs.append(out[:M])
    assert torch.equal(*outs)


def test_plan():
    """Whatever the sizes, the width is one the kernel takes."""
    from airun_b200.kernels.fast import PAIR_PARTS_BN, plan_pair
    for M in (1, 31, 129, 250, 512, 900, 1536, 2048, 8192):
        for N, K in ((32, 8), (300, 72), (2048, 2048), (6144, 2048), (24576, 4096), (151936, 4096)):
            for parts in (False, True):
                bn = plan_pair(M, N, K, in_parts=parts)
                assert bn % 32 == 0 and 32 <= bn <= (PAIR_PARTS_BN if parts else 256)
    assert plan_pair(512, 4096, 2048) == 128 and plan_pair(900, 6144, 2048) == 160 and plan_pair(2048, 2048, 6144) == 256


def test_where_pairs_run():
    """The borders of the rule: tokens, K-steps, rounds of tiles.  Where plan_gemm cuts K, no pair forms a sum over all of it."""
    from airun_b200.kernels.fast import PAIRS_NOT, PAIRS_PARTS, PAIRS_WHOLE, pair_form, plan_gemm
    for M, N, K, want in [
            (64, 1024, 1024, PAIRS_NOT), (65, 1024, 1024, PAIRS_PARTS), (65, 1024, 1025, PAIRS_NOT), (128, 1024, 1024, PAIRS_PARTS),
            (128, 12288, 2048, PAIRS_WHOLE), (128, 12288, 2056, PAIRS_NOT), (128, 20000, 2048, PAIRS_NOT), (128, 20000, 1024, PAIRS_WHOLE),
            (128, 32768, 2048, PAIRS_WHOLE), (129, 300, 2048, PAIRS_PARTS), (129, 128, 4096, PAIRS_NOT), (384, 2048, 3072, PAIRS_PARTS), (512, 2048, 6144, PAIRS_NOT),
            (512, 4096, 2048, PAIRS_WHOLE), (2048, 2048, 2048, PAIRS_WHOLE),
            (2048, 6144, 2048, PAIRS_WHOLE)]:
        assert pair_form(M, N, K) == want, (M, N, K)
    for M in (65, 100, 128, 129, 200, 256, 400, 512, 700, 1024, 2048):
        for N in (64, 300, 1024, 2048, 4096, 6144, 12288, 20000):
            for K in (512, 1024, 1536, 2048, 2816, 4096, 6144, 12288):
                assert (pair_form(M, N, K) == PAIRS_WHOLE) <= (plan_gemm(M, N, K)[2] == 1)
