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
@pytest.mark.parametrize("M,N,K,bn", SHAPES)
def test_plain_activation_and_gated(M, N, K, bn):
    from airun_b200.kernels import fast, ops
    x, w = operands(M, N, K, M + N + K)
    want, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for dtype, epi in ((torch.float32, fast.EPI_F32), (torch.bfloat16, fast.EPI_BF16)):
        out = torch.full((M, N + 8), 3.0, device="cuda", dtype=dtype)
        fast.gemm_pair(x, w, out[:, :N], epi, err, bn=bn)
        check(out[:, :N], want, most, K, dtype)
        assert bool((out[:, N:] == 3.0).all())
        fast.gemm_pair(x, w, out[:, :N], epi, err, bn=bn, act=ops.ACT_SILU)
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
            fast.gemm_pair(x, w, out[:, :N // 2], fast.EPI_SWIGLU, err, bn=bn, glu=(limit, slope))
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
    """Whatever the sizes, the width is one the kernel takes, and no narrower tile would need as few rounds."""
    from airun_b200.kernels.fast import plan_pair
    for M in (1, 31, 129, 250, 512, 900, 1536, 2048, 8192):
        for N, K in ((32, 8), (300, 72), (2048, 2048), (6144, 2048), (24576, 4096), (151936, 4096)):
            bn = plan_pair(M, N, K)
            assert bn % 32 == 0 and 32 <= bn <= 256
    assert plan_pair(512, 4096, 2048) == 128 and plan_pair(900, 6144, 2048) == 160 and plan_pair(2048, 2048, 6144) == 256
