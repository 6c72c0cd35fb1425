"""Products of few rows whose weights go straight to registers (csrc/gemm_rows.cu) against float64 products of the same bfloat16
operands: plain, with an activation, as a gated unit, per segment and per head.

Tolerance: sums of K products in float32, in 8 parts (2^-24 * K / 8 of the sum of absolute values, doubled), and for bfloat16
results half a unit of theirs (2^-8 at most: seven stored bits)."""
from types import SimpleNamespace

import pytest
import torch

gpu = pytest.mark.gpu
SHAPES = [(1, 1, 8), (1, 16, 64), (3, 100, 72), (8, 4096, 520), (9, 333, 1024), (16, 4800, 136), (7, 32, 4104), (16, 4736, 8), (5, 2048, 2816)]


def close(got, want, most, K, dtype):
    tol = 2.0 * 2.0 ** -24 * max(K / 8, 8) * most
    if dtype == torch.bfloat16:
        tol = tol + 2.0 ** -8 * want.abs()
    assert bool(((got.double() - want).abs() <= tol + 1e-6).all())


def operands(M, N, K, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.zeros(M, K + 8).to("cuda", torch.bfloat16)
    x[:, :K] = torch.randn(M, K, generator=g).to("cuda", torch.bfloat16)
    w = torch.randn(N, K, generator=g).to("cuda", torch.bfloat16)
    return x[:, :K], w


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain_and_activation(M, N, K, dtype):
    from airun_b200.kernels import fast, ops
    x, w = operands(M, N, K, M + N)
    want, most = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    out = torch.full((M, N + 8), 5.0, device="cuda", dtype=dtype)
    fast.gemm_rows(x, w, out[:, :N], fast.EPI_F32 if dtype == torch.float32 else fast.EPI_BF16)
    close(out[:, :N], want, most, K, dtype)
    assert bool((out[:, N:] == 5.0).all())
    got = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
    fast.gemm_rows(x, w, got, fast.EPI_BF16, act=ops.ACTIVATIONS["relu2"])
    z = torch.relu(want)
    close(got, z * z, 2 * most * (z + 1), K, torch.bfloat16)


@gpu
@pytest.mark.parametrize("limit", [0.0, 1.5])
@pytest.mark.parametrize("M,N,K", [(1, 32, 64), (8, 4768, 520), (16, 96, 1032)])
def test_gated_unit(M, N, K, limit):
    from airun_b200.kernels import fast
    x, w = operands(M, N, K, M * N)
    w *= K ** -0.5
    z = (x.double() @ w.double().T).view(M, N // 32, 2, 16)
    g, u = z[:, :, 0].reshape(M, -1), z[:, :, 1].reshape(M, -1)
    if limit:
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        want = g * torch.sigmoid(1.702 * g) * (u + 1)
    else:
        want = g * torch.sigmoid(g) * u
    out = torch.empty(M, N // 2, device="cuda", dtype=torch.bfloat16)
    fast.gemm_rows(x, w, out, fast.EPI_SWIGLU, glu=(limit, 1.702 if limit else 0.0))
    assert bool(((out.double() - want).abs() <= (2.0 ** -8 + 1e-5) * want.abs() + 2e-5).all())


@gpu
@pytest.mark.parametrize("lens,N,K", [((0, 3, 8, 0, 9, 1), 96, 264), ((17, 0, 30), 64, 72), ((1, 0, 0, 0), 4800, 64)])
def test_segments_and_heads(lens, N, K):
    from airun_b200.kernels import fast
    E, M = len(lens), sum(lens) + 2
    x, _ = operands(M, N, K, N)
    x = x.contiguous()
    w = torch.randn(E, N, K, generator=torch.Generator().manual_seed(E)).to("cuda", torch.bfloat16)
    seg = torch.tensor([sum(lens[:i]) for i in range(E + 1)], dtype=torch.int32, device="cuda")
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32, device="cuda"))
    out = torch.full((M, N), 5.0, device="cuda")
    assert M <= fast.GROUPED_ROWS_MAX * E or E == 3
    old, fast.GROUPED_ROWS_MAX = fast.GROUPED_ROWS_MAX, 64
    try:
        assert fast.grouped_linear_bf16(ctx, x, w, out, seg)
    finally:
        fast.GROUPED_ROWS_MAX = old
    for e, n in enumerate(lens):
        a = int(seg[e])
        close(out[a:a + n], x[a:a + n].double() @ w[e].double().T, x[a:a + n].double().abs() @ w[e].double().abs().T, K, torch.float32)
    assert bool((out[sum(lens):] == 5.0).all())
    for T in (1, 8, 16):
        xh = torch.randn(T, E, K + 8, generator=torch.Generator().manual_seed(T)).to("cuda", torch.bfloat16)[:, :, :K]
        oh = torch.full((T, E, N + 8), 5.0, device="cuda", dtype=torch.bfloat16)
        assert fast.head_linear_bf16(ctx, xh, w, oh[:, :, :N])
        close(oh[:, :, :N], torch.einsum("thk,hnk->thn", xh.double(), w.double()), torch.einsum("thk,hnk->thn", xh.double().abs(), w.double().abs()),
              K, torch.bfloat16)
        assert bool((oh[:, :, N:] == 5.0).all())


def test_which_products_of_segments_read_their_matrices_per_few_rows(monkeypatch):
    """By the rows a segment has on average and by the rows it can have: with many tokens, all of which may choose one expert, the
    matrices are read once (csrc/gemm_tcgen05.cu)."""
    from airun_b200.kernels import fast
    from airun_b200.parts.moe import grouped_linear
    went = []
    monkeypatch.setattr(fast, "_cuda", lambda *a: None)
    monkeypatch.setattr(fast, "_check", lambda *a: None)
    monkeypatch.setattr(fast, "_stream", lambda: None)
    monkeypatch.setattr(fast, "_fn", lambda lib, name, args, defines=None: lambda *a: went.append(lib))
    ctx = SimpleNamespace(err=torch.zeros(1, dtype=torch.int32))
    for E, tokens, top, want in ((16, 8, 4, "gemm_rows"), (16, 32, 4, "gemm_rows"), (16, 33, 2, "gemm_tcgen05"), (64, 512, 1, "gemm_tcgen05"),
                                 (16, 20, 8, "gemm_tcgen05"), (64, 32, 8, "gemm_rows")):
        x, w = torch.zeros(tokens * top, 64, dtype=torch.bfloat16), torch.zeros(E, 32, 64, dtype=torch.bfloat16)
        out, seg = torch.zeros(tokens * top, 32), torch.zeros(E + 1, dtype=torch.int32)
        went.clear()
        assert fast.grouped_linear_bf16(ctx, x, w, out, seg, tokens=tokens) and went == [want]
        went.clear()
        grouped_linear(ctx, x, w, out, seg)                  # without the number of tokens: by the average alone
        assert went == ["gemm_rows" if tokens * top <= fast.GROUPED_ROWS_MAX * E else "gemm_tcgen05"]
