"""Float32 products on the tensor cores (three bfloat16 parts of each operand, csrc/gemm_simt.cu) against 64-bit ones.

Tolerance, of the sum S of absolute products: the products of parts left out are below 2^-23; the tensor cores cut their running sum
off at 2^-23 of it at most, 24 times a step of 64 k-values, of which the four that add the leading products and the eight of
the next size count (the others add less than 2^-7 of S); the steps are added with 2^-24 each."""
import pytest
import torch

gpu = pytest.mark.gpu


def bound(x, w):
    return (2.0 ** -23 * (1 + 12) + 2.0 ** -24 * (x.shape[1] // 64 + 1)) * (x.double().abs() @ w.double().abs().T) + 1e-30


def operands(M, N, K, seed, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, w = (torch.randn(r, K + p, device="cuda", generator=g) for r, p in ((M, pad), (N, 2 * pad)))
    return x[:, :K], w[:, :K]


def word():
    return torch.zeros(1, dtype=torch.int32, device="cuda")


SHAPES = [(17, 1, 1024), (17, 128, 1024), (33, 130, 1100), (128, 1024, 1028), (129, 257, 1600), (300, 512, 8192), (642, 1024, 2816), (200, 5632, 1024)]


@gpu
@pytest.mark.parametrize("pad", [0, 4])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain(M, N, K, pad):
    from airun_b200.kernels import ops
    x, w = operands(M, N, K, M + N + K, pad)
    out, err = torch.full((M, N + 5), 3.0, device="cuda"), word()
    ops.gemm_simt(x, w, out[:, :N], err)
    assert bool(((out[:, :N].double() - x.double() @ w.double().T).abs() <= bound(x, w)).all()) and err.item() == 0
    assert bool((out[:, N:] == 3.0).all())


@gpu
@pytest.mark.parametrize("one_sign", [False, True])
def test_error_is_no_larger_than_the_fma_kernels(one_sign):
    from airun_b200.kernels import ops
    for M, N, K in ((642, 1024, 1024), (130, 700, 2816)):
        x, w = operands(M, N, K, 5)
        if one_sign:
            x, w = x.abs(), w.abs()
        want, parts, fma = x.double() @ w.double().T, torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
        ops.gemm_simt(x, w, parts, word())
        ops.gemm_simt(x, w, fma)
        assert (parts.double() - want).norm() <= (fma.double() - want).norm()


@gpu
def test_large_infinite_and_not_a_number():
    from airun_b200.kernels import ops
    for M, N, K in ((300, 260, 1024), (40, 130, 4096)):          # without and with slices of K
        x, w = operands(M, N, K, 6)
        x[5, 7], x[21, 3], w[100, K - 1], x[33, 0], w[3, 0] = float("inf"), float("nan"), -float("inf"), 3.3e38, 0.5
        parts, fma, err = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda"), word()
        ops.gemm_simt(x, w, parts, err)
        ops.gemm_simt(x, w, fma)
        assert torch.equal(parts.isnan(), fma.isnan()) and torch.equal(parts.isinf(), fma.isinf()) and err.item() == 0
        assert torch.equal(parts[parts.isinf()], fma[fma.isinf()]) and bool(parts[21].isnan().all())
        assert torch.allclose(parts[33][fma[33].isfinite()], fma[33][fma[33].isfinite()], rtol=1e-5)


@gpu
def test_grouped():
    from airun_b200.kernels import ops
    E, M, N, K = 5, 400, 200, 1024
    x, _ = operands(M, 1, K, 7)
    w = torch.randn(E, N, K, device="cuda")
    cuts = [0, 0, 130, 131, 260, 390]                           # an empty segment, one of a row, rows behind the last
    out, err = torch.full((M, N), 7.0, device="cuda"), word()
    ops.gemm_simt_grouped(x, w, out, torch.tensor(cuts, dtype=torch.int32, device="cuda"), err)
    for e in range(E):
        lo, hi = cuts[e], cuts[e + 1]
        assert bool(((out[lo:hi].double() - x[lo:hi].double() @ w[e].double().T).abs() <= bound(x[lo:hi], w[e])).all())
    assert bool((out[390:] == 7.0).all()) and err.item() == 0
