"""Float32 products on the tensor cores (three bfloat16 parts of each operand, csrc/gemm_simt.cu) against 64-bit ones.

Tolerance, of the sum S of absolute products: the tensor cores cut a running sum off at 2^-23 of it at most, once a product of 16 k-values: four times a
step of 64 in the sum of the leading products, and 28 times a step, over four steps, in that of the small ones, which is 2^-7 of S at most (a rounded part
leaves 2^-9 of an operand); a step is added with 2^-24, and every fourth time the small ones; the product of parts left out is below 2^-35."""
import pytest
import torch

gpu = pytest.mark.gpu


def bound(x, w):
    return (2.0 ** -23 * (4 + 112 / 128) + 2.0 ** -24 * (x.shape[1] // 50 + 3)) * (x.double().abs() @ w.double().abs().T) + 1e-30


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
@pytest.mark.parametrize("share", [1.0, 0.5, 0.1, 0.03, 0.01, 0.001])
@pytest.mark.parametrize("one_sign", [False, True])
def test_error_is_no_larger_than_the_fma_kernels(share, one_sign):
    """Dense rows and rows of few terms.  A step of 64 is rounded when it is added up, the FMA kernel's four sums when a term is: with fewer than about six terms a
    step the steps' roundings are the larger ones, up to 16 to 44 steps here."""
    from airun_b200.kernels import ops
    for M, N, K in ((642, 1024, 1024), (130, 700, 2816), (40, 512, 1024)):
        x, w = operands(M, N, K, 5)
        x = x * (torch.rand(M, K, device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)) < share)
        if one_sign:
            x, w = x.abs(), w.abs()
        want, parts, fma = x.double() @ w.double().T, torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
        ops.gemm_simt(x, w, parts, word())
        ops.gemm_simt(x, w, fma)
        got, was = (parts.double() - want).norm(), (fma.double() - want).norm()
        assert got <= (1.0 if share >= 0.1 else 1.25) * was, (got / want.norm(), was / want.norm())


@gpu
def test_a_sum_of_one_product_is_that_product_rounded():
    """Up to the cuts of the sum of seven small products, 2^-23 of 2^-7 of it."""
    from airun_b200.kernels import ops
    M, N, K = 300, 200, 1024
    x, w = operands(M, N, K, 8)
    x[0], w[0], w[1] = 1.0 + 2.0 ** -7 - 2.0 ** -16, 1.0 + 2.0 ** -7 - 2.0 ** -16, 1.0 + 2.0 ** -8 + 2.0 ** -17 - 2.0 ** -23      # parts as large as they get
    x = x * torch.nn.functional.one_hot(torch.randint(0, K, (M,), device="cuda"), K)
    want, parts, err = x.double() @ w.double().T, torch.empty(M, N, device="cuda"), word()
    ops.gemm_simt(x, w, parts, err)
    assert err.item() == 0 and bool(((parts.double() - want).abs() <= (2.0 ** -24 + 7 * 2.0 ** -30) * want.abs()).all())


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
@pytest.mark.parametrize("M,N,K", [(300, 260, 1024), (40, 130, 4096)])
def test_products_beyond_the_range(M, N, K):
    """A product that is too large in one place: an infinity as the FMA kernel has it, whatever the signs of its parts' products."""
    from airun_b200.kernels import ops
    x, w = operands(M, N, K, 10)
    at = torch.randint(0, K, (M,), device="cuda")
    x[torch.arange(M), at] = x[torch.arange(M), at].sign() * 2.0 ** 80 * (1.0 + torch.rand(M, device="cuda"))
    w[:, :] = w.sign() * (1.0 + w.abs().frac()) * torch.exp2(torch.randint(40, 75, (N, 1), device="cuda").float())
    x[7], x[8, 1:], x[8, 0], x[9, 1:], x[9, 0] = 0.0, 0.0, 3.4e38, 0.0, 2.0 ** -20
    parts, fma, err = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda"), word()
    ops.gemm_simt(x, w, parts, err)
    ops.gemm_simt(x, w, fma)
    assert err.item() == 0 and torch.equal(parts.isnan(), fma.isnan()) and torch.equal(parts.isinf(), fma.isinf()) and not parts.isnan().any()
    assert torch.equal(parts[parts.isinf()], fma[fma.isinf()]) and 0.1 < parts.isinf().float().mean() < 0.95
    fine = parts.isfinite()
    assert bool(((parts.double() - x.double() @ w.double().T).abs() <= bound(x, w))[fine].all())


@gpu
@pytest.mark.parametrize("x_exp,w_exp", [(-105, 0), (-112, 0), (-112, 60), (-120, 20), (-133, 40), (60, -115), (-60, -60), (-70, -62), (-66, -75)])
def test_small_operands_and_results(x_exp, w_exp):
    """Operands whose last part does not fit, and results near and below the smallest normal number: no further off than the FMA kernel."""
    from airun_b200.kernels import ops
    M, N, K = 70, 140, 1024
    x, w = operands(M, N, K, 11)
    x, w = (x.double() * 2.0 ** x_exp).float(), (w.double() * 2.0 ** w_exp).float()
    x[3], x[20:] = 0.0, (x[20:].double() * 2.0 ** 8).float()
    want, parts, fma, err = x.double() @ w.double().T, torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda"), word()
    ops.gemm_simt(x, w, parts, err)
    ops.gemm_simt(x, w, fma)
    assert err.item() == 0 and bool((parts[3] == 0).all())
    for rows in (slice(0, 20), slice(20, M)):
        tol = 2.0 ** -24 * (K + 1) * (x[rows].double().abs() @ w.double().abs().T) + (K + 1) * 2.0 ** -150
        assert bool(((parts[rows].double() - want[rows]).abs() <= tol).all())
        assert (parts[rows].double() - want[rows]).norm() <= 1.2 * (fma[rows].double() - want[rows]).norm() + 2.0 ** -149


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


@gpu
def test_plans_that_share_a_place():
    """Sizes in turn whose plans are kept in one place of the table (its number is 31 M + 7 N + K / 4 modulo 64)."""
    from airun_b200.kernels import ops
    sizes = [(17, 64, 1024), (81, 64, 1024), (145, 128, 1024), (17, 64, 1280)]
    assert len({(31 * M + 7 * N + K // 4) % 64 for M, N, K in sizes}) == 1
    for M, N, K in sizes * 2 + sizes[::-1]:
        x, w = operands(M, N, K, 3)
        out, err = torch.empty(M, N, device="cuda"), word()
        ops.gemm_simt(x, w, out, err)
        assert bool(((out.double() - x.double() @ w.double().T).abs() <= bound(x, w)).all()) and err.item() == 0
