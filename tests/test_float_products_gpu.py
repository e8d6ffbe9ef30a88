"""Float products by split floats: edges of the tiles and of the blocks of K, operands that are not finite, and the rule that chooses them."""
import pytest
import torch


@pytest.mark.parametrize("sizes,want", [((63, 4096, 4096), 0), ((1000, 960, 576), 64), ((1000, 960, 578), 0), ((512, 16384, 2048), 128), ((128, 2048, 8192), 0), ((128, 4096, 4096), 64)])
def test_route(sizes, want):
    """No GPU needed."""
    from cisr_b200.ops import kernels
    assert kernels.float_tile(*sizes, 148) == want


def operands(m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    return (torch.randn(r, k, generator=g, device="cuda") for r in (m, n))


@pytest.mark.gpu
@pytest.mark.parametrize("narrow", [False, True])
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (127, 63, 60), (128, 64, 64), (129, 130, 68), (300, 257, 128), (64, 1000, 1060), (257, 90, 4100)])
def test_products(m, n, k, narrow):
    from cisr_b200.ops import kernels
    a, w = operands(m, n, k)
    out = torch.full((m, n), float("nan"), device="cuda")
    kernels.gemm_float(a, w, out, narrow)
    kernels.raise_if_kernel_gave_up()
    want = a.double() @ w.double().T
    # a block of 64 terms of size 1: sums of about 8 cut a few times at 2^-24; k / 64 of them added with rounding, sums of about k^1/2
    assert ((out.double() - want).abs() <= 2.0 ** -24 * (8 * 8 * (k / 64 + 1) ** 0.5 + 4 * k ** 0.5 * (k / 64 + 1) ** 0.5)).all()


@pytest.mark.gpu
def test_large_and_small_operands():
    """Exponents far apart, and numbers near both ends of the range."""
    from cisr_b200.ops import kernels
    a, w = operands(130, 70, 192)
    a, w = a * torch.exp2(torch.randint(-40, 40, a.shape, device="cuda").float()), w * torch.exp2(torch.randint(-40, 40, w.shape, device="cuda").float())
    out = kernels.gemm_float(a, w, torch.empty(130, 70, device="cuda"))
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((out.double() - want).abs() <= 2.0 ** -20 * size).all()
    a, w = torch.full((3, 64), 3e38, device="cuda"), torch.full((2, 64), 1e-3, device="cuda")
    assert torch.allclose(kernels.gemm_float(a, w, torch.empty(3, 2, device="cuda")), torch.full((3, 2), 64 * 3e35, device="cuda"), rtol=1e-6)
    for power in (-60, -100, -112, -120):                    # results of about 2^-114 at the least: beside them a term's rounding to a subnormal's last place is 2^-35
        a, w = operands(130, 70, 192)
        small, w = a.abs() * 2.0 ** power, w.abs()
        for left, right in ((small, w), (w, small)):
            out = kernels.gemm_float(left, right, torch.empty(left.shape[0], right.shape[0], device="cuda"))
            want = left.double() @ right.double().T
            assert ((out.double() - want).abs() <= 1e-6 * want).all(), power


@pytest.mark.gpu
@pytest.mark.parametrize("narrow", [False, True])
def test_not_finite(narrow):
    from cisr_b200.ops import kernels
    a, w = operands(140, 150, 132)
    a[3, 7], a[130, 131], w[5, 9], w[149, 0], a[60, 1] = float("inf"), float("nan"), float("-inf"), 3.4028e38, 1e30
    w[60, 7] = 0.0                                           # inf x 0
    out = kernels.gemm_float(a, w, torch.empty(140, 150, device="cuda"), narrow)
    want = a.double() @ w.double().T
    want = torch.where(want.abs() > 3.4028235e38, want.sign() * float("inf"), want)
    ok = want.isfinite()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[want.isinf()].double(), want[want.isinf()])
    size = (a.double().abs() @ w.double().abs().T)[ok]
    assert ((out.double()[ok] - want[ok]).abs() <= 1e-6 * size).all()
