"""The 32-bit product in all its kernels (passes of four and eight rows, tiles of 64 and 128 rows, the any-size kernel):
against a float64 product, and bit for bit between kernels, whose choice follows the row count and the alignment."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    from catena_models_b200 import kernels

    kernels.lib()
    return kernels


# widths around the tiles' edges, inner sizes around the slices of 128 and the k-steps of 16 and 32, rows around every switch
@pytest.mark.parametrize("N,Kd", [(1, 4), (7, 20), (16, 128), (64, 176), (129, 132), (200, 260), (2047, 512), (2050, 1028), (1024, 4608)])
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 16, 17, 63, 65, 129, 300])
def test_float_product(K, M, N, Kd):
    g = torch.Generator("cuda").manual_seed(M * 7 + N + Kd)
    x = torch.randn(M, Kd, generator=g, device="cuda")
    w = torch.randn(N, Kd, generator=g, device="cuda")
    y = torch.full((M, N), float("nan"), device="cuda")
    K.gemm_simt(y, x, w)
    exact = x.double() @ w.double().T
    # a sum over slices of 128: at most 128 + K / 128 roundings of partial sums that |x| @ |w| bounds
    bound = (128 + Kd / 128 + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((y.double() - exact).abs() <= bound).all()
    # the same operands at addresses and pitches that only the any-size kernel takes: the same bits
    xu = torch.empty(M * (Kd + 1) + 1, device="cuda")[1:].view(M, Kd + 1)[:, :Kd]
    xu.copy_(x)
    yu = torch.full((M, N), float("nan"), device="cuda")
    K.gemm_simt(yu, xu, w)
    assert torch.equal(y, yu)
    # a row alone, and rows inside a wider buffer written beside others' data
    one = torch.empty(1, N, device="cuda")
    K.gemm_simt(one, x[M - 1:], w)
    assert torch.equal(one[0], y[M - 1])
    wide = torch.full((M, N + 3), 7.0, device="cuda")
    K.gemm_simt(wide[:, :N], x, w)
    assert torch.equal(wide[:, :N], y) and (wide[:, N:] == 7.0).all()


def test_many_rows_and_non_finite_values(K):
    g = torch.Generator("cuda").manual_seed(3)
    x = torch.randn(1000, 256, generator=g, device="cuda")
    w = torch.randn(9216, 256, generator=g, device="cuda")
    x[5, 17], x[700, 3] = float("inf"), float("nan")
    y = torch.empty(1000, 9216, device="cuda")
    K.gemm_simt(y, x, w)
    few = torch.empty(4, 9216, device="cuda")
    rows = [5, 6, 700, 999]
    K.gemm_simt(few, x[rows], w)
    assert torch.equal(torch.nan_to_num(few, nan=-1.0), torch.nan_to_num(y[rows], nan=-1.0))
    assert y[[i for i in range(1000) if i not in (5, 700)]].isfinite().all() and y[700].isnan().all()
    assert torch.equal(y[5].isinf(), w[:, 17] != 0)
