"""The weight-streaming product around the edges of its ring: inner sizes that fill no stage, one stage, a stage and a piece,
one turn of the block's warps and one piece more; row tiles that end early; both numbers of stages of the gated form."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def K():
    from catena_models_b200 import kernels

    kernels.lib()
    return kernels


def _operands(M, N, Kd, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    x = torch.randn(M, Kd, generator=g, device=DEV).to(torch.bfloat16)
    return x, (torch.randn(N, Kd, generator=g, device=DEV) * Kd ** -0.5).to(torch.bfloat16)


def _bound(x, w):
    """Float sums of K products in any order: K roundings of partial sums that |x| @ |w| bounds (the products are exact)."""
    return x.shape[1] * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("Kd", [8, 64, 72, 256, 264, 512, 1000, 1544, 2048, 4104])
@pytest.mark.parametrize("N", [1, 16, 23, 2600])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
def test_plain_and_parts(K, M, N, Kd):
    x, w = _operands(M, N, Kd, M + N + Kd)
    exact, bound = x.double() @ w.double().T, _bound(x, w)
    y = torch.full((M, N), float("nan"), device=DEV)
    K.gemm_skinny(y, x, w)
    assert ((y.double() - exact).abs() <= bound).all()
    one = torch.empty(1, N, device=DEV)
    K.gemm_skinny(one, x[M - 1:], w)
    assert torch.equal(one[0], y[M - 1])                               # one row and sixteen: the same sums
    for slices in (1, 3, 4):
        parts = torch.full((slices, M, N), float("nan"), device=DEV)
        K.gemm_skinny_parts(parts, x, w)
        assert ((parts.double().sum(0) - exact).abs() <= bound).all()
    rows = torch.full((M + 2, Kd + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
    rows[1:-1, :Kd] = x                                                # rows of a wider buffer: nothing beside them is read
    K.gemm_skinny(y, rows[1:-1, :Kd], w)
    assert ((y.double() - exact).abs() <= bound).all()


@pytest.mark.parametrize("F", [5, 16, 2048, 9488])                     # 9,488 outputs are 593 blocks: more than four an SM
@pytest.mark.parametrize("Kd", [64, 200, 1032])
@pytest.mark.parametrize("M", [1, 8, 13, 16])
def test_gated(K, M, F, Kd):
    x, w = _operands(M, 2 * F, Kd, M + F + Kd)
    a = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.gemm_skinny(a, x, w, swiglu=True)
    gu, b = x.double() @ w.double().T, _bound(x, w)
    g, u = gu[:, :F], gu[:, F:]
    dg, du = 2.0 ** -8 * g.abs() + b[:, :F], 2.0 ** -8 * u.abs() + b[:, F:]         # a sum near a rounding border falls either way
    silu = g * torch.sigmoid(g)
    # silu's slope lies in (-0.1, 1.1); the result is rounded once more
    bound = 1.1 * dg * (u.abs() + du) + silu.abs() * du
    assert ((a.double() - silu * u).abs() <= bound + 2.0 ** -8 * ((silu * u).abs() + bound) + 1e-30).all()


def test_nothing_of_a_neighbour_reaches_a_row(K):
    x, w = _operands(16, 40, 520, 5)
    clean = torch.empty(16, 40, device=DEV)
    K.gemm_skinny(clean, x, w)
    dirty = x.clone()
    dirty[3], dirty[11, 100] = float("nan"), float("inf")
    y = torch.empty(16, 40, device=DEV)
    K.gemm_skinny(y, dirty, w)
    keep = [i for i in range(16) if i not in (3, 11)]
    assert torch.equal(y[keep], clean[keep]) and y[3].isnan().all() and not y[11].isfinite().any()
