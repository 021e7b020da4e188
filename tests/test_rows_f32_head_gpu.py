"""Float32 products of few rows (csrc/gemm_simt.cu): two, four or eight warps share four columns, against float64."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# every number of rows a pass takes and one beyond; two warps a group in many rounds and in one, four, eight; inner sizes below a chunk
# of 128, at whole ones and beyond, columns that end inside a group of four and inside a block's turn
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 17])
@pytest.mark.parametrize("n,k", [(40001, 8), (50257, 136), (3071, 768), (2303, 768), (1601, 1600), (770, 264), (5, 3072)])
def test_wide(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * 3 + k)
    a = torch.randn(m, k + 8, generator=g, device=DEV)[:, :k]  # rows apart from one another
    w = torch.randn(n, k, generator=g, device=DEV) * k ** -0.5
    b = torch.randn(n, generator=g, device=DEV)
    out = torch.full((m, n + 1), float("nan"), device=DEV)
    K.linear(a, w, b, out[:, :n], act=K.ACT_NONE)
    want, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    # a lane adds k / 32 products, four at a time, lanes by halves, eight warps and the bias in a row: k / 32 + 18 roundings of 2^-24 of
    # the sum of magnitudes at most
    assert ((out[:, :n].double() - want).abs() <= (k / 32 + 18) * 2.0 ** -24 * size).all()
    assert out[:, n].isnan().all()
    alone = torch.empty(1, n, device=DEV)
    K.linear(a[m - 1:], w, b, alone)
    assert torch.equal(alone[0], out[m - 1, :n])  # a row's sums do not depend on the rows beside it
    x = torch.randn(m, n, generator=g, device=DEV)
    want = x.double() + want
    K.linear(a, w, b, x, residual=True)
    assert ((x.double() - want).abs() <= (k / 32 + 19) * 2.0 ** -24 * (size + want.abs())).all()
