"""Float32 products on the tensor cores (csrc/gemm_f32_tc.cu) where sums are not finite, or operands are not the sum of three bfloat16
numbers: those sums are single FMAs', in ascending order, and no other sum changes a bit."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _fmas(a, w):
    """One rounding a step: the product is exact in 64 bits, and its sum with 24 bits exact or rounded far below those."""
    t = torch.zeros(a.shape[0], w.shape[0], device=DEV)
    for i in range(a.shape[1]):
        t = (t.double() + a[:, i:i + 1].double() * w[:, i].double()).float()
    return t


def _product(a, w, width, bias=None, act=K.ACT_NONE):
    out = torch.full((a.shape[0], w.shape[0]), 7.0, device=DEV)
    K.linear(a, w, bias, out, path="f32tc", tile_width=width, act=act)
    return out


def _equal(got, want):
    return torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(nan=0.0, posinf=3e38, neginf=-3e38),
                                                                  want.nan_to_num(nan=0.0, posinf=3e38, neginf=-3e38))


# more tiles than SMs (width 32), several a block; the rows and columns with what is not finite in one tile only
@pytest.mark.parametrize("width", [32, 64, 128])
def test_rows_beside_numbers_that_are_not_finite_keep_their_bits(width):
    g = torch.Generator(device=DEV).manual_seed(width)
    a, w = torch.randn(700, 264, generator=g, device=DEV), torch.randn(1000, 264, generator=g, device=DEV)
    fine = _product(a, w, width)
    a2, w2 = a.clone(), w.clone()
    a2[3, 5], a2[300, 263], a2[699, 0], w2[17, 40] = float("inf"), float("nan"), float("-inf"), float("nan")
    odd_rows, odd_columns = torch.tensor([3, 300, 699], device=DEV), torch.tensor([17], device=DEV)
    for _ in range(2):
        got = _product(a2, w2, width)
        same = torch.ones_like(got, dtype=torch.bool)
        same[odd_rows], same[:, odd_columns] = False, False
        assert torch.equal(got[same], fine[same])
        assert _equal(got[odd_rows], _fmas(a2[odd_rows], w2)) and _equal(got[:, odd_columns], _fmas(a2, w2[odd_columns]))
    bias, x = torch.randn(1000, generator=g, device=DEV), torch.randn(700, 1000, generator=g, device=DEV)
    plain = _product(a2, w2, width, bias=bias)
    added = x.clone()
    K.linear(a2, w2, bias, added, residual=True, path="f32tc", tile_width=width)
    assert _equal(added, x + plain)
    # ahead of an activation: of what is not finite too
    act, want = _product(a2, w2, width, bias=bias, act=K.ACT_GELU_ERF), torch.empty(3, 1000, device=DEV)
    K.linear(a2[odd_rows], w2, bias, want, act=K.ACT_GELU_ERF, path="rows")
    assert torch.equal(act[odd_rows].isnan(), want.isnan()) and torch.equal(act[odd_rows].isinf(), want.isinf())


@pytest.mark.parametrize("width", [32, 128])
def test_sums_that_overflow_and_operands_of_more_than_three_parts(width):
    g = torch.Generator(device=DEV).manual_seed(width + 1)
    a, w = torch.randn(130, 296, generator=g, device=DEV), torch.randn(70, 296, generator=g, device=DEV)
    a[1] *= 3e19
    w[2] *= 3e19                           # products about float32's largest number
    a[5, 7] = 3.4e38                       # rounds to infinity in bfloat16
    a[64] *= 2.0 ** -130                   # bits below bfloat16's least number, in every part of the row that a thread cuts
    a[65, :] = 2.0 ** -140                 # subnormal
    got, want = _product(a, w, width), _fmas(a, w)
    assert _equal(got[5:6], want[5:6]) and _equal(got[64:66], want[64:66]) and _equal(got[1:2, 2:3], want[1:2, 2:3])
    fine = torch.ones_like(got, dtype=torch.bool)
    fine[[5, 64, 65]], fine[1, 2] = False, False
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # 296 roundings of partial sums at most
    assert ((got.double() - ref).abs()[fine] <= (296 * 2.0 ** -24 * size)[fine]).all()
