"""Float32 products on the tensor cores (csrc/gemm_f32_tc.cu) hold their operands in full: sums of one product and of a few, and
operands whose lower parts all have one sign, against 64 bits and against single FMAs."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WIDTHS = [32, 64, 128]


def _fmas(a, w):
    """Sums by single FMAs in ascending order: one rounding a step, the product is exact in 64 bits."""
    t = torch.zeros(a.shape[0], w.shape[0], device=DEV, dtype=torch.float64)
    for i in range(a.shape[1]):
        t = (t + a[:, i:i + 1].double() * w[:, i].double()).float().double()
    return t


def _product(a, w, width):
    out = torch.empty(a.shape[0], w.shape[0], device=DEV)
    K.linear(a, w, None, out, path="f32tc", tile_width=width)
    return out


def _sparse(rows, k, count, g):
    places = torch.rand(rows, k, generator=g, device=DEV).argsort(1)[:, :count]
    return torch.zeros(rows, k, device=DEV).scatter_(1, places, torch.randn(rows, count, generator=g, device=DEV))


@pytest.mark.parametrize("width", WIDTHS)
@pytest.mark.parametrize("k", [256, 4608])  # the small products' accumulator drained once, and twice
def test_a_row_with_a_single_one_picks_a_column(k, width):
    w = torch.randn(200, k, device=DEV) * torch.exp2(torch.randint(-60, 60, (200, k), device=DEV).float())
    a = torch.zeros(300, k, device=DEV)
    places = torch.arange(300, device=DEV) * 17 % k
    a[torch.arange(300, device=DEV), places] = 1
    assert torch.equal(_product(a, w, width), w.T[places])


@pytest.mark.parametrize("width", WIDTHS)
@pytest.mark.parametrize("count", [1, 2, 4, 16])
def test_sums_of_few_products(count, width):
    g = torch.Generator(device=DEV).manual_seed(count)
    a, w = _sparse(256, 768, count, g), torch.randn(256, 768, generator=g, device=DEV)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # one product: the rounding of hi hi plus the rest; lo lo left out and the small parts cut off at 2^-23 of themselves: a sixteenth more.  Others:
    # a rounding for each product's drain, 2^-23 cut off where two stand in one accumulator, and the rounding at the end
    assert ((_product(a, w, width).double() - ref).abs() <= (17 / 16 if count == 1 else 3 * count + 1) * 2.0 ** -24 * size).all()


# sums whose parts' signs are not random (the lower parts of all operands positive: what is left out and cut off adds up one way), rows behind
# a ReLU, operands over many orders of magnitude
@pytest.mark.parametrize("width", WIDTHS)
@pytest.mark.parametrize("kind", ["normal", "positive", "wide", "relu", "rests"])
@pytest.mark.parametrize("k", [256, 768, 3072])
def test_error_is_no_larger_than_that_of_fmas(k, kind, width):
    g = torch.Generator(device=DEV).manual_seed(k)
    a, w = torch.randn(128, k, generator=g, device=DEV), torch.randn(192, k, generator=g, device=DEV)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    elif kind == "wide":
        a = a * torch.exp(3 * torch.randn(128, k, generator=g, device=DEV))
    elif kind == "relu":
        a = a.relu()
    elif kind == "rests":
        a, w = ((torch.randint(128, 256, s, generator=g, device=DEV) / 128 + 0.0038).float() for s in (a.shape, w.shape))
    ref = a.double() @ w.double().T
    assert (_product(a, w, width).double() - ref).norm() <= (_fmas(a, w) - ref).norm()
