"""Float32 products on the tensor cores (csrc/gemm_f32_tc.cu): operands in three bfloat16 parts, against float64 and against the
CUDA-core kernels, whose error they may not exceed."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _data(m, n, k, seed=0):
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n * 3 + k + seed)
    return (torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * k ** -0.5,
            torch.randn(n, generator=g, device=DEV))


# one K block and a part of one, an odd number of them (the last chunk is short), more than stages; rows and columns one short of,
# at and beyond a tile; an output stride that is no multiple of four
@pytest.mark.parametrize("width", [32, 64, 128])
@pytest.mark.parametrize("m,n,k", [(1, 4, 8), (65, 127, 24), (128, 128, 32), (129, 129, 40), (300, 260, 96), (257, 2304, 768), (700, 768, 3072)])
def test_every_width(m, n, k, width):
    a, w, b = _data(m, n, k)
    ref = a.double() @ w.double().T
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, None, out, path="f32tc", tile_width=width)
    # a product leaves out 2^-34 of itself at most, a chunk of 32 elements adds two partial sums cut off at 2^-23 and
    # the chunks are added with a rounding each: all of it below k roundings of 2^-24 of sums of order 1
    assert (out.double() - ref).abs().max().item() <= 4 * (k + 64) * 2.0 ** -24 + 1e-6
    x = torch.randn(m, n + 3, device=DEV)[:, :n]
    want = x.double() + ref + b.double()
    K.linear(a, w, b, x, residual=True, path="f32tc", tile_width=width)
    assert (x.double() - want).abs().max().item() <= 4 * (k + 64) * 2.0 ** -24 + 1e-6
    for act in (K.ACT_GELU_TANH, K.ACT_GELU_ERF):
        got, plain = torch.empty(m, n, device=DEV), out + b
        K.linear(a, w, b, got, act=act, path="f32tc", tile_width=width)
        fn = torch.nn.functional.gelu(plain.double(), approximate="tanh" if act == K.ACT_GELU_TANH else "none")
        assert (got.double() - fn).abs().max().item() <= 1e-5
    K.check_status(torch.device(DEV))


# sums that cancel, that do not, and operands over many orders of magnitude, from the shortest sums that come here: the error against
# 64 bits is no larger than that of single FMAs in ascending order
@pytest.mark.parametrize("k", [256, 768, 3072])
@pytest.mark.parametrize("kind", ["normal", "positive", "wide"])
def test_error_is_no_larger_than_that_of_fmas(kind, k):
    a, w, _ = _data(256, 256, k, 5)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    if kind == "wide":
        a = a * torch.exp(3 * torch.randn(256, k, device=DEV))
    ref = a.double() @ w.double().T
    fma = torch.zeros(256, 256, device=DEV, dtype=torch.float64)
    for i in range(k):  # one rounding a step: the product is exact in 64 bits
        fma = (fma + a[:, i:i + 1].double() * w[:, i].double()).float().double()
    out = torch.empty(256, 256, device=DEV)
    K.linear(a, w, None, out, path="f32tc", tile_width=64)
    assert (out.double() - ref).norm() <= (fma - ref).norm()


def test_numbers_that_cannot_be_cut():
    """Infinities, NaN and magnitudes that round to infinity: the sums with them are those of FMAs."""
    a, w, b = _data(300, 200, 96)
    a[5, 7], a[200, 3], a[130, 9], w[17, 40] = float("inf"), float("nan"), 3.4028e38, float("-inf")
    out, ref = torch.empty(300, 200, device=DEV), a.double() @ w.double().T + b.double()
    K.linear(a, w, b, out, path="f32tc", tile_width=64)
    want = ref.float()  # (too large for 32 bits: an infinity)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    fine = want.isfinite()
    assert ((out.double() - ref)[fine].abs() <= 1e-5 * (1 + ref[fine].abs())).all() and torch.equal(out[want.isinf()], want[want.isinf()])


@pytest.mark.parametrize("m,n,k", [(2048, 3072, 768), (128, 4800, 1600), (65, 64, 8), (640, 129, 40)])
def test_a_row_does_not_depend_on_the_rows_beside_it(m, n, k):
    a, w, b = _data(m, n, k)
    out, fewer = torch.empty(m, n, device=DEV), torch.empty(m - 1, n, device=DEV)
    K.linear(a, w, b, out)
    K.linear(a[:m - 1], w, b, fewer, path="tile")
    assert torch.equal(fewer, out[:m - 1])


def test_operands_off_a_16_byte_boundary_are_refused():
    a, w, b = _data(200, 96, 64)
    shifted = torch.empty(200 * 64 + 1, device=DEV)[1:].view(200, 64).copy_(a)  # rows four bytes off a 16-byte boundary
    with pytest.raises(K.KernelError):
        K.linear(shifted, w, b, torch.empty(200, 96, device=DEV))  # refused as before
