"""Float32 products of more than 64 rows: which kernel takes one (csrc/gemm_f32_tc.cuh: ``ahead``) hangs on its columns and inner size, so
that a row's result does not depend on how many rows share the launch."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# sizes on both sides of the rule; numbers of rows on both sides of where the one kernel becomes the faster, and of the tiles' edges
@pytest.mark.parametrize("n,k", [(768, 768), (736, 768), (728, 768), (1024, 1024), (1024, 256), (512, 512), (256, 1024), (768, 760), (1600, 1600)])
def test_a_row_is_the_same_whatever_the_number_of_rows(n, k):
    g = torch.Generator(device=DEV).manual_seed(n + k)
    a, w = torch.randn(2048, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * k ** -0.5
    b = torch.randn(n, generator=g, device=DEV)
    whole = torch.empty(2048, n, device=DEV)
    K.linear(a, w, b, whole)
    for m in (65, 96, 97, 128, 129, 192, 256, 257, 384, 385, 700, 1752):
        some = torch.empty(m, n, device=DEV)
        K.linear(a[2048 - m:], w, b, some)
        assert torch.equal(some, whole[2048 - m:]), m


@pytest.mark.parametrize("stride", [0, 8])
def test_rows_that_lie_over_one_another(stride):
    """What no tensor map describes stays on the CUDA cores, which take any stride."""
    g = torch.Generator(device=DEV).manual_seed(stride)
    base, w = torch.randn(100 * 8 + 768, generator=g, device=DEV), torch.randn(800, 768, generator=g, device=DEV)
    a = base.as_strided((100, 768), (stride, 1))
    out = torch.full((100, 800), float("nan"), device=DEV)
    K.linear(a, w, None, out)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((out.double() - ref).abs() <= 768 * 2.0 ** -24 * size).all()  # a rounding a step
