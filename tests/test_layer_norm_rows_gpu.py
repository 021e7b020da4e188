"""Layer norm of many rows, a warp a row (csrc/embed_norm.cu): scale and shift from shared memory up to 1024 elements."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("shift", [True, False])
@pytest.mark.parametrize("hidden", [4, 508, 1020, 1024, 1028, 2048])  # the last of 1024 and the first that fetch them at the end
@pytest.mark.parametrize("rows", [1, 6, 2047])
def test_edges(rows, hidden, shift):
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    x = torch.randn(rows, hidden, generator=g, device=DEV) + 1
    gamma, beta = torch.randn(hidden, generator=g, device=DEV), torch.randn(hidden, generator=g, device=DEV)
    out = torch.empty(rows, hidden, device=DEV)
    K.layernorm(x, gamma, beta if shift else None, 1e-5, out)
    want = torch.nn.functional.layer_norm(x.double(), (hidden,), gamma.double(), beta.double() if shift else None, 1e-5)
    # float32 sums of up to 2048 values of order 1 (16 a lane, 5 halvings) and a handful of roundings of values up to 2^3 * 2^2
    assert (out.double() - want).abs().max().item() <= 32 * 2.0 ** -24 * 64
