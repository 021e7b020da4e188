"""Float32 products (csrc/gemm_simt.cu) at the edges of their tiles and of the rows kernel, against float64, and against
themselves: a row's result may not depend on the rows beside it."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _data(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n * 3 + k)
    return (torch.randn(m, k, generator=g, device=DEV), torch.randn(n, k, generator=g, device=DEV) * k ** -0.5,
            torch.randn(n, generator=g, device=DEV))


def _close(got, ref, k):
    # k additions, each rounding a partial sum below 8 or so by 2^-24 of it
    assert (got.double() - ref).abs().max().item() <= 8 * k * 2.0 ** -24 + 1e-6


# rows kernel: one row, eight, nine, 64; one chunk of K (128), a ragged one, more than the warps take at once (1024);
# groups of four columns, ragged
@pytest.mark.parametrize("m", [1, 8, 9, 64])
@pytest.mark.parametrize("n,k", [(1, 8), (5, 136), (769, 768), (2401, 1032), (768, 3072), (50257, 64)])
def test_few_rows(m, n, k):
    a, w, b = _data(m, n, k)
    ref = a.double() @ w.double().T + b.double()
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, b, out)
    _close(out, ref, k)
    one = torch.empty(1, n, device=DEV)
    K.linear(a[m - 1:], w, b, one)
    assert torch.equal(one[0], out[m - 1])
    x = torch.randn(m, n + 3, device=DEV)[:, :n]
    want = x.double() + ref
    K.linear(a, w, b, x, residual=True)
    _close(x, want, k)


# tiles: every tile shape is chosen by one of these; rows and columns one short of, at and beyond a tile's edge
@pytest.mark.parametrize("m,n,k", [(65, 64, 8), (65, 127, 24), (128, 130, 100 * 8), (257, 768, 768), (1000, 2304, 768),
                                   (2047, 768, 3072), (129, 3073, 768), (640, 129, 40)])
def test_tiles(m, n, k):
    a, w, b = _data(m, n, k)
    ref = a.double() @ w.double().T + b.double()
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, b, out)
    _close(out, ref, k)
    fewer = torch.empty(m - 1, n, device=DEV)  # perhaps on another tile: the same sums in the same order
    K.linear(a[:m - 1], w, b, fewer, path="tile")
    assert torch.equal(fewer, out[:m - 1])
    x = torch.randn(m, n, device=DEV)
    want = x.double() + ref
    K.linear(a, w, b, x, residual=True)
    _close(x, want, k)


# more rows than a grid has tiles of 32 downwards
@pytest.mark.parametrize("n", [1, 33])
def test_very_many_rows(n):
    m, k = 32 * 65535 + 1, 8
    a, w, b = _data(m, n, k)
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, b, out)
    ref = torch.addmm(b.double(), a.double(), w.double().T)
    _close(out, ref, k)


# the fastest of the three where they are far apart (csrc/gemm_simt.cu: launch_tile_f32)
@pytest.mark.parametrize("m,n,tile", [(300, 1600, (32, 64)), (100, 768, (32, 32)), (65, 256, (32, 32)), (1300, 768, (32, 64)),
                                      (2048, 3072, (64, 64)), (32 * 65535 + 1, 1, (64, 64))])
def test_which_tile(m, n, tile):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert K.f32_tile(m, n) == tile
