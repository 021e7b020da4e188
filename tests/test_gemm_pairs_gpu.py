"""tcgen05 products on pairs of SMs (tiles of 256 rows over two blocks), and the clustered kernel of few rows whose ring is
shorter than its part of K."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAIRS = -2


def _data(m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m * 5 + n * 3 + k)
    return (torch.randn(m, k, generator=g, device=DEV).bfloat16(), (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16(),
            torch.randn(n, generator=g, device=DEV))


def _close(got, ref, k):
    # float32 sums of k products with results of order 1
    assert (got.double() - ref).abs().max().item() <= 8 * k * 2.0 ** -24 + 1e-6


# the second block's rows all there, some, none; columns that end in the first or the second block's half of W; K blocks: one,
# fewer than stages, several laps; more tiles than pairs
@pytest.mark.parametrize("m,n,k,width", [(256, 256, 64, 256), (129, 72, 64, 64), (128, 96, 136, 96), (385, 1000, 200, 224), (300, 160, 1600, 160),
                                         (2048, 4800, 192, 128), (520, 776, 1544, 192), (640, 100, 768, 64)])
def test_pairs(m, n, k, width):
    a, w, b = _data(m, n, k)
    ref = a.double() @ w.double().T + b.double()
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, b, out, path="tc", tile_width=width, splits=PAIRS)
    _close(out, ref, k)
    x = torch.randn(m, n, device=DEV)
    want = x.double() + ref
    K.linear(a, w, b, x, residual=True, path="tc", tile_width=width, splits=PAIRS)
    _close(x, want, k)
    single = torch.empty_like(out)
    K.linear(a, w, b, single, path="tc", tile_width=width, splits=1)
    assert torch.equal(single, out)  # the same sums in the same order
    half = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.linear(a, w, b, half, path="tc", tile_width=width, splits=PAIRS)
    assert torch.equal(half, out.bfloat16())
    K.check_status(torch.device(DEV))


# by the library's own choice: sizes that go to pairs, beside ones that do not
@pytest.mark.parametrize("m,n,k", [(2048, 1600, 6400), (700, 3072, 2048), (257, 6400, 1600)])
def test_chosen(m, n, k):
    a, w, b = _data(m, n, k)
    x = torch.randn(m, n, device=DEV)
    want = x.double() + a.double() @ w.double().T + b.double()
    K.linear(a, w, b, x, residual=True)
    _close(x, want, k)
    K.check_status(torch.device(DEV))


# rows at the edges of the 16 that they are rounded up to; one block a cluster to eight, parts of K longer than the ring, the last
# one short; an output that ends inside a tile
@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(200, 104), (768, 768), (3072, 1024), (130, 6400), (6400, 200), (1000, 1608)])
def test_rows_in_clusters(m, n, k):
    a, w, b = _data(m, n, k)
    ref = a.double() @ w.double().T + b.double()
    out = torch.full((m, n), float("nan"), device=DEV)
    K.linear(a, w, b, out, path="tcr")
    _close(out, ref, k)
    again = torch.empty_like(out)
    K.linear(a, w, b, again, path="tcr")
    assert torch.equal(again, out)
    x = torch.randn(m, n, device=DEV)
    want = x.double() + ref
    K.linear(a, w, b, x, residual=True, path="tcr")
    _close(x, want, k)
    half = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device=DEV)
    K.linear(a, w, b, half, path="tcr")
    assert torch.equal(half, out.bfloat16())
    K.check_status(torch.device(DEV))


@pytest.mark.parametrize("rows,n,k,kw,clustered", [
    (16, 3072, 1024, {}, False), (17, 3072, 1024, {}, True), (64, 3072, 1024, {}, True), (65, 3072, 1024, {}, False), (64, 3071, 1024, {}, False),
    (64, 3072, 1023, {}, False), (64, 4800, 1600, dict(out_f32=True), False), (64, 1600, 6400, dict(residual=True, out_f32=True), True),
    (64, 1600, 6399, dict(residual=True, out_f32=True), False), (64, 4800, 8256, {}, False), (64, 9472, 1600, {}, False)])
def test_which_products_go_to_clusters(rows, n, k, kw, clustered):
    assert K.clustered_is_ahead(rows, n, k, **kw) == clustered
