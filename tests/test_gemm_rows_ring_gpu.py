"""The product of at most 16 rows fed by a ring of stages in shared memory (csrc/gemm_rows_ring.cu), at the sizes where
its cuts and remainders change, against float64."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _data(m, n, k, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    return torch.randn(m, k, generator=g, device=DEV), w, torch.randn(n, generator=g, device=DEV)


def _close(got, ref, k):
    """float32 sums of k products of bfloat16 numbers, whose results are of order 1: each of the k additions rounds by at
    most 2^-24 of a partial sum below 8 or so; a bfloat16 result rounds by 2^-9 of its size."""
    tol = 8 * k * 2.0 ** -24
    assert torch.isfinite(got).all()
    err = (got.double() - ref).abs()
    if got.dtype == torch.bfloat16:
        err = err - ref.abs() * 2.0 ** -8
    assert err.max().item() <= tol + 1e-6


# K: below a warp's 32, ragged, a stage exactly, one beyond it, two stages, more than a warp's fragments hold;
# N: a pair, a ragged group, one group a block, several rounds of groups (inner sizes that are no multiple of 64, and short
# ones, run on the register-fed kernel: test_where_the_ring_begins)
@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(2, 8), (10, 40), (66, 1000), (1600, 1024), (4800, 1088), (6400, 1600), (72, 2048),
                                 (130, 2112), (2048, 8192), (16384, 256), (10, 64)])
def test_rows_of_a_matrix(m, n, k):
    a, w, b = _data(m, n, k)
    a = a.bfloat16()
    ref = a.double() @ w.double().T + b.double()
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((m, n), float("nan"), device=DEV, dtype=dtype)
        K.linear(a, w, b, out, path="mma")
        _close(out, ref, k)
    out = torch.empty(m, n, device=DEV, dtype=torch.float32)
    K.linear(a, w, b, out, act=K.ACT_RELU_SQUARED, path="mma")
    assert torch.allclose(out.double(), ref.clamp(min=0) ** 2, rtol=1e-4, atol=1e-4)
    K.check_status(torch.device(DEV))


@pytest.mark.parametrize("m", [1, 8, 16])
@pytest.mark.parametrize("n,k", [(10, 40), (768, 3072), (1600, 1600), (1600, 6400), (24, 5120), (1202, 4160)])
def test_added_to_the_stream_in_parts_of_k(m, n, k):
    a, w, b = _data(m, n, k, 1)
    a = a.bfloat16()
    x = torch.randn(m, n + 6, device=DEV)[:, :n]  # a row stride of its own
    ref = x.double() + a.double() @ w.double().T + b.double()
    K.linear(a, w, b, x, residual=True, path="mma")
    _close(x, ref, k)
    K.check_status(torch.device(DEV))


@pytest.mark.parametrize("m,k", [(1, 8), (16, 40), (9, 1000), (16, 1024), (8, 960), (5, 64)])
def test_normalised_inside(m, k):
    n = 330
    x, w, b = _data(m, n, k, 2)
    x = x * 3 + 1
    gamma, beta = torch.randn(k, device=DEV), torch.randn(k, device=DEV)
    for bt in (beta, None):
        h = torch.nn.functional.layer_norm(x.double(), (k,), gamma.double(), None if bt is None else bt.double(), 1e-5)
        out = torch.empty(m, n, device=DEV, dtype=torch.float32)
        K.linear(K.NormInput(x, gamma, bt, 1e-5), w, b, out)
        # the rows are rounded to bfloat16 (2^-9 of each of k entries of order 1, weights of order k^-1/2: below
        # 2^-9 sqrt(k) k^-1/2 in the mean square, eight times that at most over a few thousand results)
        ref = h.bfloat16().double() @ w.double().T + b.double()
        assert (out.double() - ref).abs().max().item() < 8 * 2.0 ** -9
    K.check_status(torch.device(DEV))


@pytest.mark.parametrize("k", [64, 320, 1088])  # register-fed; five blocks for eight warps; a second piece of one block
def test_weights_that_are_not_finite_stay_in_their_column(k):
    """What a stage held before, and blocks of K that a warp does not have, never reach a sum."""
    m, n = 8, 4000
    a, w, b = _data(m, n, k, 3)
    a = a.bfloat16()
    w[::2] = float("nan")
    out = torch.empty(m, n, device=DEV, dtype=torch.float32)
    K.linear(a, w, b, out, path="mma")
    assert torch.isnan(out[:, ::2]).all()
    _close(out[:, 1::2], (a.double() @ w.double().T + b.double())[:, 1::2], k)


# short rows of W go through the ring only where a block has few groups of columns and the rows of A are few, or where the
# result is added to the stream: both sides of each line (gemm_rows_ring.cu: short_rows; six groups a block on 148 SMs)
@pytest.mark.parametrize("m,n,k,residual,norm,ring", [
    (8, 7104, 256, False, False, True), (8, 7106, 256, False, False, False), (8, 4736, 192, False, False, False),
    (9, 2368, 512, False, False, False), (9, 2368, 576, False, False, True), (8, 7106, 512, False, False, False),
    (8, 16384, 576, False, False, True), (16, 256, 256, True, False, True), (16, 256, 128, True, False, True),
    (16, 256, 64, True, False, False), (8, 7106, 512, True, False, False), (1, 2304, 256, False, True, False),
    (1, 2304, 320, False, True, True), (2, 2304, 128, False, True, False), (2, 2304, 64, False, True, True),
    (3, 2304, 128, False, True, True), (8, 10, 64, False, False, False)])
def test_where_the_ring_begins(m, n, k, residual, norm, ring):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert K.rows_are_ring_fed(m, n, k, residual=residual, norm=norm) == ring
    a, w, b = _data(m, n, k, 4)
    x = torch.randn(m, n, device=DEV) if residual else torch.full((m, n), float("nan"), device=DEV)
    if norm:
        inp = K.NormInput(a, torch.randn(k, device=DEV), None, 1e-5)
        h = torch.nn.functional.layer_norm(a.double(), (k,), inp.gamma.double(), None, 1e-5).bfloat16().double()
        # as in test_normalised_inside
        tol = 8 * 2.0 ** -9
    else:
        inp, h, tol = a.bfloat16(), a.bfloat16().double(), 8 * k * 2.0 ** -24 + 1e-6
    ref = h @ w.double().T + b.double() + (x.double() if residual else 0.0)
    K.linear(inp, w, b, x, residual=residual)
    assert (x.double() - ref).abs().max().item() <= tol
    K.check_status(torch.device(DEV))
