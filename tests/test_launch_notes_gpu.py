"""Launches noted by the library and issued again in one call; which kernel a product of few rows goes to; decode
attention in blocks of eight warps."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_noted_kernels_are_issued_again_on_new_contents():
    g = torch.Generator(device=DEV).manual_seed(0)
    x = torch.randn(40, 768, generator=g, device=DEV)
    gamma, beta = torch.randn(768, generator=g, device=DEV), torch.randn(768, generator=g, device=DEV)
    h, out = torch.empty(40, 768, dtype=torch.bfloat16, device=DEV), torch.empty(40, 2304, device=DEV)
    ws = [(torch.randn(2304, 768, generator=g, device=DEV) * 0.03).bfloat16() for _ in range(2)]

    def calls():
        K.layernorm(x, gamma, beta, 1e-5, h)
        K.linear(h, ws[0], None, out, path="smem")
        K.linear(h, ws[1], None, out, residual=True, path="tc")  # tensor maps among the arguments
        K.linear(h[:8], ws[0], None, out[:8], residual=True)
        K.linear(h, ws[1], None, out, residual=True, path="tcr")  # a cluster

    before = K.launches()
    with K.recording() as launches:
        calls()
    assert launches._notes is not None and launches.launches == K.launches() - before == 5
    x.copy_(torch.randn(40, 768, generator=g, device=DEV))
    calls()
    want = out.clone()
    out.fill_(float("nan"))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # on the stream that is current then
        launches.replay()
    torch.cuda.current_stream().wait_stream(side)
    # the sums of a product in parts of K meet in no fixed order: float32 roundings of values below 16
    assert (out - want).abs().max().item() < 16 * 8 * 2.0 ** -24 * 8
    K.check_status(torch.device(DEV))


def test_a_copy_between_the_launches_keeps_the_calls():
    src, dst = torch.arange(8, dtype=torch.int32).pin_memory(), torch.zeros(8, dtype=torch.int32, device=DEV)
    with K.recording() as launches:
        K.copy_to_device(dst, src, 8)
    assert launches._notes is None
    dst.zero_()
    launches.replay()
    assert dst.tolist() == list(range(8))


@pytest.mark.parametrize("rows,n,k,kw,path", [
    (16, 4800, 1600, {}, "mma"), (17, 4800, 1600, {}, "tc"), (64, 4800, 1600, {}, "tc"), (64, 2304, 768, {}, "smem"),
    (64, 1600, 6400, dict(residual=True, out_f32=True), "tc"), (64, 768, 3072, dict(residual=True, out_f32=True), "smem"),
    (96, 768, 768, {}, "tc"), (40, 301, 1600, dict(out_f32=True), "mma"), (64, 5003, 1600, dict(out_f32=True), "mma"),
    (40, 2048, 8192, dict(out_f32=True), "tc")])
def test_which_kernel_takes_a_product(rows, n, k, kw, path):
    assert K.bf16_path(rows, n, k, **kw) == path


@pytest.mark.parametrize("dtype,n_req,heads,dh", [(torch.bfloat16, 20, 12, 64), (torch.float32, 10, 16, 32), (torch.bfloat16, 13, 12, 128),
                                                  (torch.float32, 7, 25, 256)])
def test_decode_attention_in_blocks_of_eight_warps(dtype, n_req, heads, dh):
    """More blocks than the device holds of sixteen warps; contexts of one key, beside a round of a block's keys and beyond."""
    lens = [[1, 33, 127, 128, 129, 257, 600][i % 7] for i in range(n_req)]
    run_attention(K, dtype, [1] * n_req, lens, heads, heads, dh, 16, None, seed=dh, decode_wide=True)


def test_a_kernel_whose_limit_of_shared_memory_has_been_lowered_since_is_issued_again():
    """The norm of rows of some sizes has its kernel's limit set to what each launch needs: one of shorter rows lowers it."""
    def row(n):
        x = torch.randn(3, n, device=DEV)
        return x, torch.randn(n, device=DEV), torch.randn(n, device=DEV), torch.empty(3, n, device=DEV)

    long, short = row(30001), row(14001)  # 117 and 55 KB, both above the limit that needs no raising
    with K.recording() as launches:
        K.layernorm(*long[:3], 1e-5, long[3])
    assert launches._notes is not None
    K.layernorm(*short[:3], 1e-5, short[3])
    long[0].mul_(2).add_(1)
    long[3].fill_(float("nan"))
    launches.replay()
    for x, gamma, beta, out in (long, short):
        want = torch.nn.functional.layer_norm(x.double(), x.shape[1:], gamma.double(), beta.double(), 1e-5)
        assert (out.double() - want).abs().max().item() < 1e-4  # float32 statistics of numbers of order 1
    K.layernorm(*short[:3], 1e-5, short[3])
    launches.replay()  # and once more after the limit was lowered a second time
    torch.cuda.synchronize()
