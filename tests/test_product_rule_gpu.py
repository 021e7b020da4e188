"""Which kernel takes a bfloat16 product of 17 to 64 rows that shared memory does not hold in one round, and what it gives."""
import pytest
import torch

from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F32 = dict(out_f32=True)


@pytest.mark.parametrize("rows,n,k,kw,path", [
    # few weights: the kernels they ran on before the tiles
    (33, 768, 1600, {}, "mma"), (64, 1024, 1600, {}, "mma"), (64, 1032, 1600, {}, "tc"), (33, 1024, 2048, {}, "tcr"),
    (64, 1600, 2048, {}, "tcr"), (64, 1608, 2048, {}, "tc"), (17, 2304, 3072, {}, "mma"), (32, 2312, 3072, {}, "tc"),
    (17, 1024, 4096, {}, "mma"), (32, 1032, 4096, {}, "tc"), (64, 1024, 4096, {}, "tc"), (64, 1600, 1600, F32, "mma"),
    (33, 1600, 6400, dict(residual=True, out_f32=True), "tc"),
    # float32 outputs and heads in several rounds
    (32, 5000, 768, F32, "mma"), (33, 5000, 768, F32, "smem"), (17, 9400, 1600, F32, "smem"), (17, 7000, 1600, F32, "mma"),
    (32, 4096, 4096, dict(out_f32=True, head=True), "mma"), (64, 1600, 2048, dict(out_f32=True, head=True), "tcr"),
    (17, 9400, 2048, dict(out_f32=True, head=True), "mma"), (17, 9400, 2048, F32, "tc")])
def test_route_and_result(rows, n, k, kw, path):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert K.bf16_path(rows, n, k, **kw) == path
    g = torch.Generator(device=DEV).manual_seed(rows + n + k)
    a = torch.randn(rows, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * k ** -0.5).bfloat16()
    out = torch.randn(rows, n, generator=g, device=DEV).to(torch.float32 if kw.get("out_f32") else torch.bfloat16)
    ref = a.double() @ w.double().T + (out.double() if kw.get("residual") else 0.0)
    K.linear(a, w, None, out, residual=kw.get("residual", False), head=kw.get("head", False))
    # float32 sums of k products whose results are of order 1; a bfloat16 result rounds by 2^-9 of its size
    err = (out.double() - ref).abs() - (0.0 if kw.get("out_f32") else ref.abs() * 2.0 ** -8)
    assert err.max().item() <= 8 * k * 2.0 ** -24 + 1e-6
    K.check_status(torch.device(DEV))
