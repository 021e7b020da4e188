"""Decode attention in wide blocks: how many warps they have where blocks of sixteen would take a second round."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from rosellm_b200.parts.standard import CausalSelfAttention
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,dh,ahead,behind", [(torch.bfloat16, 64, 960, 961), (torch.float32, 64, 320, 321), (torch.bfloat16, 128, 320, 512),
                                                   (torch.float32, 128, 64, 96), (torch.bfloat16, 256, 64, 512), (torch.float32, 256, 400, 1000),
                                                   (torch.bfloat16, 16, 960, 2000)])
def test_eight_warps_for_short_walks_only(dtype, dh, ahead, behind):
    att = CausalSelfAttention(8 * dh, 8, dh)
    assert not att.decode_sixteen_for(1, ahead, dtype) and att.decode_sixteen_for(1, behind, dtype)
    assert not att.decode_sixteen_for(2, 2 * ahead, dtype) and att.decode_sixteen_for(2, 2 * behind, dtype)
    windowed = CausalSelfAttention(8 * dh, 8, dh, window=ahead)
    assert not windowed.decode_sixteen_for(1, 100_000, dtype)


@pytest.mark.parametrize("dtype,n_req,heads,dh", [(torch.bfloat16, 20, 12, 64), (torch.float32, 10, 16, 32), (torch.bfloat16, 20, 8, 128),
                                                  (torch.float32, 20, 8, 128), (torch.float32, 7, 25, 256)])
def test_sixteen_warps_in_two_rounds(dtype, n_req, heads, dh, monkeypatch):
    lens = [[1, 33, 127, 128, 129, 257, 600][i % 7] for i in range(n_req)]
    real = K.attention
    monkeypatch.setattr(K, "attention", lambda *a, **k: real(*a, **k, decode_sixteen=True))
    run_attention(K, dtype, [1] * n_req, lens, heads, heads, dh, 16, None, seed=dh, decode_wide=True)
