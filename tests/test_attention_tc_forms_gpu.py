"""Prompt attention on tcgen05 (csrc/attention_tc.cuh): how the pieces of 128 queries go over the blocks, against 64 bits."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu


# on 148 SMs: pieces that all stand at once go singly; more of them, requests of five pieces singly beside others in pairs (one of them an odd
# number, one a single piece and a row); in pairs; singly again where pairs would need a second round
@pytest.mark.parametrize("heads,kv_heads,lens", [(2, 1, [300, 70]), (12, 12, [640, 512, 300, 129]), (16, 4, [513, 512, 384, 500]), (40, 8, [600, 500])])
def test_pieces_over_blocks(heads, kv_heads, lens):
    before = [0, 37, 200, 5][:len(lens)]  # tokens that are cached already
    run_attention(K, torch.bfloat16, lens, [n + b for n, b in zip(lens, before)], heads, kv_heads, 64, 16, None, seed=heads, prefill_path="tc")
