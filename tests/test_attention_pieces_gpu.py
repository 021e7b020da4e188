"""Prompt attention on tcgen05 whose pieces of 128 queries go singly (more pairs of pieces than the device holds blocks), at
lengths beside the edges of pieces and key tiles, against float64."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens_q,lens_kv,heads,n_kv", [
    ([700, 130, 1, 520], [900, 130, 77, 520], 40, 20),     # pieces with a remainder, a decoded request between
    ([128, 129, 127, 256], [128, 257, 1000, 256], 150, 1),  # one piece, one and a row, one short of it
    ([65] * 4, [65, 128, 129, 640], 150, 150),
])
def test_pieces_that_go_singly(lens_q, lens_kv, heads, n_kv):
    tiles = sum(-(-n // 64) for n in lens_q if n > 1)
    assert (tiles + 3) // 4 * heads > K.sm_count(torch.device("cuda:0"))
    run_attention(K, torch.bfloat16, lens_q, lens_kv, heads, n_kv, 64, 16, None, seed=sum(lens_q), prefill_path="tc")


@pytest.mark.parametrize("lens_q,lens_kv,heads", [([512, 500, 449, 511], [512, 900, 449, 511], 32),  # 256 pairs: two rounds, the second well filled
                                                  ([385, 129], [385, 640], 74)])                     # 148 at most: one round
def test_pieces_that_go_in_pairs(lens_q, lens_kv, heads):
    run_attention(K, torch.bfloat16, lens_q, lens_kv, heads, heads, 64, 16, None, seed=heads, prefill_path="tc")
