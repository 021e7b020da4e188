"""Decode attention with the parts of a request's keys in the blocks of a cluster, against 64 bits."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from rosellm_b200.parts.standard import CausalSelfAttention
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu


# contexts that the first block takes alone (up to 256 keys), one key more, parts without keys (257 keys in eight parts of 64), full
# parts; a window; head sizes up to the largest, groups of heads
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("splits", [2, 3, 8])
@pytest.mark.parametrize("dh,heads,kv", [(64, 6, 2), (16, 2, 2), (128, 4, 4), (256, 2, 1)])
def test_parts_in_a_cluster(dtype, splits, dh, heads, kv, monkeypatch):
    real = K.attention
    monkeypatch.setattr(K, "attention", lambda *a, **k: real(*a, **{**k, "part_o": None, "part_ml": None}))
    lens = [700, 1, 256, 257, 1030, 33]
    run_attention(K, dtype, [1] * 6, lens, heads, kv, dh, 16, None, seed=splits, splits=splits, decode_wide=True, sharp=True)
    run_attention(K, dtype, [1] * 3, [900, 300, 40], heads, kv, dh, 8, 300, seed=splits + 1, splits=splits, decode_wide=True)


def test_parts_without_scratch_are_refused_otherwise():
    for splits, wide in ((9, True), (2, False)):
        with pytest.raises(K.KernelError, match="scratch"):
            K.attention(torch.zeros(1, 64, device="cuda"), torch.zeros(1, 2, 1, 16, 64, device="cuda"), torch.zeros(1, 1, dtype=torch.int32),
                        None, None, None, torch.zeros(1, 64, device="cuda"), n_heads=1, scale=1.0, window=None, tiles=None, n_tiles=0,
                        decode_reqs=None, n_decode=1, n_splits=splits, decode_wide=wide)


def test_which_steps_take_clusters():
    att = CausalSelfAttention(25 * 64, 25, 64)
    if K.sm_count() == 148:
        plans = {(n, span): att.decode_plan_for(n, span) for n in (1, 2, 4, 8, 11) for span in (256, 299, 300, 544, 1024)}
        assert plans[1, 256] == plans[1, 299] == (1, True) and plans[1, 300] == (3, True) and plans[1, 544] == (5, True)
        assert plans[1, 1024] == (8, True) and plans[2, 544] == (6, True) and plans[4, 1024] == (1, True)
        assert plans[8, 300] == plans[8, 1024] == (2, True) and plans[11, 1024] == (1, True)
