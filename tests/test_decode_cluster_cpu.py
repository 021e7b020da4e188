"""Which decode steps have the parts of a request's keys meet in clusters, and that all other parts get their scratch."""
from types import SimpleNamespace

import pytest
import torch

from rosellm_b200.engine.context import Workspace
from rosellm_b200.ops import kernels as K
from rosellm_b200.parts.standard import CausalSelfAttention

F32, BF16 = torch.float32, torch.bfloat16


# (heads, head size, requests, keys, dtype, whether a cluster, parts): both sides of every line of the rule
@pytest.mark.parametrize("heads,dh,n,span,dtype,clustered,parts", [
    (12, 64, 1, 299, BF16, False, 1), (12, 64, 1, 300, BF16, True, 3), (12, 64, 1, 4095, BF16, True, 8), (12, 64, 1, 4096, BF16, False, 4),
    (16, 64, 1, 8192, BF16, False, 8), (24, 64, 1, 8192, BF16, True, 8), (24, 64, 1, 8193, BF16, False, 8), (37, 64, 1, 8192, BF16, True, 8),
    (38, 64, 1, 499, BF16, False, 1), (38, 64, 1, 8192, BF16, True, 6), (66, 64, 1, 500, F32, True, 6), (67, 64, 1, 2100, BF16, False, 2),
    (16, 64, 9, 4100, BF16, False, 2), (148, 64, 1, 2100, BF16, False, 2), (149, 64, 1, 2100, BF16, True, 2), (222, 64, 1, 300, F32, True, 2),
    (223, 64, 1, 900, BF16, False, 1), (16, 128, 1, 2100, F32, False, 2), (16, 128, 4, 4100, F32, False, 4), (16, 128, 1, 2100, BF16, True, 8),
    (12, 64, 1, 20000, BF16, False, 19)])
def test_scratch_goes_with_the_parts_that_are_merged(monkeypatch, heads, dh, n, span, dtype, clustered, parts):
    monkeypatch.setattr(K, "device_facts_given", (148, 233472))
    calls = []
    monkeypatch.setattr(K, "linear", lambda *a, **k: None)
    monkeypatch.setattr(K, "kv_write", lambda *a, **k: None)
    monkeypatch.setattr(K, "attention", lambda *a, **k: calls.append(k))
    att = CausalSelfAttention(heads * dh, heads, dh)
    run = SimpleNamespace(writes_cache=False, cache_key=0)
    ctx = SimpleNamespace(n_tokens=n, n_decode=n, n_reqs=n, n_tiles=0, n_tiles_wide=0, max_kv_len=span, max_tile_kv_len=0, act_dtype=dtype, extras={},
                          workspace=Workspace(torch.device("cpu")), kv_pool=lambda k: None, block_table=lambda k: None,
                          position=SimpleNamespace(rotate=lambda *a: None), q_start=None, kv_len=None, slots=None, tiles=None, tiles_wide=None,
                          decode_reqs=None, positions=None, req_of_token=None)
    for extras in ({}, {"decode_plan": att.decode_plan_for(n, span, dtype), "decode_span": span}):  # as the step goes, and as a captured one is laid out
        ctx.extras = extras
        att.forward(ctx, run, None, None)
        call = calls.pop()
        assert call["n_splits"] == parts and call["decode_wide"]
        assert (parts > 1 and call["part_o"] is None) == clustered
        if parts > 1 and not clustered:
            assert call["part_o"].numel() == n * heads * parts * dh and call["part_ml"].numel() == n * heads * parts * 2
        assert att.launch_key(ctx)[1] == clustered
