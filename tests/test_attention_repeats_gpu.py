"""Prompt attention on tcgen05 gives the same bits every time: nothing of a tile is overwritten while a product reads it,
however late the next tile's keys arrive."""
import pytest
import torch

from rosellm_b200.engine.context import build_host_batch
from rosellm_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("heads,lens", [(25, (1024, 1024)), (12, (1024, 1024)), (3, (900, 130, 640))])  # singly; in pairs
def test_the_same_bits_with_warm_and_with_cold_caches(heads, lens):
    g = torch.Generator(device=DEV).manual_seed(heads)
    dh, ps, per = 64, 16, 64
    pool = torch.randn(len(lens) * per, 2, heads, ps, dh, generator=g, device=DEV).bfloat16()
    table = torch.arange(len(lens) * per, dtype=torch.int32, device=DEV).view(len(lens), per)
    hb = build_host_batch([(r, 0, [0] * n, []) for r, n in enumerate(lens)])
    i32 = lambda a: torch.as_tensor(a, dtype=torch.int32).contiguous().to(DEV)
    qs, kl, sl, tiles, wide = i32(hb.q_start), i32(hb.kv_len), i32(hb.slots), i32(hb.tiles.reshape(-1)), i32(hb.tiles_wide.reshape(-1))
    q = (torch.randn(sum(lens), heads * dh, generator=g, device=DEV) * 3).bfloat16()
    flush = torch.empty(160 << 20, dtype=torch.uint8, device=DEV)  # more than the second-level cache
    want = None
    for i in range(150):
        if i % 3:
            flush.fill_(i)
        out = torch.empty_like(q)
        K.attention(q, pool, table, qs, kl, sl, out, n_heads=heads, scale=dh ** -0.5, window=None, tiles=tiles, n_tiles=len(hb.tiles),
                    decode_reqs=None, n_decode=0, n_splits=1, part_o=None, part_ml=None, tiles_wide=wide,
                    n_tiles_wide=len(hb.tiles_wide), decode_wide=False, old_keys_settled=True, prefill_path="tc")
        want = out if want is None else want
        assert torch.equal(out, want), f"run {i}: {int((out != want).sum())} entries differ"
    K.check_status(torch.device(DEV))
