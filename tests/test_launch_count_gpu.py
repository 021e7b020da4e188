"""``K.launches()`` counts the kernels that attention launches: parts that meet in a cluster take none to merge them."""
import pytest
import torch

from rosellm_b200.ops import kernels as K
from test_kernels_gpu import run_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("prompts,splits,wide,scratch,kernels", [
    ([], 1, True, True, 1), ([], 4, True, False, 1), ([], 4, True, True, 2), ([], 4, False, True, 2), ([], 9, True, True, 2), ([40], 4, True, False, 2),
    ([40], 4, True, True, 3), ([40], 1, True, True, 2)])
def test_attention(monkeypatch, prompts, splits, wide, scratch, kernels):
    real, counted = K.attention, []

    def attention(*args, **kw):
        if not scratch:
            kw.update(part_o=None, part_ml=None)
        before = K.launches()
        real(*args, **kw)
        counted.append(K.launches() - before)

    monkeypatch.setattr(K, "attention", attention)
    run_attention(K, torch.bfloat16, prompts + [1, 1], prompts + [600, 90], 6, 2, 64, 16, None, seed=1, splits=splits, decode_wide=wide)
    assert counted == [kernels]


@pytest.mark.parametrize("requests,splits,kernels", [(2, 1, 1), (2, 2, 2), (2, 4, 1), (2, 9, 2), (40, 4, 2)])  # 160 blocks: not all at once
def test_latent_attention(requests, splits, kernels):
    heads, rank, width, page = 4, 64, 72, 16
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pool = torch.randn(4, 1, 1, page, width, device=DEV).bfloat16()
    ids = ints(list(range(requests)))
    scratch = [torch.empty(requests * heads * splits, w, device=DEV) for w in (rank, 2)]
    before = K.launches()
    K.latent_attention(torch.randn(requests, heads * width, device=DEV).bfloat16(), pool, ints([[0, 1, 2, 3]] * requests),
                       ints(list(range(requests + 1))), ints([60] * requests), ids, torch.empty(requests, heads * rank, device=DEV).bfloat16(),
                       sink=torch.zeros(heads, device=DEV), n_heads=heads, rank=rank, scale=0.1, tiles=None, n_tiles=0, decode_reqs=ids,
                       n_decode=requests, decode_by_request=True, n_splits=splits, part_o=scratch[0], part_ml=scratch[1])
    assert K.launches() - before == kernels
    K.check_status(torch.device(DEV))
