"""Which form a decode layer of few rows takes (two fused kernels or kernels of its own), and what the parts keep for it."""
import pytest
import torch

from rosellm_b200.engine.context import standalone_context
from rosellm_b200.models.model import _build_layer
from rosellm_b200.ops import kernels as K
from rosellm_b200.ops.microbench import _fused_kernels_of
from rosellm_b200.parts.spec import LayerSpec, PartSpec, RunEntry
from rosellm_b200.parts.standard import NoPositions
from test_parts_gpu import bind_random, make_cache

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BOTH, FEED_FORWARD = ["attn_block_fused", "mlp_fused"], ["mlp_fused"]


def _layer(hidden, heads):
    spec = LayerSpec(PartSpec("pre_norm", {}, {}), (
        ("norm_mixer", "norm", PartSpec("layer_norm", dict(hidden_size=hidden, eps=1e-5), {})),
        ("mixer", "mixer", PartSpec("causal_self_attention", dict(hidden_size=hidden, num_heads=heads, head_dim=hidden // heads), {})),
        ("norm_feed_forward", "norm", PartSpec("layer_norm", dict(hidden_size=hidden, eps=1e-5), {})),
        ("feed_forward", "feed_forward", PartSpec("dense_mlp", dict(hidden_size=hidden, inner_size=4 * hidden, activation="gelu_tanh"), {}))))
    layer = _build_layer(spec)
    for i, part in enumerate(layer.parts.values()):
        bind_random(part, torch.bfloat16, i, scale=0.02)
    return layer


@pytest.mark.parametrize("hidden,heads,decoded,prompt", [
    # rows of a decode step -> what it launches; tokens of a short prompt -> the same
    (576, 9, {1: BOTH, 4: BOTH, 8: BOTH, 16: BOTH}, {8: [], 9: FEED_FORWARD}),
    (768, 12, {1: BOTH, 2: BOTH, 4: BOTH, 5: [], 8: [], 9: BOTH, 16: BOTH}, {1: [], 12: [], 13: FEED_FORWARD}),
    (896, 14, {1: BOTH, 8: BOTH, 16: BOTH}, {8: [], 9: FEED_FORWARD, 16: FEED_FORWARD}),
    (128, 2, {1: BOTH, 8: BOTH}, {1: FEED_FORWARD, 8: FEED_FORWARD}),
    (1024, 16, {1: [], 8: [], 16: []}, {4: [], 16: []})])
def test_form_of_a_layer(hidden, heads, decoded, prompt):
    layer = _layer(hidden, heads)
    # the second copy of the output weights is kept only where some row count reads it
    kept = hidden <= K.FUSED_LAYER_MAX_WIDTH
    assert (layer.mixer._out_weight_packed is not None) == kept and (layer.feed_forward._out_weight_packed is not None) == kept
    cache = make_cache({0: layer.mixer.cache_spec()}, page=16, pages=80, slots=18, seq=64, dtype=torch.bfloat16)
    slots = [cache.new_request() for _ in range(16)]
    for s in slots:
        assert cache.reserve(s, 32)
    cache.sync_to_device()
    for entries, want in [([(s, 3, [0], []) for s in slots[:rows]], w) for rows, w in decoded.items()] + \
                         [([(slots[0], 3, [0] * n, [])], w) for n, w in prompt.items() if n > 1]:
        ctx = standalone_context(cache, entries, torch.bfloat16)
        ctx.position = NoPositions()
        x = torch.randn(sum(len(e[2]) for e in entries), hidden, device=DEV)
        assert _fused_kernels_of(lambda: layer.block.forward(ctx, RunEntry(0), layer, x)) == want, (len(entries), len(x))
    K.check_status(torch.device(DEV))
