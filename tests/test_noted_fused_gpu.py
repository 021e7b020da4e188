"""Steps of sizes seen before whose noted launches are the fused decode kernels (clusters, additions in no fixed order)."""
import numpy as np
import pytest
import torch

from rosellm_b200.config import EngineConfig
from rosellm_b200.engine.runner import ModelRunner, StepEntry
from rosellm_b200.ops.microbench import _fused_kernels_of
from tiny import TINY, write_tiny

pytestmark = pytest.mark.gpu


def test_noted_launches_of_the_fused_kernels(tmp_path):
    folder, vocab = write_tiny("B_sharp", str(tmp_path)), TINY["B_sharp"]["config"].vocab_size

    def run(reuse):
        r = ModelRunner.from_folder(folder, EngineConfig(dtype="bfloat16", page_size=8, max_num_seqs=16, max_num_batched_tokens=96,
                                                         kv_cache_tokens=2048, cuda_graphs=False, reuse_launch_lists=reuse))
        rng, out, ran = np.random.default_rng(3), [], {}
        ids = lambda n: rng.integers(0, vocab, n).tolist()
        for _ in range(3):
            slots = [r.cache.new_request() for _ in range(14)]
            for s in slots:
                r.step([StepEntry(s, ids(int(rng.integers(17, 40))), [])])
            for rows in (1, 2, 4, 14, 14):  # decoded requests alone
                names = _fused_kernels_of(lambda: out.append(r.step([StepEntry(s, ids(1), [0]) for s in slots[:rows]]).clone()))
                ran.setdefault(rows, []).append(names)
            for s in slots:
                r.cache.release(s)
        r.check_status()
        return out, ran, r.launch_list_replays

    want, ran, none = run(False)
    both = ["attn_block_fused", "mlp_fused"] * TINY["B_sharp"]["config"].n_layer
    assert none == 0 and all(names == both for n in ran.values() for names in n)
    got, ran, replays = run(True)
    # walked through once a size (and again where a buffer of the workspace has moved), then issued in one native call
    assert replays >= 11 and all(n[0] == both and n[-1] == [] and n.count(both) + n.count([]) == len(n) for n in ran.values())
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, atol=5e-2, rtol=0)  # as where the same kernels are compared with the separate ones
