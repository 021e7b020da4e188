"""What the library's C entry points refuse before anything is launched (no device is needed to be told so)."""
import pytest
import torch

from rosellm_b200.ops import kernels as K


@pytest.mark.parametrize("splits,wide,part_o,part_ml", [
    (2, 1, True, False), (8, 2, True, False), (2, 1, False, True),  # one half of the scratch
    (2, 0, False, False), (9, 1, False, False), (9, 1, True, False), (3, 0, True, False), (0, 1, True, True)])
def test_decode_parts_need_both_halves_of_their_scratch(splits, wide, part_o, part_ml):
    some = torch.zeros(64)
    at = some.data_ptr()
    rc = K._lib().rl_attention(0, at, 16, at, at, 1, at, at, at, at, 16, 1, 1, 16, 16, 0, 1.0, None, 0, None, 0, at, 1, splits, wide,
                               at if part_o else None, at if part_ml else None, 1, 1, 0, 0, at, None)
    assert rc == -4
