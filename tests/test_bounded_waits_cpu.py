"""Waits on barriers that give up after a while, read in the sources: a warp leaves a loop by them as a whole."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rosellm_b200", "csrc")
# `ok = wait(...)` by each lane for itself, followed by an end of the loop: a lane that gave up would be gone where the others meet it again
ALONE = re.compile(r"\bok\s*=\s*(?:tc::)?(?:mbar|att)_wait\([^;]*;[^\n]*\n\s*if \(!ok\) (?:break|return)")
# what is one lane's own loop: (file, what stands before it)
ONE_LANE = {"gemm_rows_ring.cu": "if (lap > 0) {"}


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_a_wait_that_ends_a_loop_is_the_whole_warps(path):
    source = open(path).read()
    for m in ALONE.finditer(source):
        before = source[:m.start()].rstrip()
        assert before.endswith(ONE_LANE.get(os.path.basename(path), "\0")), source[:m.start()].count("\n") + 1
