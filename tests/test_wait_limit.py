"""What follows a wait that has run out, read from the sources: a run shows a thread left behind at a barrier only by hanging."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "gpt.c_b200", "csrc")
# The flag changes at any time, so threads that each look at it for themselves need not decide the same.
LEAVES_ALONE = re.compile(r"if \([^;{]*(?:cta_abort|abort_flag)[^;{]*\)\s*\{?\s*(?:return|break|continue)\b")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_no_thread_leaves_by_its_own_look_at_the_flag(path):
    assert not LEAVES_ALONE.search(open(path).read())


def test_cross_entropy_waits_for_its_copies_before_it_ends():
    text = open(os.path.join(CSRC, "xent_sm100.cu")).read()
    body = text[text.index("xent_forward_rows_kernel("):]
    assert re.search(r"drain\(sm, load_rows\(", body[:body.index("\n}\n")])
