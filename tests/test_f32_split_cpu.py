"""What can be shown without a GPU of float32 work on the tensor cores."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "foundation-model-stack_b200", "csrc")


def one_lane_blocks(text):
    """(start, end) of what only an elected lane runs."""
    out = []
    for m in re.finditer(r"elect_one\(\)\)\s*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        out.append((m.end(), at))
    return out


@pytest.mark.parametrize("name", ["gemm_f32_tc.cu", "attention_f32_tc.cuh"])
def test_a_warp_waits_and_gives_up_as_one(name):
    """The lanes of a warp poll a barrier each for itself; where the whole warp waits, what follows takes all of its lanes (shuffles,
    loads of tensor memory), so they have to agree on whether the wait ended or was given up."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    lanes, uses = one_lane_blocks(text), [m.start() for m in re.finditer(r"\bwait_or_abort\(", text)]
    assert lanes and uses
    for at in uses:
        statement = text[max(text.rfind(c, 0, at) for c in ";{}"):at]
        assert any(a <= at < b for a, b in lanes) or "__all_sync(0xffffffffu, " in statement, text[at - 120:at + 60]
    for loop in re.finditer(r"for \([^;]*;[^;]*;[^)]*\)", text):  # nor may lanes leave a loop one by one
        assert "!*failed" not in loop.group() or any(a <= loop.start() < b for a, b in lanes), loop.group()
