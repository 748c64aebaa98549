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


def test_rows_of_either_side_of_a_limit():
    """Which rows a float32 product takes together: neighbours as they lie, a side of several runs by its places."""
    from fms_b200.engine.batch import Batch, row_sides

    def plain(sides):
        return [(many, first, rows, None if places is None else places.tolist()) for many, first, rows, places in sides]

    assert plain(row_sides([3, 0, 4], 3, "cpu")) == [(True, 0, 7, None)]
    assert plain(row_sides([3, 4, 1, 1], 3, "cpu")) == [(True, 0, 7, None), (False, 7, 2, None)]
    assert plain(row_sides([1, 0, 3, 2, 4, 0], 3, "cpu")) == [(True, 0, 7, [1, 2, 3, 6, 7, 8, 9]), (False, 0, 3, [0, 4, 5])]
    assert plain(row_sides([2, 3, 2], 3, "cpu", True)) == [(True, 2, 3, None), (False, 0, 2, None), (False, 5, 2, None)]
    batch = Batch.from_lists([0, 1, 2], [0, 0, 0], [[1], [2, 3], [4]], [[], [], []], "cpu")
    assert batch.row_sides(2, True) is not batch.row_sides(2) and batch.row_sides(2, True) is batch.row_sides(2)


def test_scratch_of_a_product_gives_way(monkeypatch):
    """A card without room for a product's scratch takes fewer rows at a time, down to 32, and every row once."""
    import torch

    from fms_b200.kernels import ops

    room, taken = [0], []
    empty = torch.empty

    def scratch(shape, dtype=None, device=None):
        if shape[0] > room[0]:
            raise torch.OutOfMemoryError("no room")
        return empty(shape, dtype=dtype, device=device)

    monkeypatch.setattr(ops, "error_flag", lambda device: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "_call", lambda library, name, x, w, b, y, s, have, rows, n, k, *_: (
        taken.append((x.shape[0], rows)), y.fill_(1.0), have >= rows * (-(-k // 64) * 384 + 1) + n or pytest.fail("too little scratch")))
    x, w = torch.zeros(1000, 128), torch.zeros(7, 128)
    for at_a_time in (1000, 999, 300, 100, 32):
        y = torch.zeros(1000, 7)
        room[0], taken[:] = at_a_time * 769 + 7, []
        monkeypatch.setattr(torch, "empty", scratch)
        ops._split_product(x, w, None, y)
        monkeypatch.setattr(torch, "empty", empty)
        assert bool((y == 1).all()) and sum(r for _, r in taken) == 1000 and max(r for _, r in taken) <= at_a_time
        assert all(a == r for a, r in taken)
    monkeypatch.setattr(torch, "empty", scratch)
    room[0] = 31 * 769 + 7
    with pytest.raises(torch.OutOfMemoryError):
        ops._split_product(x, w, None, torch.zeros(1000, 7))
