"""A step's index arrays are there when the call that makes them returns: for any stream, and without a wait for the current one."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_index_arrays_made_on_one_stream_and_used_on_another():
    from fms_b200.engine.batch import Batch

    def arrays(offset):
        b = Batch.from_lists([3, 1, 2], [offset, 5, 9], [[7 + offset] * 70, [8] * 40, [9] * 3], [[1], [2], [0]], "cuda", [1, 0, 0])
        tiles = [b.query_tiles(64), b.query_tiles(64, [0, 2]), *b.row_chunks(32), *b.key_rows(0)[:3], b.row_sides(50)[1][3], b.row_sides(4)[1][3]]
        return [b.tokens, b.positions, b.token_seq, b.first_row, b.slots, b.len_after, b.position_ids, b.want_rows] + [t for t in tiles if t is not None]

    want = [t.cpu() for t in arrays(11)]
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    arrays(12)  # memory of the same sizes with other values, given back
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1 << 29)  # some 0.3 s
        start = time.monotonic()
        made = arrays(11)
        waited = time.monotonic() - start
    with torch.cuda.stream(other):
        got = [t.clone() for t in made]
    other.synchronize()
    assert not busy.query() and waited < 0.1
    assert all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
    torch.cuda.synchronize()


def test_index_arrays_are_not_given_out_again_while_their_stream_may_read_them():
    from fms_b200.engine.batch import int32_on

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        first = int32_on("cuda", list(range(1000)))
        torch.cuda._sleep(1 << 27)
        read = first.clone()
        del first
        others = [int32_on("cuda", [-1] * 1000) for _ in range(20)]
    stream.synchronize()
    assert torch.equal(read.cpu(), torch.arange(1000, dtype=torch.int32)) and len(others) == 20


def test_a_capture_refuses_the_copy():
    from fms_b200.engine.batch import Batch

    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(graph):
            Batch.from_lists([0], [0], [[1, 2, 3]], [[2]], "cuda")
    torch.cuda.synchronize()
