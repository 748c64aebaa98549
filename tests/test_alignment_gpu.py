"""Tensors that do not lie on 16 bytes: the kernels with wide loads leave them to the others, with the same results."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def shifted(t):
    """The same values, contiguous, four bytes further on than a 16-byte boundary."""
    room = torch.empty(t.numel() + 16 // t.element_size(), dtype=t.dtype, device=t.device)
    at = 4 // t.element_size()
    out = room[at:at + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.is_contiguous() and out.data_ptr() % 16 == 4
    return out


def batch_of(lengths):
    from fms_b200.engine.batch import Batch

    return Batch.from_lists(list(range(len(lengths))), [0] * len(lengths), [[0] * n for n in lengths], [[] for _ in lengths], "cuda")


@pytest.mark.parametrize("rows,hd", [(64, 128), (65, 16), (70, 12), (63, 128)])
def test_rotation_of_shifted_float32_rows(rows, hd):
    """Whole pieces of four values or not (12: pairs only in the general kernel's width), just below and above the number of
    rows from which the vector kernel takes over.  The angles and products are the same; a multiply-add may be contracted
    differently, half a unit of 2^-24 of a sum of two terms of at most 5."""
    from fms_b200.cache import Cache, KVRequest
    from fms_b200.kernels import ops

    nheads, kvheads = 3, 1
    g = torch.Generator().manual_seed(rows)
    qkv = torch.randn(rows, (nheads + 2 * kvheads) * hd, generator=g).cuda()
    inv = (1.0 / (10000.0 ** (torch.arange(0, hd, 2).float() / hd))).cuda()
    results = []
    for x in (qkv, shifted(qkv)):
        cache = Cache([KVRequest(kvheads, hd)], 256, 256, torch.float32, "cuda", max_slots=1)
        slots = cache.begin(1)
        lengths = cache.prepare(slots, [rows])
        from fms_b200.engine.batch import Batch

        batch = Batch.from_lists(slots, lengths, [[0] * rows], [[]], "cuda")
        view = cache.layer_view(0)
        view.keys.zero_()
        view.values.zero_()
        results.append((ops.rope_store(x, inv, batch, view, nheads, kvheads, hd), view.keys.clone(), view.values.clone()))
    for a, b in zip(*results):
        assert float((a - b).abs().max()) <= 5 * 2.0 ** -23
    assert torch.equal(results[0][2], results[1][2])  # values are only moved


@pytest.mark.parametrize("rows,n,k", [(1, 33, 132), (8, 96, 1024), (32, 31, 4), (33, 130, 260), (70, 129, 1056)])
def test_float32_products_of_shifted_operands(rows, n, k):
    """Few rows and many; x, the matrix or both four bytes off.  The sums run in the same order, so they are the same bits."""
    from fms_b200.kernels import ops

    g = torch.Generator().manual_seed(rows)
    x, w, b = torch.randn(rows, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    want = ops.linear(x, w, b)
    for a, m in ((shifted(x), w), (x, shifted(w)), (shifted(x), shifted(w))):
        assert torch.equal(ops.linear(a, m, shifted(b)), want)


def test_scans_of_shifted_rows(monkeypatch):
    """The walk over tokens takes them; beside the runs that the same values on 16 bytes take, as in the test of the runs."""
    from fms_b200.kernels import ops

    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: True)
    heads, dim, vdim, n = 2, 128, 128, 150
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    batch, rows, logits, state = batch_of([100, 50]), r(n, heads * vdim + 2 * dim) * 0.3, r(n, 2 * heads), r(2, heads, vdim, dim)
    qkv, bias, rates, skip = r(n, 2 * dim + heads * vdim), r(heads) - 2.0, r(heads).abs(), r(heads)
    results = []
    for move in (lambda t: t.clone(), shifted):
        s0, s1, x0, x1 = state.clone(), state.clone(), move(rows), move(qkv)
        y0 = ops.selective_scan(x0, logits, 0, bias, rates, skip, s0, batch, heads, vdim, dim, 1)
        y1 = ops.delta_rule_scan(x1, logits, 0, None, bias, rates, s1, batch, heads, 1, dim, vdim, decay_offset=heads)
        results.append((y0, y1, s0, s1))
    for a, b in zip(*results):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
        assert float((a - b).norm()) <= 2e-6 * float(b.norm())
