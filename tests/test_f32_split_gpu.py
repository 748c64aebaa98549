"""Float32 products of many rows on the tensor cores (operands in three bfloat16 parts), against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fms_b200.kernels import ops

    yield ops
    ops.check_error_flag("cuda:0")


def made(m, n, k, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(*s, generator=g, device="cuda") for s in ((m, k), (n, k), (n,))]


def bound(x, w, b):
    """Of an element's error, from its terms' magnitudes: an accumulator cuts off at most 2^-23 of what it holds, twice at the large
    products and ten times at 2^-8 of it; parts left out are 3 * 2^-26 of a term; every 32 k, every run and the bias round once."""
    k = x.shape[1]
    return ((2 + 10 * 2.0 ** -7) * 2.0 ** -23 + 3 * 2.0 ** -26 + (k / 4 / 32 + 8) * 2.0 ** -24) * (x.double().abs() @ w.double().abs().T + b.double().abs())


@pytest.mark.parametrize("n,k", [(1024, 1024), (1153, 1050), (1030, 2052), (4100, 3072)])
@pytest.mark.parametrize("m", [33, 64, 65, 129, 256, 257, 600])
def test_edges_of_tiles_runs_and_steps(ops, m, n, k):
    """Tiles of 128 rows of w by up to 256 of x, clusters and single blocks, K of no multiple of 4 or of a step; a row's
    result is the same bits however many rows are beside it."""
    x, w, b = made(m, n, k)
    got = ops.linear(x, w, b, None, [m])
    assert bool(((got.double() - (x.double() @ w.double().T + b.double())).abs() <= bound(x, w, b)).all())
    few = max(m // 2, ops.f32_split_tokens(w))
    assert torch.equal(ops.linear(x[:few].contiguous(), w, b, None, [few]), got[:few])
    assert torch.equal(ops.linear(x, w, None, None, [m]) + b, got)


def test_a_sequence_chooses_by_its_own_rows(ops):
    """Sequences of one row to 300 together and each alone: the same bits, and those of a row alone below the limit."""
    x, w, b = made(500, 4096, 3072, 1)
    counts = [1, 300, 16, 17, 1, 1, 164]
    got, at = ops.linear(x, w, b, None, counts), 0
    for c in counts:
        own = x[at:at + c].contiguous()
        assert torch.equal(ops.linear(own, w, b, None, [c]), got[at:at + c])
        if c < ops.f32_split_tokens(w):
            assert torch.equal(ops.linear(own, w, b), got[at:at + c])
        at += c


@pytest.mark.parametrize("m", [40, 300])
def test_values_that_do_not_split(ops, m):
    """Infinities, NaN, values near the largest and rows of tiny values: what multiply-adds give."""
    x, w, b = made(m, 1200, 1024, 2)
    b.zero_()
    x[3, 5], x[7, 9], x[11], x[12], w[40, 3], w[41], w[300, 700] = float("inf"), float("nan"), x[11] * 1e-30, 0.0, 3e38, w[41] * 1e-25, float("-inf")
    got, want = ops.linear(x, w, b, None, [m]), ops.linear(x, w, b)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine = torch.isfinite(want) & torch.isfinite((x.double().abs() @ w.double().abs().T).float())
    limit = 2e-6 * (x.double().abs() @ w.double().abs().T)
    assert bool(((got.double() - want.double()).abs() <= limit)[fine].all())
    x.fill_(float("nan"))
    assert bool(torch.isnan(ops.linear(x, w, b, None, [m])).all())


def test_shifted_operands_and_scratch_at_a_time(ops, monkeypatch):
    """Operands off 16 bytes, and rows taken a few at a time: the same bits."""
    x, w, b = made(600, 1100, 1056, 3)
    want = ops.linear(x, w, b, None, [600])
    shifted = lambda t: torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)  # noqa: E731
    assert torch.equal(ops.linear(shifted(x), shifted(w), shifted(b), None, [600]), want)
    monkeypatch.setattr(ops, "F32_SPLIT_BYTES", 1)
    assert torch.equal(ops.linear(x, w, b, None, [600]), want)
