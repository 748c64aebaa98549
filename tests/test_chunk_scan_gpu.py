"""The scans that go run by run (csrc/chunk_scan.cu) beside the kernels that walk a sequence token by token, which stay for
short prompts and other sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = ["fixed", "gated", "space", "delta"]
LENGTHS = [[64], [1, 65], [127, 3, 128], [200, 64, 129]]


def batch_of(lengths):
    from fms_b200.engine.batch import Batch

    # slots in another order than the sequences
    slots = list(range(len(lengths)))[::-1]
    return Batch.from_lists(slots, [0] * len(lengths), [[0] * n for n in lengths], [[] for _ in lengths], "cuda")


def run(kind, batch, n, slots, vdim, seed, change=None, writes_state=True):
    """(outputs, what the slots hold afterwards) of two key heads' worth of heads."""
    from fms_b200.kernels import ops

    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    dim, heads = 128, 4 if kind == "space" else 2
    state = r(slots, heads, vdim, dim)
    if kind == "space":
        xbc, proj = r(n, heads * vdim + 2 * 2 * dim) * 0.3, r(n, heads).bfloat16()
        if change:
            change(xbc)
        y = ops.selective_scan(xbc, proj, 0, r(heads) - 2.0, r(heads).abs(), r(heads), state, batch, heads, vdim, dim, 2, writes_state)
        return y, [state]
    if kind == "delta":  # two heads over one key head
        qkv, proj = r(n, 2 * dim + heads * vdim), r(n, 2 * heads).bfloat16()
        if change:
            change(qkv)
        y = ops.delta_rule_scan(qkv, proj, 0, None, r(heads) - 2.0, r(heads).abs(), state, batch, heads, 1, dim, vdim, writes_state, decay_offset=heads)
        return y, [state]
    proj = r(n, heads * (2 * dim + vdim) + 2 * heads)
    if change:
        change(proj)
    if kind == "fixed":
        y = ops.decay_scan(proj, state, batch, heads, dim, vdim, ops.ACT_SILU, decay=torch.tensor([0.999, 0.3]).cuda(), writes_state=writes_state)
        return y, [state]
    norm = r(slots, heads, dim + 1)
    y = ops.decay_scan(proj, state, batch, heads, dim, vdim, q_scale=dim ** -0.5, gate_offset=heads * (2 * dim + vdim),
                       gate_bias=torch.tensor([0.0, 0.5, 4.0, 1.0]).cuda(), gate_cap=15.0, norm_state=norm, writes_state=writes_state)
    return y, [state, norm]


def both(monkeypatch, *args, **kw):
    from fms_b200.kernels import ops

    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: False)
    want = run(*args, **kw)
    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: True)
    return run(*args, **kw), want


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("vdim", [128, 64])
@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("pass_runs", [1, 2, 1000])
def test_runs_equal_the_walk_over_tokens(monkeypatch, kind, vdim, lengths, pass_runs):
    """Remainders of runs, sequences cut by a pass, states that are not zero before the step.  Both sides are sums of the
    same up to 200 terms in float32, in another order: a few units of 2^-24 of the largest partial sums."""
    from fms_b200.kernels import ops

    monkeypatch.setattr(ops, "CHUNK_STATE_BYTES", pass_runs * 4 * vdim * 128 * 4)
    batch = batch_of(lengths)
    for writes in (True, False):
        (y, left), (y0, left0) = both(monkeypatch, kind, batch, sum(lengths), len(lengths) + 1, vdim, 7, writes_state=writes)
        for a, b in zip([y] + left, [y0] + left0):
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
            assert float((a - b).norm()) <= 2e-6 * float(b.norm())


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(monkeypatch, kind, value):
    """One value of one token's v (of its k, of its q) is not finite: the tokens before it in the same run come out as they do
    without it, and the first touched row is the same as in the walk over tokens."""
    at = 70  # the seventh token of the second run
    for column in (300, 130, 5):
        def change(m):
            m[at, column] = value

        (y, _), (y0, _) = both(monkeypatch, kind, batch_of([150]), 150, 2, 128, 9, change=change)
        clean = run(kind, batch_of([150]), 150, 2, 128, 9)[0]
        assert bool(torch.isfinite(y[:at]).all()) and torch.allclose(y[:at], clean[:at], rtol=0, atol=1e-5 * float(clean.abs().max()))
        assert bool((torch.isfinite(y[at]) == torch.isfinite(y0[at])).all())
