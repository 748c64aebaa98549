"""The scans that go run by run (csrc/chunk_scan.cu) beside the kernels that walk a sequence token by token, which stay for
short prompts and other sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = ["fixed", "gated", "space", "delta"]
TAKEN = [(kind, 128) for kind in KINDS] + [("space", 64)]  # what the runs' kernels take; the others walk with 64 values
LENGTHS = [[64], [1, 65], [127, 3, 128], [200, 64, 129], [330, 5]]  # the last: one sequence over three passes and more


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
    dim, heads = 128, heads_of(kind)
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


def heads_of(kind):
    return 4 if kind == "space" else 2


def both(monkeypatch, *args, **kw):
    """(by runs, walked); that each went the way it was sent is looked at."""
    from fms_b200.kernels import ops

    calls, entry = [], ops._call
    monkeypatch.setattr(ops, "_call", lambda library, name, *a: (calls.append((name, a)), entry(library, name, *a))[1])
    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: False)
    want = run(*args, **kw)
    assert "fms_chunk_scan" not in [name for name, _ in calls]
    calls.clear()
    monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: True)
    got = run(*args, **kw)
    names = [name for name, _ in calls]
    assert names.count("fms_chunk_scan") == 1 and not {"fms_decay_scan", "fms_selective_scan", "fms_delta_rule_scan"} & set(names)
    monkeypatch.setattr(ops, "_call", entry)
    return got, want, next(a for name, a in calls if name == "fms_chunk_scan")


@pytest.mark.parametrize("kind,vdim", TAKEN)
@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("pass_runs", [1, 2, 1000])
def test_runs_equal_the_walk_over_tokens(monkeypatch, kind, vdim, lengths, pass_runs):
    """Remainders of runs, sequences cut by one pass and by several, states that are not zero before the step.  Both sides are sums of the
    same up to 200 terms in float32, in another order: a few units of 2^-24 of the largest partial sums."""
    from fms_b200.kernels import ops

    monkeypatch.setattr(ops, "CHUNK_STATE_BYTES", pass_runs * heads_of(kind) * vdim * 128 * 4)
    batch, runs = batch_of(lengths), sum((n + 63) // 64 for n in lengths)
    for writes in (True, False):
        (y, left), (y0, left0), sent = both(monkeypatch, kind, batch, sum(lengths), len(lengths) + 1, vdim, 7, writes_state=writes)
        assert sent[7:9] == (runs, min(pass_runs, runs))  # runs of the step and of a pass
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

        (y, _), (y0, _), _ = both(monkeypatch, kind, batch_of([150]), 150, 2, 128, 9, change=change)
        clean = run(kind, batch_of([150]), 150, 2, 128, 9)[0]
        assert bool(torch.isfinite(y[:at]).all()) and torch.allclose(y[:at], clean[:at], rtol=0, atol=1e-5 * float(clean.abs().max()))
        assert bool((torch.isfinite(y[at]) == torch.isfinite(y0[at])).all())


def in_64_bits(kind, n, heads, vdim, seed):
    """Inputs as a trained layer has them, what ``ops`` makes of one sequence of them, and the recurrence in 64 bits."""
    from fms_b200.kernels import ops

    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    silu, softplus, dim = torch.nn.functional.silu, torch.nn.functional.softplus, 128
    u = torch.rand(heads, generator=g, device="cuda")
    bias, rates = torch.log(torch.expm1(torch.exp(-6.9 + 4.6 * u))), torch.log(1 + 15 * torch.rand(heads, generator=g, device="cuda"))
    state, batch = torch.zeros(1, heads, vdim, dim, device="cuda"), batch_of([n])
    ones, norm = torch.ones(n, heads, dtype=torch.float64, device="cuda"), None
    if kind == "space":
        x, logits, skip = silu(r(n, heads * vdim + 2 * dim)), 0.5 * r(n, heads), torch.ones(heads, device="cuda")
        dt = softplus(logits.double() + bias.double())
        keep, give = torch.exp(-torch.exp(rates.double()) * dt), dt
        v, k, q = x[:, : heads * vdim].double().view(n, heads, vdim), *(t.double()[:, None].expand(n, heads, dim) for t in (x[:, -2 * dim: -dim], x[:, -dim:]))
        make = lambda: ops.selective_scan(x, logits, 0, bias, rates, skip, state, batch, heads, vdim, dim, 1)  # noqa: E731
    elif kind == "delta":
        x, logits = silu(r(n, heads * (2 * dim + vdim))), r(n, 2 * heads)
        q, k, v = (t.double().view(n, heads, -1) for t in torch.split(x, [heads * dim, heads * dim, heads * vdim], 1))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q * 1.0, k))
        q, give = q * dim ** -0.5, torch.sigmoid(logits[:, :heads].double())
        keep = torch.exp(-torch.exp(rates.double()) * softplus(logits[:, heads:].double() + bias.double()))
        make = lambda: ops.delta_rule_scan(x.clone(), logits, 0, None, bias, rates, state, batch, heads, heads, dim, vdim, decay_offset=heads)  # noqa: E731
    else:
        x = r(n, heads * (2 * dim + vdim) + 2 * heads)
        q, k, v = (t.double().view(n, heads, -1) for t in torch.split(x[:, : heads * (2 * dim + vdim)], [heads * dim, heads * dim, heads * vdim], 1))
        if kind == "fixed":
            q, k, v = silu(q), silu(k), silu(v)
            decay = torch.exp(-(2.0 ** (-8.0 * torch.arange(1, heads + 1, device="cuda") / heads)))
            keep, give = decay.double() * ones, ones
            make = lambda: ops.decay_scan(x, state, batch, heads, dim, vdim, ops.ACT_SILU, decay=decay)  # noqa: E731
        else:
            gate_bias = torch.cat([torch.zeros(heads), torch.linspace(3, 6, heads)]).cuda()
            gi, gf = torch.split(15.0 * torch.tanh((x[:, heads * (2 * dim + vdim):].double() + gate_bias.double()) / 15.0), heads, 1)
            gf, top, keep, give, tops = torch.nn.functional.logsigmoid(gf), torch.zeros_like(gi[0]), ones.clone(), ones.clone(), ones.clone()
            for t in range(n):
                to = torch.maximum(gf[t] + top, gi[t])
                keep[t], give[t], tops[t] = torch.exp(gf[t] + top - to), torch.exp(gi[t] - to), to
                top = to
            q, norm, held = q * dim ** -0.5, torch.zeros(heads, dim, dtype=torch.float64, device="cuda"), torch.zeros(1, heads, dim + 1, device="cuda")
            make = lambda: ops.decay_scan(x, state, batch, heads, dim, vdim, q_scale=dim ** -0.5, gate_offset=heads * (2 * dim + vdim),  # noqa: E731
                                          gate_bias=gate_bias, gate_cap=15.0, norm_state=held.zero_())
    S, out = torch.zeros(heads, vdim, dim, dtype=torch.float64, device="cuda"), []
    for t in range(n):
        S = S * keep[t][:, None, None]
        vt = v[t] - torch.einsum("hvk,hk->hv", S, k[t]) if kind == "delta" else v[t]
        S = S + (give[t][:, None] * vt)[..., None] * k[t][:, None]
        o = torch.einsum("hvk,hk->hv", S, q[t])
        if kind == "gated":
            norm = norm * keep[t][:, None] + give[t][:, None] * k[t]
            o = o / (torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-tops[t])) + 1e-6)[:, None]
        out.append((o + v[t] if kind == "space" else o).flatten())
    return make, state, torch.stack(out), S


@pytest.mark.parametrize("kind", KINDS)
def test_runs_are_no_further_from_64_bits_than_the_walk(monkeypatch, kind):
    """Outputs and states of a sequence long enough to go run by run, the walk's and the runs' errors over two draws.  Under a
    normalizer a head's row may be divided by next to nothing, and one such row is most of the whole's error: there the
    median over the rows."""
    from fms_b200.kernels import ops

    def apart(a, b):
        if kind != "gated":
            return float((a - b).norm() / b.norm())
        a, b = a.view(-1, 128), b.view(-1, 128)
        return float(((a - b).norm(dim=1) / b.norm(dim=1)).median())

    errors = []
    for seed in (1, 2):
        make, state, want, S = in_64_bits(kind, 400, 8, 64 if kind == "space" else 128, seed)
        for pays in (False, True):
            monkeypatch.setattr(ops, "chunk_scan_pays", lambda *_: pays)
            state.zero_()
            y = make()
            errors.append([apart(y.double(), want), float((state[0].double() - S).norm() / S.norm())])
    for walk, runs in zip(*[[sum(e[j] for e in errors[i::2]) for j in range(2)] for i in range(2)]):
        assert walk < 1e-5 and runs <= walk, (walk, runs)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("vdim", [128, 64])
def test_a_sequence_comes_out_alike_alone_and_among_others(kind, vdim):
    """Sequences below and above the number of tokens from which they go run by run, together and each alone: the same bits."""
    from fms_b200.kernels import ops

    g = torch.Generator().manual_seed(4)
    least = ops.CHUNK_SCAN_FROM[kind]
    lengths, dim, heads = [100, least + 44, 1, least - 1, least, 257], 128, 4
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    n = sum(lengths)
    key_heads = 2 if kind == "space" else heads
    rows = r(n, heads * vdim + 2 * key_heads * dim + (2 * heads if kind in ("fixed", "gated") else 0)) * 0.3
    logits, bias, rates, skip = r(n, 2 * heads), r(heads) - 2.0, r(heads).abs(), r(heads)
    start = r(len(lengths), heads, vdim, dim)
    norms, gate_bias = r(len(lengths), heads, dim + 1), torch.cat([r(heads), r(heads) + 4.0])
    decay = torch.tensor([0.999, 0.9, 0.5, 0.97]).cuda()

    def scan(which):
        x = torch.cat([rows[sum(lengths[:i]): sum(lengths[: i + 1])] for i in which])
        z = torch.cat([logits[sum(lengths[:i]): sum(lengths[: i + 1])] for i in which])
        batch = batch_of([lengths[i] for i in which])
        state, norm = start[which[::-1]].clone(), norms[which[::-1]].clone()  # the slots are in the other order
        if kind == "space":
            y = ops.selective_scan(x, z, 0, bias, rates, skip, state, batch, heads, vdim, dim, key_heads)
        elif kind == "delta":
            y = ops.delta_rule_scan(x, z, 0, None, bias, rates, state, batch, heads, heads, dim, vdim, decay_offset=heads)
        elif kind == "fixed":
            y = ops.decay_scan(x, state, batch, heads, dim, vdim, ops.ACT_SILU, decay=decay)
        else:
            y = ops.decay_scan(x, state, batch, heads, dim, vdim, q_scale=dim ** -0.5, gate_offset=heads * (2 * dim + vdim),
                               gate_bias=gate_bias, gate_cap=15.0, norm_state=norm)
        return [(t, state[len(which) - 1 - j], norm[len(which) - 1 - j]) for j, t in enumerate(torch.split(y, [lengths[i] for i in which]))]

    together = scan(list(range(len(lengths))))
    for i in range(len(lengths)):
        for a, b in zip(scan([i])[0], together[i]):
            assert torch.equal(a, b)
    for a, b in zip(scan([0, 2, 3]), (together[0], together[2], together[3])):  # none goes run by run
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("group", [128, 132, 260, 512, 1000, 1024, 1028])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_row_is_normed_alike_alone_and_among_many(group, dtype):
    """Few long groups take a block each, many a warp each: the same bits."""
    from fms_b200.kernels import ops

    g = torch.Generator().manual_seed(group)
    x, gate, w = (torch.randn(*s, generator=g).cuda() for s in ((700, 2 * group), (700, 2 * group), (2 * group,)))
    gate = gate.to(dtype)
    for mode in (ops.GATE_SILU_BEFORE, ops.GATE_SIGMOID_AFTER):
        norm = lambda n: ops.gated_group_rmsnorm(x[:n].contiguous(), gate[:n].contiguous(), 0, mode, w, 1e-5, group, dtype)  # noqa: E731
        many = norm(700)
        assert torch.equal(norm(3), many[:3])
        y = x[:3].double() * torch.nn.functional.silu(gate[:3].double()) if mode == ops.GATE_SILU_BEFORE else x[:3].double()
        y = y.view(3, 2, group)
        y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)).flatten(1) * w.double()
        if mode == ops.GATE_SIGMOID_AFTER:
            y = y * torch.sigmoid(gate[:3].double())
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 16 * 2.0 ** -24
        assert float((many[:3].double() - y).abs().max()) <= eps * float(y.abs().max())
