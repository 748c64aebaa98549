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


def attended(ops, num_new, lens_before, nheads, kvheads, hd, window=0, chunk=0, sink=None, seed=0, scale=None):
    """A step's attention, its queries and the keys and values of every sequence in order."""
    from test_kernels_gpu import make_cache_case

    _, view, batch = make_cache_case(torch.float32, nheads, kvheads, hd, lens_before, num_new, seed, window)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = sum(num_new)
    qkv = torch.randn(n, (nheads + 2 * kvheads) * hd, generator=g, device="cuda")
    q = ops.rope_store(qkv, None, batch, view, nheads, kvheads, hd)
    return ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, window, sink, chunk), q, view, batch


@pytest.mark.parametrize("nheads,kvheads,hd", [(4, 2, 64), (8, 2, 128)])
@pytest.mark.parametrize("num_new,lens_before", [([17, 64, 65], [0, 0, 63]), ([128, 1, 16, 200], [5, 300, 64, 129])])
@pytest.mark.parametrize("window,chunk,sinks", [(0, 0, False), (70, 0, True), (0, 96, False)])
def test_attention_at_the_edges_of_its_tiles(ops, monkeypatch, nheads, kvheads, hd, num_new, lens_before, window, chunk, sinks):
    """Remainders of 64 queries and of 64 keys, windows that skip blocks, sequences that stay on the CUDA cores beside others; everything
    that no query sees is NaN.  Beside the CUDA cores' kernel: an output is an average of values, both sides' errors some 2^-24 of the
    largest score's size and of the values' each."""
    sink = torch.randn(nheads, device="cuda") if sinks else None
    calls, entry = [], ops._call
    monkeypatch.setattr(ops, "_call", lambda library, name, *a: (calls.append(name), entry(library, name, *a))[1])
    got, q, view, batch = attended(ops, num_new, lens_before, nheads, kvheads, hd, window, chunk, sink)
    assert "fms_attention_prefill_f32_split" in calls
    monkeypatch.setattr(ops, "F32_SPLIT_ATTENTION_TOKENS", 1 << 30)
    calls.clear()
    want = ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, window, sink, chunk)
    assert "fms_attention_prefill_f32_split" not in calls
    assert float((got - want).abs().max()) <= 2.0 ** -24 * 64 * float(want.abs().max())
    assert float((got - want).norm()) <= 2.0 ** -24 * 16 * float(want.norm())
    at = 0
    for n in num_new:  # few rows: the same kernel, the same bits
        if n < 17:
            assert torch.equal(got[at:at + n], want[at:at + n])
        at += n


def test_attention_of_a_sequence_alone_and_among_others(ops):
    """The same bits, also where a tile's other rows are other ones; and no further from 64 bits than the CUDA cores' kernel."""
    nheads, kvheads, hd = 8, 2, 128
    got, q, view, batch = attended(ops, [150, 40, 300], [10, 0, 100], nheads, kvheads, hd, seed=3)
    from fms_b200.engine.batch import Batch

    slots = batch.slots.tolist()
    for i, (first, n, before) in enumerate(((0, 150, 10), (150, 40, 0), (190, 300, 100))):
        alone = Batch.from_lists([slots[i]], [before], [[0] * n], [[]], "cuda")
        assert torch.equal(ops.attention(q[first:first + n].contiguous(), alone, view, nheads, kvheads, hd, hd ** -0.5, 0), got[first:first + n])
        rest = Batch.from_lists([slots[i]], [before + 13], [[0] * (n - 13)], [[]], "cuda")
        assert torch.equal(ops.attention(q[first + 13:first + n].contiguous(), rest, view, nheads, kvheads, hd, hd ** -0.5, 0), got[first + 13:first + n])
    table, errors = view.table.tolist(), []
    keys, values = (torch.cat([t[b] for b in table[slots[2]][:7]], 1)[:, :400].double() for t in (view.keys, view.values))
    scores = torch.einsum("thd,hkd->htk", q[190:].double().view(300, nheads, hd), keys.repeat_interleave(4, 0)) * hd ** -0.5
    scores = scores.masked_fill(torch.arange(400, device="cuda")[None] > 100 + torch.arange(300, device="cuda")[:, None], -float("inf"))
    want = torch.einsum("htk,hkd->thd", torch.softmax(scores, -1), values.repeat_interleave(4, 0)).flatten(1)
    for least in (17, 1 << 30):
        ops.F32_SPLIT_ATTENTION_TOKENS, kept = least, ops.F32_SPLIT_ATTENTION_TOKENS
        try:
            out = ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, 0)[190:]
        finally:
            ops.F32_SPLIT_ATTENTION_TOKENS = kept
        errors.append(float((out.double() - want).norm() / want.norm()))
    assert errors[0] <= errors[1], errors


@pytest.mark.parametrize("value", [float("nan"), float("inf"), 3e38])
@pytest.mark.parametrize("what", ["query", "key", "value"])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_keeps_what_does_not_split_to_the_rows_that_see_it(ops, what, value, window):
    """The rows that do not see it come out as they do without it, bit for bit; the others as on the CUDA cores."""
    nheads, kvheads, hd, n, before, at = 4, 2, 128, 200, 37, 120
    clean, q, view, batch = attended(ops, [n], [before], nheads, kvheads, hd, window, seed=5)
    q = q.clone()
    if what == "query":
        q[at, 2 * hd + 3] = value
    else:
        table = view.table[batch.slots[0]]
        (view.keys if what == "key" else view.values)[table[(before + at) // 64], 1, (before + at) % 64, 3] = value
    got, limit = ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, window), ops.F32_SPLIT_ATTENTION_TOKENS
    try:
        ops.F32_SPLIT_ATTENTION_TOKENS = 1 << 30
        want = ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, window)
    finally:
        ops.F32_SPLIT_ATTENTION_TOKENS = limit
    sees = torch.zeros(n, dtype=torch.bool, device="cuda")
    sees[at: at + 1 if what == "query" else (at + window if window else n)] = True
    assert torch.equal(got[~sees], clean[~sees])
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    fine = torch.isfinite(want)
    assert float((got - want)[fine].abs().max()) <= 2.0 ** -24 * 64 * float(want[fine].abs().max())


def beside_the_cuda_cores(ops, monkeypatch, q, view, batch, nheads, kvheads, hd, window=0, scale=None):
    """A step's attention as it is and on the CUDA cores."""
    scale = hd ** -0.5 if scale is None else scale
    got = ops.attention(q, batch, view, nheads, kvheads, hd, scale, window)
    with monkeypatch.context() as m:
        m.setattr(ops, "F32_SPLIT_ATTENTION_TOKENS", 1 << 30)
        return got, ops.attention(q, batch, view, nheads, kvheads, hd, scale, window)


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("scale", [None, 3e38])
def test_attention_of_scores_beyond_float32(ops, monkeypatch, sign, scale):
    """A query and a key of 1e21, whose score overflows either way, and a scale that makes every score do so: no number where the
    multiply-adds give none, weight zero where they give -inf; such a row equals theirs but for the order of its sums."""
    nheads, kvheads, hd, n, before, at = 4, 2, 128, 200, 37, 120
    _, q, view, batch = attended(ops, [n], [before], nheads, kvheads, hd, seed=6)
    signs = torch.where(torch.randn(hd, device="cuda") < 0, -1.0, 1.0)
    q = q.clone()
    q[at, 2 * hd:3 * hd] = 1e21 * signs
    block = view.table[batch.slots[0]][(before + at - 30) // 64]
    view.keys[block, 1, (before + at - 30) % 64] = sign * 1e21 * signs
    got, want = beside_the_cuda_cores(ops, monkeypatch, q, view, batch, nheads, kvheads, hd, scale=scale)
    row = want[at, 2 * hd:3 * hd]
    assert bool(torch.isnan(row).all() if sign > 0 or scale else (torch.isfinite(row) & (row != 0)).all())
    assert torch.equal(torch.isfinite(got), torch.isfinite(want))
    fine = torch.isfinite(want)
    assert scale or float((got - want)[fine].abs().max()) <= 2.0 ** -24 * 64 * float(want[fine].abs().max())


@pytest.mark.parametrize("what", ["key", "value"])
@pytest.mark.parametrize("window,chunk", [(16, 0), (0, 16)])
def test_attention_rows_between_positions_that_do_not_split(ops, what, window, chunk):
    """Bad positions on both sides of what a row sees leave its bits as they are."""
    nheads, kvheads, hd, n, bad = 4, 2, 64, 150, (5, 62, 127)
    clean, q, view, batch = attended(ops, [n], [0], nheads, kvheads, hd, window, chunk, seed=7)
    for at in bad:
        (view.keys if what == "key" else view.values)[view.table[batch.slots[0]][at // 64], :, at % 64, 3] = float("nan")
    got = ops.attention(q, batch, view, nheads, kvheads, hd, hd ** -0.5, window, None, chunk)
    sees = torch.tensor([any(a <= p and (p - a < window if window else p // chunk == a // chunk) for a in bad) for p in range(n)], device="cuda")
    assert torch.equal(got[~sees], clean[~sees])
    assert bool(torch.isnan(got[sees]).any(1).all())


@pytest.mark.parametrize("small,gap", [(2.0 ** -126, 0.0), (1.0, 86.0)])
def test_attention_of_small_values(ops, monkeypatch, small, gap):
    """Values, and probabilities of e^-86 beside one whose value is zero, whose last bits lie below 2^-133: nothing of them is lost."""
    nheads, kvheads, hd, n = 4, 2, 128, 130
    _, q, view, batch = attended(ops, [n], [0], nheads, kvheads, hd, seed=8)
    q = torch.zeros_like(q)
    q.view(n, nheads, hd)[:, :, 0] = gap * hd ** 0.5
    blocks = view.table[batch.slots[0]][:3].long()
    view.keys[blocks] = 0.0
    view.keys[blocks[0], :, 0, 0] = 1.0
    view.values[blocks] *= small
    view.values[blocks[0], :, 0] = 0.0
    got, want = beside_the_cuda_cores(ops, monkeypatch, q, view, batch, nheads, kvheads, hd)
    # both sides' sums of up to 130 terms and their exponentials: some 2^-24 of the terms' magnitudes each; a result's spacing
    values = view.values[blocks].double().abs().transpose(0, 1).reshape(kvheads, -1, hd)[:, :n].repeat_interleave(nheads // kvheads, 0)
    size = torch.cumsum(values, 1).transpose(0, 1) * float(torch.exp(torch.tensor(-gap).double()))
    if not gap:
        size /= torch.arange(1, n + 1, device="cuda")[:, None, None]
    a, b = (t.view(n, nheads, hd).double() for t in (got, want))
    assert float(b.abs().max()) > 2.0 ** -126
    assert bool(((a - b).abs() <= 2.0 ** -24 * 64 * size + 2.0 ** -148).all())


def split_product(ops, x, w, b=None):
    """The product by ``gemm_f32_tc`` whatever the number of rows and the size of the matrix."""
    m, (n, k) = x.shape[0], w.shape
    y, scratch = torch.empty(m, n, device="cuda"), torch.empty(m * ((k + 63) // 64 * 64 * 6 + 1) + n, dtype=torch.uint8, device="cuda")
    ops._call("gemm_f32_tc", "fms_gemm_f32_tc", x, w, b, y, scratch, scratch.numel(), m, n, k, ops.error_flag(x.device), ops._stream())
    return y


@pytest.mark.parametrize("m,n,k", [(40, 1200, 1024), (300, 1200, 1024), (700, 6144, 1024)])
def test_operands_of_any_size(ops, m, n, k):
    """Products that overflow, operands near 2^63, rows of values below 2^-110, of subnormal ones, and results down to float32's
    smallest: what multiply-adds give, with 2^-150 for every rounding of theirs.  Clusters, single blocks, and many tiles."""
    x, w, _ = made(m, n, k, 9)
    x[3], x[4], x[5], w[7], w[8] = x[3] * 1e21, x[4] * 2.0 ** 63, x[5] * 2.0 ** 28, w[7] * 1e21, w[8].sign() * 1.998 * 2.0 ** 63
    x[6, 1:], x[9], x[10, ::2], w[11], w[12, ::2] = x[6, 1:] * 2.0 ** -120, x[9] * 2.0 ** -135, 0.0, w[11] * 2.0 ** -128, 0.0
    x[10, 1::2] *= 2.0 ** -126
    x[13], w[13], x[14] = x[13] * 2.0 ** -70, w[13] * 2.0 ** -70, x[14] * 2.0 ** -147
    w[14, 0] = 0.0  # beside x[6]: what only the small values make
    got, want = split_product(ops, x, w), ops.linear(x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine, size = torch.isfinite(want), x.double().abs() @ w.double().abs().T
    assert bool(((got.double() - want.double()).abs() <= 2e-6 * size + k * 2.0 ** -150)[fine].all())
    few = split_product(ops, x[:33].contiguous(), w)  # another form: the same bits, those of subnormal results among them
    assert torch.equal(few.nan_to_num(7.0), got[:33].nan_to_num(7.0))


@pytest.mark.parametrize("m,n,k", [(64, 1024, 1024), (600, 1536, 4096)])
def test_what_multiply_adds_make_exactly(ops, m, n, k):
    """Rows that pick an element, whole numbers, equal terms: no sum that float32 holds is cut off."""
    _, w, _ = made(m, n, k, 10)
    at = torch.randint(0, k, (m,), device="cuda")
    x = torch.nn.functional.one_hot(at, k).float()
    assert torch.equal(split_product(ops, x, w), w[:, at].T)
    x, w = torch.randint(-7, 8, (m, k), device="cuda").float(), torch.randint(-2047, 2048, (n, k), device="cuda").float()
    assert torch.equal(split_product(ops, x, w).double(), x.double() @ w.double().T)
    assert torch.equal(split_product(ops, torch.ones_like(x), torch.full_like(w, 1 + 2.0 ** -23)), torch.full((m, n), k * (1 + 2.0 ** -23), device="cuda"))


@pytest.mark.parametrize("m,n,k", [(300, 28672, 4096), (2048, 4096, 14336)])
def test_many_rows_that_do_not_split(ops, m, n, k):
    """Several tiles a block, whose rows are none split: they are made behind all tiles, and no warp gives up waiting meanwhile."""
    x, w, b = made(m, n, k, 11)
    want = ops.linear(x, w, b, None, [m])
    x[:, 0], rows = float("nan"), [5, m - 1]
    x[rows, 0] = 1.0
    x[rows[1], 1], w[:, 1] = 2e30, 0.0
    got = ops.linear(x, w, b, None, [m])
    ops.check_error_flag("cuda:0")
    others = torch.ones(m, dtype=torch.bool, device="cuda")
    others[rows] = False
    assert bool(torch.isnan(got[others]).all()) and bool(torch.isfinite(got[rows]).all())
    x[rows[1], 1] = 0.0
    assert torch.equal(got[rows[0]], ops.linear(x[rows[0]].repeat(64, 1), w, b, None, [64])[0])
    assert bool(((got[rows].double() - (x[rows].double() @ w.double().T + b.double())).abs() <= bound(x[rows], w, b) + 2e-6 * (x[rows].double().abs() @ w.double().abs().T)).all())
    assert not torch.isnan(want).any()
    x[:] = 2e30
    w.fill_(1.0)
    b.zero_()
    got = ops.linear(x[:, :1024].contiguous(), w[:, :1024].contiguous(), b, None, [m])
    ops.check_error_flag("cuda:0")
    assert bool(((got.double() / (1024 * 2e30) - 1).abs() <= 2.0 ** -20).all())


@pytest.mark.parametrize("kind", ["glu", "mlp"])
def test_rows_of_a_feed_forward_stand_alone(ops, kind):
    """Called as ``forward(x)`` a feed-forward does not know whose rows they are: 40 rows are what each is alone.  Told so, they
    are a prompt's."""
    from fms_b200.config.specs import FeedForwardSpec
    from fms_b200.parts.registry import build_feed_forward

    part = build_feed_forward(FeedForwardSpec(kind, dim=2048, hidden=4096))
    g = torch.Generator(device="cuda").manual_seed(12)
    for _, owner, local, d in list(part.named_decls()):
        owner.set_tensor(local, torch.randn(d.shape, generator=g, device="cuda") * 0.02)
    part.finalize("cuda", torch.float32)
    x = torch.randn(40, 2048, generator=g, device="cuda")
    got = part.forward(x)
    assert torch.equal(torch.cat([part.forward(x[i:i + 1]) for i in range(40)]), got)
    assert torch.equal(part.forward(x, [40]), part.forward(torch.cat([x, x]), [40, 40])[:40])
    assert not torch.equal(part.forward(x, [40]), got)


# rows alone and together: up to 64, or more (the norms' forms); decode steps of 4, 5 and 20 sequences
@pytest.mark.parametrize("lengths", [[33, 17, 2, 12], [70, 100, 65, 129, 80], [2, 3, 4] * 6 + [3, 4]])
def test_requests_of_a_float32_model_together_and_alone(ops, lengths):
    """A model whose products go to the tensor cores: a prompt's logits among other prompts, and a decode step's, are the
    bits that each sequence gets alone."""
    from fms_b200.models.llama import LLaMA, LLaMAConfig
    from fms_b200.weights import RandomSource

    model = LLaMA(LLaMAConfig(src_vocab_size=512, emb_dim=2048, nheads=16, kvheads=8, nlayers=2, hidden_dim=2048, multiple_of=1,
                              max_expected_seq_len=512))
    model.load(RandomSource(model.checkpoint_layout(), 13, dtype=torch.float32, device="cuda", std=0.05), "hf", "cuda", torch.float32)
    prompts = [[(7 * i + 3 * j) % 512 for j in range(n)] for i, n in enumerate(lengths)]
    calls, entry = [], ops._call
    ops._call = lambda library, name, *a: (calls.append(name), entry(library, name, *a))[1]
    try:
        engine = model.new_engine(max_tokens=64 * 20, max_slots=20)
        slots = engine.begin(len(lengths))
        together = [engine.step(slots, prompts), engine.step(slots, [[i] for i in range(len(lengths))])]
        engine.release(slots)
    finally:
        ops._call = entry
    on_tensor_cores = {"fms_gemm_f32_tc", "fms_attention_prefill_f32_split"}
    assert on_tensor_cores & set(calls) == (on_tensor_cores if max(lengths) > 32 else set())
    for i, prompt in enumerate(prompts):
        slot = engine.begin(1)
        alone = [engine.step(slot, [prompt]), engine.step(slot, [[i]])]
        engine.release(slot)
        assert all(torch.equal(t[i], a[0]) for t, a in zip(together, alone)), i
    engine.check()


@pytest.mark.parametrize("k", [2048, 2051])
def test_sequences_on_either_side_of_the_limit_in_turn(ops, monkeypatch, k):
    """One product a side, whatever the order; each sequence's rows are what it gets alone; the same under capture."""
    from fms_b200.engine.batch import Batch

    counts = [33, 1, 40, 32, 32, 64, 2]
    x, w, b = made(sum(counts), 2050, k, 14)
    batch = Batch.from_lists(list(range(7)), [0] * 7, [[0] * c for c in counts], [[]] * 7, "cuda")
    calls, entry = [], ops._call
    monkeypatch.setattr(ops, "_call", lambda library, name, *a: (calls.append(name), entry(library, name, *a))[1])
    got = ops.linear(x, w, b, None, counts)
    assert calls.count("fms_gemm_f32_tc") == 1 and calls.count("fms_gemm_f32") == 1
    graph, held = torch.cuda.CUDAGraph(), torch.empty_like(got)
    with torch.cuda.graph(graph):
        held.copy_(ops.linear(x, w, b, None, batch))
    graph.replay()
    assert torch.equal(held, got) and torch.equal(ops.linear(x, w, b, None, batch), got)
    at = 0
    for c in counts:
        assert torch.equal(ops.linear(x[at:at + c].contiguous(), w, b, None, [c]), got[at:at + c])
        at += c


@pytest.fixture
def every_size(ops, monkeypatch):
    """Matrices of fewer values go to the tensor cores from 33 tokens on as well."""
    monkeypatch.setattr(ops, "F32_SPLIT_LINES", ((12 << 20, 17), (0, 33)))


@pytest.mark.parametrize("n,k", [(1024, 1024), (1153, 1050), (1030, 2052)])
@pytest.mark.parametrize("m", [33, 64, 65, 129, 256, 257, 600])
def test_edges_with_small_matrices(ops, every_size, m, n, k):
    test_edges_of_tiles_runs_and_steps(ops, m, n, k)


@pytest.mark.parametrize("m", [40, 300])
def test_values_that_do_not_split_with_small_matrices(ops, every_size, m):
    test_values_that_do_not_split(ops, m)


def test_shifted_operands_and_scratch_with_small_matrices(ops, every_size, monkeypatch):
    test_shifted_operands_and_scratch_at_a_time(ops, monkeypatch)


def test_lines_by_the_values_of_a_matrix(ops):
    """The tokens from which a matrix' products change, at the edges of its sizes."""
    shapes = {(1023, 1 << 20): 0, (1024, 1024): 1025, (1024, 2048): 257, (1024, 4096): 33, (3072, 4096): 17, (3071, 4096): 33, (1024, 1 << 18): 17,
              (1024, (1 << 18) + 1): 0}
    assert {s: ops.f32_split_tokens(torch.empty(s, device="meta")) for s in shapes} == shapes
