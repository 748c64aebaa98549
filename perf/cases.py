"""The work by which this library's speed is judged: single layers of its architectures and one whole request, each
through the entry point that a program calls (a part's ``forward`` over a ``Batch`` and a ``Cache``, ``Engine.step``).

Sizes are those of ``bench.py``: the Llama-3-8B layer, and the layers of Goletar, Niletar, Figonex and Giganex at the same
width.  Prompts are unequal, as requests are: most lengths are no multiple of any tile.  Weights are N(0, 0.02) and vectors
as a trained layer has them (gains around 1, decay rates spread over decades).  What a step's layers share (the ``Batch``
with its index arrays) is made in ``prepare``, once a step in a running engine; what it caches for one step is
emptied before every pass, as the decoder does when a step starts.
"""
import math
import zlib

import torch

EPS = 1e-5
WIDTH = 4096


# ---- cases -------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a request's whole way through Llama: four prompts in one step, then five decode steps (captured graphs), two layers
        {"name": "llama_request", "kind": "request", "dtype": "bf16", "seqs": 4, "new": 601, "steps": 5},
        # the attention layer of a decode step of eight requests, as bench.py's headline has it (1,190 cached tokens on average)
        {"name": "attention_decode_8", "kind": "attention", "dtype": "bf16", "seqs": 8, "cached": 9520, "new": 8},
        # the attention layer of one prompt of the benchmark's length
        {"name": "attention_prompt_2048", "kind": "attention", "dtype": "bf16", "seqs": 1, "cached": 0, "new": 2048},
        # the feed-forward of a decode step of one request: the smallest call a server makes, all weights for one row
        {"name": "mlp_decode_1", "kind": "mlp", "dtype": "bf16", "new": 1},
        # the true 32-bit path (data_type="fp32"), a feed-forward in a decode step of eight
        {"name": "mlp_fp32_decode_8", "kind": "mlp", "dtype": "fp32", "new": 8},
        # the true 32-bit path, an attention layer over three unequal prompts
        {"name": "attention_fp32_prompts", "kind": "attention", "dtype": "fp32", "seqs": 3, "cached": 0, "new": 1100},
        # Goletar's latent attention over two unequal prompts
        {"name": "latent_prompts", "kind": "latent", "dtype": "bf16", "seqs": 2, "cached": 0, "new": 2048, "query_latent": False},
        # Giganex's latent attention (queries through a latent of their own, a window) in a decode step of eight
        {"name": "latent_decode_8", "kind": "latent", "dtype": "bf16", "seqs": 8, "cached": 8192, "new": 8, "query_latent": True},
        # Niletar's state-space layer over one prompt
        {"name": "state_space_prompt_2048", "kind": "state_space", "dtype": "bf16", "seqs": 1, "new": 2048, "steps": 0},
        # Giganex's delta rule (one decay a head) over short prompts and four decode steps: many small launches
        {"name": "delta_rule_requests", "kind": "delta_rule", "dtype": "bf16", "seqs": 4, "new": 333, "steps": 4},
        # Figonex's matrix memory under exponential gates over two unequal prompts
        {"name": "matrix_memory_prompts", "kind": "matrix_memory", "dtype": "bf16", "seqs": 2, "new": 1700, "steps": 0},
        # Goletar's routed experts in a decode step of eight: most experts are hit, by a row or two each
        {"name": "experts_decode_8", "kind": "experts", "dtype": "bf16", "new": 8},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng):
    kind = rng.choice(["request", "attention", "attention", "mlp", "mlp", "latent", "latent", "state_space", "delta_rule",
                       "matrix_memory", "decayed_memory", "experts"])
    dtype = "fp32" if kind in ("attention", "mlp") and rng.random() < 0.5 else "bf16"
    if kind == "request":
        seqs = rng.randint(1, 8)
        return {"kind": kind, "dtype": dtype, "seqs": seqs, "new": _spread(rng, 8 * seqs, 900), "steps": rng.randint(2, 6)}
    if kind == "mlp":
        return {"kind": kind, "dtype": dtype, "new": _spread(rng, 1, 2048 if dtype == "bf16" else 256)}
    if kind == "experts":
        return {"kind": kind, "dtype": dtype, "new": _spread(rng, 1, 512)}
    seqs = rng.randint(1, 8)
    if kind in ("attention", "latent"):
        case = {"kind": kind, "dtype": dtype, "seqs": seqs}
        if rng.random() < 0.5:  # a decode step
            case.update(cached=_spread(rng, 64 * seqs, 1190 * seqs), new=seqs)
        else:  # prompts, half of them onto what is cached already
            case.update(cached=rng.choice([0, _spread(rng, 16 * seqs, 1024)]),
                        new=_spread(rng, 16 * seqs, 2048 if dtype == "bf16" else 1000))
        if kind == "latent":
            case["query_latent"] = rng.random() < 0.5
        return case
    return {"kind": kind, "dtype": dtype, "seqs": seqs, "new": _spread(rng, 12 * seqs, 2048), "steps": rng.choice([0, 0, 3])}


# ---- what a case is made of --------------------------------------------------------------------------------------------
# kind -> sizes of its layer (bench.py's)
HEADS, KV_HEADS, HEAD, FF = 32, 8, 128, 14336
LATENT = dict(heads=32, dim=96, rot=32, vdim=128, rank=512, q_rank=1536, window=4096)
SPACE = dict(heads=128, vdim=64, state=128, groups=8, taps=4)
DELTA = dict(heads=16, dim=128, vdim=128, taps=4)
MEMORY = dict(heads=32, dim=128, vdim=128, cap=15.0)
EXPERTS = dict(experts=16, top=4, hidden=3584, limit=7.0, alpha=1.702)
VOCAB, LAYERS, THETA = 128256, 2, 500000.0
DECAYS = tuple(math.exp(-(2.0 ** (-8.0 * (i + 1) / MEMORY["heads"]))) for i in range(MEMORY["heads"]))


def _type(case):
    return torch.float32 if case["dtype"] == "fp32" else torch.bfloat16


def _shares(total, n):
    """``total`` tokens over n unequal sequences, at least one each."""
    weights = [1.0 + (5 * i + 2) % 7 / 3.0 for i in range(n)]
    out, rest = [], total - n
    for w in weights[:-1]:
        out.append(1 + int((total - n) * w / sum(weights)))
        rest -= out[-1] - 1
    return out + [1 + rest]


def _made(seed, name, shape, how, dtype, device):
    """A tensor of its own generator, by the seed and its name."""
    g = torch.Generator(device=device)
    g.manual_seed((zlib.crc32(name.encode()) + 1000003 * int(seed)) & 0x7FFFFFFF)
    if how == "tokens":
        return torch.randint(0, VOCAB, shape, generator=g, device=device)
    if how in ("rows", "matrix", "taps", "bias"):
        scale = {"rows": 1.0, "matrix": 0.02, "taps": 0.5, "bias": 0.1}[how]
        if len(shape) == 3:  # a stack of matrices: one at a time, for the sake of memory
            out = torch.empty(shape, dtype=dtype, device=device)
            for i in range(shape[0]):
                out[i] = torch.empty(shape[1:], dtype=torch.float32, device=device).normal_(0.0, scale, generator=g)
            return out
        return torch.empty(shape, dtype=torch.float32, device=device).normal_(0.0, scale, generator=g).to(dtype)
    u = torch.empty(shape, dtype=torch.float32, device=device).uniform_(0.0, 1.0, generator=g)
    if how == "gain":
        u = 0.9 + 0.2 * u
    elif how == "rates":  # logarithms of decay rates from 1 to 16
        u = torch.log(1.0 + 15.0 * u)
    elif how == "steps":  # what softplus takes to step sizes from 0.001 to 0.1
        u = torch.exp(math.log(1e-3) + u * math.log(100.0))
        u = u + torch.log(-torch.expm1(-u))
    elif how == "gates":  # input gates around 0, forget gates open
        half = shape[0] // 2
        u[:half] = 0.2 * u[:half] - 0.1
        u[half:] = 3.0 + 3.0 * u[half:]
    else:
        raise ValueError(how)
    return u.to(dtype)


def _round8(n):
    return (n + 7) // 8 * 8


def _tensors(case):
    """name in the part -> (shape, how it is made)"""
    kind, d = case["kind"], WIDTH
    if kind == "attention":
        return {"in_proj.qkv_fused.weight": (((HEADS + 2 * KV_HEADS) * HEAD, d), "matrix"),
                "dense.weight": ((d, HEADS * HEAD), "matrix")}
    if kind == "mlp":
        return {"wg1_fused.weight": ((2 * FF, d), "matrix"), "w2.weight": ((d, FF), "matrix")}
    if kind == "latent":
        s = LATENT
        q = s["heads"] * (s["dim"] + s["rot"])
        out = {"latent_norm": ((s["rank"],), "gain"), "uk": ((s["heads"] * s["dim"], s["rank"]), "matrix"),
               "uv": ((s["heads"] * s["vdim"], s["rank"]), "matrix"), "dense.weight": ((d, s["heads"] * s["vdim"]), "matrix")}
        if case["query_latent"]:
            out.update({"in_proj.weight": ((s["rank"] + s["rot"] + s["q_rank"], d), "matrix"), "q_norm": ((s["q_rank"],), "gain"),
                        "q_up.weight": ((q, s["q_rank"]), "matrix")})
        else:
            out.update({"in_proj.weight": ((q + s["rank"] + s["rot"] + s["heads"], d), "matrix"), "sink": ((s["heads"],), "bias")})
        return out
    if kind == "state_space":
        s = SPACE
        inner = s["heads"] * s["vdim"]
        ch = inner + 2 * s["groups"] * s["state"]
        return {"in_proj.weight": ((inner + ch + s["heads"], d), "matrix"), "conv": ((ch, s["taps"]), "taps"),
                "conv_bias": ((ch,), "bias"), "dt_bias": ((s["heads"],), "steps"), "A_log": ((s["heads"],), "rates"),
                "D": ((s["heads"],), "gain"), "norm": ((inner,), "gain"), "dense.weight": ((d, inner), "matrix")}
    if kind == "delta_rule":
        s = DELTA
        ch = s["heads"] * (2 * s["dim"] + s["vdim"])
        gate = _round8(ch + 2 * s["heads"])
        return {"in_proj.weight": ((gate + s["heads"] * s["vdim"], d), "matrix"), "conv": ((ch, s["taps"]), "taps"),
                "dt_bias": ((s["heads"],), "steps"), "A_log": ((s["heads"],), "rates"), "norm": ((s["vdim"],), "gain"),
                "dense.weight": ((d, s["heads"] * s["vdim"]), "matrix")}
    if kind in ("matrix_memory", "decayed_memory"):
        s = MEMORY
        per_head = 2 * s["dim"] + 2 * s["vdim"] + (2 if kind == "matrix_memory" else 0)
        out = {"in_proj.weight": ((_round8(s["heads"] * per_head), d), "matrix"), "norm": ((s["heads"] * s["vdim"],), "gain"),
               "dense.weight": ((d, s["heads"] * s["vdim"]), "matrix")}
        if kind == "matrix_memory":
            out["gate_bias"] = ((2 * s["heads"],), "gates")
        return out
    if kind == "experts":
        s = EXPERTS
        return {"router.weight": ((s["experts"], d), "matrix"), "gate_up": ((s["experts"], 2 * s["hidden"], d), "matrix"),
                "down": ((s["experts"], d, s["hidden"]), "matrix")}
    raise ValueError(kind)


def _weights(case, seed, device):
    return {n: _made(seed, n, shape, how, _type(case), device) for n, (shape, how) in _tensors(case).items()}


def _rows(case, seed, device):
    """(rows of the cached tokens or None, rows of the new ones, rows of the decode steps [steps, seqs] or None)"""
    make = lambda name, shape: _made(seed, name, shape, "rows", _type(case), device)  # noqa: E731
    return (make("cached rows", (case["cached"], WIDTH)) if case.get("cached") else None, make("rows", (case["new"], WIDTH)),
            make("later rows", (case["steps"], case["seqs"], WIDTH)) if case.get("steps") else None)


def _part(case):
    from fms_b200.config.specs import FeedForwardSpec, MixerSpec, PositionSpec
    from fms_b200.parts.registry import build_feed_forward, build_mixer
    import fms_b200.engine.decoder  # noqa: F401  (registers the built-in kinds)
    import fms_b200.parts.experts  # noqa: F401
    import fms_b200.parts.latent_attention  # noqa: F401
    import fms_b200.parts.linear_attention  # noqa: F401
    import fms_b200.parts.state_space  # noqa: F401

    kind, d = case["kind"], WIDTH
    if kind == "mlp":
        return build_feed_forward(FeedForwardSpec("glu", dim=d, hidden=FF, activation="silu"))
    if kind == "experts":
        s = EXPERTS
        return build_feed_forward(FeedForwardSpec("routed_experts", dim=d, hidden=s["hidden"], activation="swish_clamped", options=(
            ("experts", s["experts"]), ("top", s["top"]), ("limit", s["limit"]), ("alpha", s["alpha"]))))
    if kind == "attention":
        return build_mixer(MixerSpec("attention", dim=d, nheads=HEADS, kvheads=KV_HEADS, head_dim=HEAD, position=PositionSpec(
            "rope", head_dim=HEAD, theta=THETA, max_positions=8192)))
    if kind == "latent":
        s = LATENT
        options = [("rot", s["rot"]), ("vdim", s["vdim"]), ("rank", s["rank"]), ("rot_dims", s["rot"]), ("eps", EPS)]
        if case["query_latent"]:
            options += [("q_rank", s["q_rank"]), ("sink", False), ("gate", False), ("pairing", "halves")]
        return build_mixer(MixerSpec("latent_attention", dim=d, nheads=s["heads"], kvheads=1, head_dim=s["dim"],
                                     scale=(s["dim"] + s["rot"]) ** -0.5, window=s["window"] if case["query_latent"] else 0,
                                     position=PositionSpec("rope", head_dim=s["rot"], theta=10000.0), options=tuple(options)))
    if kind == "state_space":
        s = SPACE
        return build_mixer(MixerSpec("selective_state_space", dim=d, nheads=s["heads"], options=(
            ("vdim", s["vdim"]), ("state", s["state"]), ("groups", s["groups"]), ("conv", s["taps"]),
            ("norm_groups", s["groups"]), ("eps", EPS))))
    if kind == "delta_rule":
        s = DELTA
        return build_mixer(MixerSpec("gated_delta_rule", dim=d, nheads=s["heads"], kvheads=s["heads"], head_dim=s["dim"], options=(
            ("vdim", s["vdim"]), ("conv", s["taps"]), ("eps", EPS), ("decay", "head"))))
    s = MEMORY
    if kind == "matrix_memory":
        return build_mixer(MixerSpec("mlstm", dim=d, nheads=s["heads"], head_dim=s["dim"], options=(
            ("vdim", s["vdim"]), ("gate_cap", s["cap"]), ("eps", EPS))))
    return build_mixer(MixerSpec("lightning_attention", dim=d, nheads=s["heads"], head_dim=s["dim"], options=(
        ("vdim", s["vdim"]), ("decay", DECAYS), ("eps", EPS))))


# ---- a program's preparations ------------------------------------------------------------------------------------------
class _Checkpoint:
    """Made tensors under a checkpoint's names, as the loader reads them."""

    def __init__(self, case, seed, device):
        from fms_b200.models.llama import LLaMA

        self.of, self.seed, self.dtype, self.device = {t.name: t for t in LLaMA(_config()).checkpoint_layout()}, seed, _type(case), device

    def keys(self):
        return list(self.of)

    def spec(self, name):
        return self.dtype, tuple(self.of[name].shape)

    def get(self, name):
        return _made(self.seed, name, tuple(self.of[name].shape), "gain" if "norm" in name else "matrix", self.dtype, self.device)


def _config():
    from fms_b200.models.llama import LLaMAConfig

    return LLaMAConfig(src_vocab_size=VOCAB, emb_dim=WIDTH, norm_eps=EPS, nheads=HEADS, kvheads=KV_HEADS, nlayers=LAYERS,
                       hidden_dim=FF, multiple_of=1, max_expected_seq_len=8192, rope_theta=THETA)


def _prompts(case, seed):
    """(the prompts, the tokens of the decode steps) as lists; a request's tokens do not depend on its logits here."""
    flat = _made(seed, "tokens", (case["new"] + case["steps"] * case["seqs"],), "tokens", None, "cpu").tolist()
    prompts, at = [], 0
    for n in _shares(case["new"], case["seqs"]):
        prompts.append(flat[at:at + n])
        at += n
    later = [flat[at + i * case["seqs"]: at + (i + 1) * case["seqs"]] for i in range(case["steps"])]
    return prompts, later


def prepare(case, seed):
    from fms_b200.cache.cache import Cache
    from fms_b200.engine.batch import Batch

    device = "cuda"
    if case["kind"] == "request":
        from fms_b200.models.llama import LLaMA

        model = LLaMA(_config()).load(_Checkpoint(case, seed, device), "hf", device, _type(case))
        prompts, later = _prompts(case, seed)
        room = sum((len(p) + case["steps"] + 63) // 64 * 64 for p in prompts)
        return {"case": case, "engine": model.new_engine(max_tokens=room, max_slots=case["seqs"]), "prompts": prompts, "later": later}
    part = _part(case)
    for name, owner, local, _ in list(part.named_decls()):
        owner.set_tensor(local, _made(seed, name, *_tensors(case)[name], _type(case), device))
    part.finalize(device, _type(case))
    cached, rows, later = _rows(case, seed, device)
    state = {"case": case, "part": part, "rows": rows, "later": later}
    if case["kind"] in ("mlp", "experts"):
        return state
    n = case["seqs"]
    new, before, steps = _shares(case["new"], n), _shares(case["cached"], n) if case.get("cached") else [0] * n, case.get("steps", 0)
    room = sum((a + b + steps + 63) // 64 * 64 for a, b in zip(before, new))
    cache = Cache([part.cache_request()], room, 16384, _type(case), device, max_slots=n)
    slots = cache.begin(n)

    def batch_of(counts):
        lengths = cache.prepare(slots, counts)
        b = Batch.from_lists(slots, lengths, [[0] * c for c in counts], [[] for _ in counts], device)
        cache.commit(slots, counts)
        return b

    if cached is not None:
        part.forward(cached, batch_of(before), cache.layer_view(0))
    batches = [batch_of(new)] + [batch_of([1] * n) for _ in range(steps)]
    state.update(cache=cache, slots=slots, batches=batches)
    return state


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "request":
        engine = state["engine"]
        slots = engine.begin(case["seqs"])
        try:
            out = [engine.step(slots, state["prompts"])]
            for tokens in state["later"]:
                out.append(engine.step(slots, [[t] for t in tokens]))
        finally:
            engine.release(slots)
        return {"logits": out}
    part = state["part"]
    if case["kind"] in ("mlp", "experts"):
        return {"y": part.forward(state["rows"])}
    cache = state["cache"]
    view = cache.layer_view(0)
    if "steps" in case:  # requests start from nothing: their states are zero
        for group in cache.groups:
            for slot in state["slots"]:
                group.reset(slot)
    rows = [state["rows"]] + (list(state["later"]) if state["later"] is not None else [])
    y = []
    for x, batch in zip(rows, state["batches"]):
        batch.scratch.clear()
        y.append(part.forward(x, batch, view))
    out = {"y": y}
    if "steps" in case:
        out["state"] = [v.state[: case["seqs"]] for v in (view if isinstance(view, tuple) else (view,))]
    else:
        out["cache"] = cache.groups[0].storage
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def work(case):
    size, kind, d, new = 4 if case["dtype"] == "fp32" else 2, case["kind"], WIDTH, case["new"]
    if kind == "request":
        matrices = LAYERS * d * ((HEADS + 2 * KV_HEADS) * HEAD + HEADS * HEAD + 3 * FF)
        rows, steps, n = new + case["steps"] * case["seqs"], case["steps"] + 1, case["seqs"]
        pairs = sum(p * p / 2.0 + p * case["steps"] for p in _shares(new, n))
        read = sum(p + case["steps"] / 2.0 for p in _shares(new, n)) * case["steps"] * LAYERS * 2 * KV_HEADS * HEAD * size
        return {"bytes": float(steps * (matrices + VOCAB * d) * size + read + steps * n * VOCAB * 4),
                "flops": float(2.0 * rows * matrices + 2.0 * steps * n * VOCAB * d + LAYERS * 4.0 * pairs * HEADS * HEAD)}
    weights = sum(math.prod(shape) for shape, _ in _tensors(case).values())
    if kind == "mlp":
        return {"bytes": float(size * (weights + 2 * new * d)), "flops": 2.0 * new * weights}
    if kind == "experts":
        s = EXPERTS
        hit = s["experts"] * (1.0 - (1.0 - s["top"] / s["experts"]) ** new)
        one = 3 * s["hidden"] * d
        return {"bytes": size * (hit * one + s["experts"] * d + 2.0 * new * d),
                "flops": 2.0 * new * (s["top"] * one + s["experts"] * d)}
    if kind in ("attention", "latent"):
        counts = list(zip(_shares(case["cached"], case["seqs"]) if case["cached"] else [0] * case["seqs"], _shares(new, case["seqs"])))
        pairs = sum(b * n + n * (n + 1) / 2.0 for b, n in counts)
        s = LATENT
        per_key = 2 * KV_HEADS * HEAD if kind == "attention" else s["rank"] + s["rot"]
        per_pair = 4.0 * HEADS * HEAD if kind == "attention" else 2.0 * s["heads"] * (s["dim"] + s["rot"] + s["vdim"])
        return {"bytes": float(size * (weights + 2 * new * d + per_key * (case["cached"] + new))),
                "flops": 2.0 * new * weights + pairs * per_pair}
    rows = new + case["steps"] * case["seqs"]
    s = {"state_space": SPACE, "delta_rule": DELTA}.get(kind, MEMORY)
    held = s["heads"] * s["vdim"] * s["state" if kind == "state_space" else "dim"]
    each = {"state_space": 6.0, "delta_rule": 8.0}.get(kind, 5.0)
    return {"bytes": float(size * ((1 + case["steps"]) * weights + 2 * rows * d) + 4 * case["seqs"] * held * (1 + 2 * case["steps"])),
            "flops": 2.0 * rows * weights + each * rows * held}


def tolerance(case):
    # four times what this library shows against the same formulas in 64 bits
    # (measured: 3e-6 in 32 bits, 0.005 through a layer in bfloat16, 0.013 through two layers and the head)
    if case["dtype"] == "fp32":
        return {"rel": 1.2e-5}
    return {"rel": 5e-2 if case["kind"] == "request" else 2e-2}


# ---- the same in 64 bits, plainly --------------------------------------------------------------------------------------
def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turn(x, positions, theta, halves):
    """x [tokens, heads, dims] turned by the angles position * theta^(-2i / dims); pairs (i, i + dims / 2) or neighbours."""
    dims = x.shape[-1]
    f = theta ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    angle = positions.double()[:, None, None] * f
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = (x[..., : dims // 2], x[..., dims // 2:]) if halves else (x[..., 0::2], x[..., 1::2])
    a, b = a * c - b * s, a * s + b * c
    return torch.cat([a, b], -1) if halves else torch.stack([a, b], -1).flatten(-2)


def _attend(q, k, v, first, scale, window=0, sink=None):
    """q [new, heads, ..], k and v [all, kv heads, ..]; query i stands at position first + i.  A head at a time."""
    new, heads = q.shape[:2]
    at, of = first + torch.arange(new, device=q.device)[:, None], torch.arange(k.shape[0], device=q.device)[None]
    hidden = (of > at) | ((of <= at - window) if window else torch.zeros((), dtype=torch.bool, device=q.device))
    out = []
    for h in range(heads):
        g = h * k.shape[1] // heads
        scores = ((q[:, h] @ k[:, g].T) * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            scores = torch.cat([scores, sink[h].expand(new, 1)], 1)
        p = torch.softmax(scores, -1)
        out.append(p[:, : k.shape[0]] @ v[:, g])
    return torch.stack(out, 1)


def _conv(x, taps, bias=None):
    """x [sequences, time, channels], zeros before the start."""
    t = taps.shape[1]
    padded = torch.cat([x.new_zeros(x.shape[0], t - 1, x.shape[2]), x], 1)
    y = sum(padded[:, j: j + x.shape[1]] * taps[:, j] for j in range(t))
    return _silu(y if bias is None else y + bias)


def _exact_attention(case, w, cached, rows):
    new, before = _shares(case["new"], case["seqs"]), _shares(case["cached"], case["seqs"]) if case["cached"] else [0] * case["seqs"]
    out, at, at_c, s = [], 0, 0, LATENT
    for n, b in zip(new, before):
        x = rows[at: at + n] if not b else torch.cat([cached[at_c: at_c + b], rows[at: at + n]])
        at, at_c, pos = at + n, at_c + b, torch.arange(b + n, device=x.device)
        if case["kind"] == "attention":
            q, k, v = torch.split(x @ w["in_proj.qkv_fused.weight"].T, [HEADS * HEAD, KV_HEADS * HEAD, KV_HEADS * HEAD], 1)
            q, k = (_turn(t.view(b + n, -1, HEAD), pos, THETA, False) for t in (q, k))
            o = _attend(q[b:], k, v.view(b + n, -1, HEAD), b, HEAD ** -0.5)
        else:
            h, dim, rot, own = s["heads"], s["dim"], s["rot"], not case["query_latent"]
            p = x @ w["in_proj.weight"].T
            if own:
                q, c, kr, gate = torch.split(p, [h * (dim + rot), s["rank"], rot, h], 1)
            else:
                c, kr, q = torch.split(p, [s["rank"], rot, s["q_rank"]], 1)
                q = (_rms(q) * w["q_norm"]) @ w["q_up.weight"].T
            q, c = q.view(b + n, h, dim + rot), _rms(c) * w["latent_norm"]
            q = torch.cat([q[..., :dim], _turn(q[..., dim:], pos, 10000.0, not own)], -1)
            kr = _turn(kr.view(b + n, 1, rot), pos, 10000.0, not own).expand(-1, h, -1)
            k, v = torch.cat([(c @ w["uk"].T).view(b + n, h, dim), kr], -1), (c @ w["uv"].T).view(b + n, h, s["vdim"])
            o = _attend(q[b:], k, v, b, (dim + rot) ** -0.5, 0 if own else s["window"], w["sink"] if own else None)
            if own:
                o = o * torch.sigmoid(gate[b:])[..., None]
        out.append(o.flatten(1) @ w["dense.weight"].T)
    return {"y": [torch.cat(out)], "cache": None}


def _exact_memory(case, w, rows, later):
    """The mixers with a state: every sequence's rows, those of its decode steps behind its prompt's, side by side."""
    kind, new, steps = case["kind"], _shares(case["new"], case["seqs"]), case["steps"]
    n, longest = len(new), max(new) + steps
    x, at = rows.new_zeros(n, longest, WIDTH), 0
    for i, c in enumerate(new):
        x[i, :c] = rows[at: at + c]
        if steps:
            x[i, c: c + steps] = later[:, i]
        at += c
    live = torch.tensor([c + steps for c in new], device=x.device)
    p = x @ w["in_proj.weight"].T
    tails = None
    if kind == "state_space":
        s = SPACE
        h, vd, gs, inner = s["heads"], s["vdim"], s["groups"] * s["state"], s["heads"] * s["vdim"]
        z, raw, dt = torch.split(p, [inner, inner + 2 * gs, h], -1)
        xs, bs, cs = torch.split(_conv(raw, w["conv"], w["conv_bias"]), [inner, gs, gs], -1)
        xs = xs.view(n, longest, h, vd)
        k, q = (t.view(n, longest, s["groups"], s["state"]).repeat_interleave(h // s["groups"], 2) for t in (bs, cs))
        dt = torch.nn.functional.softplus(dt + w["dt_bias"])
        keep, v = torch.exp(-torch.exp(w["A_log"]) * dt), xs * dt[..., None]
    elif kind == "delta_rule":
        s = DELTA
        h, ch = s["heads"], s["heads"] * (2 * s["dim"] + s["vdim"])
        raw, gate = p[..., :ch], p[..., _round8(ch + 2 * h):]
        q, k, v = (t.view(n, longest, h, -1) for t in torch.split(_conv(raw, w["conv"]), [h * s["dim"], h * s["dim"], h * s["vdim"]], -1))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, beta = q * s["dim"] ** -0.5, torch.sigmoid(p[..., ch: ch + h])
        keep = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(p[..., ch + h: ch + 2 * h] + w["dt_bias"]))
    else:
        s = MEMORY
        h = s["heads"]
        q, k, v, gate, more = torch.split(p, [h * s["dim"], h * s["dim"], h * s["vdim"], h * s["vdim"],
                                              p.shape[-1] - 2 * h * (s["dim"] + s["vdim"])], -1)
        q, k, v = (t.view(n, longest, h, -1) for t in (q, k, v))
        if kind == "matrix_memory":
            q = q * s["dim"] ** -0.5
            gi, gf = (s["cap"] * torch.tanh(t / s["cap"]) for t in torch.split(more[..., : 2 * h] + w["gate_bias"], h, -1))
            gf = torch.nn.functional.logsigmoid(gf)
        else:
            q, k, v = _silu(q), _silu(k), _silu(v)
            keep = torch.tensor(DECAYS, dtype=torch.float64, device=x.device).expand(n, longest, h)
    if kind in ("state_space", "delta_rule"):
        t = w["conv"].shape[1]
        tails = torch.stack([raw[i, c + steps - t + 1: c + steps] for i, c in enumerate(new)])
    S = x.new_zeros(n, h, v.shape[-1], k.shape[-1])
    top, norm, out = x.new_zeros(n, h), x.new_zeros(n, h, k.shape[-1]), []
    for t in range(longest):
        on = (t < live)[:, None]
        kt, vt, qt = k[:, t], v[:, t], q[:, t]
        if kind == "matrix_memory":
            to = torch.maximum(gf[:, t] + top, gi[:, t])
            a, kt = torch.exp(gf[:, t] + top - to), kt * torch.exp(gi[:, t] - to)[..., None]
            top = torch.where(on, to, top)
            norm = torch.where(on[..., None], a[..., None] * norm + kt, norm)
        else:
            a = keep[:, t]
        T = S * a[..., None, None]
        if kind == "delta_rule":
            vt = beta[:, t][..., None] * (vt - torch.einsum("nhvk,nhk->nhv", T, kt))
        T = T + vt[..., None] * kt[..., None, :]
        o = torch.einsum("nhvk,nhk->nhv", T, qt)
        if kind == "matrix_memory":
            o = o / (torch.maximum(((norm * qt).sum(-1)).abs(), torch.exp(-top)) + 1e-6)[..., None]
        S = torch.where(on[..., None, None], T, S)
        out.append(o)
    o = torch.stack(out, 1)
    if kind == "state_space":
        o = ((o + xs * w["D"][:, None]).flatten(2) * _silu(z)).view(n, longest, s["groups"], -1)
        o = _rms(o).flatten(2) * w["norm"]
    elif kind == "delta_rule":
        o = (_rms(o) * w["norm"]).flatten(2) * _silu(gate)
    elif kind == "matrix_memory":
        o = _rms(o).flatten(2) * w["norm"] * torch.sigmoid(gate)
    else:
        o = _rms(o.flatten(2)) * w["norm"] * torch.sigmoid(gate)
    y = o @ w["dense.weight"].T
    outs = [torch.cat([y[i, :c] for i, c in enumerate(new)])]
    outs += [torch.stack([y[i, c + j] for i, c in enumerate(new)]) for j in range(steps)]
    states = [S] + ([tails] if tails is not None else []) + ([torch.cat([norm, top[..., None]], -1)] if kind == "matrix_memory" else [])
    return {"y": outs, "state": states}


def _exact_request(case, seed, device):
    get = lambda name, shape: _made(seed, name, shape, "gain" if "norm" in name else "matrix", _type(case), device).double()  # noqa: E731
    prompts, later = _prompts(case, seed)
    whole = [p + [t[i] for t in later] for i, p in enumerate(prompts)]
    table = get("model.embed_tokens.weight", (VOCAB, WIDTH))
    xs = [table[torch.tensor(t, device=device)] for t in whole]
    del table
    for layer in range(LAYERS):
        p = "model.layers.%d." % layer
        norm = [get(p + n + "_layernorm.weight", (WIDTH,)) for n in ("input", "post_attention")]
        wq, wk, wv = (get(p + "self_attn.%s_proj.weight" % n, (h * HEAD, WIDTH)) for n, h in (("q", HEADS), ("k", KV_HEADS), ("v", KV_HEADS)))
        wo = get(p + "self_attn.o_proj.weight", (WIDTH, HEADS * HEAD))
        wg, wu = (get(p + "mlp.%s_proj.weight" % n, (FF, WIDTH)) for n in ("gate", "up"))
        wd = get(p + "mlp.down_proj.weight", (WIDTH, FF))
        for i, x in enumerate(xs):
            h, pos = _rms(x) * norm[0], torch.arange(x.shape[0], device=device)
            q, k = (_turn((h @ m.T).view(x.shape[0], -1, HEAD), pos, THETA, True) for m in (wq, wk))
            x = x + _attend(q, k, (h @ wv.T).view(x.shape[0], -1, HEAD), 0, HEAD ** -0.5).flatten(1) @ wo.T
            h = _rms(x) * norm[1]
            xs[i] = x + (_silu(h @ wg.T) * (h @ wu.T)) @ wd.T
    gain, head = get("model.norm.weight", (WIDTH,)), get("lm_head.weight", (VOCAB, WIDTH))
    last = [[x[len(p) - 1 + j] for x, p in zip(xs, prompts)] for j in range(case["steps"] + 1)]
    return {"logits": [(_rms(torch.stack(rows)) * gain) @ head.T for rows in last]}


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "request":
        return _exact_request(case, seed, device)
    cached, rows, later = (None if t is None else t.double() for t in _rows(case, seed, device))
    if kind == "experts":  # a matrix at a time: the stacks would take 11 GB
        s, w = EXPERTS, _weights(case, seed, device)
        scores, chosen = torch.topk(torch.sigmoid(rows @ w["router.weight"].double().T), s["top"], -1)
        y = torch.zeros_like(rows)
        for e in range(s["experts"]):
            r, c = torch.nonzero(chosen == e, as_tuple=True)
            x = rows[r] * scores[r, c][:, None]
            gate, up = torch.split(x @ w["gate_up"][e].double().T, s["hidden"], -1)
            gate, up = gate.clamp(max=s["limit"]), up.clamp(-s["limit"], s["limit"])
            y.index_add_(0, r, (gate * torch.sigmoid(s["alpha"] * gate) * (up + 1.0)) @ w["down"][e].double().T)
        return {"y": y}
    w = {n: t.double() for n, t in _weights(case, seed, device).items()}
    if kind == "mlp":
        gate, up = torch.split(rows @ w["wg1_fused.weight"].T, FF, -1)
        return {"y": (_silu(gate) * up) @ w["w2.weight"].T}
    if kind in ("attention", "latent"):
        return _exact_attention(case, w, cached, rows)
    return _exact_memory(case, w, rows, later)
