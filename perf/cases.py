"""The calls whose speed is followed: layers of the decoders, and whole steps of the flagship, over their range.

A case names a layer (or a whole model), the sizes of one of the shapes that ``bench.py`` and the tests use, a data type
and the step: ``prompt`` (sequences of unequal lengths that start together) or ``decode`` (one more token for every
sequence).  Layers run through the parts that the registry hands out, as the engine runs them: ``begin_step`` and
``forward`` on a step context and a cache entry, for a decode step captured once in a CUDA graph and replayed, as
``Engine.generate`` does.  Whole models run through ``Engine.step``, launch by launch.
"""

import dataclasses
import math
import random

import torch

DEV = "cuda"
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
F64 = torch.float64

# ---------------------------------------------------------------------------------------------------------------- sizes
# attention of the flagship: (width, query heads, key heads, head size); widths of its three benchmark shapes, and heads of 64
ATTENTION = {"0.6b": (1024, 16, 8, 128), "4b": (2560, 32, 8, 128), "8b": (4096, 32, 8, 128), "d64": (2048, 32, 8, 64)}
# attention with a window that keeps the first tokens and a gate per head: (..., rotated values, window, kept)
WINDOW = {"1b": (2048, 16, 8, 128, 64, 1024, 4), "2b": (2560, 20, 10, 128, 128, 512, 64)}
# attention through a latent: (width, heads, head size, rotated, value size, query latent, key/value latent)
LATENT = {"1b": (2048, 16, 128, 64, 128, 768, 192), "2b": (2560, 20, 128, 64, 128, 1024, 192)}
# routed experts: (width, expert size, experts, chosen, gated)
EXPERTS = {"1b": (2048, 1024, 32, 4, True), "1b-plain": (2048, 1024, 32, 4, False), "2b": (2560, 1536, 16, 2, True)}
# delta rule with a decay per key channel: (width, heads, key heads, key size, value size, taps, inner size of the low ranks)
DELTA = {"1b": (2048, 16, 16, 128, 128, 4, 64), "2b": (2560, 20, 20, 128, 128, 4, 64)}
# state space: (width, heads, value size, state, groups, taps, parts of the norm)
SSM = {"1b": (2048, 32, 128, 128, 8, 4, 8), "2b": (2560, 40, 128, 128, 4, 4, 1)}
# whole models of the flagship: (width, heads, key heads, head size, feed-forward)
MODEL = {"0.6b": (1024, 16, 8, 128, 3072), "4b": (2560, 32, 8, 128, 9728)}
VOCAB, EPS = 151936, 1e-6


def listed():
    return [
        # the smallest call: one user, one token, short context, the smallest model - launches and latency
        dict(name="attention_token", kind="attention", shape="0.6b", dtype="bfloat16", step="decode", seqs=1, longest=300),
        # the headline decode step's attention layer: eight users with contexts of 2,048
        dict(name="attention_decode", kind="attention", shape="4b", dtype="bfloat16", step="decode", seqs=8, longest=2048),
        # one prompt of 2,048 tokens through the same layer
        dict(name="attention_prompt", kind="attention", shape="4b", dtype="bfloat16", step="prompt", seqs=1, longest=2048),
        # a few prompts of unequal lengths under a window, some longer than it, some shorter
        dict(name="window_prompts", kind="window", shape="1b", dtype="bfloat16", step="prompt", seqs=3, longest=2500),
        # one prompt through latent attention, and eight users decoding over cached latents
        dict(name="latent_prompt", kind="latent", shape="1b", dtype="bfloat16", step="prompt", seqs=1, longest=2048),
        dict(name="latent_decode", kind="latent", shape="1b", dtype="bfloat16", step="decode", seqs=8, longest=2048),
        # a prompt through routed experts, and eight users decoding
        dict(name="experts_prompt", kind="experts", shape="1b", dtype="bfloat16", step="prompt", seqs=1, longest=2048),
        dict(name="experts_decode", kind="experts", shape="1b", dtype="bfloat16", step="decode", seqs=8, longest=1),
        # the two kinds of recurrent layers: a long prompt alone, and a ragged batch of prompts
        dict(name="delta_prompt", kind="delta", shape="1b", dtype="bfloat16", step="prompt", seqs=1, longest=2048),
        dict(name="state_space_prompts", kind="state_space", shape="1b", dtype="bfloat16", step="prompt", seqs=4, longest=1500),
        # whole steps: the check in true 32-bit at batch 4, and the flagship's ragged batch of prompts with two tokens behind
        dict(name="model_f32", kind="model", shape="0.6b", dtype="float32", step="prompt", seqs=4, longest=512, layers=4),
        dict(name="model_bf16", kind="model", shape="4b", dtype="bfloat16", step="prompt", seqs=8, longest=2048, layers=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "window", "latent", "experts", "delta", "state_space", "model"])
    shapes = {"attention": ATTENTION, "window": WINDOW, "latent": LATENT, "experts": EXPERTS, "delta": DELTA,
              "state_space": SSM, "model": MODEL}[kind]
    shape = rng.choice(sorted(shapes))
    dtype = "float32" if rng.random() < 0.15 else "bfloat16"
    step = "prompt" if kind == "model" or rng.random() < 0.6 else "decode"
    case = dict(kind=kind, shape=shape, dtype=dtype, step=step)
    if step == "decode":
        case["seqs"] = _log(rng, 1, 64 if dtype == "bfloat16" else 8)
        recurrent = kind in ("delta", "state_space")
        case["longest"] = 1 if kind == "experts" else _log(rng, 5, 600 if recurrent else min(4096, 65536 // case["seqs"]))
    else:
        case["seqs"] = _log(rng, 1, 8)
        most = 4096 if dtype == "bfloat16" else 400
        if kind == "model":
            most, case["layers"] = most // 2, rng.randint(1, 4)
        case["longest"] = _log(rng, 9, most if case["seqs"] <= 3 else most // 2)
    return case


def _lengths(case):
    """Tokens of every sequence (of a decode step: behind the new one), the first the longest, down to a sixteenth."""
    rng = random.Random(1000 * case["longest"] + case["seqs"])
    n = case["longest"]
    return [n] + [max(1, _log(rng, max(1, n / 16), n)) for _ in range(case["seqs"] - 1)]


# --------------------------------------------------------------------------------------------------------------- inputs
def _generator(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + sum(ord(c) for c in case["kind"] + case["shape"] + case["dtype"])) % (1 << 62))
    return g


def _weights(case, seed):
    """A checkpoint's tensors of the layer: (part kind, its parameters, tensors by name in bfloat16)."""
    g = _generator(case, seed)

    def mat(*s):
        return (torch.randn(*s, generator=g, device=DEV) * 0.02).to(torch.bfloat16)

    def gain(*s):
        return (1 + 0.1 * torch.randn(*s, generator=g, device=DEV)).to(torch.bfloat16)

    def rand(*s):
        return torch.rand(*s, generator=g, device=DEV)

    def dt_bias(n):                                   # the inverse softplus of steps between 0.001 and 0.1
        dt = torch.exp(rand(n) * math.log(100.0) + math.log(0.001))
        return torch.log(torch.expm1(dt)).to(torch.bfloat16)

    kind = case["kind"]
    if kind == "attention":
        h, nh, nkv, d = ATTENTION[case["shape"]]
        w = dict(q=mat(nh * d, h), k=mat(nkv * d, h), v=mat(nkv * d, h), o=mat(h, nh * d), q_norm=gain(d), k_norm=gain(d))
        p = dict(hidden_size=h, num_heads=nh, num_kv_heads=nkv, head_dim=d, scale=d ** -0.5, qk_norm_eps=EPS, window=None,
                 position=("rope_neox", dict(head_dim=d, theta=1000000.0, rotary_dim=d)))
        return "attention", p, w
    if kind == "window":
        h, nh, nkv, d, rot, window, keep = WINDOW[case["shape"]]
        w = dict(q=mat(nh * d, h), k=mat(nkv * d, h), v=mat(nkv * d, h), o=mat(h, nh * d), gate=mat(nh, h))
        p = dict(hidden_size=h, num_heads=nh, num_kv_heads=nkv, head_dim=d, value_dim=d, scale=d ** -0.5 * 1.5, window=window,
                 keep_first=keep, unit_norm_after_rotation=EPS, head_gate=True, keep_all_keys=True,
                 position=("rope_stretched", dict(rotary_dim=rot, theta=500000.0, divide=1.0)))
        return "attention", p, w
    if kind == "latent":
        h, nh, d, r, e, a, c = LATENT[case["shape"]]
        w = dict(dq=mat(a, h), dq_norm=gain(a), uq=mat(nh * (d + r), a), dkv=mat(c + r, h), dkv_norm=gain(c),
                 uk=mat(nh * d, c), uv=mat(nh * e, c), o=mat(h, nh * e),
                 sink=torch.randn(nh, generator=g, device=DEV).to(torch.bfloat16))
        p = dict(hidden_size=h, num_heads=nh, head_dim=d, rot_dim=r, v_dim=e, q_rank=a, kv_rank=c, scale=(d + r) ** -0.5,
                 eps=EPS, sink=True, position=("rope_neox", dict(head_dim=r, theta=10000.0, rotary_dim=r)))
        return "latent_attention", p, w
    if kind == "experts":
        h, i, n, top, gated = EXPERTS[case["shape"]]
        w = dict(router=mat(n, h))
        for e in range(n):
            if gated:
                w[f"gate_{e}"] = mat(i, h)
            w[f"up_{e}"], w[f"down_{e}"] = mat(i, h), mat(h, i)
        p = dict(hidden_size=h, intermediate_size=i, experts=n, top=top, activation="silu" if gated else "relu2", gated=gated,
                 weights="softmax_of_chosen" if gated else "scores_of_chosen")
        return "routed_experts", p, w
    if kind == "delta":
        h, nh, ng, d, e, taps, rank = DELTA[case["shape"]]
        conv = lambda n: (0.5 * torch.randn(n, taps, generator=g, device=DEV)).to(torch.bfloat16)
        w = dict(q=mat(ng * d, h), k=mat(ng * d, h), v=mat(nh * e, h), q_conv=conv(ng * d), k_conv=conv(ng * d),
                 v_conv=conv(nh * e), b=mat(nh, h), A_log=torch.log(1 + 15 * rand(nh)).to(torch.bfloat16),
                 dt_bias=dt_bias(nh * d), a1=mat(rank, h), a2=mat(nh * d, rank), g1=mat(rank, h), g2=mat(nh * e, rank),
                 norm=gain(e), o=mat(h, nh * e))
        p = dict(hidden_size=h, num_heads=nh, num_kv_heads=ng, head_dim=d, v_dim=e, conv=taps, eps=EPS)
        return "channel_delta", p, w
    assert kind == "state_space"
    h, nh, e, n, ng, taps, parts = SSM[case["shape"]]
    inner, ch = nh * e, nh * e + 2 * ng * n
    w = {"in": mat(2 * inner + 2 * ng * n + nh, h), "conv": (0.5 * torch.randn(ch, taps, generator=g, device=DEV)).to(torch.bfloat16),
         "conv_bias": mat(ch), "dt_bias": dt_bias(nh), "A_log": torch.log(1 + 15 * rand(nh)).to(torch.bfloat16), "D": gain(nh),
         "norm": gain(inner), "o": mat(h, inner)}
    p = dict(hidden_size=h, num_heads=nh, v_dim=e, state=n, groups=ng, conv=taps, norm_groups=parts, eps=EPS)
    return "state_space", p, w


def _activations(case, seed, width):
    """Normalised activations of the step's sequences, one row a token (of a decode step: the new token's is the last)."""
    g = _generator(case, seed + 7919)
    more = 1 if case["step"] == "decode" else 0
    return [torch.randn(n + more, width, generator=g, device=DEV).to(DTYPES[case["dtype"]]) for n in _lengths(case)]


def _prompt_ids(case, seed):
    """Token ids of every sequence of a whole model's step, two more behind the prompt."""
    rng = random.Random(seed * 31 + 5)
    return [[rng.randrange(151000) for _ in range(n + 2)] for n in _lengths(case)]


def _context(case, starts, counts, slots, dtype, workspace):
    from enginekernel_b200.parts.base import StepContext
    pos = [p for s, n in zip(starts, counts) for p in range(s, s + n)]
    slot = [s for s, n in zip(slots, counts) for _ in range(n)]
    cu = [0]
    for n in counts:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    return StepContext(
        n_tokens=cu[-1], n_seqs=len(counts), token_ids=torch.zeros(cu[-1], **i32), positions=torch.tensor(pos, **i32),
        token_slot=torch.tensor(slot, **i32), cu_seqlens=torch.tensor(cu, **i32), is_decode=max(counts) == 1,
        max_new=max(counts), max_context=max(s + n for s, n in zip(starts, counts)), dtype=dtype,
        device=torch.device(DEV), workspace=workspace, host_positions=pos, host_token_slot=slot, host_cu_seqlens=cu)


@dataclasses.dataclass
class Layer:
    part: object
    x: torch.Tensor
    ctx: object
    cache: object = None
    recurrent: bool = False
    graph: object = None          # of a decode step, and what it writes
    outputs: list = None


@dataclasses.dataclass
class Whole:
    engine: object
    prompts: list
    tails: list


def _config(case):
    h, nh, nkv, d, ff = MODEL[case["shape"]]
    return dict(num_hidden_layers=case["layers"], hidden_size=h, num_attention_heads=nh, num_key_value_heads=nkv, head_dim=d,
                intermediate_size=ff, vocab_size=VOCAB, rope_theta=1000000.0, rms_norm_eps=EPS, max_position_embeddings=8192,
                tie_word_embeddings=True)


def prepare(case, seed):
    if case["kind"] == "model":
        from enginekernel_b200 import Engine
        from enginekernel_b200.config.qwen3 import Qwen3Config
        ids = _prompt_ids(case, seed)
        tokens = sum(-(-len(i) // 64) * 64 for i in ids)
        engine = Engine.from_config(Qwen3Config(**_config(case)), seed=seed, dtype=case["dtype"], max_tokens=tokens,
                                    max_batch=len(ids))
        return Whole(engine, [i[:-2] for i in ids], [i[-2:] for i in ids])
    from enginekernel_b200.cache import SequenceCache
    from enginekernel_b200.parts.base import Workspace
    from enginekernel_b200.parts.spec import PartSpec
    from enginekernel_b200.registry import lookup_part
    dtype = DTYPES[case["dtype"]]
    kind, params, w = _weights(case, seed)
    if params.get("position"):
        params = dict(params, position=PartSpec(*params["position"]))
    role = "feed_forward" if case["kind"] == "experts" else "mixer"
    part = lookup_part(role, kind)(PartSpec(kind, params, {n: n for n in w}), dtype, DEV)
    part.load(w)
    xs = _activations(case, seed, params["hidden_size"])
    lens, decode = _lengths(case), case["step"] == "decode"
    workspace = Workspace(torch.device(DEV))
    if role == "feed_forward":
        x = torch.cat([x[-1:] if decode else x for x in xs])
        n = [1] * len(xs) if decode else lens
        return _captured(Layer(part, x, _context(case, [0] * len(n), n, range(len(n)), dtype, workspace)), decode)
    part.prepare(max(lens) + 64)
    cache = SequenceCache([part.cache_spec()], dtype, DEV, max_tokens=sum(-(-(n + 1) // 64) * 64 for n in lens),
                          max_slots=len(lens), max_len=max(lens) + 64)
    slots = [cache.open() for _ in lens]
    cache.reserve_all((s, n + 1) for s, n in zip(slots, lens))
    cache.upload_tables()
    recurrent = cache.entry(0).spec.kind == "state"
    ctx = _context(case, [0] * len(lens), lens, slots, dtype, workspace)
    if not decode:
        return Layer(part, torch.cat(xs), ctx, cache, recurrent)
    part.begin_step(ctx)
    part.forward(torch.cat([x[:-1] for x in xs]), ctx, cache.entry(0), True)
    ctx = _context(case, lens, [1] * len(lens), slots, dtype, Workspace(torch.device(DEV)))
    return _captured(Layer(part, torch.cat([x[-1:] for x in xs]), ctx, cache, recurrent), True)


@torch.inference_mode()
def _captured(layer, wanted):
    """The layer with its step in a graph; a first pass, which makes the workspace, leaves recurrent state as it was."""
    if wanted:
        state = layer.cache.entry(0).state if layer.recurrent else None
        before = state.clone() if state is not None else None
        _forward(layer)
        if state is not None:
            state.copy_(before)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outputs = _forward(layer)
        layer.graph, layer.outputs = graph, outputs
    return layer


def _forward(layer):
    part, ctx = layer.part, layer.ctx
    if layer.cache is None:
        return [part.forward(layer.x, ctx)]
    entry = layer.cache.entry(0)
    if layer.recurrent and not ctx.is_decode:
        entry.state.zero_()                       # as a sequence's state is when its slot is opened
    ctx.shared = {}
    part.begin_step(ctx)
    out = part.forward(layer.x, ctx, entry, True)
    if layer.recurrent:
        return [out, entry.state[:, :part.s_values], entry.state[:, part.s_values:]]
    return [out, entry.k_pages, entry.v_pages] if entry.spec.planes == 2 else [out, entry.k_pages]


def run(state):
    if isinstance(state, Whole):
        e = state.engine
        slots = [e.open_sequence() for _ in state.prompts]
        logits = [e.step([(s, p, [len(p) - 1]) for s, p in zip(slots, state.prompts)])]
        for i in range(2):
            logits.append(e.step([(s, [t[i]], [0]) for s, t in zip(slots, state.tails)]))
        for s in slots:
            e.close_sequence(s)
        return logits
    if state.graph is not None:
        state.graph.replay()
        return state.outputs
    return _forward(state)


# ------------------------------------------------------------------------------------------------- work and tolerances
def _pairs(case, window=None, keep=0):
    """Pairs of a query and a key that it sees, over the step's sequences."""
    def seen(i):
        return i + 1 if window is None or i < window else window + max(0, min(keep, i + 1 - window))
    if case["step"] == "decode":
        return sum(seen(n) for n in _lengths(case))
    return sum(sum(seen(i) for i in range(n)) for n in _lengths(case))


def work(case):
    lens, decode = _lengths(case), case["step"] == "decode"
    t = len(lens) if decode else sum(lens)
    b = 2 if case["dtype"] == "bfloat16" else 4
    kind = case["kind"]
    if kind == "model":
        h, nh, nkv, d, ff = MODEL[case["shape"]]
        per = h * d * (2 * nh + 2 * nkv) + 3 * h * ff
        n, runs = len(lens), 3
        flops = 2.0 * (t + 2 * n) * per * case["layers"] + 2.0 * 3 * n * h * VOCAB + 4.0 * _pairs(case) * nh * d * case["layers"]
        # a pass is three steps; every step reads the layers and the head
        return dict(bytes=runs * b * (per * case["layers"] + h * VOCAB) + 4.0 * runs * n * VOCAB, flops=flops)
    if kind in ("attention", "window"):
        h, nh, nkv, d = (ATTENTION if kind == "attention" else WINDOW)[case["shape"]][:4]
        window, keep = WINDOW[case["shape"]][5:] if kind == "window" else (None, 0)
        weights = h * d * (2 * nh + 2 * nkv) + (nh * h if kind == "window" else 0)
        pairs = _pairs(case, window, keep)
        cached = 2 * nkv * d * (pairs if decode else t)
        return dict(bytes=float(b * (weights + 2 * t * h + cached)), flops=2.0 * t * weights + 4.0 * pairs * nh * d)
    if kind == "latent":
        h, nh, d, r, e, a, c = LATENT[case["shape"]]
        weights = (a + c + r) * h + nh * (d + r) * a + nh * d * c + nh * e * c + h * nh * e
        pairs = _pairs(case)
        cached = (c + r) * (pairs if decode else t)
        # per pair the cheaper of the two forms: keys and values expanded per head, or rows of the latent
        per_pair = 2 * (2 * c + r) if decode else 2 * (d + r + e)
        return dict(bytes=float(b * (weights + 2 * t * h + cached)), flops=2.0 * t * weights + float(per_pair) * pairs * nh)
    if kind == "experts":
        h, i, n, top, gated = EXPERTS[case["shape"]]
        per = (3 if gated else 2) * h * i
        touched = n * (1 - (1 - top / n) ** t)         # experts that t tokens choose, on average
        return dict(bytes=float(b * (n * h + touched * per + 2 * t * h)), flops=2.0 * t * (n * h + top * per))
    if kind == "delta":
        h, nh, ng, d, e, taps, rank = DELTA[case["shape"]]
        ch = 2 * ng * d + nh * e
        weights = (ch + nh + 2 * rank) * h + nh * (d + e) * rank + h * nh * e
        scan = 6.0 * nh * d * e
        state = nh * d * e + ch * (taps - 1)
    else:
        h, nh, e, d, ng, taps, _ = SSM[case["shape"]]
        ch = nh * e + 2 * ng * d
        weights = (nh * e + ch + nh) * h + h * nh * e
        scan = 4.0 * nh * d * e
        state = nh * d * e + ch * (taps - 1)
    moved = 4 * state * len(lens) * (2 if decode else 1)
    return dict(bytes=float(b * (weights + 2 * t * h) + moved), flops=2.0 * t * (weights + ch * taps) + t * scan)


def tolerance(case):
    """bfloat16: operands of the products and the cached rows are rounded to 8 bits of mantissa on the way; another order
    of the sums moves some of these roundings by one place.  32-bit: sums of up to 4,096 terms in another order."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 2e-2 if case["kind"] == "model" else 1e-2}


# ----------------------------------------------------------------------------------------------------- plain, in 64 bits
def _rotate(x, positions, rot, theta):
    """Values (i, i + rot / 2) of the last axis turn by p theta^(-2i / rot); x [T, heads, .]."""
    half = rot // 2
    f = theta ** (-torch.arange(half, dtype=F64, device=x.device) * 2 / rot)
    angle = positions.to(F64)[:, None, None] * f
    c, s = torch.cos(angle), torch.sin(angle)
    a, b = x[..., :half], x[..., half:rot]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., rot:]], -1)


def _rms(x, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale, first, window=None, keep=0, sink=None):
    """q [T, H, d] at positions first .., k [N, G, d], v [N, G, e] at 0 ..: softmax attention, [T, H, e]."""
    t, nh, _ = q.shape
    i = torch.arange(first, first + t, device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    mask = j <= i
    if window is not None:
        mask &= (i - j < window) | (j < keep)
    out = torch.empty(t, nh, v.shape[-1], dtype=F64, device=q.device)
    for a in range(nh):
        g = a // (nh // k.shape[1])
        s = (q[:, a] @ k[:, g].T) * scale
        s = s.masked_fill(~mask, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[a].expand(t, 1)], 1)
        out[:, a] = torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, g]
    return out


def _conv(x, taps, bias=None):
    """Causal convolution per channel, the last column of ``taps`` for the current token; x [T, C]."""
    k = taps.shape[1]
    pad = torch.cat([x.new_zeros(k - 1, x.shape[1]), x], 0)
    y = sum(pad[j:j + x.shape[0]] * taps[:, j] for j in range(k))
    return y if bias is None else y + bias


def _exact_attention(case, w, x):
    nh, nkv, d = (ATTENTION if case["kind"] == "attention" else WINDOW)[case["shape"]][1:4]
    t = x.shape[0]
    pos = torch.arange(t, device=DEV)
    first = t - 1 if case["step"] == "decode" else 0
    q = (x[first:] @ w["q"].T).view(-1, nh, d)
    k = (x @ w["k"].T).view(t, nkv, d)
    v = (x @ w["v"].T).view(t, nkv, d)
    if case["kind"] == "attention":
        q = _rotate(_rms(q) * w["q_norm"], pos[first:], d, 1000000.0)
        k = _rotate(_rms(k) * w["k_norm"], pos, d, 1000000.0)
        o = _attend(q, k, v, d ** -0.5, first)
    else:
        rot, window, keep = WINDOW[case["shape"]][4:]
        q = _rms(_rotate(q, pos[first:], rot, 500000.0))
        k = _rms(_rotate(k, pos, rot, 500000.0))
        o = _attend(q, k, v, d ** -0.5 * 1.5, first, window, keep) * torch.sigmoid(x[first:] @ w["gate"].T)[:, :, None]
    return o.reshape(-1, nh * d) @ w["o"].T


def _exact_latent(case, w, x):
    _, nh, d, r, e, _, c = LATENT[case["shape"]]
    t = x.shape[0]
    pos = torch.arange(t, device=DEV)
    first = t - 1 if case["step"] == "decode" else 0
    q = ((_rms(x[first:] @ w["dq"].T) * w["dq_norm"]) @ w["uq"].T).view(-1, nh, d + r)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], pos[first:], r, 10000.0)], -1)
    kv = x @ w["dkv"].T
    lat = _rms(kv[:, :c]) * w["dkv_norm"]
    k_rot = _rotate(kv[:, None, c:], pos, r, 10000.0)
    k = torch.cat([(lat @ w["uk"].T).view(t, nh, d), k_rot.expand(t, nh, r)], -1)
    v = (lat @ w["uv"].T).view(t, nh, e)
    return _attend(q, k, v, (d + r) ** -0.5, first, sink=w["sink"]).reshape(-1, nh * e) @ w["o"].T


def _exact_experts(case, w, x):
    h, _, n, top, gated = EXPERTS[case["shape"]]
    z = x @ w["router"].T
    best, chosen = z.topk(top, -1)
    weight = torch.softmax(best, -1)           # (scores over the chosen scores' sum are the same numbers)
    out = torch.zeros_like(x)
    for e in range(n):
        at, k = (chosen == e).nonzero(as_tuple=True)
        if at.numel():
            up = x[at] @ w[f"up_{e}"].T
            act = _silu(x[at] @ w[f"gate_{e}"].T) * up if gated else torch.relu(up).square()
            out.index_add_(0, at, (act @ w[f"down_{e}"].T) * weight[at, k][:, None])
    return out


def _padded(seqs):
    n = max(s.shape[0] for s in seqs)
    return torch.stack([torch.cat([s, s.new_zeros(n - s.shape[0], *s.shape[1:])]) for s in seqs], 1)


def _exact_delta(case, w, xs):
    _, nh, ng, d, e, _, _ = DELTA[case["shape"]]
    unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
    qs, ks, vs, bs, gs = [], [], [], [], []
    for x in xs:
        t = x.shape[0]
        heads = lambda y: y.repeat_interleave(nh // ng, 1)
        qs.append(heads(unit(_silu(_conv(x @ w["q"].T, w["q_conv"])).view(t, ng, d)) * d ** -0.5))
        ks.append(heads(unit(_silu(_conv(x @ w["k"].T, w["k_conv"])).view(t, ng, d))))
        vs.append(_silu(_conv(x @ w["v"].T, w["v_conv"])).view(t, nh, e))
        bs.append(torch.sigmoid(x @ w["b"].T))
        a = (x @ w["a1"].T) @ w["a2"].T + w["dt_bias"]
        gs.append(torch.exp(-torch.exp(w["A_log"])[None, :, None] * torch.nn.functional.softplus(a).view(t, nh, d)))
    lens = [x.shape[0] for x in xs]
    # a padded token leaves the state alone: decay 1, beta 0
    q, k, v, beta = _padded(qs), _padded(ks), _padded(vs), _padded(bs)
    g = _padded([y - 1 for y in gs]) + 1
    s = x.new_zeros(len(xs), nh, d, e)
    o = torch.empty(max(lens), len(xs), nh, e, dtype=F64, device=DEV)
    for i in range(max(lens)):
        s = s * g[i][..., None]
        u = beta[i][..., None] * (v[i] - (s * k[i][..., None]).sum(-2))
        s = s + k[i][..., None] * u[..., None, :]
        o[i] = (s * q[i][..., None]).sum(-2)
    outs = []
    for b, x in enumerate(xs):
        y = _rms(o[:lens[b], b]) * w["norm"] * torch.sigmoid((x @ w["g1"].T) @ w["g2"].T).view(-1, nh, e)
        outs.append(y.reshape(lens[b], -1) @ w["o"].T)
    return outs, s.transpose(-1, -2).reshape(len(xs), -1)


def _exact_state_space(case, w, xs):
    _, nh, e, n, ng, _, parts = SSM[case["shape"]]
    inner = nh * e
    ps, cs, dts = [], [], []
    for x in xs:
        p = x @ w["in"].T
        ps.append(p)
        cs.append(_silu(_conv(p[:, inner:2 * inner + 2 * ng * n], w["conv"], w["conv_bias"])))
        dts.append(torch.nn.functional.softplus(p[:, 2 * inner + 2 * ng * n:] + w["dt_bias"]))
    lens = [x.shape[0] for x in xs]
    c, dt = _padded(cs), _padded(dts)              # a padded token's step is 0: the state stays
    a = torch.exp(-torch.exp(w["A_log"]) * dt)
    s = x.new_zeros(len(xs), nh, n, e)
    o = torch.empty(max(lens), len(xs), nh, e, dtype=F64, device=DEV)
    for i in range(max(lens)):
        v = c[i][:, :inner].view(-1, nh, e)
        k = c[i][:, inner:inner + ng * n].view(-1, ng, n).repeat_interleave(nh // ng, 1)
        q = c[i][:, inner + ng * n:].view(-1, ng, n).repeat_interleave(nh // ng, 1)
        s = a[i][..., None, None] * s + (dt[i][..., None] * k)[..., None] * v[..., None, :]
        o[i] = (s * q[..., None]).sum(-2)
    outs = []
    for b in range(len(xs)):
        y = o[:lens[b], b] + w["D"][:, None] * cs[b][:, :inner].view(-1, nh, e)
        y = y.reshape(lens[b], inner) * _silu(ps[b][:, :inner])
        y = _rms(y.view(lens[b], parts, -1)).reshape(lens[b], inner) * w["norm"]
        outs.append(y @ w["o"].T)
    return outs, s.transpose(-1, -2).reshape(len(xs), -1)


def _exact_model(case, seed):
    """The decoder over each whole sequence, its weights drawn as a seeded engine says it draws them: tensor by tensor in
    the order of their names from one generator on the device, in 32-bit, rounded to bfloat16."""
    h, nh, nkv, d, ff = MODEL[case["shape"]]
    shapes = {"model.embed_tokens.weight": (VOCAB, h), "model.norm.weight": (h,)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        shapes.update({p + "self_attn.q_proj.weight": (nh * d, h), p + "self_attn.k_proj.weight": (nkv * d, h),
                       p + "self_attn.v_proj.weight": (nkv * d, h), p + "self_attn.o_proj.weight": (h, nh * d),
                       p + "self_attn.q_norm.weight": (d,), p + "self_attn.k_norm.weight": (d,),
                       p + "mlp.gate_proj.weight": (ff, h), p + "mlp.up_proj.weight": (ff, h),
                       p + "mlp.down_proj.weight": (h, ff), p + "input_layernorm.weight": (h,),
                       p + "post_attention_layernorm.weight": (h,)})
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    w = {}
    for name in sorted(shapes):
        y = torch.randn(shapes[name], generator=g, device=DEV, dtype=torch.float32)
        y = y.mul_(0.1).add_(1.0) if "norm" in name else y.mul_(0.02)
        w[name] = y.to(torch.bfloat16)
    rows = []
    for ids in _prompt_ids(case, seed):
        ids = torch.tensor(ids, device=DEV)
        x = w["model.embed_tokens.weight"][ids].to(F64)
        pos = torch.arange(len(ids), device=DEV)
        for i in range(case["layers"]):
            l = {n[len(f"model.layers.{i}."):]: y.to(F64) for n, y in w.items() if n.startswith(f"model.layers.{i}.")}
            y = _rms(x) * l["input_layernorm.weight"]
            q, k, v = ((y @ l[f"self_attn.{n}_proj.weight"].T).view(len(ids), -1, d) for n in "qkv")
            q = _rotate(_rms(q) * l["self_attn.q_norm.weight"], pos, d, 1000000.0)
            k = _rotate(_rms(k) * l["self_attn.k_norm.weight"], pos, d, 1000000.0)
            x = x + _attend(q, k, v, d ** -0.5, 0).reshape(len(ids), -1) @ l["self_attn.o_proj.weight"].T
            y = _rms(x) * l["post_attention_layernorm.weight"]
            y = _silu(y @ l["mlp.gate_proj.weight"].T) * (y @ l["mlp.up_proj.weight"].T)
            x = x + y @ l["mlp.down_proj.weight"].T
        rows.append((_rms(x[-3:]) * w["model.norm.weight"].to(F64)) @ w["model.embed_tokens.weight"].to(F64).T)
    return [torch.stack([r[i] for r in rows]) for i in range(3)]


@torch.inference_mode()
def exact(case, seed):
    if case["kind"] == "model":
        return _exact_model(case, seed)
    _, params, w = _weights(case, seed)
    w = {n: y.to(F64) for n, y in w.items()}
    xs = [x.to(F64) for x in _activations(case, seed, params["hidden_size"])]
    decode = case["step"] == "decode"
    if case["kind"] == "experts":
        return [_exact_experts(case, w, torch.cat([x[-1:] if decode else x for x in xs]))]
    if case["kind"] in ("delta", "state_space"):
        outs, s = (_exact_delta if case["kind"] == "delta" else _exact_state_space)(case, w, xs)
        return [torch.cat([o[-1:] if decode else o for o in outs]), s, None]
    layer = _exact_latent if case["kind"] == "latent" else _exact_attention
    return [torch.cat([layer(case, w, x) for x in xs]), *([None] if case["kind"] == "latent" else [None, None])]
