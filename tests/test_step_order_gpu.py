"""What a layer's kernels read of a step - its table of tiles, positions, slots - is that step's, not an earlier one's."""

import pytest
import torch

from tests import helpers

pytestmark = pytest.mark.gpu

DEV = "cuda"
H, EPS = 256, 1e-5


def layer(kind, heads=4):
    """A layer with weights of its own, small enough for every launch of a short prompt to be a programmatic one."""
    from enginekernel_b200.parts.spec import PartSpec
    from enginekernel_b200.registry import lookup_part
    g = torch.Generator().manual_seed(11)
    rand = lambda *s: (torch.randn(*s, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    rope = lambda d: PartSpec("rope_neox", dict(head_dim=d, theta=10000.0, rotary_dim=d))
    if kind == "latent":
        d, r, e, c, a = 32, 64, 32, 192, 64
        p = dict(hidden_size=H, num_heads=heads, head_dim=d, rot_dim=r, v_dim=e, q_rank=a, kv_rank=c,
                 scale=(d + r) ** -0.5, eps=EPS, position=rope(r))
        w = dict(dq=rand(a, H), dq_norm=rand(a), uq=rand(heads * (d + r), a), dkv=rand(c + r, H), dkv_norm=rand(c),
                 uk=rand(heads * d, c), uv=rand(heads * e, c), o=rand(H, heads * e))
        kind = "latent_attention"
    else:
        d, kv = 64, heads // 2
        p = dict(hidden_size=H, num_heads=heads, num_kv_heads=kv, head_dim=d, scale=d ** -0.5, qk_norm_eps=EPS,
                 window=None, position=rope(d))
        w = dict(q=rand(heads * d, H), k=rand(kv * d, H), v=rand(kv * d, H), o=rand(H, heads * d), q_norm=rand(d),
                 k_norm=rand(d))
        if kind == "window":
            p.update(window=70, keep_first=3, head_gate=True, keep_all_keys=True)
            w["gate"] = rand(heads, H)
        kind = "attention"
    part = lookup_part("mixer", kind)(PartSpec(kind, p, {n: n for n in w}), torch.bfloat16, DEV)
    part.load(w)
    part.prepare(512)
    return part


def prompts(part, lens, seed):
    """A step of prompts of these lengths with a cache of its own: (input rows, context, entry)."""
    from enginekernel_b200.cache import SequenceCache
    cache = SequenceCache([part.cache_spec()], torch.bfloat16, DEV, max_tokens=64 * sum(-(-n // 64) for n in lens),
                          max_slots=len(lens))
    slots = [cache.open() for _ in lens]
    for s, n in zip(slots, lens):
        cache.reserve(s, n)
    cache.upload_tables()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ctx = helpers.make_context(torch.bfloat16, DEV, [i for n in lens for i in range(n)],
                               [s for s, n in zip(slots, lens) for _ in range(n)], cu)
    x = torch.randn(cu[-1], H, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).to(DEV)
    return x, ctx, cache.entry(0)


@pytest.mark.parametrize("kind", ["attention", "window", "latent"])
def test_a_layer_driven_alone_reads_its_own_steps_table(kind):
    """``begin_step`` and ``forward`` with nothing in between and one workspace for steps of unequal sequences, none
    waited for: every result is the one of the step alone in a workspace of its own, with the table waited for."""
    from enginekernel_b200.parts.base import Workspace
    part = layer(kind)
    steps = [prompts(part, lens, i) for i, lens in enumerate([[9], [3, 13], [1, 2, 5, 1], [130, 40], [2, 14]])]
    wants = []
    for x, ctx, entry in steps:
        ctx.workspace = Workspace(torch.device(DEV))
        ctx.shared = {}
        part.begin_step(ctx)
        torch.cuda.synchronize()
        wants.append(part.forward(x, ctx, entry, True).clone())
        torch.cuda.synchronize()
    shared = Workspace(torch.device(DEV))
    got = []
    for _ in range(4):
        for x, ctx, entry in steps:
            ctx.workspace, ctx.shared = shared, {}
            part.begin_step(ctx)
            got.append(part.forward(x, ctx, entry, True).clone())
    torch.cuda.synchronize()
    for i, y in enumerate(got):
        assert torch.equal(y, wants[i % len(steps)]), (i // len(steps), i % len(steps))


@pytest.mark.parametrize("seqs", [1, 3])
def test_a_latent_layer_driven_alone_decodes_over_rows_that_earlier_steps_wrote(seqs):
    """Decode steps over a page's border (62 to 67 rows, and 126 to 131) with contexts made ahead, nothing between the steps
    and none waited for: rows that a step wrote to a page are there in the next steps, which read it as an older one."""
    from enginekernel_b200.cache import SequenceCache
    from enginekernel_b200.parts.base import Workspace
    part = layer("latent", heads=20)
    for past in (62, 126):
        def decode(waited):
            cache = SequenceCache([part.cache_spec()], torch.bfloat16, DEV, max_tokens=192 * seqs, max_slots=seqs)
            slots = [cache.open() for _ in range(seqs)]
            for s in slots:
                cache.reserve(s, past + 6)
            cache.upload_tables()
            entry, shared = cache.entry(0), Workspace(torch.device(DEV))
            g = torch.Generator().manual_seed(past)
            rows = lambda n: torch.randn(n, H, generator=g).to(torch.bfloat16).to(DEV)
            prompt = helpers.make_context(torch.bfloat16, DEV, [i for _ in slots for i in range(past)],
                                          [s for s in slots for _ in range(past)], [past * i for i in range(seqs + 1)])
            steps = [(rows(past * seqs), prompt)]
            for i in range(6):
                steps.append((rows(seqs), helpers.make_context(torch.bfloat16, DEV, [past + i] * seqs, slots, list(range(seqs + 1)))))
            torch.cuda.synchronize()
            got = []
            for x, ctx in steps:
                ctx.workspace = Workspace(torch.device(DEV)) if waited else shared
                ctx.shared = {}
                part.begin_step(ctx)
                got.append(part.forward(x, ctx, entry, True).clone())
                if waited:
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            return got[1:]
        want = decode(True)
        for _ in range(4):
            for i, (a, b) in enumerate(zip(decode(False), want)):
                assert torch.equal(a, b), (past, i)


@pytest.mark.parametrize("kind", ["attention", "window"])
def test_tiles_found_by_the_blocks_are_those_of_the_table(kind):
    """A step with a table of tiles and without one: the same results, for sequences of one token to several tiles."""
    from enginekernel_b200.parts.attention import make_prefill_tiles
    part = layer(kind)
    x, ctx, entry = prompts(part, [1, 300, 64, 65, 17, 128, 2], 5)
    ctx.shared = {}
    alone = part.forward(x, ctx, entry, True).clone()
    make_prefill_tiles(ctx, part._tiles_key, part.num_heads, part.num_kv_heads, part.padded_dim)
    assert torch.equal(part.forward(x, ctx, entry, True), alone)


@pytest.mark.parametrize("d,n_splits", [(64, 1), (64, 4), (128, 2), (256, 1), (256, 4)])
def test_a_captured_decode_step_reads_this_steps_places(d, n_splits):
    """Positions, slots and pages that change from step to step, looked up ahead of the wait: in a captured step of few
    blocks, replayed back to back, every step's attention is the one of its own places (taken eagerly, the device idle)."""
    from enginekernel_b200.ops import kernels as k
    nq, nkv, past = 4, (1 if d == 256 else 2), 190
    g = torch.Generator().manual_seed(3)
    rand = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)
    pages = rand(9, nkv, 64, d)
    values = pages if d == 256 else rand(9, nkv, 64, d)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table = i32([[0, 2, 4, 6], [1, 3, 5, 7]])
    positions, slots = i32([past, past - 70]), i32([0, 1])
    q, out = rand(2, nq * d), torch.zeros(2, nq * d, dtype=torch.bfloat16, device=DEV)
    stream, ids, vocab = torch.zeros(2, 64, device=DEV), i32([3, 5]), rand(8, 64)
    normed, gain = torch.zeros(2, 64, dtype=torch.bfloat16, device=DEV), torch.ones(64, device=DEV)

    def attend(to):
        k.attention_decode_tma(to, q, 2, positions, slots, pages, values, table, nq, nkv, d, d ** -0.5, n_splits=n_splits)

    def step():
        positions.add_(1)                      # plain launches: what a step's state advance leaves behind
        slots.copy_(1 - slots)
        table.copy_(table.roll(1, 0))
        k.embed(stream, vocab, ids, 2)         # the step's first kernel, a plain launch; the next are programmatic
        k.rmsnorm(normed, stream, gain, 1e-5, n_rows=2)
        attend(out)

    at = lambda: [t.clone() for t in (positions, slots, table)]
    start = at()
    step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for t, s in zip((positions, slots, table), start):
        t.copy_(s)
    got, places = [], []
    for _ in range(12):
        graph.replay()
        got.append(out.clone())
        places.append(at())
    torch.cuda.synchronize()
    for y, place in zip(got, places):
        for t, s in zip((positions, slots, table), place):
            t.copy_(s)
        torch.cuda.synchronize()
        want = torch.zeros_like(out)
        attend(want)
        torch.cuda.synchronize()
        assert torch.equal(y, want)
