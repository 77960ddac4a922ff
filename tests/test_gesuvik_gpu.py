"""The Gesuvik decoder in the engine against the plain implementation, mechanism by mechanism and then whole models
under every way of cutting the work.

Part one drives the new kernels and options alone: the norm of queries and keys over the whole projection (plain,
padded and odd heads), sinks per head in every attention kernel, latent attention with plain queries, window and
gate, rotation in place and the gated norm per head around the retention scan, the corrected router, identity experts,
the soft cap on logits.  Part two runs one-mixer models with a key at every edge of a window, and part three four small
models of unlike shapes (tests/plain/gesuvik_models.py) through ``Engine``: whole prompts, prompts in portions down to
two tokens, token-by-token decoding, unequal batches, slots, pages and states used again, long decoding, and greedy
generation through the scheduler.
"""

import json

import pytest
import torch

from tests import helpers
from tests.plain import gesuvik_models as models
from tests.plain import gesuvik_plain as plain
from tests.test_kernels_gpu import DEV, DTYPES, TOL, K, Pages, rel, rnd

pytestmark = pytest.mark.gpu
F32, F64, BF16 = torch.float32, torch.float64, torch.bfloat16


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def tables(rot, n):
    speeds, factor = plain.rotation_speeds(rot)
    ang = torch.arange(n, dtype=F64)[:, None] * speeds[None]
    return (factor * ang.cos()).float().to(DEV), (factor * ang.sin()).float().to(DEV)


# ===================================================================== mechanisms alone
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("nq,nkv,d,real,rot", [(4, 2, 64, 64, 16), (16, 8, 128, 128, 128), (6, 1, 16, 10, 0), (3, 3, 20, 20, 10),
                                               (5, 5, 32, 24, 24), (40, 2, 128, 120, 64), (2, 1, 500, 500, 40), (1, 1, 6, 6, 2)])
def test_norm_of_queries_and_keys_over_the_projection(dtype, nq, nkv, d, real, rot):
    """Heads of ``real`` values padded with zeros to ``d``: one mean over all query heads, one over all key heads, gains
    per value of the projection, rotation behind it; values stored as projected; rows of finished sequences stay."""
    k, t = K(), 70
    heads = nq + 2 * nkv
    rows = rnd(t, heads, d, dtype=dtype, seed=1, scale=2.0)
    rows[:, :, real:] = 0
    gq, gk = 1 + 0.2 * rnd(nq * d, seed=6), 1 + 0.2 * rnd(nkv * d, seed=7)
    pos = [p if p != 5 else -1 for p in range(t)]
    spec = models.rotation(rot, 1e4, (2.0, 64, 4.0, 1.0)) if rot else None
    cos, sin = tables(spec, t) if rot else (torch.zeros(1, 0, device=DEV), torch.zeros(1, 0, device=DEV))
    cpu = rows.double().cpu()

    def want(part, gain):
        flat = part[:, :, :real].reshape(t, -1)
        g = gain.double().cpu().view(-1, d)[:, :real].reshape(-1)
        return plain.rotate((plain.rms_unit(flat, 1e-5) * g).view(t, -1, real), torch.arange(t), spec, False)

    pages = Pages(2, t, nkv, d, dtype, seed=3)
    got = rows.view(t, heads * d).clone()
    k.qk_whole_norm_kv(got, t, gq, gk, cos, sin, rot, i32(pos), i32([1] * t), pages.k, pages.v, pages.table, nq, nkv, d, 1e-5,
                       norm_dim=real)
    live = [i for i in range(t) if i != 5]
    kk, vv = pages.dense(1, t)
    assert rel(got.view(t, heads, d)[live, :nq, :real], want(cpu[:, :nq], gq)[live]) <= TOL[dtype]
    assert rel(kk[live][:, :, :real], want(cpu[:, nq:nq + nkv], gk)[live]) <= TOL[dtype]
    assert torch.equal(vv[live].cpu(), rows[live][:, nq + nkv:].cpu())
    assert torch.equal(got[5], rows.view(t, -1)[5])
    before = pages.k.clone()                              # queries alone, nothing stored
    alone = rows[:, :nq].reshape(t, nq * d).clone()
    k.qk_whole_norm_kv(alone, t, gq, None, cos, sin, rot, i32(pos), i32([1] * t), pages.k, pages.v, pages.table, nq, nkv, d,
                       1e-5, norm_dim=real, write_kv=False)
    assert torch.equal(alone[live], got[live, :nq * d]) and torch.equal(pages.k, before)


def _plain_row(q, keys, values, pos, scale, window, sinks):
    nh, g = q.shape[0], keys.shape[1]
    idx = [j for j in range(pos + 1) if plain.sees(pos, j, window)]
    kk = keys[idx].double().cpu().repeat_interleave(nh // g, 1)
    vv = values[idx].double().cpu().repeat_interleave(nh // g, 1)
    s = torch.einsum("hd,khd->hk", q.double().cpu(), kk) * scale
    p = torch.softmax(torch.cat([s, sinks.double().cpu()[:, None]], 1), -1)[:, :-1]
    return torch.einsum("hk,khd->hd", p, vv).reshape(-1)


def _kernels_for(dtype, d, nq, nkv):
    k = K()
    out = ["generic", "generic_split"]
    if k.attention_prefill_supported(dtype, d, nq, nkv):
        out.append("prefill")
    if dtype == BF16 and k.attention_prefill_tc_supported(dtype, d, nq, nkv):
        out.append("prefill_tc")
    if k.attention_decode_supported(dtype, d):
        out += ["decode", "decode_split"]
    if dtype == BF16 and k.attention_decode_tma_supported(dtype, d, nq, nkv):
        out += ["decode_tma", "decode_tma_split"]
    return out


def _attend(which, q, pos, pages, nq, nkv, d, scale, window, sinks):
    k = K()
    n = len(pos)
    out = torch.full((n, nq * d), 7.0, dtype=q.dtype, device=DEV)
    args = (out, q, n, i32(pos), i32([1] * n))
    tail = (pages.k, pages.v, pages.table, nq, nkv, d, scale, window)
    splits = 3 if which.endswith("split") else 1
    acc = torch.empty(n, nq, splits, d, device=DEV) if splits > 1 else None
    ml = torch.empty(n, nq, splits, 2, device=DEV) if splits > 1 else None
    if which.startswith("generic"):
        per = -(-(max(pos) + 1) // splits) if splits > 1 else 0
        k.attention_generic(*args, *tail, n_splits=splits, keys_per_split=per, part_acc=acc, part_ml=ml, sinks=sinks)
    elif which.startswith("decode_tma"):
        k.attention_decode_tma(*args, *tail, n_splits=2 if splits > 1 else 1, sinks=sinks)
        k.check_tc_status(DEV)
    elif which.startswith("decode"):
        k.attention_decode_bf16(*args, *tail, n_splits=splits, part_acc=acc, part_ml=ml, sinks=sinks)
    else:
        fn = k.attention_prefill_tc if which == "prefill_tc" else k.attention_prefill_bf16
        fn(*args, i32([0, n]), 1, *tail, sinks=sinks)
        if which == "prefill_tc":
            k.check_tc_status(DEV)
    return out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d,nq,nkv", [(20, 3, 1), (64, 4, 2), (64, 6, 6), (96, 6, 1), (128, 8, 2), (256, 2, 2)])
@pytest.mark.parametrize("window", [1, 9, 64, 96, None])
def test_sinks_per_head_under_a_window(dtype, d, nq, nkv, window):
    """Every attention kernel against the plain rule, with sinks from far below to far above the scores (a head whose
    sink takes nearly everything, one whose sink takes nothing), at the windows' and pages' edges, a prompt whole and
    behind a cached prefix."""
    length, scale = 300, 0.4
    pages = Pages(2, length, nkv, d, dtype, seed=d)
    keys, values = rnd(length, nkv, d, dtype=dtype, seed=1), rnd(length, nkv, d, dtype=dtype, seed=2)
    pages.fill(1, keys, values)
    q = rnd(length, nq * d, dtype=dtype, seed=3)
    sinks = torch.tensor([(-30.0, 1.0, 3.0, 5.0, -2.0, 0.0)[h % 6] for h in range(nq)], device=DEV)
    edge = window or 128
    picks = sorted({0, 1, edge - 1, edge, edge + 1, 63, 64, 65, 127, 128, 255, 256, length - 1} & set(range(length)))
    want = torch.stack([_plain_row(q[p].view(nq, d), keys, values, p, scale, window, sinks) for p in picks])
    cut = 101
    for which in _kernels_for(dtype, d, nq, nkv):
        if which.startswith("decode"):
            got = _attend(which, q[picks].contiguous(), picks, pages, nq, nkv, d, scale, window, sinks)
            assert rel(got, want) <= TOL[dtype], which
            continue
        got = _attend(which, q, list(range(length)), pages, nq, nkv, d, scale, window, sinks)
        assert rel(got[picks], want) <= TOL[dtype], which
        late = [i for i, p in enumerate(picks) if p >= cut]
        got = _attend(which, q[cut:], list(range(cut, length)), pages, nq, nkv, d, scale, window, sinks)
        assert rel(got[[picks[i] - cut for i in late]], want[late]) <= TOL[dtype], (which, "behind a prefix")


@pytest.mark.parametrize("d,nq,nkv", [(64, 4, 2), (96, 4, 2), (128, 4, 1)])
@pytest.mark.parametrize("window", [50, 64, 100])
def test_one_key_that_stands_out_at_every_edge_of_a_window(d, nq, nkv, window):
    length = 230
    pos, lo = length - 1, length - window
    keys, values = 0.1 * rnd(length, nkv, d, seed=1), rnd(length, nkv, d, seed=2)
    q = 0.1 * rnd(length, nq * d, seed=3)
    direction = torch.ones(d, device=DEV)
    q[pos] = direction.repeat(nq)
    sinks = torch.tensor([-1.0, 0.0, 1.0, 2.0][:nq], device=DEV)
    for key_pos in sorted({0, lo - 1, lo, lo + 1, pos - 1, pos}):
        kk, vv = keys.clone(), values.clone()
        kk[key_pos] = direction
        vv[key_pos] = 50.0
        pages = Pages(2, length, nkv, d, BF16, seed=key_pos)
        pages.fill(1, kk.to(BF16), vv.to(BF16))
        for which in _kernels_for(BF16, d, nq, nkv):
            if which.startswith("decode"):
                row = _attend(which, q[pos:].to(BF16), [pos], pages, nq, nkv, d, 0.3, window, sinks)[0]
            else:
                row = _attend(which, q.to(BF16), list(range(length)), pages, nq, nkv, d, 0.3, window, sinks)[pos]
            if key_pos >= lo:
                assert (row.float() - 50.0).abs().max() <= 0.5, (which, key_pos)
            else:
                assert row.float().abs().max() < 10.0, (which, key_pos)


@pytest.mark.parametrize("heads,dim,rot,col0", [(4, 64, 64, 0), (3, 12, 6, 5), (32, 128, 32, 128), (2, 256, 256, 4), (1, 40, 10, 0)])
def test_rotation_of_heads_in_place(heads, dim, rot, col0):
    k, t = K(), 9
    x = rnd(t, col0 + heads * dim + 8, seed=1)
    pos = [0, 1, 2, 700, -1, 63, 64, 5, 6]
    spec = models.rotation(rot, 1e4)
    cos, sin = tables(spec, 701)
    got = x.clone()
    k.rotate_heads(got, col0, heads, dim, rot, cos, sin, i32(pos), t)
    want = x.double().cpu()
    want[:, col0:col0 + heads * dim] = plain.rotate(want[:, col0:col0 + heads * dim].reshape(t, heads, dim),
                                                    torch.tensor(pos).clamp(min=0), spec, False).reshape(t, -1)
    live = [i for i in range(t) if i != 4]
    assert rel(got[live], want[live]) <= 1e-6 and torch.equal(got[4], x[4])
    outside = [c for c in range(x.shape[1]) if not col0 <= c < col0 + heads * dim]
    assert torch.equal(got[:, outside], x[:, outside])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,vdim,col", [(4, 64, 8), (3, 24, 3), (2, 256, 4), (5, 33, 1), (1, 400, 0), (16, 128, 16)])
def test_gated_norm_per_head(dtype, heads, vdim, col):
    k, n = K(), heads * vdim
    o, proj, w = rnd(6, n, seed=1, scale=3.0), rnd(6, n + col + 4, seed=2, scale=2.0), 1 + 0.2 * rnd(n, seed=3)
    unit = plain.rms_unit(o.double().cpu().view(6, heads, vdim), 1e-3).reshape(6, n)
    gate = proj[:, col:col + n].double().cpu()
    live = [0, 1, 3, 4, 5]
    for weight in (None, w):
        for act, fn in (("silu", plain.silu), ("sigmoid", torch.sigmoid)):
            y = torch.full((6, n), 7.0, dtype=dtype, device=DEV)
            k.head_norm_gate_out(y, o, proj, col, weight, 1e-3, i32([0, 5, -1, 3, 2, 9]), 6, heads, vdim, gate_activation=act)
            want = unit * fn(gate) * (1.0 if weight is None else weight.double().cpu())
            assert rel(y[live], want[live]) <= TOL[dtype] and (y[2] == 7.0).all()


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,ones", [(2, 2, 20, 12, False), (4, 2, 64, 33, True), (3, 3, 128, 40, False),
                                                          (2, 1, 200, 16, True), (1, 1, 256, 256, False)])
def test_scan_in_segments_is_the_scan(heads, kv_heads, dim, vdim, ones):
    """Unequal sequences cut into segments that run side by side, from carried states, with decays per token and per head
    (some of them 0 and 1): outputs and states as the plain walk gives them, whatever the cut."""
    from enginekernel_b200.parts.base import Workspace
    k, cols = K(), vdim + (1 if ones else 0)
    lens, slots = [300, 1, 64, 129], [2, 0, 3, 1]
    n, cu = sum(lens), [0]
    for ln in lens:
        cu.append(cu[-1] + ln)
    tok_slots = [s for s, ln in zip(slots, lens) for _ in range(ln)]
    pos = [5 + j for ln in lens for j in range(ln)]
    q, kk, v = rnd(n, kv_heads * dim + 4, seed=1), rnd(n, kv_heads * dim, seed=2, scale=0.5), rnd(n, heads * vdim, seed=3)
    rows = k.decay_scan_rows(dim)
    start = torch.zeros(4, heads, cols, rows, device=DEV)
    start[..., :dim] = rnd(4, heads, cols, dim, seed=4)
    start = start.view(4, -1)
    per_token = (0.5 + 0.5 * torch.rand(n, heads, generator=torch.Generator().manual_seed(5))).to(DEV)
    per_token[70], per_token[200:210] = 0.0, 1.0
    b_token = rnd(n, heads, seed=6)
    fixed = torch.tensor([0.995, 1.0, 0.0, 0.9][:heads], device=DEV)
    for a, b in ((per_token, b_token), (fixed, torch.full((heads,), 0.3, device=DEV))):
        full_a, full_b = (x if x.dim() > 1 else x.expand(n, heads) for x in (a, b))
        want, ends = torch.empty(n, heads, cols, dtype=F64), {}
        for s, (ln, slot) in enumerate(zip(lens, slots)):
            S = start[slot].double().cpu().view(heads, cols, rows)[..., :dim].clone()
            for t in range(cu[s], cu[s + 1]):
                kt = kk[t].double().cpu().view(kv_heads, dim).repeat_interleave(heads // kv_heads, 0)
                qt = q[t, :kv_heads * dim].double().cpu().view(kv_heads, dim).repeat_interleave(heads // kv_heads, 0)
                vt = v[t].double().cpu().view(heads, vdim)
                if ones:
                    vt = torch.cat([vt, torch.ones(heads, 1, dtype=F64)], 1)
                at, bt = full_a[t].double().cpu(), full_b[t].double().cpu()
                S = at[:, None, None] * S + bt[:, None, None] * vt[:, :, None] * kt[:, None, :]
                want[t] = (S * qt[:, None, :]).sum(-1)
            ends[slot] = S
        for segments in ((1, 300), (2, 192), (5, 64), (19, 16), (3, 101)):
            state = start.clone()
            out = torch.full((n, heads * cols), 7.0, device=DEV)
            k.decay_scan(out, q, kk, v, a, b, state, i32(cu), i32(pos), i32(tok_slots), 4, heads, kv_heads, dim, vdim,
                         ones_column=ones, n_tokens=n, max_new=300, workspace=Workspace(DEV), segments=segments)
            assert rel(out.view(n, heads, cols), want) <= 1e-5, segments
            for slot, S in ends.items():
                assert rel(state[slot].view(heads, cols, rows)[..., :dim], S) <= 1e-5, (segments, slot)
            keep = start.clone()
            k.decay_scan(out, q, kk, v, a, b, keep, i32(cu), i32(pos), i32(tok_slots), 4, heads, kv_heads, dim, vdim,
                         ones_column=ones, write_state=False, n_tokens=n, max_new=300, workspace=Workspace(DEV), segments=segments)
            assert torch.equal(keep, start)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim,ones", [(2, 1, 128, 130, False), (3, 3, 60, 64, True), (2, 2, 20, 33, False), (1, 1, 200, 40, False)])
def test_decay_scan_columns_a_lane(heads, kv_heads, dim, vdim, ones):
    """One, two and four columns a lane: groups of eight tokens whose decays' product is within the range that is walked
    divided by it, at its edge, beyond it on both sides and zero; sequences of 1, 7, 8, 9 and 150 tokens."""
    from enginekernel_b200.parts.base import Workspace
    k = K()
    lens, slots = [150, 1, 9, 7, 8], [1, 0, 2, 4, 3]
    n, cols, rows = sum(lens), vdim + int(ones), k.decay_scan_rows(dim)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    tok_slots = [s for s, ln in zip(slots, lens) for _ in range(ln)]
    pos = [3 + j for ln in lens for j in range(ln)]
    q, kk, v = rnd(n, kv_heads * dim, seed=1), rnd(n, kv_heads * dim, seed=2, scale=0.5), rnd(n, heads * vdim, seed=3)
    start = torch.zeros(5, heads, cols, rows, device=DEV)
    start[..., :dim] = rnd(5, heads, cols, dim, seed=4)
    start = start.view(5, -1)
    a, b = 0.3 + 0.7 * torch.rand(n, heads, generator=torch.Generator().manual_seed(5)), torch.randn(n, heads, generator=torch.Generator().manual_seed(6))
    a[8:16], a[16:24], a[24:32], a[32:40], a[45] = 2.0 ** -5, 2.0 ** -4.99, 2.0 ** -12, 1.5, 0.0
    a, b = a.to(DEV), b.to(DEV)
    want, ends = torch.empty(n, heads, cols, dtype=F64), {}
    for s, (ln, slot) in enumerate(zip(lens, slots)):
        S = start[slot].double().cpu().view(heads, cols, rows)[..., :dim].clone()
        for t in range(cu[s], cu[s + 1]):
            kt, qt = (x[t].double().cpu().view(kv_heads, dim).repeat_interleave(heads // kv_heads, 0) for x in (kk, q))
            vt = torch.cat([v[t].double().cpu().view(heads, vdim), torch.ones(heads, int(ones), dtype=F64)], 1)
            S = a[t].double().cpu()[:, None, None] * S + (b[t].double().cpu()[:, None] * vt)[:, :, None] * kt[:, None, :]
            want[t] = (S * qt[:, None, :]).sum(-1)
        ends[slot] = S
    for lane_columns in (1, 2, 4) if dim > 32 else (1, 2):
        for segments in ((1, 150), (3, 50)):
            state, out = start.clone(), torch.full((n, heads * cols), 7.0, device=DEV)
            k.decay_scan(out, q, kk, v, a, b, state, i32(cu), i32(pos), i32(tok_slots), 5, heads, kv_heads, dim, vdim,
                         ones_column=ones, n_tokens=n, max_new=150, workspace=Workspace(DEV), segments=segments,
                         lane_columns=lane_columns)
            assert rel(out.view(n, heads, cols), want) <= 1e-5, (lane_columns, segments)
            for slot, S in ends.items():
                assert rel(state[slot].view(heads, cols, rows)[..., :dim], S) <= 1e-5, (lane_columns, segments, slot)


@pytest.mark.parametrize("lane_columns", [1, 2, 4])
def test_an_infinite_value_stays_in_its_column(lane_columns):
    """In a group of eight tokens it reaches no earlier token and no other column, and a column whose state overflowed is
    infinite, not NaN, where every product with it is: keys and queries of one sign."""
    from enginekernel_b200.parts.base import Workspace
    k, heads, dim, n = K(), 2, 64, 43
    g = torch.Generator(device=DEV).manual_seed(3)
    draw = lambda *s: torch.rand(*s, generator=g, device=DEV) + 0.1
    q, kk, v, a, b = draw(n, dim), draw(n, dim), draw(n, heads * dim), 0.9 * draw(n, heads).clamp(max=1.0), draw(n, heads)

    def run(values):
        state, out = torch.zeros(1, heads * dim * dim, device=DEV), torch.empty(n, heads * dim, device=DEV)
        k.decay_scan(out, q, kk, values, a, b, state, i32([0, n]), i32(list(range(n))), i32([0] * n), 1, heads, 1, dim, dim,
                     n_tokens=n, max_new=n, workspace=Workspace(DEV), segments=(1, n), lane_columns=lane_columns)
        return out, state.view(heads, dim, dim)

    (clean, clean_state), spoilt = run(v), v.clone()
    spoilt[20, 3] = float("inf")
    out, state = run(spoilt)
    assert clean.isfinite().all() and torch.isposinf(out[20:, 3]).all() and torch.isposinf(state[0, 3]).all()
    out[20:, 3], state[0, 3] = clean[20:, 3], clean_state[0, 3]
    assert torch.equal(out, clean) and torch.equal(state, clean_state)


@pytest.mark.parametrize("low", [0.5, 0.95, 0.05])
def test_prompts_are_as_exact_as_single_tokens(low):
    """The scan of a prompt, eight tokens at a time, against 64 bits, beside the same tokens one a step, each a product and a
    sum a value of S: no larger an error.  (Both are the norms of tens of thousands of independent roundings, of outputs
    over all tokens, of S at the end of 8 sequences: 2 % and 4 % for what chance moves them.)"""
    from enginekernel_b200.parts.base import Workspace
    k, heads, kv_heads, dim, n_seqs, ln = K(), 4, 2, 128, 8, 400
    n = n_seqs * ln
    g = torch.Generator(device=DEV).manual_seed(7)
    draw = lambda *s: torch.randn(*s, generator=g, device=DEV)
    uniform = lambda *s: torch.rand(*s, generator=g, device=DEV)
    q, kk, v = draw(n, kv_heads * dim), draw(n, kv_heads * dim), draw(n, heads * dim)
    a, b = uniform(n, heads) * (1 - low) + low, uniform(n, heads)
    by_seq = lambda x: x.double().view(n_seqs, ln, *x.shape[1:])
    twice = lambda x: by_seq(x).view(n_seqs, ln, kv_heads, dim).repeat_interleave(heads // kv_heads, 2)
    q64, k64, v64, a64, b64 = twice(q), twice(kk), by_seq(v).view(n_seqs, ln, heads, dim), by_seq(a), by_seq(b)
    S, want = torch.zeros(n_seqs, heads, dim, dim, dtype=F64, device=DEV), []
    for t in range(ln):
        S = a64[:, t, :, None, None] * S + (b64[:, t, :, None] * v64[:, t])[..., None] * k64[:, t, :, None, :]
        want.append((S * q64[:, t, :, None, :]).sum(-1))
    want = torch.stack(want, 1)
    off = lambda got, ref: ((got.double().view_as(ref) - ref).norm() / ref.norm()).item()
    slots, pos = [s for s in range(n_seqs) for _ in range(ln)], list(range(ln)) * n_seqs
    errors = []
    for segments, lane_columns in ((None, None), ((1, ln), 2), ((4, 128), 4)):
        state, out = torch.zeros(n_seqs, heads * dim * dim, device=DEV), torch.empty(n, heads * dim, device=DEV)
        k.decay_scan(out, q, kk, v, a, b, state, i32([s * ln for s in range(n_seqs + 1)]), i32(pos), i32(slots), n_seqs, heads,
                     kv_heads, dim, dim, n_tokens=n, max_new=ln, workspace=Workspace(DEV), segments=segments,
                     lane_columns=lane_columns)
        errors.append((off(out, want), off(state, S)))
    state, out = torch.zeros(n_seqs, heads * dim * dim, device=DEV), torch.empty(n_seqs, ln, heads * dim, device=DEV)
    for t in range(ln):
        step = lambda x: x.view(n_seqs, ln, -1)[:, t].contiguous()
        one = torch.empty(n_seqs, heads * dim, device=DEV)
        k.decay_scan(one, step(q), step(kk), step(v), step(a), step(b), state, i32(list(range(n_seqs + 1))), i32([t] * n_seqs),
                     i32(list(range(n_seqs))), n_seqs, heads, kv_heads, dim, dim, n_tokens=n_seqs, max_new=1)
        out[:, t] = one
    of_out, of_state = off(out, want), off(state, S)
    print(low, errors, of_out, of_state)
    for e_out, e_state in errors:
        assert e_out <= 1.02 * of_out and e_state <= 1.04 * of_state, (errors, of_out, of_state)


def test_how_a_step_is_cut_into_segments():
    k = K()
    for n_seqs, heads, cols, longest in ((1, 16, 128, 2048), (1, 2, 16, 130), (8, 16, 128, 2048), (1, 16, 128, 1), (3, 1, 20, 100000)):
        parts, length = k.decay_scan_segments(n_seqs, heads, cols, longest)
        assert parts >= 1 and parts * length >= longest > (parts - 1) * length
        assert parts == 1 or (length % 64 == 0 and length >= k.SCAN_MIN_SEGMENT)
    assert k.decay_scan_segments(1, 16, 128, 2048)[0] > 1 and k.decay_scan_segments(1, 4, 64, 1)[0] == 1


@pytest.mark.parametrize("experts,top", [(12, 3), (5, 5), (16, 6), (40, 33), (7, 1)])
def test_corrected_router(experts, top):
    """The largest corrected scores in order, the bare softmax scores as weights: corrections of both signs, beyond any
    score, and none; logits so far apart that scores vanish."""
    k = K()
    for scale, size in ((1.0, 0.2), (30.0, 0.5), (1.0, 4.0), (2.0, 0.0)):
        logits = rnd(70, experts, seed=experts + top, scale=scale)
        corr = rnd(experts, seed=9, scale=size) - (3.0 if size == 4.0 else 0.0)
        chosen = torch.empty(70, top, dtype=torch.int32, device=DEV)
        weight = torch.empty(70, top, device=DEV)
        k.moe_route(chosen, weight, logits, 70, 1, 1, top, 1.5, weights="softmax", correction=corr if size else None)
        s = torch.softmax(logits.double().cpu(), -1)
        keyed = s + (corr.double().cpu() if size else 0)
        picked = keyed.gather(1, chosen.cpu().long())
        assert (picked - keyed.topk(top, -1).values).abs().max() <= 1e-6            # (ties of vanished scores either way)
        assert all(len(set(r)) == top for r in chosen.tolist())
        assert (weight.double().cpu() - 1.5 * s.gather(1, chosen.cpu().long())).abs().max() <= 1e-6


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,ff,experts,identity,top,shared,tokens", [
    (96, 48, 8, 4, 3, 56, 50), (100, 36, 2, 6, 2, None, 7), (256, 32, 16, 1, 6, 128, 300), (128, 40, 6, 2, 3, 20, 1),
    (96, 20, 3, 0, 1, 96, 130), (128, 64, 1, 3, 4, 64, 9)])
def test_experts_with_the_identity_among_them(dtype, width, ff, experts, identity, top, shared, tokens):
    from enginekernel_b200.parts.moe import RoutedExperts
    from enginekernel_b200.parts.spec import PartSpec
    mlp = models.moe(experts, identity, top, ff, shared)
    names = {"router": "router", "correction": "correction"}
    w = {"router": rnd(experts + identity, width, dtype=BF16, seed=1, scale=4 * width ** -0.5),
         "correction": rnd(experts + identity, dtype=BF16, seed=2, scale=0.3)}
    for i, e in enumerate(list(range(experts)) + (["shared"] if shared else [])):
        p, size = (f"e{e}.", ff) if e != "shared" else ("shared.", shared)
        if e != "shared":
            names[f"gate_{e}"], names[f"up_{e}"], names[f"down_{e}"] = p + "gate", p + "up", p + "down"
        w[p + "gate"] = rnd(size, width, dtype=BF16, seed=200 + i, scale=2 * width ** -0.5)
        w[p + "up"] = rnd(size, width, dtype=BF16, seed=10 + i, scale=2 * width ** -0.5)
        w[p + "down"] = rnd(width, size, dtype=BF16, seed=100 + i, scale=size ** -0.5)
    shared_spec = None if not shared else PartSpec(
        "gated_mlp", {"hidden_size": width, "intermediate_size": shared, "activation": "clamped", "limit": 1.3, "name": "shared_expert"},
        {"gate": "shared.gate", "up": "shared.up", "down": "shared.down"})
    part = RoutedExperts(PartSpec("routed_experts", {
        "hidden_size": width, "intermediate_size": ff, "experts": experts, "identity": identity, "top": top,
        "activation": "clamped", "limit": 0.8, "gated": True, "weights": "softmax", "corrected": True,
        "shared": shared_spec}, names), dtype, DEV)
    part.load(w)
    x = rnd(tokens, width, dtype=dtype, seed=5)
    ctx = helpers.make_context(dtype, DEV, list(range(tokens)), [0] * tokens, [0, tokens])
    cpu = {n: v.cpu() for n, v in w.items()}
    for _ in range(2):                                     # a second run finds the scratch of the first
        got = part.forward(x, ctx)
    want = plain.experts_ff(x.double().cpu(), cpu, "", mlp)
    rows = ((got.double().cpu() - want).abs().amax(-1) / want.abs().max()) <= TOL[dtype] * 2
    assert rows.float().mean().item() >= (1.0 if dtype == F32 else 0.97)
    # the choice, the identity and the correction all matter here
    expert, _ = plain.choose(x.double().cpu(), cpu, "", mlp)
    if identity and tokens >= 7:
        assert (expert >= experts).any() and (expert < experts).any()
    if tokens >= 50:
        bare, _ = plain.choose(x.double().cpu(), dict(cpu, correction=torch.zeros(experts + identity)), "", mlp)
        assert (expert.sort(-1).values != bare.sort(-1).values).any()


@pytest.mark.parametrize("n,offset", [(640, 0), (1023, 1), (5, 0), (151936, 2)])
def test_soft_cap_on_logits(n, offset):
    k = K()
    x = rnd(n + offset + 3, seed=1, scale=20.0)
    got = x.clone()
    k.scale_cap_(got[offset:], 0.25, 3.0, n=n)
    want = x.double().cpu()
    want[offset:offset + n] = plain.cap(0.25 * want[offset:offset + n], 3.0)
    assert (got.double().cpu() - want)[offset:offset + n].abs().max() <= 2e-6
    assert torch.equal(got[:offset], x[:offset]) and torch.equal(got[offset + n:], x[offset + n:])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("heads,d,r,e,c,window", [(3, 24, 16, 20, 40, 11), (4, 64, 32, 80, 64, 72), (2, 12, 6, 28, 10, 1),
                                                  (20, 32, 16, 8, 240, 40), (2, 16, 8, 24, 300, 100), (8, 64, 64, 96, 160, None)])
def test_latent_attention_with_plain_queries(dtype, heads, d, r, e, c, window):
    """The part alone, prompt (beyond and up to the rows that share one product), then single tokens, rows of the cache
    narrower and wider than the 16-bit kernels take; sinks and gates that decide."""
    from enginekernel_b200.cache.store import SequenceCache
    from enginekernel_b200.parts.latent_attention import LatentAttention
    from enginekernel_b200.parts.spec import PartSpec
    width, n = 96, 150
    m = models.latent(heads, d, r, e, c, window)["mixer"]
    cfg = models.config(width, 11, [({"type": "latent_attention", "mixer": m}, None)])
    w = {k: t.to(DEV) for k, t in models.make_tensors(cfg, 3).items()}
    p = "l0.mix."
    part = LatentAttention(PartSpec("latent_attention", {
        "hidden_size": width, "num_heads": heads, "head_dim": d, "rot_dim": r, "v_dim": e, "q_rank": None, "kv_rank": c,
        "scale": m["scale"], "eps": 1e-5, "window": window, "pairing": "neighbours", "sink": True, "head_gate": True,
        "position": PartSpec("rope_stretched", {"rotary_dim": r, "theta": 1e4})},
        {"q": p + "q", "dkv": p + "dkv", "dkv_norm": p + "dkv.norm", "uk": p + "uk", "uv": p + "uv", "sink": p + "sink",
         "gate": p + "g", "o": p + "o"}), dtype, DEV)
    part.load(w)
    part.prepare(256)
    x = rnd(n, width, dtype=dtype, seed=5, scale=1.5)
    want = plain.latent_mixer(x.double().cpu(), {k: t.cpu() for k, t in w.items()}, p, m, 1e-5, torch.arange(n))
    tol = TOL[dtype] * (1 if dtype == F32 else 3)
    for cuts in ((n,), (100, 30, 1, 1, 18), (64, 65) + (1,) * 21):
        cache = SequenceCache([part.cache_spec()], dtype, DEV, max_tokens=512, max_slots=2)
        slot, at, rows = cache.open(), 0, []
        for step in cuts:
            cache.reserve(slot, at + step)
            cache.upload_tables()
            ctx = helpers.make_context(dtype, DEV, list(range(at, at + step)), [slot] * step, [0, step], max_context=at + step)
            rows.append(part.forward(x[at:at + step].contiguous(), ctx, cache.entry(0)).clone())
            cache.advance(slot, step)
            at += step
        assert rel(torch.cat(rows), want) <= tol, cuts


# ===================================================================== one-mixer models
def _one_layer(mixer_entry, width, vocab):
    return models.config(width, vocab, [(mixer_entry, None)], logit_softcap=50.0)


ONE_LAYER = {
    # sharp attentions: scores spread over tens, so one key can hold nearly all the weight
    "window": _one_layer(models.attention(4, 2, 24, 40, models.rotation(16, 1e4, (4.0, 128, 8.0, 1.0)), 50, scale=1.0), 96, 600),
    "window_fast": _one_layer(models.attention(4, 2, 128, 128, models.rotation(128, 1e6), 100, scale=0.4), 128, 600),
    "window_64": _one_layer(models.attention(4, 4, 64, 64, models.rotation(16, 1e5, (2.0, 64, 4.0, 1.0)), 64, scale=0.6), 128, 600),
    "no_window": _one_layer(models.attention(6, 1, 40, 12, models.rotation(10), None, scale=0.5), 100, 600),
    "latent": _one_layer(models.latent(4, 32, 16, 24, 48, 72, scale=0.8), 96, 600),
    "latent_page": _one_layer(models.latent(3, 20, 12, 40, 52, 64, scale=0.8), 100, 600),
    "latent_wide": _one_layer(models.latent(2, 32, 32, 16, 288, 90, scale=0.8), 96, 600),
    "retention": _one_layer(models.retention(4, 24, 16, models.rotation(12), [0.99, 0.995, 1.0, 0.5]), 96, 83),
    "retention_wide": _one_layer(models.retention(4, 128, 64, models.rotation(128, 1e6), [0.999, 0.98, 1.0, 0.9]), 128, 83),
    "retention_tall": _one_layer(models.retention(2, 16, 300, models.rotation(16)), 64, 83),
}
SEEN_BY_WINDOW = ["window", "window_fast", "window_64", "no_window", "latent", "latent_page", "latent_wide"]


@pytest.fixture(scope="module")
def one_layer_engines(tmp_path_factory):
    from enginekernel_b200 import Engine
    made = {}

    def get(tag, dtype):
        if (tag, dtype) not in made:
            cfg = ONE_LAYER[tag]
            w = models.make_tensors(cfg, 5)
            folder = models.write_folder(str(tmp_path_factory.mktemp("one_" + tag)), cfg, w)
            made[(tag, dtype)] = (Engine(folder, dtype, max_tokens=2048, max_batch=4), cfg, w)
        return made[(tag, dtype)]
    return get


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", list(ONE_LAYER))
def test_one_mixer_whole_then_token_by_token(one_layer_engines, tag, dtype):
    eng, cfg, w = one_layer_engines(tag, dtype)
    ids = models.random_prompts(cfg, [330], seed=2)[0]
    want = plain.forward(cfg, w, ids)
    tol = helpers.TOL[dtype] * (1 if dtype == "float32" else 2)
    assert helpers.rel_err(helpers.whole(eng, ids), want) <= tol
    assert helpers.rel_err(helpers.tail_one_by_one(eng, ids, 140), want) <= tol       # a window passes over decoded tokens


def _best_key_token(cfg, w, last_token, last_pos, key_pos):
    """The vocabulary token whose key at ``key_pos`` scores highest against the query of ``last_token`` at ``last_pos``
    in some head of layer 0 (from the plain pieces)."""
    layer, eps, v = cfg["layers"][0], cfg["norm"]["eps"], cfg["vocab"]
    m, p = layer["mixer"], "l0.mix."
    make = plain.latent_queries_keys_values if layer["type"] == "latent_attention" else plain.make_queries_keys_values
    h = plain.rms_norm(w["embed"].double(), w, "l0.norm1", eps)
    _, keys, _ = make(h, w, p, m, eps, torch.full((v,), key_pos))
    q = make(h[last_token:last_token + 1], w, p, m, eps, torch.tensor([last_pos]))[0][0]
    s = torch.einsum("hd,vhd->vh", q, keys.repeat_interleave(m["heads"] // keys.shape[1], 1)) * m["scale"]
    s[:v // 2] = -1e9                                       # the prompts are drawn from the lower half
    return int(s.amax(-1).argmax())


@pytest.mark.parametrize("tag", SEEN_BY_WINDOW)
def test_one_key_at_every_edge_decides_or_is_not_seen(one_layer_engines, tag):
    """The token whose key fits the last query best is put at the first places, just inside and just outside the last
    token's window, and on both sides of page borders, among 320 others: the last logits follow it where the plain
    rule sees it, in a prompt and when the last tokens are decoded alone."""
    eng, cfg, w = one_layer_engines(tag, "float32")
    n, window = 320, (cfg["layers"][0]["mixer"].get("mask") or {}).get("size")
    a = [t % (cfg["vocab"] // 2) for t in models.random_prompts(cfg, [n], seed=3)[0]]
    wa = plain.forward(cfg, w, a)[-1]
    runs = (helpers.whole, lambda e, ids: helpers.tail_one_by_one(e, ids, 3))
    ga = [run(eng, a)[-1] for run in runs]
    edges = {0, 1, 63, 64, 255, 256, n - 2}
    if window:
        edges |= {n - window - 1, n - window, n - window + 1}
    moved = {}
    for key_pos in sorted(edges & set(range(n - 1))):
        b = list(a)
        b[key_pos] = _best_key_token(cfg, w, a[-1], n - 1, key_pos)         # a token that is nowhere else
        wb = plain.forward(cfg, w, b)[-1]
        moved[key_pos] = (float((wa - wb).abs().max() / wa.abs().max()), plain.sees(n - 1, key_pos, window))
        for run, base in zip(runs, ga):
            gb = run(eng, b)[-1]
            assert helpers.rel_err(gb, wb) <= helpers.TOL["float32"], key_pos
            assert (base - gb - (wa - wb).float()).abs().max().item() <= 1e-3 * float((wa - wb).abs().max()) + 2e-5 * float(wa.abs().max()), key_pos
    # the test's weights do what they are made for: a seen key moves the logits, an unseen one does not
    assert min(m for m, seen in moved.values() if seen) > 1e-3, moved
    if window:
        assert max(m for m, seen in moved.values() if not seen) < 1e-9, moved


@pytest.mark.parametrize("tag", ["retention", "retention_wide"])
@pytest.mark.parametrize("changed", [0, 63, 64, 300, 318])
def test_one_changed_token_moves_the_last_logits(one_layer_engines, tag, changed):
    """What the state carries of one changed token moves the logits at the end in the engine as in the plain model."""
    eng, cfg, w = one_layer_engines(tag, "float32")
    a = models.random_prompts(cfg, [320], seed=3)[0]
    b = list(a)
    b[changed] = (a[changed] + 1) % cfg["vocab"]
    wa, wb = plain.forward(cfg, w, a)[-1], plain.forward(cfg, w, b)[-1]
    assert (wa - wb).abs().max() > 1e-4 * wa.abs().max()
    for run in (helpers.whole, lambda e, ids: helpers.tail_one_by_one(e, ids, 3)):
        ga, gb = run(eng, a)[-1], run(eng, b)[-1]
        assert (ga - gb - (wa - wb).float()).abs().max().item() <= 2e-2 * float((wa - wb).abs().max()) + 2e-5 * float(wa.abs().max())


@pytest.mark.parametrize("tag", ["window", "window_fast", "latent", "latent_wide"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_sink_left_out_would_show(one_layer_engines, tag, dtype):
    """Sinks as large as the scores: the first tokens' logits follow the plain model, and without sinks they would not."""
    eng, cfg, w = one_layer_engines(tag, dtype)
    ids = models.random_prompts(cfg, [6], seed=12)[0]
    want = plain.forward(cfg, w, ids)
    without = plain.forward(cfg, dict(w, **{"l0.mix.sink": torch.full_like(w["l0.mix.sink"], -1e4)}), ids)
    tol = helpers.TOL[dtype] * (1 if dtype == "float32" else 2)
    for got in (helpers.whole(eng, ids), helpers.tail_one_by_one(eng, ids, 5)):
        assert helpers.rel_err(got, want) <= tol
    assert helpers.rel_err(without, want) > 0.05


# ===================================================================== whole models
TAGS = list(models.SHAPES)
SEEDS = {"early": 11, "flat": 12, "odd": 13, "wide": 14}
# in bfloat16 a router's score can round the other way than in 64-bit, and a row then takes another expert
ALLOWED = {"float32": 1.0, "bfloat16": 0.9}


@pytest.fixture(scope="module")
def weights():
    return {tag: models.make_tensors(cfg, SEEDS[tag]) for tag, cfg in models.SHAPES.items()}


@pytest.fixture(scope="module")
def engines(tmp_path_factory, weights):
    from enginekernel_b200 import Engine
    made = {}

    def get(tag, dtype):
        if (tag, dtype) not in made:
            folder = models.write_folder(str(tmp_path_factory.mktemp("gesuvik_" + tag)), models.SHAPES[tag], weights[tag])
            made[(tag, dtype)] = Engine(folder, dtype, max_tokens=4096, max_batch=8)
        return made[(tag, dtype)]
    return get


def close(got, want, dtype, what=""):
    got, want = got.double().cpu(), want.double().cpu()
    err = (got - want).abs().amax(-1) / want.abs().max()
    limit = helpers.TOL[dtype] * (3 if dtype == "bfloat16" else 1)
    inside = (err <= limit).sum().item()
    assert inside >= ALLOWED[dtype] * err.numel() or err.numel() - inside <= (1 if dtype == "bfloat16" else 0), \
        f"{what} {dtype}: {inside} of {err.numel()} rows within {limit}, worst {err.max():.3e}"
    if dtype == "bfloat16" and err.numel() >= 3:
        assert err.median().item() <= helpers.TOL[dtype], f"{what}: median {err.median():.3e}"


_WANT = {}


def want_logits(weights, tag, ids):
    key = (tag, tuple(ids))
    if key not in _WANT:
        _WANT[key] = plain.forward(models.SHAPES[tag], weights[tag], ids)
    return _WANT[key]


def in_portions(engine, tokens, sizes):
    slot = engine.open_sequence()
    try:
        rows, at = [], 0
        for n in list(sizes) + [len(tokens)]:
            part = tokens[at:at + n]
            if not part:
                break
            rows.append(engine.step([(slot, part, list(range(len(part))))]).cpu())
            at += len(part)
        return torch.cat(rows, 0)
    finally:
        engine.close_sequence(slot)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", TAGS)
def test_whole_prompts(engines, weights, tag, dtype):
    eng = engines(tag, dtype)
    for j, n in enumerate((1, 2, 7, 33, 64, 65, 130, 260)):
        ids = models.random_prompts(models.SHAPES[tag], [n], seed=40 + j)[0]
        close(helpers.whole(eng, ids), want_logits(weights, tag, ids), dtype, f"{tag} length {n}")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", TAGS)
def test_prompt_then_token_by_token(engines, weights, tag, dtype):
    eng = engines(tag, dtype)
    ids = models.random_prompts(models.SHAPES[tag], [150], seed=77)[0]
    got = helpers.tail_one_by_one(eng, ids, 80)
    close(got, want_logits(weights, tag, ids), dtype, tag)
    if dtype == "float32":
        assert helpers.rel_err(got, helpers.whole(eng, ids)) <= 1e-5


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", TAGS)
def test_prompts_in_portions(engines, weights, tag, dtype):
    eng = engines(tag, dtype)
    ids = models.random_prompts(models.SHAPES[tag], [210], seed=78)[0]
    want = want_logits(weights, tag, ids)
    for sizes in ((2, 2, 2, 3, 17), (64, 64, 2), (63, 2, 65), (1, 127, 2), (129,)):
        close(in_portions(eng, ids, sizes), want, dtype, f"{tag} portions {sizes}")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", TAGS)
def test_unequal_batches_and_reuse(engines, weights, tag, dtype):
    """Requests of unequal lengths start together and end at different steps; three such batches in a row through the
    same few slots, pages and states, then everything is free again."""
    eng = engines(tag, dtype)
    shapes = [((5, 9, 13), (3, 9, 1)), ((1, 70, 31, 16), (1, 64, 20, 16)), ((66, 2, 140), (65, 1, 100))]
    for j, (lens, heads) in enumerate(shapes):
        seqs = models.random_prompts(models.SHAPES[tag], lens, seed=200 + j)
        got = helpers.batch_then_steps(eng, seqs, heads)
        for ids, g in zip(seqs, got):
            close(g, want_logits(weights, tag, ids), dtype, f"{tag} batch {j} length {len(ids)}")
            if dtype == "float32":                       # what else is in the batch does not matter beyond rounding
                assert helpers.rel_err(g, helpers.whole(eng, ids)) <= 1e-5
    assert eng.cache.book.open_slots() == []
    assert eng.cache.free_tokens() == eng.cache.num_pages * 64


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", ["odd", "early"])
def test_first_tokens_one_by_one(engines, weights, tag, dtype):
    eng = engines(tag, dtype)
    ids = models.random_prompts(models.SHAPES[tag], [7], seed=5)[0]
    close(helpers.tail_one_by_one(eng, ids, tail=6), want_logits(weights, tag, ids), dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", ["early", "flat"])
def test_long_decoding(engines, weights, tag, dtype):
    """Pages in front of the windows go back while the sequence grows, and are used again."""
    eng = engines(tag, dtype)
    ids = models.random_prompts(models.SHAPES[tag], [300], seed=9)[0]
    close(helpers.tail_one_by_one(eng, ids, tail=290), want_logits(weights, tag, ids), dtype, tag)


def test_a_step_too_large_for_one_pass_is_cut(tmp_path, weights):
    from enginekernel_b200 import Engine
    cfg = models.SHAPES["early"]
    eng = Engine(models.write_folder(str(tmp_path / "m"), cfg, weights["early"]), "float32", max_tokens=1024, max_batch=4)
    eng.runner.max_step_tokens = 50
    seqs = models.random_prompts(cfg, (70, 33), seed=6)
    slots = [eng.open_sequence() for _ in seqs]
    got = eng.step([(s, t, list(range(len(t)))) for s, t in zip(slots, seqs)]).cpu()
    close(got[:70], want_logits(weights, "early", seqs[0]), "float32")
    close(got[70:], want_logits(weights, "early", seqs[1]), "float32")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("tag", ["early", "wide"])
def test_greedy_generation_through_the_scheduler(tmp_path, tag, dtype):
    """``Engine.generate_all``: five requests of unequal lengths through two slots, so the scheduler forms several
    batches and the captured decode step runs on slots, states and pages used before."""
    from enginekernel_b200 import Engine
    cfg = models.SHAPES[tag]
    w = models.make_tensors(cfg, 21)
    folder = models.write_folder(str(tmp_path / "m"), cfg, w)
    eng = Engine(folder, dtype, max_tokens=2048, max_batch=2)
    prompts = models.random_prompts(cfg, [3, 70, 17, 64, 1], seed=8)
    got = eng.generate_all(prompts, 12)
    distinct = set()
    for ids, out in zip(prompts, got):
        assert len(out) == 12
        want = plain.greedy(cfg, w, ids, 12)
        distinct.update(want)
        if dtype == "float32":
            assert out == want
    assert len(distinct) > 3
    assert eng.cache.book.open_slots() == []
    eager = Engine(folder, dtype, max_tokens=2048, max_batch=2, use_graph=False)
    assert eager.generate_all(prompts, 12) == got             # without the captured graph: the same tokens


def test_unused_tensors_and_missing_ones(tmp_path):
    """A layer without experts may still carry its second norm; a file that lacks a tensor is refused by name, and so is
    one that holds tensors for a layer that runs on another's."""
    from enginekernel_b200 import Engine
    from enginekernel_b200.weights.checkpoint import WeightsError
    cfg = models.SHAPES["early"]
    w = models.make_tensors(cfg, 2)
    w["l1.norm2"] = torch.zeros(cfg["width"], dtype=BF16)
    eng = Engine(models.write_folder(str(tmp_path / "a"), cfg, w), "float32", max_tokens=256, max_batch=2)
    ids = models.random_prompts(cfg, [20], seed=1)[0]
    assert helpers.rel_err(helpers.whole(eng, ids), plain.forward(cfg, w, ids)) <= helpers.TOL["float32"]
    for name in ("l0.mix.sink", "l0.mix.g", "l0.mix.dkv.norm", "l1.mix.v", "l2.mix.k.norm", "l2.mlp.correction", "l0.mlp.e3.up"):
        less = dict(w)
        del less[name]
        with pytest.raises(WeightsError, match=name):
            Engine(models.write_folder(str(tmp_path / ("b" + name)), cfg, less), "float32", max_tokens=256, max_batch=2)
    with pytest.raises(WeightsError, match="l3.mix.uk"):
        Engine(models.write_folder(str(tmp_path / "c"), cfg, dict(w, **{"l3.mix.uk": w["l0.mix.uk"].clone()})), "float32",
               max_tokens=256, max_batch=2)


def test_command_line_and_trace_replay(tmp_path):
    """``random-model`` writes a Gesuvik folder from a configuration file, ``generate`` prints the plain model's greedy
    tokens for it, and ``bin/trace_run`` replays steps over the same folder."""
    import os
    import subprocess
    import sys

    import numpy as np
    from safetensors import safe_open
    from tests.test_cli_gpu import ROOT, run_cli
    cfg = models.SHAPES["flat"]
    config_file = tmp_path / "config.json"
    config_file.write_text(json.dumps(cfg))
    folder = tmp_path / "model"
    run_cli("random-model", "--config", str(config_file), "--seed", "5", "--out", str(folder))
    with safe_open(str(folder / "model.safetensors"), framework="pt", device="cpu") as f:
        w = {name: f.get_tensor(name) for name in f.keys()}
    assert {n: tuple(t.shape) for n, t in w.items()} == models.tensor_shapes(cfg)
    prompts = models.random_prompts(cfg, (3, 40), seed=4)
    ids = ";".join(",".join(str(t) for t in p) for p in prompts)
    out = run_cli("generate", "--model", str(folder), "--dtype", "float32", "--prompt-ids", ids, "--out-len", "5")
    rows = [json.loads(line) for line in out.strip().splitlines()]
    assert [r["tokens"] for r in rows] == [plain.greedy(cfg, w, p, 5) for p in prompts]

    steps = [{"step": 0, "entries": [{"id": "a", "tokens": prompts[1][:30], "want": [0, 29]},
                                     {"id": "b", "tokens": prompts[0][:1], "want": []}], "end": []},
             {"step": 1, "entries": [{"id": "a", "tokens": prompts[1][30:31], "want": [0]},
                                     {"id": "b", "tokens": prompts[0][1:2], "want": [0]}], "end": ["b"]},
             {"step": 2, "entries": [{"id": "a", "tokens": prompts[1][31:32], "want": [0]}], "end": ["a"]}]
    out_dir = tmp_path / "out"
    p = subprocess.run([sys.executable, os.path.join(ROOT, "bin", "trace_run"), "--model", str(folder), "--dtype",
                        "float32", "--out", str(out_dir), "--max-tokens", "128"],
                       input="".join(json.dumps(s) + "\n" for s in steps), capture_output=True, text=True,
                       timeout=900)
    assert p.returncode == 0, p.stderr[-2000:]
    assert [l for l in p.stdout.splitlines() if l.startswith("done")] == ["done 0", "done 1", "done 2"]
    a, b = plain.forward(cfg, w, prompts[1][:32]), plain.forward(cfg, w, prompts[0][:2])
    want = {0: torch.stack([a[0], a[29]]), 1: torch.stack([a[30], b[1]]), 2: a[31:32]}
    for n, rows_wanted in want.items():
        got = torch.from_numpy(np.fromfile(str(out_dir / f"{n}.f32"), dtype="<f4").reshape(rows_wanted.shape))
        assert helpers.rel_err(got, rows_wanted) <= helpers.TOL["float32"], n
