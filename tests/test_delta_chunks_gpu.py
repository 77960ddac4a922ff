"""The delta rule by chunks, and the kernels that feed it with many tokens, against the plain recurrence in 64 bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
F64 = torch.float64


def K():
    from enginekernel_b200.ops import kernels
    return kernels


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def rel(got, want):
    return (got.double() - want).abs().max().item() / want.abs().max().item()


def _walk(q, k, v, beta, g, s):
    """Token by token: q, k, g [T, H, d], v [T, H, e], beta [T, H], s [H, e, d]."""
    s, out = s.transpose(1, 2).clone(), []
    for t in range(q.shape[0]):
        s = s * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - (s * k[t][:, :, None]).sum(1))
        s = s + k[t][:, :, None] * u[:, None, :]
        out.append((s * q[t][:, :, None]).sum(1))
    return torch.stack(out), s.transpose(1, 2)


@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(2, 1, 64, 4), (3, 3, 128, 20), (4, 2, 128, 128), (1, 1, 64, 128),
                                                     (2, 2, 128, 256)])
@pytest.mark.parametrize("decays", ["mild", "strong", "zero", "per head"])
def test_delta_rule_by_chunks(heads, kv_heads, dim, vdim, decays):
    """Sequences of 1, 31, 32, 33 and 97 tokens and a finished one, from carried states, in slots out of order.  Sums of
    up to 128 + 32 terms in 32-bit, in another order than token by token: 2e-5 of the largest value, the bound the walk
    token by token is held to.  Decays of 0 and products that vanish divide nothing; an infinite value reaches no
    earlier token and no other column."""
    k = K()
    from enginekernel_b200.parts.base import Workspace
    lens, dead = [33, 1, 97, 31, 32, 5], 5
    t, n = sum(lens), len(lens)
    g_ = torch.Generator().manual_seed(dim + vdim)
    rnd = lambda *s: torch.randn(*s, generator=g_)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, kk, v = unit(rnd(t, kv_heads, dim)) * dim ** -0.5, unit(rnd(t, kv_heads, dim)), rnd(t, heads, vdim)
    beta = torch.rand(t, heads, generator=g_)
    per_head = decays == "per head"
    decay = torch.rand(t, heads, 1 if per_head else dim, generator=g_)
    decay = decay ** 0.1 if decays in ("mild", "per head") else decay ** 40
    if decays == "zero":
        decay[::7] = 0
    q, kk, v, beta, decay = (x.to(DEV) for x in (q, kk, v, beta, decay))
    slots = [4, 0, 6, 2, 1, 3]
    per_slot = heads * vdim * dim + 8
    start = (rnd(7, per_slot) * 0.3).to(DEV)
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    pos = [(-1 if b == dead else 10 + j) for b, m in enumerate(lens) for j in range(m)]
    slot = [slots[b] for b, m in enumerate(lens) for _ in range(m)]

    def run(values):
        state, out = start.clone(), torch.full((t, heads * vdim), 7.0, device=DEV)
        assert k.delta_by_chunks(k.DELTA_CHUNK_TOKENS * n, n, dim, vdim)
        k.delta_scan(out, q.reshape(t, -1).contiguous(), kk.reshape(t, -1).contiguous(), values.reshape(t, -1).clone(), beta,
                     decay.reshape(t, -1).clone(), state, i32(cu), i32(pos), i32(slot), n, heads, kv_heads, dim, vdim,
                     n_tokens=t, decay_per_head=per_head, workspace=Workspace(torch.device(DEV)))
        return out.view(t, heads, vdim), state

    k.DELTA_CHUNK_TOKENS, before = 1, k.DELTA_CHUNK_TOKENS
    try:
        out, state = run(v)
        v2 = v.clone()
        v2[cu[2] + 40, 0, 1] = float("inf")
        spoilt, _ = run(v2)
    finally:
        k.DELTA_CHUNK_TOKENS = before
    rep = heads // kv_heads
    for b in range(n):
        rows, s0 = slice(cu[b], cu[b + 1]), start[slots[b], :-8].view(heads, vdim, dim)
        if b == dead:
            assert torch.equal(out[rows], torch.full_like(out[rows], 7.0)) and torch.equal(state[slots[b]], start[slots[b]])
            continue
        want, s = _walk(q[rows].double().repeat_interleave(rep, 1), kk[rows].double().repeat_interleave(rep, 1),
                        v[rows].double(), beta[rows].double(), decay[rows].double().expand(-1, heads, dim), s0.double())
        assert rel(out[rows], want) <= 2e-5 and rel(state[slots[b], :-8].view_as(s), s) <= 2e-5
    assert torch.equal(state[:, -8:], start[:, -8:]) and torch.equal(state[5], start[5])
    first = cu[2] + 40
    keep = torch.ones_like(out, dtype=torch.bool)
    keep[first:cu[3], 0, 1] = False
    assert torch.equal(spoilt[keep], out[keep])


@pytest.mark.parametrize("per_head", [False, True])
def test_a_sequence_alone_in_company_and_in_portions(per_head):
    """The form of the recurrence goes by a step's tokens a sequence, and chunks start at a step's first token: one sequence
    of 300 tokens alone (chunks), beside five of 9 tokens (token by token), beside one of 200 (chunks), and in portions of
    130, 70 and 100 tokens.  What differs is the order of 32-bit sums: each run is within 2e-7 (2-norm) of 64 bits, so two
    runs are within 1e-6 of one another."""
    from enginekernel_b200.parts.base import Workspace
    k, heads, kv_heads, dim, vdim, n = K(), 4, 2, 128, 128, 300
    g_ = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g_)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    t = n + 200
    q, kk, v = unit(rnd(t, kv_heads, dim)) * dim ** -0.5, unit(rnd(t, kv_heads, dim)), rnd(t, heads, vdim)
    beta, decay = torch.rand(t, heads, generator=g_), torch.rand(t, heads, 1 if per_head else dim, generator=g_) ** 0.1
    q, kk, v, beta, decay = (x.reshape(t, -1).to(DEV) for x in (q, kk, v, beta, decay))
    start = (rnd(8, heads * vdim * dim) * 0.3).to(DEV)

    def run(lens, first, state):
        """A step of sequences of these tokens, the first one's from ``first`` on, the others' behind token 300."""
        rows, at = list(range(first, first + lens[0])), n
        for m in lens[1:]:
            rows += range(at, at + m)
            at += m
        cu, slot, pos = [0], [], []
        for b, m in enumerate(lens):
            cu.append(cu[-1] + m)
            slot += [b] * m
            pos += [j + (first if b == 0 else 0) for j in range(m)]
        out = torch.empty(len(rows), heads * vdim, device=DEV)
        args = [x[rows].contiguous() for x in (q, kk, v, beta, decay)]
        k.delta_scan(out, *args, state, i32(cu), i32(pos), i32(slot), len(lens), heads, kv_heads, dim, vdim, n_tokens=len(rows),
                     decay_per_head=per_head, workspace=Workspace(torch.device(DEV)))
        return out[:lens[0]]

    runs = []
    for steps in ([[n]], [[n] + [9] * 5], [[n, 200]], [[130], [70], [100]]):
        state, first, outs = start.clone(), 0, []
        for lens in steps:
            outs.append(run(lens, first, state))
            first += lens[0]
        runs.append((torch.cat(outs), state[0]))
    assert k.delta_by_chunks(n, 1, dim, vdim) and not k.delta_by_chunks(n + 45, 6, dim, vdim) and k.delta_by_chunks(t, 2, dim, vdim)
    far = lambda got, want: ((got.double() - want.double()).norm() / want.double().norm()).item()
    for out, state in runs[1:]:
        assert far(out, runs[0][0]) <= 1e-6 and far(state, runs[0][1]) <= 1e-6


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("heads,kv_heads,dim,vdim", [(8, 8, 40, 24), (12, 4, 64, 100)])
def test_convolution_and_unit_vectors_of_many_tokens(heads, kv_heads, dim, vdim, taps):
    """Tiles of eight tokens over sequences of 1, 2, 3, 170 and 30 tokens, some behind earlier inputs, some finished:
    the same values as the plain formulas to a few 32-bit roundings."""
    k = K()
    lens, first = [1, 2, 170, 3, 30], [0, 5, 0, 1, 7]
    t, ch = sum(lens), 2 * kv_heads * dim + heads * vdim
    g = torch.Generator().manual_seed(taps)
    proj = torch.randn(t, ch + heads + 3, generator=g).to(DEV)
    w = torch.randn(ch, taps, generator=g).to(DEV)
    s_values = 16
    state = torch.randn(5, s_values + ch * (taps - 1), generator=g).to(DEV)
    pos = [p for n, p0 in zip(lens, first) for p in range(p0, p0 + n)]
    slot = [s for s, n in enumerate(lens) for _ in range(n)]
    pos[-4:] = [-1] * 4
    outs = [torch.full(s, 7.0, device=DEV) for s in ((t, kv_heads * dim), (t, kv_heads * dim), (t, heads * vdim), (t, heads))]
    k.delta_prepare(*outs, proj, t, w, state, s_values, i32(pos), i32(slot), (heads, kv_heads, dim, vdim, taps, 1, 1))
    cu = 0
    x64, w64 = proj.double(), w.double()
    for s, n in enumerate(lens):
        tail = state[s, s_values:].view(ch, taps - 1).t().double()
        x = torch.cat([tail, x64[cu:cu + n, :ch]])
        y = sum(x[j:j + n] * w64[:, j] for j in range(taps))
        y = y * torch.sigmoid(y)
        live = n - 4 if s == len(lens) - 1 else n
        cq = kv_heads * dim
        unit = lambda z: (z.view(n, kv_heads, dim) / torch.sqrt((z.view(n, kv_heads, dim) ** 2).sum(-1, keepdim=True) + 1e-6)).reshape(n, -1)
        for got, want in zip(outs, (unit(y[:, :cq]) * dim ** -0.5, unit(y[:, cq:2 * cq]), y[:, 2 * cq:],
                                    torch.sigmoid(x64[cu:cu + n, ch:ch + heads]))):
            assert rel(got[cu:cu + live], want[:live]) <= 2e-6
            assert torch.equal(got[cu + live:cu + n], torch.full_like(got[cu + live:cu + n], 7.0))
        cu += n


@pytest.mark.parametrize("channels,rank,tokens", [(1024, 64, 1200), (1028, 7, 1500), (516, 130, 2401)])
def test_low_rank_halves_of_many_tokens(channels, rank, tokens):
    """Four channels a thread: ranks that are no multiple of 4, channels that fill no tile.  Sums of `rank` products of
    32-bit values of size one: 1e-6 of what comes out."""
    k = K()
    g = torch.Generator().manual_seed(rank)
    proj = torch.randn(tokens, rank + 9, generator=g).to(DEV)
    w = (torch.randn(rank, channels, generator=g) * rank ** -0.5).to(DEV)
    bias, a_log = torch.randn(channels, generator=g).to(DEV), torch.randn(4, generator=g).to(DEV)
    out = torch.empty(tokens, channels, device=DEV)
    z = proj[:, 5:5 + rank].double() @ w.double()
    k.delta_low_rank(out, proj, tokens, 5, w)
    assert (out.double() - torch.sigmoid(z)).abs().max() <= 2e-6
    k.delta_low_rank(out, proj, tokens, 5, w, bias=bias, a_log=a_log, dim=-(-channels // 4))
    rate = torch.exp(a_log.double())[torch.arange(channels, device=DEV) // -(-channels // 4)]
    assert (out.double() - torch.exp(-rate * torch.nn.functional.softplus(z + bias.double()))).abs().max() <= 4e-6


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels,col0,in_bias,act", [(1024, 0, False, True), (1027, 3, True, False), (516, 8, True, True)])
def test_convolution_of_many_tokens_with_biases(channels, col0, in_bias, act, taps):
    """Tiles of eight tokens, four channels a thread and one, over sequences of 1, 2, 1,300, 3 and 1,900 tokens, some behind
    earlier inputs, some finished: the plain formulas to a few 32-bit roundings of sums of five terms."""
    k = K()
    lens, first = [1, 2, 1300, 3, 1900], [0, 5, 0, 1, 7]
    t = sum(lens)
    g = torch.Generator().manual_seed(taps)
    proj = torch.randn(t, channels + col0 + 4 - (channels + col0) % 4, generator=g).to(DEV)
    w, b, xb = (torch.randn(*s, generator=g).to(DEV) for s in ((channels, taps), (channels,), (channels,)))
    state = torch.randn(5, 16 + channels * (taps - 1), generator=g).to(DEV)
    pos = [p for n, p0 in zip(lens, first) for p in range(p0, p0 + n)]
    slot = [s for s, n in enumerate(lens) for _ in range(n)]
    pos[-4:] = [-1] * 4
    out = torch.full((t, channels), 7.0, device=DEV)
    k.conv_act(out, proj, col0, w, b, state, 16, i32(pos), i32(slot), t, channels, taps, in_bias=xb if in_bias else None,
               activation="silu" if act else None)
    cu = 0
    for s, n in enumerate(lens):
        live = n - 4 if s == len(lens) - 1 else n
        x = torch.cat([state[s, 16:].view(channels, taps - 1).t(), proj[cu:cu + n, col0:col0 + channels]]).double()
        if in_bias:                              # inputs before position 0 do not belong to a token
            x[max(0, taps - 1 - first[s]):] += xb.double()
        y = sum(x[j:j + n] * w[:, j].double() for j in range(taps)) + b.double()
        y = y * torch.sigmoid(y) if act else y
        assert rel(out[cu:cu + live], y[:live]) <= 2e-6
        assert torch.equal(out[cu + live:cu + n], torch.full_like(out[cu + live:cu + n], 7.0))
        cu += n


@pytest.mark.parametrize("inner,vdim,parts", [(512, 64, 1), (520, 20, 2), (768, 4, 1), (96, 32, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_state_space_output_norm(inner, vdim, parts, offset):
    """Four channels a thread, and one by one where the gate's column is not on a 16-byte boundary: 32-bit results to a few
    roundings."""
    k = K()
    t = 40
    g = torch.Generator().manual_seed(inner)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    o, x, proj, d, w = rnd(t, inner), rnd(t, inner + 8), rnd(t, inner + 12), rnd(inner // vdim), rnd(inner)
    y = torch.empty(t, inner, device=DEV)
    k.ssm_out(y, o, x, proj, offset, d, w, 1e-5, i32(list(range(t))), t, inner, vdim, parts)
    z = proj[:, offset:offset + inner].double()
    u = (o.double() + d.double().repeat_interleave(vdim) * x[:, :inner].double()) * z * torch.sigmoid(z)
    p = u.view(t, parts, -1)
    want = (p * torch.rsqrt((p * p).mean(-1, keepdim=True) + 1e-5)).reshape(t, inner) * w.double()
    assert rel(y, want) <= 2e-6
