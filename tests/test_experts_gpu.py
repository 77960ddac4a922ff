"""The experts' products on pairs of SMs (wide plans) against the plain formulas."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _activation(name, g, u, limit):
    if name == "clamped":
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    f = {"silu": torch.nn.functional.silu, "gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh"),
         "relu2": lambda z: torch.relu(z).square(), "none": lambda z: z}[name]
    return f(g) if u is None else f(g) * u


@pytest.mark.parametrize("hidden,inter,top", [(264, 72, 3), (256, 136, 1), (72, 520, 2)])
@pytest.mark.parametrize("act,gated,weigh", [("silu", True, "output"), ("clamped", True, "input"), ("gelu_tanh", True, "input"),
                                             ("relu2", False, "output"), ("none", False, "input")])
@pytest.mark.parametrize("gather", [False, True])
def test_wide_expert_products(monkeypatch, hidden, inter, top, act, gated, weigh, gather):
    """Experts with 0, 1, 31, 32, 33, 255, 256, 257 and 600 pairs, and pairs that name no expert of the plan; sizes that
    fill no tile.  Operands are bfloat16, sums 32-bit: the up result is one rounding (2^-9) from the plain one, with the
    sum's own error (a few 2^-24 of its terms' norm) beside it; the down result has the 32-bit sum's error alone."""
    from enginekernel_b200.ops import kernels as k
    counts = [0, 1, 31, 32, 33, 255, 256, 257, 600]
    e = len(counts)
    pairs = -(-(sum(counts) + 7) // top) * top
    owner = torch.cat([torch.full((n,), i) for i, n in enumerate(counts)])
    owner = torch.cat([owner, torch.full((pairs - owner.numel(),), e + 1)])       # choices without weights
    g = torch.Generator().manual_seed(hidden + inter)
    owner = owner[torch.randperm(pairs, generator=g)]
    rnd = lambda *s: torch.randn(*s, generator=g)
    x = rnd(pairs // top, hidden).bfloat16().to(DEV)
    w_up = (rnd(e, (2 if gated else 1) * inter, hidden) * 0.1).bfloat16().to(DEV)
    w_down = (rnd(e, hidden, inter) * 0.1).bfloat16().to(DEV)
    weight = torch.rand(pairs, generator=g).to(DEV)
    chosen = owner.to(torch.int32).to(DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    order = torch.empty(pairs, **i32)
    tiles, n_tiles = torch.empty(k.moe_max_tiles(pairs, e, True), 3, **i32), torch.empty(1, **i32)
    k.moe_plan(order, tiles, n_tiles, chosen, pairs, e, wide=True)
    plan = tiles[:int(n_tiles)].cpu().tolist()
    assert [sum(r for ee, _, r in plan if ee == i) for i in range(e)] == counts and max(r for _, _, r in plan) <= 256
    monkeypatch.setattr(k, "MOE_GATHER_PAIRS", 0 if gather else 1 << 30)
    assert k.moe_on_pairs(x, w_up, w_down)
    act_out = torch.full((pairs, inter), 7.0, dtype=torch.bfloat16, device=DEV)
    pair_out = torch.full((pairs, hidden), 7.0, device=DEV)
    k.moe_expert_up(act_out, x, w_up, tiles, n_tiles, order, pairs, top, act, gated=gated, limit=1.5,
                    input_weight=weight if weigh == "input" else None, wide=True, scratch=pair_out)
    pair_out.fill_(7.0)
    k.moe_expert_down(pair_out, act_out, w_down, tiles, n_tiles, order, weight if weigh == "output" else None, pairs,
                      wide=True)
    k.check_tc_status(DEV)
    real = sum(counts)
    assert torch.equal(act_out[real:], torch.full_like(act_out[real:], 7.0))
    row_pair = order[:real].long()
    assert torch.equal(owner.to(DEV)[row_pair], torch.sort(owner[owner < e]).values.to(DEV))
    for i in range(e):
        rows = (owner.to(DEV)[row_pair] == i).nonzero()[:, 0]
        if not rows.numel():
            continue
        p = row_pair[rows]
        z = x[p // top].double() @ w_up[i].double().t()
        if weigh == "input":
            z = z * weight[p, None].double()
        want = _activation(act, z[:, 0::2], z[:, 1::2], 1.5) if gated else _activation(act, z, None, 0)
        got = act_out[rows].double()
        # (relu2 and the gated forms multiply two such sums)
        assert ((got - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all(), (i, (got - want).abs().max())
        down = got @ w_down[i].double().t() * (weight[p, None].double() if weigh == "output" else 1)
        assert (pair_out[p].double() - down).abs().max() <= 1e-5 * down.abs().max()
    assert (pair_out[owner.to(DEV) > e] == 7.0).all()
