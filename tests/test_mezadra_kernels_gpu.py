"""The kernels that came with the Mezadra decoder, one by one, against plain PyTorch float32."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

DEVICE = "cuda:0"


def _silu(x):
    return x * torch.sigmoid(x)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,experts,top,hidden,inter", [(300, 40, 3, 64, 24), (37, 5, 2, 50, 22), (1, 3, 3, 32, 8), (200, 1, 1, 40, 16),
                                                             (150, 2, 2, 200, 72)])
def test_products_over_pairs_grouped_by_expert(tokens, experts, top, hidden, inter, dtype, wide):
    """Given choices and weights, plan + gated product + down product + sum equal the experts run pair by pair; on the
    plain tiles and on the pipelined bfloat16 ones (``wide``; inner sizes that are no multiples of their chunk too)."""
    from rapid_llm_b200.ops import kernels

    if wide and not kernels.moe_wide_takes(dtype, hidden, inter):
        pytest.skip("the pipelined tiles take bfloat16 with 16-byte rows")

    g = torch.Generator().manual_seed(tokens + experts)
    x = torch.randn(tokens, hidden, generator=g).to(dtype).to(DEVICE)
    gate_up = (torch.randn(experts, 2 * inter, hidden, generator=g) / hidden ** 0.5).to(dtype).to(DEVICE)
    down = (torch.randn(experts, hidden, inter, generator=g) / inter ** 0.5).to(dtype).to(DEVICE)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(tokens)]).to(torch.int32).to(DEVICE)
    weights = torch.rand(tokens, top, generator=g).to(DEVICE)
    shared = torch.randn(tokens, hidden, generator=g).to(dtype).to(DEVICE)
    gate = torch.rand(tokens, 1, generator=g).to(DEVICE)
    fault = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    pairs = tokens * top
    order = torch.empty(pairs, dtype=torch.int32, device=DEVICE)
    place = torch.empty(pairs, dtype=torch.int32, device=DEVICE)
    meta = torch.zeros(1 + 3 * kernels.moe_max_tiles(pairs, experts, wide), dtype=torch.int32, device=DEVICE)
    max_tiles = kernels.moe_plan(ids, experts, order, place, meta, fault, wide=wide)
    act = torch.empty(pairs, inter, dtype=dtype, device=DEVICE)
    kernels.grouped_linear(x, gate_up, order, meta, top=top, by_token=True, max_tiles=max_tiles, pair_weight=weights.view(-1), out_act=act, wide=wide)
    each = torch.full((pairs, hidden), float("nan"), device=DEVICE)
    kernels.grouped_linear(act, down, order, meta, top=top, by_token=False, max_tiles=max_tiles, out_y=each, wide=wide)
    out = torch.empty(tokens, hidden, dtype=dtype, device=DEVICE)
    kernels.moe_combine(each, top, out, shared=shared, gate=gate)
    assert int(fault.item()) == 0
    # every pair has one place, and the places of an expert are consecutive
    assert sorted(order.tolist()) == list(range(pairs))
    assert torch.equal(order[place.long()].cpu(), torch.arange(pairs, dtype=torch.int32))
    by_place = ids.view(-1)[order.long()].tolist()
    assert by_place == sorted(by_place)
    want = torch.zeros(tokens, hidden, device=DEVICE)
    xf, wf, df = x.float(), gate_up.float(), down.float()
    for t in range(tokens):
        for j in range(top):
            e, w = int(ids[t, j]), weights[t, j]
            wide = wf[e] @ xf[t]
            a = _silu(w * wide[:inter]) * (w * wide[inter:])
            if dtype == torch.bfloat16:
                a = a.to(dtype).float()
            want[t] += df[e] @ a
    want += gate * shared.float()
    bound = {"rtol": 1e-4, "atol": 1e-5} if dtype == torch.float32 else {"rtol": 2e-2, "atol": 2e-2}
    torch.testing.assert_close(out.float(), want, **bound)


@pytest.mark.parametrize("kind", ["few", "tensor"])
@pytest.mark.parametrize("tokens,experts,top,hidden,inter", [(1, 3, 2, 64, 32), (8, 16, 2, 2048, 512), (17, 1, 1, 40, 24), (130, 2, 2, 200, 136),
                                                             (400, 3, 1, 64, 264), (2048, 16, 2, 256, 64), (300, 40, 3, 72, 8)])
def test_products_over_few_and_over_many_pairs(tokens, experts, top, hidden, inter, kind):
    """The kernels for few pairs a tile and on the tensor cores, at edges of their tiles (16 and 128 pairs, 16 and 128 gated
    columns, 32 and 256 plain ones, 32 and 64 inner columns) with unit, clamp and pair weights, against each expert's rows in
    float32; identity experts' pairs are in no tile, and nothing is written past the pairs."""
    from rapid_llm_b200.ops import kernels

    torch.manual_seed(tokens)
    bf = torch.bfloat16
    x = torch.randn(tokens, hidden + 8, device=DEVICE).to(bf)[:, :hidden]
    gate_up = (torch.randn(experts, 2 * inter, hidden, device=DEVICE) / hidden ** 0.5).to(bf)
    down = (torch.randn(experts, hidden, inter, device=DEVICE) / inter ** 0.5).to(bf)
    ids = torch.rand(tokens, experts + 1, device=DEVICE).argsort(-1)[:, :top].to(torch.int32).contiguous()      # id `experts`: an identity expert
    weights = torch.rand(tokens, top, device=DEVICE)
    pairs = tokens * top
    fault = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    order, place = torch.zeros(pairs, dtype=torch.int32, device=DEVICE), torch.zeros(pairs, dtype=torch.int32, device=DEVICE)
    meta = torch.zeros(1 + 3 * kernels.moe_max_tiles(pairs, experts, kind), dtype=torch.int32, device=DEVICE)
    tiles = kernels.moe_plan(ids, experts, order, place, meta, fault, wide=kind)
    chosen = ids.view(-1).long()
    mine = chosen < experts
    for clamp in (None, (0.5, 1.702)):
        act = torch.full((pairs + 1, inter), 7.0, dtype=bf, device=DEVICE)
        kernels.grouped_linear(x, gate_up, order, meta, top=top, by_token=True, max_tiles=tiles, pair_weight=weights.view(-1),
                               out_act=act[:pairs], wide=kind, clamp=clamp, fault=fault)
        each = torch.full((pairs + 1, hidden), 7.0, device=DEVICE)
        kernels.grouped_linear(act[:pairs], down, order, meta, top=top, by_token=False, max_tiles=tiles, out_y=each[:pairs], wide=kind, fault=fault)
        assert int(fault.item()) == 0
        assert bool((act[pairs] == 7.0).all()) and bool((each[pairs] == 7.0).all()) and bool((each[:pairs][~mine] == 7.0).all())
        rows = x.float().repeat_interleave(top, dim=0)
        for e in range(experts):
            at = (chosen == e).nonzero(as_tuple=True)[0]
            if not at.numel():
                continue
            both = (rows[at] @ gate_up[e].float().t()) * weights.view(-1)[at][:, None]
            g, u = both[:, :inter], both[:, inter:]
            if clamp is None:
                unit = g * torch.sigmoid(g) * u
            else:
                g, u = g.clamp(max=clamp[0]), u.clamp(-clamp[0], clamp[0])
                unit = g * torch.sigmoid(clamp[1] * g) * (u + 1.0)
            got = act[place.long()[at]].float()
            torch.testing.assert_close(got, unit, rtol=2.0 ** -7, atol=1e-3)            # one rounding to bfloat16
            torch.testing.assert_close(each[at], got @ down[e].float().t(), rtol=1e-4, atol=1e-4)      # float32 sums
    # a row does not depend on what else is in its tile
    alone_ids = ids[:1].contiguous()
    order1, place1 = torch.zeros(top, dtype=torch.int32, device=DEVICE), torch.zeros(top, dtype=torch.int32, device=DEVICE)
    meta1 = torch.zeros(1 + 3 * kernels.moe_max_tiles(top, experts, kind), dtype=torch.int32, device=DEVICE)
    tiles1 = kernels.moe_plan(alone_ids, experts, order1, place1, meta1, fault, wide=kind)
    act1 = torch.empty(top, inter, dtype=bf, device=DEVICE)
    kernels.grouped_linear(x[:1], gate_up, order1, meta1, top=top, by_token=True, max_tiles=tiles1, pair_weight=weights.view(-1)[:top],
                           out_act=act1, wide=kind, clamp=(0.5, 1.702), fault=fault)
    for j in range(top):
        if int(chosen[j]) < experts:
            assert torch.equal(act1[int(place1[j])], act[int(place[j])])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("experts,top,gates,hidden", [(12, 1, 1, 64), (40, 3, 0, 50), (2, 2, 2, 33), (70, 8, 1, 128)])
def test_router_scores_choices_and_gates(experts, top, gates, hidden, dtype):
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(experts)
    tokens = 45
    x = (4 * torch.randn(tokens, hidden, generator=g)).to(dtype).to(DEVICE)
    w = torch.randn(experts + gates, hidden, generator=g).to(DEVICE)
    ids = torch.empty(tokens, top, dtype=torch.int32, device=DEVICE)
    weights = torch.empty(tokens, top, device=DEVICE)
    gate_out = torch.empty(tokens, gates, device=DEVICE) if gates else None
    scores = torch.empty(tokens, experts, device=DEVICE)
    kernels.router_topk(x, w, experts=experts, top=top, ids=ids, weights=weights, gates=gate_out, scores=scores)
    logits = x.double() @ w.double().T
    want = torch.topk(logits[:, :experts], top, dim=-1)
    assert torch.equal(ids.long().cpu(), want.indices.cpu())       # large logits: sigmoid saturates, the order must not
    torch.testing.assert_close(weights.double(), torch.sigmoid(want.values), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(scores.double(), torch.sigmoid(logits[:, :experts]), rtol=1e-5, atol=1e-6)
    if gates:
        torch.testing.assert_close(gate_out.double(), torch.sigmoid(logits[:, experts:]), rtol=1e-5, atol=1e-6)


def test_equal_logits_go_to_the_lower_index():
    from rapid_llm_b200.ops import kernels

    x = torch.ones(3, 8, device=DEVICE)
    w = torch.zeros(6, 8, device=DEVICE)
    w[4], w[1] = 0.5, 0.5
    ids = torch.empty(3, 3, dtype=torch.int32, device=DEVICE)
    weights = torch.empty(3, 3, device=DEVICE)
    kernels.router_topk(x, w, experts=6, top=3, ids=ids, weights=weights)
    assert ids.tolist() == [[1, 4, 0]] * 3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [64, 50, 1032])
def test_a_norm_that_joins_the_stream_and_the_norm_of_the_stream(hidden, dtype):
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(hidden)
    y = torch.randn(9, hidden, generator=g).to(dtype).to(DEVICE)
    stream = (5 * torch.randn(9, hidden, generator=g)).to(DEVICE)
    weight = (1 + 0.2 * torch.randn(hidden, generator=g)).to(DEVICE)
    before = stream.clone()
    out = torch.empty(9, hidden, dtype=dtype, device=DEVICE)
    kernels.join_rmsnorm(y, stream, weight, out, 1e-5)
    yf = y.float()
    want = before + yf * torch.rsqrt((yf * yf).mean(-1, keepdim=True) + 1e-5) * weight
    torch.testing.assert_close(stream, want, rtol=1e-5, atol=1e-5)
    assert torch.equal(out, stream.to(dtype))
    rows = torch.tensor([7, 0, 3], dtype=torch.int32, device=DEVICE)
    normed = torch.empty(3, hidden, dtype=dtype, device=DEVICE)
    kernels.stream_rmsnorm(stream, weight, normed, 1e-5, rows)
    picked = stream[rows.long()]
    want = picked * torch.rsqrt((picked * picked).mean(-1, keepdim=True) + 1e-5) * weight
    torch.testing.assert_close(normed.float(), want, **({"rtol": 1e-5, "atol": 1e-5} if dtype == torch.float32 else {"rtol": 1e-2, "atol": 1e-2}))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_the_clamped_gated_unit_and_the_scaled_embedding(dtype):
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(2)
    wide = (2 * torch.randn(11, 2 * 37, generator=g)).to(dtype).to(DEVICE)
    out = torch.empty(11, 37, dtype=dtype, device=DEVICE)
    kernels.clamped_glu(wide, out, 0.8, 1.702)
    gate, up = wide.float()[:, :37].clamp(max=0.8), wide.float()[:, 37:].clamp(-0.8, 0.8)
    want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
    torch.testing.assert_close(out.float(), want, **({"rtol": 1e-5, "atol": 1e-6} if dtype == torch.float32 else {"rtol": 1e-2, "atol": 1e-2}))
    table = torch.randn(20, 24, generator=g).to(dtype).to(DEVICE)
    ids = torch.tensor([3, 19, 0, 3], dtype=torch.int32, device=DEVICE)
    rows = torch.empty(4, 24, dtype=dtype, device=DEVICE)
    stream = torch.empty(4, 24, device=DEVICE)
    fault = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    kernels.embedding(rows, table, ids, fault, scale=13.5, stream=stream)
    assert torch.equal(stream, table[ids.long()].float() * 13.5) and torch.equal(rows, stream.to(dtype)) and int(fault.item()) == 0


@pytest.mark.parametrize("tokens", [5, 64, 300, 1100])
def test_the_clamped_unit_rides_on_the_gate_up_product(tokens):
    """Small steps: the streaming tcgen05 product's epilogue; a thousand tokens and more: the pair kernel's; between
    them the library product and the unit's own kernel.  All against float32 arithmetic on the same bfloat16 operands."""
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import gemm

    g = torch.Generator().manual_seed(tokens)
    hidden, inter, limit, alpha = 256, 384, 0.8, 1.702
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16).to(DEVICE)
    w = (2 * torch.randn(2 * inter, hidden, generator=g) / hidden ** 0.5).to(torch.bfloat16).to(DEVICE)
    fault = torch.zeros(1, dtype=torch.int32, device=DEVICE)
    act = torch.empty(tokens, inter, dtype=torch.bfloat16, device=DEVICE)
    gemm.gated_linear(x, w, act, Workspace(tokens, torch.device(DEVICE)), fault, clamp=(limit, alpha))
    wide = x.float() @ w.float().T
    gate, up = wide[:, :inter].clamp(max=limit), wide[:, inter:].clamp(-limit, limit)
    want = gate * torch.sigmoid(alpha * gate) * (up + 1)
    assert int(fault.item()) == 0
    assert float((gate == limit).float().mean()) > 0.05 and float((up.abs() == limit).float().mean()) > 0.05      # the limits bite
    torch.testing.assert_close(act.float(), want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("clamp", [None, (7.0, 1.702)])
def test_the_gated_unit_is_the_same_to_the_last_bit_in_every_product_kernel(clamp):
    """Rows with a single one pick a weight each, so that the kernels' sums are exact and what differs is the unit alone: over
    ordinary gates, tiny ones, zeros and ones so far below zero that their sigmoid leaves the normal range."""
    from rapid_llm_b200.ops import kernels

    torch.manual_seed(5)
    tokens, hidden, inter, bf = 320, 64, 256, torch.bfloat16
    gate = torch.randn(inter, hidden, device=DEVICE)
    gate[:64] *= 6.0
    gate[64:128] = -70.0 - 25.0 * torch.rand(64, hidden, device=DEVICE)
    gate[128:160] *= 2.0 ** torch.randint(-126, 0, (32, hidden), device=DEVICE).float()
    gate[160:164] = 0.0
    up = torch.randn(inter, hidden, device=DEVICE) * 2.0 ** torch.randint(0, 40, (inter, hidden), device=DEVICE).float()
    gate_up = torch.cat([gate, up])[None].to(bf).contiguous()
    x = torch.zeros(tokens, hidden, device=DEVICE)
    x[torch.arange(tokens), torch.arange(tokens) % hidden] = 1.0
    x, weights = x.to(bf), torch.rand(tokens, 1, device=DEVICE) + 0.5
    ids, fault = torch.zeros(tokens, 1, dtype=torch.int32, device=DEVICE), torch.zeros(1, dtype=torch.int32, device=DEVICE)
    results = []
    for kind in (False, True, "few", "tensor"):
        order, place = torch.zeros(tokens, dtype=torch.int32, device=DEVICE), torch.zeros(tokens, dtype=torch.int32, device=DEVICE)
        meta = torch.zeros(1 + 3 * kernels.moe_max_tiles(tokens, 1, kind), dtype=torch.int32, device=DEVICE)
        tiles = kernels.moe_plan(ids, 1, order, place, meta, fault, wide=kind)
        act = torch.empty(tokens, inter, dtype=bf, device=DEVICE)
        kernels.grouped_linear(x, gate_up, order, meta, top=1, by_token=True, max_tiles=tiles, pair_weight=weights.view(-1), out_act=act,
                               wide=kind, clamp=clamp, fault=fault)
        results.append(act[place.long()])
    assert int(fault.item()) == 0
    assert clamp is not None or bool((results[0][:, 64:128] != 0).any())
    assert all(torch.equal(results[0], other) for other in results[1:])
