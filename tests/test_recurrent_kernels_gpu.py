"""The kernels of the recurrent mixers, each alone, against plain float64 restatements."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch
from plain_kopatar import causal_conv, rotate_halves, silu, softplus, unit_rms, xielu

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _batch(lengths, slots, starts):
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    return SimpleNamespace(
        cu_seqlens=cu, entry_slot=torch.tensor(slots, dtype=torch.int32, device=DEV),
        entry_start=torch.tensor(starts, dtype=torch.int32, device=DEV), num_entries=len(lengths),
        fault=torch.zeros(1, dtype=torch.int32, device=DEV),
    )


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("width", [1, 2, 4])
def test_short_convolution_over_steps_of_any_length(dtype, width):
    """Two requests fed in steps of 1, 2 and more tokens (fewer than the taps reach back, too); the tail kept in the
    slot carries each over; a slot that changes hands starts from zeros whatever it holds."""
    from rapid_llm_b200.ops import kernels

    channels, slots = 10, 3
    generator = torch.Generator().manual_seed(width)
    taps = torch.randn(channels, width, generator=generator)
    bias = torch.randn(channels, generator=generator)
    sequences = [torch.randn(n, channels + 4, generator=generator).to(dtype) for n in (23, 17)]
    want = [silu(causal_conv(s[:, 2 : 2 + channels].double(), taps.double(), bias.double())) for s in sequences]
    tail = torch.full((slots, (width - 1) * channels + 5), 7.0, device=DEV)      # garbage: position 0 must not read it
    cuts = [[1, 2, 1, 5, 3, 1, 1, 9], [2, 1, 1, 1, 6, 4, 2]]
    fed, got = [0, 0], [[], []]
    for step in range(max(len(c) for c in cuts)):
        live = [i for i in (0, 1) if step < len(cuts[i])]
        lengths = [cuts[i][step] for i in live]
        rows = torch.cat([sequences[i][fed[i] : fed[i] + n] for i, n in zip(live, lengths)]).to(DEV)
        out = torch.empty(rows.shape[0], channels, device=DEV)
        batch = _batch(lengths, [2 - i for i in live], [fed[i] for i in live])
        kernels.causal_conv_silu(rows[:, 2 : 2 + channels], taps.to(DEV), bias.to(DEV), tail[:, 5:], out, batch)
        at = 0
        for i, n in zip(live, lengths):
            got[i].append(out[at : at + n].cpu())
            at, fed[i] = at + n, fed[i] + n
        assert int(batch.fault.item()) == 0
    for i in (0, 1):
        torch.testing.assert_close(torch.cat(got[i]).double(), want[i], rtol=1e-5, atol=1e-5)
    assert torch.all(tail[:, :5] == 7.0)


def _plain_scan(q, k, v, decay, beta, v_scale, skip, heads, kv_heads, dim, vdim):
    length = q.shape[0]
    out = torch.zeros(length, heads, vdim, dtype=torch.float64)
    q, k, v = q.view(length, kv_heads, dim), k.view(length, kv_heads, dim), v.view(length, heads, vdim)
    for h in range(heads):
        S = torch.zeros(dim, vdim, dtype=torch.float64)
        for t in range(length):
            kh = h // (heads // kv_heads)
            if decay.dim() == 1:
                S = decay[h] * S
            elif decay.shape[1] == heads:
                S = decay[t, h] * S
            else:
                S = decay[t].view(heads, dim)[h].unsqueeze(1) * S
            if beta is not None:
                u = beta[t, h] * (v[t, h] - S.T @ k[t, kh])
            else:
                u = v[t, h] * (1.0 if v_scale is None else v_scale[t, h])
            S = S + torch.outer(k[t, kh], u)
            out[t, h] = S.T @ q[t, kh] + (0.0 if skip is None else skip[h]) * v[t, h]
    return out.view(length, heads * vdim)


@pytest.mark.parametrize("dim,vdim,heads,kv_heads", [(20, 7, 4, 2), (64, 64, 2, 2), (128, 48, 2, 1), (5, 130, 3, 3), (300, 16, 1, 1)])
@pytest.mark.parametrize("kind", ["fixed", "per_token", "per_row_delta", "per_token_scaled_skip"])
def test_the_recurrence_over_steps_and_slots(kind, dim, vdim, heads, kv_heads):
    from rapid_llm_b200.ops import kernels

    generator = torch.Generator().manual_seed(dim + vdim)
    lengths_total = (37, 12)
    data = []
    fixed = torch.rand(heads, generator=generator) * 0.2 + 0.8
    skips = torch.randn(heads, generator=generator)
    for n in lengths_total:
        q, k = torch.randn(n, kv_heads * dim, generator=generator) / dim ** 0.5, torch.randn(n, kv_heads * dim, generator=generator)
        v = torch.randn(n, heads * vdim, generator=generator)
        beta = v_scale = skip = None
        if kind == "fixed":
            decay = fixed
        elif kind == "per_token":
            decay = torch.rand(n, heads, generator=generator) * 0.5 + 0.5
        elif kind == "per_row_delta":
            decay = torch.rand(n, heads * dim, generator=generator) * 0.3 + 0.7
            beta = torch.rand(n, heads, generator=generator)
            k = k / k.view(n, kv_heads, dim).norm(dim=-1).repeat_interleave(dim, dim=1)
        else:
            decay = torch.rand(n, heads, generator=generator) * 0.5 + 0.5
            v_scale, skip = torch.rand(n, heads, generator=generator), skips
        data.append((q, k, v, decay, beta, v_scale, skip))
    want = [_plain_scan(*(None if t is None else t.double() for t in item), heads, kv_heads, dim, vdim) for item in data]
    state = torch.full((3, heads * dim * vdim + 3), float("nan"), device=DEV)      # position 0 must not read it
    cuts = [[5, 1, 1, 17, 2, 11], [1, 1, 10]]
    fed, got = [0, 0], [[], []]
    for step in range(max(len(c) for c in cuts)):
        live = [i for i in (0, 1) if step < len(cuts[i])]
        lengths = [cuts[i][step] for i in live]
        batch = _batch(lengths, [i + 1 for i in live], [fed[i] for i in live])

        def rows(index):
            if data[0][index] is None:
                return None
            return torch.cat([data[i][index][fed[i] : fed[i] + n] for i, n in zip(live, lengths)]).to(DEV).contiguous()

        q, k, v = rows(0), rows(1), rows(2)
        decay = data[0][3].to(DEV) if kind == "fixed" else rows(3)
        skip = None if data[0][6] is None else data[0][6].to(DEV)
        out = torch.empty(v.shape, device=DEV)
        kernels.linear_scan(q, k, v, decay, out, state[:, 3:], batch, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim,
                            beta=rows(4), v_scale=rows(5), skip=skip)
        assert int(batch.fault.item()) == 0
        at = 0
        for i, n in zip(live, lengths):
            got[i].append(out[at : at + n].cpu())
            at, fed[i] = at + n, fed[i] + n
    for i in (0, 1):
        torch.testing.assert_close(torch.cat(got[i]).double(), want[i], rtol=2e-4, atol=2e-4)


@pytest.mark.parametrize("kind", ["fixed", "per_token", "per_row", "bonus", "delta"])
@pytest.mark.parametrize("dim,vdim", [(36, 44), (64, 64), (128, 128), (100, 132)])
def test_prompts_walked_in_pieces(kind, dim, vdim):
    """Entries of whole pieces, of pieces with a remainder, of fewer tokens than are cut and of a single one, from zeros and from
    a carried state, in pieces against the walk from end to end (the same sums in another order) and its final states; and single tokens
    of the same heads, alone and behind another entry, bit for bit as the walk takes them.  With a correction nothing is cut."""
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import kernels

    heads, kv_heads = 4, 2
    piece, first = kernels.scan_piece(heads, vdim), kernels.scan_pieces_from(heads, dim, vdim)
    lengths, starts, slots = [first + 37, 1, first - 1, -(-first // piece) * piece], [0, 9, 5, 700], [3, 1, 0, 2]
    tokens = sum(lengths)
    torch.manual_seed(dim)
    q, k = torch.randn(tokens, kv_heads * dim, device=DEV) / dim ** 0.5, torch.randn(tokens, kv_heads * dim, device=DEV)
    k = (k.view(tokens, kv_heads, dim) / k.view(tokens, kv_heads, dim).norm(dim=-1, keepdim=True)).reshape(tokens, -1).contiguous()
    v, options = torch.randn(tokens, heads * vdim, device=DEV), {}
    if kind == "fixed":
        decay = torch.rand(heads, device=DEV) * 0.1 + 0.9
    elif kind == "per_token":
        decay = torch.rand(tokens, heads, device=DEV) * 0.1 + 0.9
        options = {"v_scale": torch.rand(tokens, heads, device=DEV), "skip": torch.rand(heads, device=DEV)}
    else:
        decay = torch.rand(tokens, heads * dim, device=DEV) * 0.1 + 0.9
        if kind == "bonus":
            options = {"bonus": torch.randn(heads, dim, device=DEV)}
        elif kind == "delta":
            options = {"beta": torch.rand(tokens, heads, device=DEV)}
    given = torch.randn(4, heads * dim * vdim, device=DEV) * 0.3
    results = []
    for pieces in (None, Workspace(64, torch.device(DEV))):
        batch = _batch(lengths, slots, starts)
        batch.max_query_len = max(lengths)
        out, state = torch.empty(tokens, heads * vdim, device=DEV), given.clone()
        kernels.linear_scan(q, k, v, decay, out, state, batch, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, pieces=pieces, **options)
        assert int(batch.fault.item()) == 0
        results.append((out, state))
    (walked, walked_state), (out, state) = results
    if kind == "delta":
        assert torch.equal(out, walked) and torch.equal(state, walked_state)
    # two float32 sums of over a thousand terms each, decayed to about 20 that count: 20 * 2^-24 of a value's size, ten-fold
    size = float(walked.abs().max())
    assert float((out - walked).abs().max()) <= 200 * 2.0 ** -24 * max(size, 1.0)
    assert float((state - walked_state).abs().max()) <= 200 * 2.0 ** -24 * max(float(walked_state.abs().max()), 1.0)
    if dim % 4 == 0 and vdim % 4 == 0:
        per_token = {name: t for name, t in options.items() if t.shape[0] == tokens}
        fixed = {name: t for name, t in options.items() if t.shape[0] != tokens}
        rows = torch.tensor([3, first + 37, 5], device=DEV)      # any three tokens, as single tokens and in an entry of two

        def taken(index):
            return (q[index].contiguous(), k[index].contiguous(), v[index].contiguous(), decay if kind == "fixed" else decay[index].contiguous(),
                    {**fixed, **{name: t[index].contiguous() for name, t in per_token.items()}})

        singles, mixed = [], []
        for index, cut, into in ((rows, [1, 1, 1], singles), (torch.cat([rows, rows[:1]]), [1, 1, 2], mixed)):
            a, b, c, d, more = taken(index)
            batch = _batch(cut, [1, 2, 0], [4, 0, 8])
            out, state = torch.empty(len(index), heads * vdim, device=DEV), given.clone()
            kernels.linear_scan(a, b, c, d, out, state, batch, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, **more)
            into.extend([out[:3], state[1:3]])
        assert all(torch.equal(one, other) for one, other in zip(singles, mixed))


@pytest.mark.parametrize("kind", ["fixed", "per_token", "per_row", "bonus"])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (128, 128), (36, 44)])
def test_an_entry_is_the_same_alone_and_beside_others(kind, dim, vdim):
    """A long prompt, a single token and shorter entries, to the last bit: which of them is cut is a matter of its own length."""
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import kernels

    heads, first = 3, kernels.scan_pieces_from(3, dim, vdim)
    lengths, starts = [1, first + 150, 201, first - 1, first, 2], [8, 0, 40, 0, 7, 3]
    tokens, count = sum(lengths), len(lengths)
    generator = torch.Generator(device=DEV).manual_seed(dim)
    draw = lambda *shape: torch.randn(*shape, generator=generator, device=DEV)      # noqa: E731
    q, k, v, given = draw(tokens, heads * dim), draw(tokens, heads * dim) * dim ** -0.5, draw(tokens, heads * vdim), draw(count, heads * dim * vdim)
    decay = 1 - 0.1 * torch.rand({"fixed": (heads,), "per_token": (tokens, heads)}.get(kind, (tokens, heads * dim)), generator=generator, device=DEV)
    options = {"bonus": draw(heads, dim)} if kind == "bonus" else {}
    space = Workspace(tokens, torch.device(DEV))

    def walk(rows, entries):
        batch = _batch([lengths[e] for e in entries], list(range(len(entries))), [starts[e] for e in entries])
        batch.max_query_len = max(lengths[e] for e in entries)
        part = lambda t: t[rows].contiguous()      # noqa: E731
        out, state = torch.empty_like(part(v)), given[entries].clone()
        kernels.linear_scan(part(q), part(k), part(v), decay if kind == "fixed" else part(decay), out, state, batch, heads=heads,
                            kv_heads=heads, dim=dim, vdim=vdim, pieces=space, **options)
        assert int(batch.fault.item()) == 0
        return out, state

    together, states = walk(slice(0, tokens), list(range(count)))
    at = 0
    for e, n in enumerate(lengths):
        out, state = walk(slice(at, at + n), [e])
        assert torch.equal(out, together[at : at + n]) and torch.equal(state[0], states[e]), n
        at += n


@pytest.mark.parametrize("kind", ["fixed", "per_row", "bonus"])
@pytest.mark.parametrize("heads,dim", [(16, 128), (16, 64)])
def test_pieces_lose_no_digits(kind, heads, dim):
    """Read-outs and final states in pieces are no further from 64-bit sums than those of the walk from end to end: decays
    up to 1 - 2^-10, whose product over a piece is still near 1.  A run's figure is a mean over 10^5 roundings and more; 2 %
    covers what another order of the same sums does to it."""
    from rapid_llm_b200.engine.batch import Workspace
    from rapid_llm_b200.ops import kernels

    tokens = 1024 + 2 * kernels.scan_piece(heads, dim) + 19
    generator = torch.Generator(device=DEV).manual_seed(dim)
    draw = lambda *shape: torch.randn(*shape, generator=generator, device=DEV)      # noqa: E731
    q, k, v, given = draw(tokens, heads * dim), draw(tokens, heads * dim) * dim ** -0.5, draw(tokens, heads * dim), draw(1, heads * dim * dim) * 0.3
    options = {"bonus": draw(heads, dim) * 0.5} if kind == "bonus" else {}
    if kind == "fixed":
        decay = 1 - 2.0 ** (-3 - 7 * torch.arange(heads, device=DEV) / (heads - 1))
        rows = decay.double().view(1, heads, 1).expand(tokens, heads, dim)
    else:
        decay = torch.sigmoid(draw(tokens, heads * dim) + 2) ** (1 / 16)
        rows = decay.double().view(tokens, heads, dim)
    S, want = given.double().view(heads, dim, dim).transpose(1, 2).contiguous(), []
    for t in range(tokens):
        qt, kt, vt = (x[t].double().view(heads, dim) for x in (q, k, v))
        pair = kt[:, :, None] * vt[:, None, :]
        if options:
            want.append(torch.einsum("hk,hkv->hv", qt, S + options["bonus"].double()[:, :, None] * pair))
        S = S * rows[t][:, :, None] + pair
        if not options:
            want.append(torch.einsum("hk,hkv->hv", qt, S))
    want, final = torch.stack(want).view(tokens, heads * dim), S.transpose(1, 2).reshape(1, -1)
    off = []
    for pieces in (None, Workspace(tokens, torch.device(DEV))):
        batch = _batch([tokens], [0], [9])
        batch.max_query_len = tokens
        out, state = torch.empty_like(v), given.clone()
        kernels.linear_scan(q, k, v, decay, out, state, batch, heads=heads, kv_heads=heads, dim=dim, vdim=dim, pieces=pieces, **options)
        off.append([float((got.double() - exact).norm() / exact.norm()) for got, exact in ((out, want), (state, final))])
    (walked, walked_state), (read, left) = off
    assert read <= 1.02 * walked and left <= 1.02 * walked_state, off


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_and_gate_in_their_three_orders(dtype):
    from rapid_llm_b200.ops import kernels

    generator = torch.Generator().manual_seed(0)
    tokens, groups, size = 5, 3, 20
    y = torch.randn(tokens, groups * size, generator=generator)
    gate = torch.randn(tokens, groups * size + 6, generator=generator).to(dtype)
    g = gate[:, 6:].double()
    per_group, whole = torch.randn(size, generator=generator), torch.randn(groups * size, generator=generator)
    yd = y.double().view(tokens, groups, size)
    cases = [
        (dict(act=kernels.GATE_SIGMOID, weight=per_group.to(DEV), eps=1e-5),
         (unit_rms(yd, 1e-5) * per_group.double()).reshape(tokens, -1) * torch.sigmoid(g)),
        (dict(act=kernels.GATE_SILU, eps=1e-6), unit_rms(yd, 1e-6).reshape(tokens, -1) * silu(g)),
        (dict(act=kernels.GATE_SILU, gate_first=True, weight=whole.to(DEV), eps=1e-5),
         unit_rms((y.double() * silu(g)).view(tokens, groups, size), 1e-5).reshape(tokens, -1) * whole.double()),
    ]
    for options, want in cases:
        out = torch.empty(tokens, groups * size, dtype=dtype, device=DEV)
        kernels.gated_norm(y.to(DEV), out, group=size, gate=gate.to(DEV)[:, 6:], **options)
        tolerance = dict(rtol=1e-5, atol=1e-5) if dtype == torch.float32 else dict(rtol=1e-2, atol=1e-2)
        torch.testing.assert_close(out.double().cpu(), want, **tolerance)
    # the gate alone, on rows of the engine's dtype (an attention's output gate)
    rows = y.to(dtype)
    out = torch.empty_like(rows, device=DEV)
    kernels.gated_norm(rows.to(DEV), out, group=groups * size, gate=gate.to(DEV)[:, 6:], act=kernels.GATE_SIGMOID, norm=False)
    torch.testing.assert_close(out.double().cpu(), rows.double() * torch.sigmoid(g), rtol=1e-2 if dtype == torch.bfloat16 else 1e-6, atol=1e-6)


@pytest.mark.parametrize("group,groups", [(4, 3), (32, 5), (36, 2), (64, 7), (128, 2), (132, 3), (512, 2), (516, 1), (2048, 2), (4100, 1), (8192, 1), (8196, 1)])
def test_norms_and_unit_vectors_at_the_edges_of_their_groups(group, groups):
    """Each number of lanes, columns a lane and block size of the gated norm, the sizes behind them, on rows that start on a
    vector's boundary and on rows that do not; unit vectors and plain activations of the same sizes."""
    from rapid_llm_b200.ops import kernels

    torch.manual_seed(group)
    tokens, width = 9, group * groups
    for shift in (0, 1):
        wide_y = torch.randn(tokens, width + 4, device=DEV)
        wide_g = torch.randn(tokens, width + 4, device=DEV).to(torch.bfloat16)
        y, gate = wide_y[:, shift : shift + width], wide_g[:, shift : shift + width]
        weight = torch.randn(width, device=DEV)
        out = torch.empty(tokens, width, dtype=torch.bfloat16, device=DEV)
        kernels.gated_norm(y, out, group=group, gate=gate, act=kernels.GATE_SILU, weight=weight, eps=1e-5)
        want = (unit_rms(y.double().cpu().reshape(tokens, groups, group), 1e-5).reshape(tokens, width) * weight.double().cpu()
                * silu(gate.double().cpu()))
        torch.testing.assert_close(out.double().cpu(), want, rtol=2.0 ** -8, atol=1e-5)      # half a step of bfloat16, twice
        plain = kernels.activate_rows(gate, torch.empty(tokens, width, device=DEV), act=True)
        torch.testing.assert_close(plain.double().cpu(), silu(gate.double().cpu()), rtol=1e-5, atol=1e-6)
        if group <= 512:
            rows = wide_y.clone()
            raw, beta = torch.randn(tokens, 3, device=DEV).to(torch.bfloat16), torch.empty(tokens, 3, device=DEV)
            kernels.unit_heads(rows[:, shift : shift + width], heads=groups, dim=group, eps=1e-6, split=1, scale_low=0.5, scale_high=2.0,
                               gate_in=raw, gate_out=beta)
            v = y.double().cpu().reshape(tokens, groups, group)
            v = v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6) * torch.tensor([0.5] + [2.0] * (groups - 1)).view(1, -1, 1)
            torch.testing.assert_close(rows[:, shift : shift + width].double().cpu(), v.reshape(tokens, width), rtol=1e-5, atol=1e-6)
            torch.testing.assert_close(beta.double().cpu(), torch.sigmoid(raw.double().cpu()), rtol=1e-5, atol=1e-6)
            assert torch.equal(rows[:, shift + width :], wide_y[:, shift + width :])


def test_activation_decays_unit_heads_and_rotation():
    from rapid_llm_b200.ops import kernels

    generator = torch.Generator().manual_seed(1)
    z = torch.randn(7, 33, generator=generator) * 3
    pq = torch.tensor([0.3, -0.8])
    out = torch.empty_like(z, device=DEV)
    kernels.xielu(z.to(DEV), out, pq.to(DEV))
    torch.testing.assert_close(out.cpu().double(), xielu(z.double(), pq[0].double(), pq[1].double()), rtol=1e-5, atol=1e-6)

    heads, per, tokens = 3, 4, 6
    x = torch.randn(tokens, heads * per + 2, generator=generator) * 2
    a_log, bias = torch.randn(heads, generator=generator), torch.randn(heads * per, generator=generator)
    decay, step = torch.empty(tokens, heads * per, device=DEV), torch.empty(tokens, heads * per, device=DEV)
    kernels.decay_gate(x.to(DEV)[:, 2:], torch.exp(a_log).to(DEV), bias.to(DEV), per, decay, step)
    dt = softplus(x[:, 2:].double() + bias.double())
    torch.testing.assert_close(step.cpu().double(), dt, rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(decay.cpu().double(), torch.exp(-torch.exp(a_log.double()).repeat_interleave(per) * dt), rtol=1e-5, atol=1e-6)

    dim = 12
    rows = torch.randn(tokens, 1 + 4 * dim, generator=generator)
    raw = torch.randn(tokens, 5, generator=generator)
    work, gates = rows.to(DEV), torch.empty(tokens, 3, device=DEV)
    kernels.unit_heads(work[:, 1:], heads=4, dim=dim, eps=1e-6, split=2, scale_low=dim ** -0.5, scale_high=1.0,
                       gate_in=raw.to(DEV)[:, 2:], gate_out=gates)
    v = rows[:, 1:].double().view(tokens, 4, dim)
    want = v / torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-6)
    want[:, :2] *= dim ** -0.5
    torch.testing.assert_close(work[:, 1:].cpu().double(), want.reshape(tokens, -1), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(gates.cpu().double(), torch.sigmoid(raw[:, 2:].double()), rtol=1e-5, atol=1e-6)
    assert torch.equal(work[:, 0].cpu(), rows[:, 0])

    heads, dim, vdim, rot, base = 2, 10, 6, 6, 50.0
    proj = torch.randn(tokens, 2 * heads * dim + heads * vdim + 3, generator=generator)
    positions = torch.tensor([0, 1, 2, 900, 31, 7], dtype=torch.int32)
    inv_freq = 1.0 / (torch.tensor(base) ** (torch.arange(0, rot, 2, dtype=torch.float32) / rot))
    out = torch.empty(tokens, 2 * heads * dim + heads * vdim, device=DEV)
    on = proj.to(DEV)
    hd = heads * dim
    kernels.rotate_heads(on[:, 3 : 3 + hd], on[:, 3 + hd : 3 + 2 * hd], on[:, 3 + 2 * hd :], out, positions.to(DEV), inv_freq.to(DEV),
                         heads=heads, dim=dim, vdim=vdim, k_scale=0.25)
    q = rotate_halves(proj[:, 3 : 3 + hd].double().view(tokens, heads, dim), positions, rot, base).reshape(tokens, -1)
    k = rotate_halves(proj[:, 3 + hd : 3 + 2 * hd].double().view(tokens, heads, dim), positions, rot, base).reshape(tokens, -1) * 0.25
    torch.testing.assert_close(out.cpu().double(), torch.cat([q, k, proj[:, 3 + 2 * hd :].double()], dim=1), rtol=1e-4, atol=1e-4)


@pytest.mark.parametrize("hidden", [64, 60])
def test_the_norm_takes_addends_into_the_stream(hidden):
    from rapid_llm_b200.ops import kernels

    generator = torch.Generator().manual_seed(2)
    tokens = 5
    x, residual, rows = (torch.randn(tokens, hidden, generator=generator) for _ in range(3))
    vector, weight = torch.randn(hidden, generator=generator), torch.randn(hidden, generator=generator)
    stream = residual.to(DEV)
    out = torch.empty(tokens, hidden, device=DEV)
    kernels.add_rmsnorm(x.to(DEV), stream, weight.to(DEV), out, 1e-5, mode=1, write_residual=True,
                        extra_rows=rows.to(DEV), extra_vector=vector.to(DEV))
    total = x.double() + residual.double() + rows.double() + vector.double()
    torch.testing.assert_close(stream.cpu().double(), total, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(out.cpu().double(), unit_rms(total, 1e-5) * weight.double(), rtol=1e-5, atol=1e-5)
