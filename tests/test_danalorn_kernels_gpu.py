"""The kernels that came with the Danalorn decoder, or got a new form for it, one by one, against plain PyTorch."""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEVICE = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def _word():
    return torch.zeros(1, dtype=torch.int32, device=DEVICE)


def _tolerance(dtype):
    return dict(rtol=2e-5, atol=2e-5) if dtype == torch.float32 else dict(rtol=1.6e-2, atol=1.6e-2)


# ------------------------------------------------------------------------------------ embedding -- #
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("scale", [1.0, 7.5])
def test_a_scaled_token_row_and_a_pair_row_without_positions(scale, dtype):
    """Entries at position 0 take the last row, others the token their slot kept; multipliers whose products pass 32 bits."""
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(1)
    vocab, buckets, hidden, mul_prev, mul_cur = 50, 31, 40, 1_000_000_007, 998_244_353
    lengths, starts, slots = [3, 1, 5], [0, 2_000_000, 7], [2, 0, 3]
    ids = torch.randint(0, vocab, (sum(lengths),), generator=g)
    kept = torch.randint(0, vocab, (4, 1), generator=g)
    table, pair = torch.randn(vocab, hidden, generator=g).to(dtype), torch.randn(buckets + 1, hidden, generator=g).to(dtype)
    rows, at = [], 0
    for length, start, slot in zip(lengths, starts, slots):
        before = int(kept[slot])
        for place in range(length):
            token = int(ids[at])
            row = buckets if start + place == 0 else (before * mul_prev + token * mul_cur) % buckets
            rows.append(scale * table[token].float() + pair[row].float())
            before, at = token, at + 1
    want = torch.stack(rows)
    positions = torch.cat([start + torch.arange(length) for length, start in zip(lengths, starts)]).to(torch.int32)
    batch = SimpleNamespace(token_ids=ids.to(torch.int32).to(DEVICE), feedback=None, positions=positions.to(DEVICE),
                            cu_seqlens=torch.tensor([0, 3, 4, 9], dtype=torch.int32, device=DEVICE),
                            entry_slot=torch.tensor(slots, dtype=torch.int32, device=DEVICE), num_entries=3, fault=_word())
    out = torch.empty(9, hidden, dtype=dtype, device=DEVICE)
    stream = torch.empty(9, hidden, device=DEVICE)
    last = kept.to(torch.int32).to(DEVICE)
    kernels.embedding_sum(out, stream, table.to(DEVICE), pair.to(DEVICE), None, batch, last, mul_prev=mul_prev, mul_cur=mul_cur, scale=scale)
    assert int(batch.fault.item()) == 0
    torch.testing.assert_close(stream.cpu(), want, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(out.cpu().float(), want.to(dtype).float(), **_tolerance(dtype))
    assert last.flatten().tolist() == [int(ids[3]), int(kept[1]), int(ids[2]), int(ids[8])]


# --------------------------------------------------------------------------------- query and key -- #
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens", [1, 9, 700])
@pytest.mark.parametrize("hq,hkv,d,true_d,rotary,temperature", [
    (6, 2, 16, 10, 0, (0.5, 7.0)), (4, 2, 32, 32, 0, (0.3, 128.0)), (8, 8, 64, 60, 0, None), (5, 5, 96, 90, 0, (1.5, 1.0)), (12, 4, 128, 128, 0, (0.5, 64.0)),
    (12, 4, 128, 128, 128, (0.5, 64.0)), (2, 1, 256, 200, 0, (0.25, 33.0)), (12, 4, 128, 128, 128, None), (4, 2, 96, 96, 96, None), (3, 3, 48, 40, 16, (0.7, 10.0))])
def test_norm_per_head_without_rotation_and_with_a_temperature(hq, hkv, d, true_d, rotary, temperature, tokens, dtype):
    """q, k and v as the first columns of wider rows; a head's padding holds zeros; the temperature steps at multiples of
    its stretch, whatever the kernel's form (registers, pairs of heads, through shared memory)."""
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(hq * d + tokens)
    page_size, extra = 16, 24
    pages = -(-tokens // page_size) + 2
    heads = hq + 2 * hkv
    inner = torch.randn(tokens, heads, d, generator=g)
    inner[:, :, true_d:] = 0.0
    wide = torch.full((tokens, heads * d + extra), float("nan"))
    wide[:, : heads * d] = inner.view(tokens, -1)
    wide = wide.to(dtype).to(DEVICE)
    q_weight, k_weight = (torch.cat([1 + 0.3 * torch.randn(true_d, generator=g), torch.zeros(d - true_d)]) for _ in range(2))
    positions = torch.randint(0, 2000, (tokens,), generator=g).to(torch.int32)
    if temperature:
        edges = [int(temperature[1]) * n + off for n in (1, 2, 9) for off in (-2, -1, 0)]
        for place, position in enumerate(edges[:tokens]):
            positions[place] = max(position, 0)
    angles = torch.outer(torch.arange(2304, dtype=torch.float32), 50.0 ** (-torch.arange(0, rotary, 2, dtype=torch.float32) / max(rotary, 1)))
    cos, sin = torch.cos(angles).contiguous(), torch.sin(angles).contiguous()
    dest = (torch.randperm(page_size * (pages - 1), generator=g)[:tokens] + page_size).to(torch.int32)
    cache = torch.zeros(pages, 2, hkv, page_size, d, dtype=dtype, device=DEVICE)
    q_out, fault = torch.empty(tokens, hq * d, dtype=dtype, device=DEVICE), _word()
    kernels.qk_norm_rope_write(wide, q_out, num_heads=hq, num_kv_heads=hkv, head_dim=d, rotary_dim=rotary, cos=cos.to(DEVICE), sin=sin.to(DEVICE),
                               positions=positions.to(DEVICE), eps=1e-5, fault=fault, q_weight=q_weight.to(DEVICE), k_weight=k_weight.to(DEVICE),
                               kv_dest=dest.to(DEVICE), cache=cache, page_size=page_size, norm_size=true_d, temperature=temperature)
    assert int(fault.item()) == 0
    rows = inner.to(dtype).double()

    def finished(part, weight):
        out = part * torch.rsqrt((part * part).sum(-1, keepdim=True) / true_d + 1e-5) * weight.double()
        if rotary:
            c, s = (t[positions.long()].double()[:, None] for t in (cos, sin))
            u, v = out[..., : rotary // 2].clone(), out[..., rotary // 2 : rotary].clone()
            out[..., : rotary // 2], out[..., rotary // 2 : rotary] = u * c - v * s, v * c + u * s
        return out

    q = finished(rows[:, :hq], q_weight)
    if temperature:
        coef, every = temperature
        q = q * torch.tensor([1.0 + coef * math.log((int(p) + 1) // int(every) + 1) for p in positions]).double()[:, None, None]
    bound = dict(rtol=2e-5, atol=5e-5) if dtype == torch.float32 else dict(rtol=1.2e-2, atol=1.2e-2)
    torch.testing.assert_close(q_out.cpu().double().view(tokens, hq, d), q, **bound)
    stored = cache.cpu().double().permute(0, 3, 1, 2, 4).reshape(-1, 2, hkv, d)[dest.long()]
    torch.testing.assert_close(stored[:, 0], finished(rows[:, hq : hq + hkv], k_weight), **bound)
    assert torch.equal(stored[:, 1], rows[:, hq + hkv :])


@pytest.mark.parametrize("rotary", [0, 96])
def test_every_head_of_an_odd_multiple_of_32_is_written_at_many_tokens(rotary):
    """Heads of 96 have no form in registers: at tens of thousands of heads a step each still gets a warp of its own."""
    from rapid_llm_b200.ops import kernels

    tokens, hq, hkv, d, page_size = 10_000, 6, 1, 96, 16
    g = torch.Generator(device=DEVICE).manual_seed(2)
    qkv = torch.randn(tokens, (hq + 2 * hkv) * d, generator=g, device=DEVICE).to(torch.bfloat16)
    table = torch.zeros(64, rotary // 2, device=DEVICE)
    cache = torch.zeros(tokens // page_size + 1, 2, hkv, page_size, d, dtype=torch.bfloat16, device=DEVICE)
    q_out, fault = torch.full((tokens, hq * d), 7.0, dtype=torch.bfloat16, device=DEVICE), _word()
    kernels.qk_norm_rope_write(qkv, q_out, num_heads=hq, num_kv_heads=hkv, head_dim=d, rotary_dim=rotary, cos=table + 1.0, sin=table,
                               positions=torch.arange(tokens, dtype=torch.int32, device=DEVICE) % 64, eps=1e-6, fault=fault,
                               kv_dest=page_size + torch.arange(tokens, dtype=torch.int32, device=DEVICE), cache=cache, page_size=page_size)
    assert int(fault.item()) == 0
    assert torch.equal(q_out, qkv[:, : hq * d])
    stored = cache.permute(0, 3, 1, 2, 4).reshape(-1, 2 * d)[page_size : page_size + tokens]
    assert torch.equal(stored, qkv[:, hq * d :])


# -------------------------------------------------------------------------------------- latents -- #
@pytest.mark.parametrize("dtype", DTYPES)
def test_a_query_latent_alone_is_normed_without_a_cache(dtype):
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(3)
    down = torch.randn(19, 24, generator=g).to(dtype).to(DEVICE)
    weight = (1 + 0.2 * torch.randn(21, generator=g)).to(DEVICE)
    out, fault = torch.empty(19, 21, dtype=dtype, device=DEVICE), _word()
    kernels.latent_norm_write(down, q_col0=0, q_rank=21, c_col0=24, kv_rank=50, rot=6, q_weight=weight, c_weight=None, eps=1e-5, q_out=out,
                              cache=None, kv_dest=None, positions=torch.zeros(19, dtype=torch.int32, device=DEVICE), freq=torch.ones(3, device=DEVICE),
                              magnitude=1.0, layout=kernels.ROTATE_NEIGHBOURS, fault=fault)
    assert int(fault.item()) == 0
    x = down.float()[:, :21]
    torch.testing.assert_close(out.float(), (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * weight).to(dtype).float(), **_tolerance(dtype))


# --------------------------------------------------------------------------------------- decays -- #
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tokens", [1, 7, 8, 130])
@pytest.mark.parametrize("copied,channels,rank,tau", [(36, 24, 5, 6.0), (33, 130, 1, 1.0), (512, 256, 32, 16.0), (40, 129, 64, 2.5), (1300, 7, 41, 0.5), (8, 300, 16, 16.0)])
def test_decays_from_a_low_rank_product(copied, channels, rank, tau, tokens, dtype):
    """``sigmoid(z) ** (1 / tau)`` in float32 for z from far below to far above zero, columns copied as float32, everything
    between the two left alone; a row's result is the same whatever rows are beside it."""
    from rapid_llm_b200.ops import kernels

    g = torch.Generator().manual_seed(copied + rank)
    low_col0 = -(-copied // 8) * 8 + 16
    buffer = torch.randn(tokens, low_col0 + -(-rank // 8) * 8, generator=g).to(dtype).to(DEVICE)
    weight = (torch.randn(channels, rank, generator=g) * 2 / math.sqrt(rank)).to(dtype).to(DEVICE)
    bias = (torch.randn(channels, generator=g) * 6).to(DEVICE)
    rows, decay = torch.full((tokens, copied), 7.0, device=DEVICE), torch.full((tokens, channels), 7.0, device=DEVICE)
    kernels.low_rank_decay(buffer[:, :copied], buffer[:, low_col0 : low_col0 + rank], weight, bias, tau, rows, decay)
    assert torch.equal(rows, buffer[:, :copied].float())
    z = buffer[:, low_col0 : low_col0 + rank].double() @ weight.double().T + bias.double()
    torch.testing.assert_close(decay.double(), torch.exp(torch.nn.functional.logsigmoid(z) / tau), rtol=3e-6, atol=1e-6)
    again_rows, again = torch.empty(1, copied, device=DEVICE), torch.empty(1, channels, device=DEVICE)
    one = buffer[-1:].clone()
    kernels.low_rank_decay(one[:, :copied], one[:, low_col0 : low_col0 + rank], weight, bias, tau, again_rows, again)
    assert torch.equal(again[0], decay[-1])


# ------------------------------------------------------------------------------------- attention -- #
def _case(dtype, hq, hkv, d, page, lengths, new, seed, planes=2):
    """A paged cache in which request r has ``lengths[r]`` tokens of which the last ``new[r]`` are this step's; page ids are
    shuffled, unused places hold numbers that must not count."""
    g = torch.Generator().manual_seed(seed)
    per = [-(-length // page) for length in lengths]
    order = (torch.randperm(sum(per), generator=g) + 1).tolist()
    cache = torch.full((sum(per) + 1, planes, hkv, page, d), 50.0, dtype=dtype)
    table = torch.zeros(len(lengths) + 1, max(per) + 1, dtype=torch.int32)
    slots = torch.randperm(len(lengths), generator=g).tolist()
    out = {"keys": [], "values": [], "queries": [], "positions": [], "token_slot": []}
    for length, fresh, count, slot in zip(lengths, new, per, slots):
        pages = [order.pop() for _ in range(count)]
        table[slot, :count] = torch.tensor(pages, dtype=torch.int32)
        rows = torch.randn(length, planes, hkv, d, generator=g).to(dtype)
        for j in range(length):
            cache[pages[j // page], :, :, j % page] = rows[j]
        out["keys"].append(rows[:, 0].double())
        out["values"].append(rows[:, -1].double())
        out["queries"].append((torch.randn(fresh, hq, d, generator=g)).to(dtype))
        out["positions"] += list(range(length - fresh, length))
        out["token_slot"] += [slot] * fresh
    return {**out, "q": torch.cat(out["queries"]).reshape(-1, hq * d).to(DEVICE), "cache": cache.to(DEVICE), "table": table.to(DEVICE),
            "slots": torch.tensor(slots, dtype=torch.int32, device=DEVICE), "positions": torch.tensor(out["positions"], dtype=torch.int32, device=DEVICE),
            "token_slot": torch.tensor(out["token_slot"], dtype=torch.int32, device=DEVICE)}


def _plain(case, hq, hkv, lengths, new, scale, window=0, sink=None, slopes=None):
    rows = []
    for key, value, query, length, fresh in zip(case["keys"], case["values"], case["queries"], lengths, new):
        for offset in range(fresh):
            i = length - fresh + offset
            first = max(0, i - window + 1) if window else 0
            k, v = (t[first : i + 1].repeat_interleave(hq // hkv, dim=1) for t in (key, value))
            scores = torch.einsum("hd,jhd->hj", query[offset].double(), k) * scale
            if slopes is not None:
                scores = scores - slopes.double().cpu()[:, None] * (i - torch.arange(first, i + 1)).double()[None]
            if sink is not None:
                scores = torch.cat([scores, sink.double().cpu()[:, None]], dim=1)
            weights = torch.softmax(scores, dim=1)[:, : k.shape[0]]
            rows.append(torch.einsum("hj,jhd->hd", weights, v).reshape(-1))
    return torch.stack(rows).float()


def _slopes(heads):
    return torch.tensor([2.0 ** (-8.0 * (h + 1) / heads) for h in range(heads)], device=DEVICE)


def _tiles(case, hq, hkv, d, page, lengths, new, out, *, window=0, sink=None, slopes=None, splits=None, decode_kernel="auto", tensor_core=True):
    from rapid_llm_b200.ops import kernels
    from rapid_llm_b200.parts.attention import AttentionItems
    from rapid_llm_b200.parts.base import StepShape

    starts = np.asarray(lengths, np.int32) - np.asarray(new, np.int32)
    planner = AttentionItems(hq // hkv, hkv, d, tensor_core=tensor_core, window=window)
    plan = planner.plan(StepShape(np.asarray(new, np.int32), starts, decode_only=max(new) == 1, page_size=page))
    if splits is not None and splits != plan["splits"]:
        def respread(items):
            base = items[items[:, 2] == 0]
            again = np.repeat(base, splits, axis=0)
            again[:, 2] = np.tile(np.arange(splits, dtype=np.int32), len(base))
            return again
        assert plan["chunk_rows"] == kernels.CHUNK_TILE_ROWS or not len(plan["chunk_items"])
        plan = dict(plan, chunk_items=respread(plan["chunk_items"]), decode_items=respread(plan["decode_items"]), splits=splits, decode_splits=splits)
    tokens, count = case["q"].shape[0], plan["splits"]
    part_out = torch.full((tokens * hq * count, d), float("nan"), device=DEVICE) if count > 1 else None
    part_lse = torch.full((tokens * hq * count,), float("nan"), device=DEVICE) if count > 1 else None
    fault = _word()
    kernels.attention_mma(
        case["q"], case["cache"], out, chunk_items=torch.from_numpy(plan["chunk_items"]).to(DEVICE), decode_items=torch.from_numpy(plan["decode_items"]).to(DEVICE),
        splits=count, part_out=part_out, part_lse=part_lse, cu_seqlens=torch.tensor([0] + list(np.cumsum(new)), dtype=torch.int32, device=DEVICE),
        entry_start=torch.from_numpy(starts).to(DEVICE), entry_slot=case["slots"], block_table=case["table"], num_heads=hq, num_kv_heads=hkv, head_dim=d,
        window=window, scale=d ** -0.5, fault=fault, decode_kernel=decode_kernel, decode_rows=plan["decode_rows"], chunk_rows=plan["chunk_rows"],
        decode_splits=plan["decode_splits"], sink=sink, slopes=slopes)
    assert int(fault.item()) == 0
    return plan


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hq,hkv,d,page,planes,window", [(6, 2, 16, 8, 2, 0), (3, 3, 48, 16, 2, 0), (8, 1, 128, 16, 2, 70), (5, 1, 272, 16, 1, 31), (4, 1, 80, 4, 1, 0)])
def test_one_warp_per_row_attention_with_slopes_and_a_sink(hq, hkv, d, page, planes, window, dtype):
    from rapid_llm_b200.ops import kernels

    lengths, new = [1, 15, 24, 25, 129, 200], [1, 15, 1, 2, 129, 33]
    case = _case(dtype, hq, hkv, d, page, lengths, new, seed=d + page, planes=planes)
    sink, slopes, fault = torch.zeros(hq, device=DEVICE), _slopes(hq), _word()
    out = torch.empty_like(case["q"])
    kernels.attention_generic(case["q"], case["cache"], out, positions=case["positions"], token_slot=case["token_slot"], block_table=case["table"],
                              num_heads=hq, num_kv_heads=hkv, head_dim=d, window=window, scale=d ** -0.5, fault=fault, sink=sink, slopes=slopes)
    assert int(fault.item()) == 0
    bound = {"rtol": 1e-4, "atol": 2e-5} if dtype == torch.float32 else {"rtol": 3e-2, "atol": 8e-3}
    torch.testing.assert_close(out.float().cpu(), _plain(case, hq, hkv, lengths, new, d ** -0.5, window, sink, slopes), **bound)


@pytest.mark.parametrize("fixed_sink", [True, False])
@pytest.mark.parametrize("hq,hkv,d,page,splits", [
    (8, 2, 128, 16, None), (12, 3, 128, 8, None), (4, 4, 128, 64, None), (5, 5, 128, 16, None), (6, 1, 32, 8, None), (6, 1, 32, 8, 3), (7, 7, 48, 4, 2),
    (4, 2, 64, 16, None), (3, 1, 256, 64, None), (40, 2, 64, 16, 4)])
def test_prompt_and_decode_tiles_with_slopes(hq, hkv, d, page, splits, fixed_sink):
    """Portions of prompts beside single tokens: the tcgen05 tiles at heads of 128, the mma.sync tiles elsewhere, whole and
    with split key ranges; the first head's slope leaves a handful of keys, the last one's reaches hundreds back."""
    lengths, new = [1, 15, 16, 17, 129, 200, 64, 700, 333, 301], [1, 15, 1, 2, 129, 1, 33, 1, 170, 1]
    case = _case(torch.bfloat16, hq, hkv, d, page, lengths, new, seed=d + page)
    sink = torch.zeros(hq, device=DEVICE) if fixed_sink else None
    out = torch.full_like(case["q"], 7.0)
    plan = _tiles(case, hq, hkv, d, page, lengths, new, out, sink=sink, slopes=_slopes(hq), splits=splits)
    assert plan["chunk_rows"] == (256 if d == 128 else 64)
    want = _plain(case, hq, hkv, lengths, new, d ** -0.5, 0, sink, _slopes(hq))
    torch.testing.assert_close(out.float().cpu(), want, rtol=3e-2, atol=8e-3)


@pytest.mark.parametrize("decode_kernel", ["auto", "mma", "deep", "shallow"])
@pytest.mark.parametrize("hq,hkv,page,splits,lengths", [
    (32, 8, 16, None, [1, 5, 128, 513, 1000, 257, 2049]), (8, 2, 16, 3, [700, 701, 1]), (40, 2, 64, 2, [400, 90]), (8, 1, 16, 10, [5000]),
    (4, 4, 8, 1, [131, 260, 130]), (16, 16, 16, None, [900, 3])])
def test_single_tokens_on_the_decode_tiles_with_slopes(hq, hkv, page, splits, lengths, decode_kernel):
    d, new = 128, [1] * len(lengths)
    case = _case(torch.bfloat16, hq, hkv, d, page, lengths, new, seed=page + hq)
    sink, out = torch.zeros(hq, device=DEVICE), torch.full_like(case["q"], 7.0)
    _tiles(case, hq, hkv, d, page, lengths, new, out, sink=sink, slopes=_slopes(hq), splits=splits, decode_kernel=decode_kernel)
    want = _plain(case, hq, hkv, lengths, new, d ** -0.5, 0, sink, _slopes(hq))
    torch.testing.assert_close(out.float().cpu(), want, rtol=3e-2, atol=8e-3)


@pytest.mark.parametrize("hq,d,page,window,splits", [(6, 128, 16, 100, None), (6, 128, 16, 100, 3), (16, 256, 16, 65, None), (3, 48, 8, 1, None), (9, 32, 4, 64, 2), (40, 64, 16, 200, None),
                                                     (5, 128, 16, 0, None)])
def test_tiles_over_one_plane_with_a_window_and_a_sink(hq, d, page, window, splits):
    """Rows that are keys and values at once, shared by all heads: windows that begin inside, on and behind a block of keys
    and a page, in portions and single tokens, with a sink a head."""
    lengths, new = [1, 15, 16, 17, 129, 200, 64, 700, 333, 301], [1, 15, 1, 2, 129, 1, 33, 1, 170, 1]
    case = _case(torch.bfloat16, hq, 1, d, page, lengths, new, seed=d + page, planes=1)
    sink = torch.linspace(-4.0, 3.0, hq, device=DEVICE)
    out = torch.full_like(case["q"], 7.0)
    _tiles(case, hq, 1, d, page, lengths, new, out, window=window, sink=sink, splits=splits, decode_kernel="mma", tensor_core=False)
    want = _plain(case, hq, 1, lengths, new, d ** -0.5, window, sink)
    torch.testing.assert_close(out.float().cpu(), want, rtol=3e-2, atol=8e-3)
    lengths = [1, 99, 100, 101, 650, 64, 65]
    new = [1] * len(lengths)
    case = _case(torch.bfloat16, hq, 1, d, page, lengths, new, seed=d, planes=1)
    out = torch.full_like(case["q"], 7.0)
    _tiles(case, hq, 1, d, page, lengths, new, out, window=window, sink=sink, splits=splits, decode_kernel="mma", tensor_core=False)
    torch.testing.assert_close(out.float().cpu(), _plain(case, hq, 1, lengths, new, d ** -0.5, window, sink), rtol=3e-2, atol=8e-3)


@pytest.mark.parametrize("hq,hkv,d,page,window,splits", [
    (16, 1, 256, 16, 0, None), (16, 1, 256, 8, 65, 3), (6, 2, 256, 48, 0, 1), (40, 1, 240, 64, 0, None), (16, 1, 208, 24, 130, 1), (5, 1, 144, 128, 0, 5),
    (128, 1, 128, 16, 0, 2), (1, 1, 80, 16, 96, 1), (12, 3, 64, 32, 0, None)])
def test_tensor_core_tiles_over_one_plane(hq, hkv, d, page, window, splits):
    """Portions that end inside and on a tile of 128 rows, ranges that end inside and on a block of 96 keys and on a box,
    more key ranges than blocks, rows that are no multiple of 64 numbers; places that nothing wrote hold NaN."""
    from rapid_llm_b200.ops import kernels
    from rapid_llm_b200.parts.attention import AttentionItems
    from rapid_llm_b200.parts.base import StepShape

    lengths, new = [17, 96, 97, 129, 200, 64, 700, 301, 288, 5], [17, 96, 1, 129, 33, 64, 300, 1, 3, 5]
    case = _case(torch.bfloat16, hq, hkv, d, page, lengths, new, seed=d + page, planes=1)
    case["cache"][case["cache"] == 50.0] = float("nan")
    starts = np.asarray(lengths, np.int32) - np.asarray(new, np.int32)
    plan = AttentionItems(hq // hkv, hkv, d, tensor_core=False, window=window, one_plane=True).plan(
        StepShape(np.asarray(new, np.int32), starts, decode_only=False, page_size=page))
    assert plan["chunk_rows"] == kernels.CHUNK_TILE_ROWS_PLANE and len(plan["chunk_items"])

    def spread(items, count):
        base = items[items[:, 2] == 0]
        again = np.repeat(base, count, axis=0)
        again[:, 2] = np.tile(np.arange(count, dtype=np.int32), len(base))
        return torch.from_numpy(again).to(DEVICE)

    count = splits or plan["splits"]
    sink = torch.linspace(-4.0, 3.0, hq, device=DEVICE) if page != 16 else None
    gate = torch.randn(case["q"].shape[0], hq, device=DEVICE).to(torch.bfloat16) if page == 64 else None
    part_out = torch.full((case["q"].shape[0] * hq * count, d), float("nan"), device=DEVICE)
    part_lse = torch.full((case["q"].shape[0] * hq * count,), float("nan"), device=DEVICE)
    wide = torch.full((case["q"].shape[0], hq * d + 8), 7.0, dtype=torch.bfloat16, device=DEVICE)
    fault = _word()
    kernels.attention_mma(
        case["q"], case["cache"], wide[:, : hq * d], chunk_items=spread(plan["chunk_items"], count), decode_items=spread(plan["decode_items"], count),
        splits=count, part_out=part_out, part_lse=part_lse, cu_seqlens=torch.tensor([0] + list(np.cumsum(new)), dtype=torch.int32, device=DEVICE),
        entry_start=torch.from_numpy(starts).to(DEVICE), entry_slot=case["slots"], block_table=case["table"], num_heads=hq, num_kv_heads=hkv,
        head_dim=d, window=window, scale=d ** -0.5, fault=fault, decode_kernel="mma", decode_rows=plan["decode_rows"], chunk_rows=plan["chunk_rows"],
        sink=sink, gate=gate)
    assert int(fault.item()) == 0
    want = _plain(case, hq, hkv, lengths, new, d ** -0.5, window, sink)
    if gate is not None:
        want = (want.view(-1, hq, d) * torch.sigmoid(gate.float().cpu())[:, :, None]).reshape(want.shape)
    torch.testing.assert_close(wide[:, : hq * d].float().cpu(), want, rtol=3e-2, atol=8e-3)
    assert bool((wide[:, hq * d :] == 7.0).all())


def test_slopes_over_one_plane_are_refused_by_the_tiles():
    from rapid_llm_b200.ops import kernels

    case = _case(torch.bfloat16, 2, 1, 32, 8, [20], [20], seed=1, planes=1)
    with pytest.raises(kernels.KernelError, match="invalid value"):
        _tiles(case, 2, 1, 32, 8, [20], [20], torch.empty_like(case["q"]), slopes=_slopes(2), decode_kernel="mma", tensor_core=False)
    with pytest.raises(kernels.KernelError, match="slopes"):
        _tiles(case, 2, 1, 32, 8, [20], [20], torch.empty_like(case["q"]), slopes=_slopes(3), decode_kernel="mma", tensor_core=False)


@pytest.mark.parametrize("heads,requests,new,start,d", [(16, 1, 600, 0, 256), (16, 8, 1, 1000, 256), (32, 16, 1, 300, 256), (8, 2, 100, 250, 256),
                                                        (16, 4, 1, 2000, 192), (12, 2, 333, 0, 128)])
def test_tensor_core_tiles_over_one_plane_are_as_precise_as_the_others(heads, requests, new, start, d):
    """Against 64 bits the tiles of 128 rows are no further off than the mma.sync tiles, which take a row's largest weight
    without an error; half a percent is what the means over 10^5 roundings and more vary by."""
    from rapid_llm_b200.ops import kernels
    from rapid_llm_b200.parts.attention import AttentionItems
    from rapid_llm_b200.parts.base import StepShape

    page, scale = 16, 0.072 * (256 / d) ** 0.5
    length = start + new
    per = -(-length // page)
    generator = torch.Generator(device=DEVICE).manual_seed(new + d)
    cache = torch.randn(requests * per, 1, 1, page, d, generator=generator, device=DEVICE).to(torch.bfloat16)
    q = torch.randn(requests * new, heads * d, generator=generator, device=DEVICE).to(torch.bfloat16)
    table = torch.arange(requests * per, dtype=torch.int32, device=DEVICE).view(requests, per)
    keys = cache.view(requests, per * page, d)[:, :length].double()
    scores = torch.einsum("nthd,nkd->nhtk", q.view(requests, new, heads, d).double(), keys) * scale
    hidden = torch.arange(length, device=DEVICE)[None, :] > (start + torch.arange(new, device=DEVICE))[:, None]
    want = torch.einsum("nhtk,nkd->nthd", torch.softmax(scores.masked_fill(hidden, float("-inf")), -1), keys).reshape(requests * new, -1)
    off = []
    for plane in (False, True):
        plan = AttentionItems(heads, 1, d, tensor_core=False, one_plane=plane).plan(
            StepShape(np.full(requests, new, np.int32), np.full(requests, start, np.int32), decode_only=new == 1, page_size=page))
        assert (plan["chunk_rows"] == kernels.CHUNK_TILE_ROWS_PLANE) == plane
        rows, fault, out = requests * new * heads * plan["splits"], _word(), torch.empty_like(q)
        kernels.attention_mma(
            q, cache, out, chunk_items=torch.from_numpy(plan["chunk_items"]).to(DEVICE), decode_items=torch.from_numpy(plan["decode_items"]).to(DEVICE),
            splits=plan["splits"], part_out=torch.empty(rows, d, device=DEVICE), part_lse=torch.empty(rows, device=DEVICE),
            cu_seqlens=torch.arange(0, requests * new + 1, new, dtype=torch.int32, device=DEVICE),
            entry_start=torch.full((requests,), start, dtype=torch.int32, device=DEVICE), entry_slot=torch.arange(requests, dtype=torch.int32, device=DEVICE),
            block_table=table, num_heads=heads, num_kv_heads=1, head_dim=d, window=0, scale=scale, fault=fault, decode_kernel="mma",
            decode_rows=plan["decode_rows"], chunk_rows=plan["chunk_rows"])
        assert int(fault.item()) == 0
        off.append(float((out.double() - want).norm() / want.norm()))
    assert off[1] <= 1.005 * off[0], off


@pytest.mark.parametrize("lift", [-3.0, 60.0, 100.0, float("inf")])
def test_a_sink_far_above_the_keys_leaves_their_sum_its_digits(lift):
    """Large rows make what the sink leaves of them a number of the result's range: e^-100 of 10^30 is one.  One rounding of
    the result and of the weights' sums, 2^-8, twice."""
    from rapid_llm_b200.ops import kernels
    from rapid_llm_b200.parts.attention import AttentionItems
    from rapid_llm_b200.parts.base import StepShape

    heads, d, page, tokens = 16, 256, 16, 40
    generator = torch.Generator(device=DEVICE).manual_seed(3)
    rows = (torch.randn(48, d, generator=generator, device=DEVICE) * 1e30).to(torch.bfloat16)
    q = (torch.randn(tokens, heads * d, generator=generator, device=DEVICE) * 1e-30).to(torch.bfloat16)
    scores = torch.einsum("thd,kd->thk", q.view(tokens, heads, d).double(), rows[:tokens].double()) / 16
    scores.masked_fill_((torch.arange(tokens, device=DEVICE)[None] > torch.arange(tokens, device=DEVICE)[:, None])[:, None], float("-inf"))
    sink = torch.full((heads,), lift, device=DEVICE)
    with_sink = torch.cat([scores, sink.double().view(1, heads, 1).expand(tokens, heads, 1)], -1)
    weights = torch.softmax(with_sink, -1)[..., :tokens] if math.isfinite(lift) else torch.zeros_like(scores)
    want = torch.einsum("thk,kd->thd", weights, rows[:tokens].double()).reshape(tokens, -1)
    plan = AttentionItems(heads, 1, d, tensor_core=False, one_plane=True).plan(
        StepShape(np.asarray([tokens], np.int32), np.asarray([0], np.int32), decode_only=False, page_size=page))
    assert plan["chunk_rows"] == kernels.CHUNK_TILE_ROWS_PLANE and plan["splits"] == 1
    out, fault = torch.empty_like(q), _word()
    call = lambda scale: kernels.attention_mma(      # noqa: E731
        q, rows.view(3, 1, 1, page, d), out, chunk_items=torch.from_numpy(plan["chunk_items"]).to(DEVICE),
        decode_items=torch.from_numpy(plan["decode_items"]).to(DEVICE), splits=1, part_out=None, part_lse=None,
        cu_seqlens=torch.tensor([0, tokens], dtype=torch.int32, device=DEVICE), entry_start=torch.zeros(1, dtype=torch.int32, device=DEVICE),
        entry_slot=torch.zeros(1, dtype=torch.int32, device=DEVICE), block_table=torch.arange(3, dtype=torch.int32, device=DEVICE).view(1, 3),
        num_heads=heads, num_kv_heads=1, head_dim=d, window=0, scale=scale, fault=fault, decode_kernel="mma", decode_rows=plan["decode_rows"],
        chunk_rows=plan["chunk_rows"], sink=sink)
    call(1 / 16)
    assert int(fault.item()) == 0
    assert float((out.double() - want).norm()) <= 2.0 ** -7 * float(want.norm())
    for scale in (0.0, -0.5):      # refused: the kernel masks and takes maxima before it scales
        with pytest.raises(kernels.KernelError):
            call(scale)
