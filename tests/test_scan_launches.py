"""How many CTAs and launches a step's recurrence asks for, by the lengths of its entries (no GPU: the library is a stand-in)."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from rapid_llm_b200.engine.batch import Workspace
from rapid_llm_b200.ops import kernels
from rapid_llm_b200.parts.recurrent import _Recurrent

# what `rl_linear_scan` is given, by place from the end
TAKEN, BLOCKS, BLOCKS_FROM, OTHERS = -5, -6, -7, -10


def asked_for(monkeypatch, lengths, blocks_from, with_host_lengths=True):
    heads, dim, tokens, seen = 2, 128, sum(lengths), []
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_stream", lambda: None)
    monkeypatch.setattr(kernels, "recurrent", lambda: SimpleNamespace(rl_linear_scan=lambda *args: seen.append(args) or 0))
    batch = SimpleNamespace(cu_seqlens=torch.zeros(1), entry_slot=torch.zeros(1), entry_start=torch.zeros(1), fault=torch.zeros(1),
                            num_entries=len(lengths), max_query_len=max(lengths))
    if with_host_lengths:
        batch.h_cu_seqlens = np.cumsum([0] + lengths).astype(np.int32)
    rows, out = torch.empty(tokens, heads * dim), torch.empty(tokens, heads * dim)
    before = kernels.LAUNCHES.count
    kernels.linear_scan(rows, rows, rows, torch.ones(heads), out, torch.empty(len(lengths), heads * dim * dim), batch, heads=heads,
                        kv_heads=heads, dim=dim, vdim=dim, pieces=Workspace(tokens, torch.device("cpu")), blocks_from=blocks_from)
    (args,) = seen
    return args, kernels.LAUNCHES.count - before


@pytest.mark.parametrize("lengths", [[600] + [1] * 64, [256, 255, 1, 300], [256] * 5, [1024], [3, 2000, 700, 1]])
def test_entries_that_are_not_taken_in_blocks_get_no_ctas(monkeypatch, lengths):
    first = 256
    long = [n for n in lengths if n >= first]
    args, _ = asked_for(monkeypatch, lengths, first)
    assert args[BLOCKS_FROM] == first
    # enough for those that are, and no more than could be so long with as many tokens
    assert len(long) <= args[TAKEN] <= sum(lengths) // first
    assert sum(-(-n // kernels.SCAN_BLOCK) for n in long) <= args[BLOCKS] <= sum(lengths) // kernels.SCAN_BLOCK + args[TAKEN]


@pytest.mark.parametrize("host", [True, False])
@pytest.mark.parametrize("lengths", [[700, 333, 1015], [600] + [1] * 64, [256, 255], [300] * 4, [256]])
def test_a_walk_is_launched_for_shorter_entries_alone(monkeypatch, lengths, host):
    args, launched = asked_for(monkeypatch, lengths, 256, with_host_lengths=host)
    shorter, uneven = min(lengths) < 256, len(set(lengths)) > 1
    assert args[OTHERS] == int(shorter if host else uneven)      # (without the host's lengths, where there may be some)
    assert launched == 2 + args[OTHERS]


@pytest.mark.parametrize("heads,dim,vdim", [(8, 128, 128), (16, 128, 128), (32, 64, 64), (32, 128, 128), (64, 64, 64), (64, 128, 128)])
@pytest.mark.parametrize("max_tokens", [64, 640, 2048, 8192, 65536])
def test_with_a_correction_no_step_holds_two_entries_in_blocks(heads, dim, vdim, max_tokens):
    """Several prompts are walked as fast as one, blocks of several take turns: what a step can hold beside an entry in blocks is
    short enough for its walk to cost no more than the blocks gain."""
    first = kernels.scan_blocks_from(heads, dim, vdim, True, max_tokens)
    if heads * vdim > 4096:
        assert first == 0
        return
    assert first >= kernels.scan_blocks_from(heads, dim, vdim, True) >= 640
    # the share of its walk that a prompt takes in blocks, as measured: taken with the rest walked, or walked with it
    share = 0.47 if heads * vdim <= 2048 else 0.88
    if first <= max_tokens:
        assert share * first + (max_tokens - first) <= first * 1.02


@pytest.mark.parametrize("corrected", [False, True])
@pytest.mark.parametrize("heads,dim,vdim", [(32, 128, 128), (16, 128, 128), (32, 64, 64), (4, 100, 132), (48, 128, 128)])
def test_records_are_allocated_once_and_within_the_reserve(heads, dim, vdim, corrected):
    most = 8192
    first = kernels.scan_blocks_from(heads, dim, vdim, corrected, most)
    reserve = _Recurrent._blocks_elements(SimpleNamespace(dtype=torch.bfloat16), heads, dim, vdim, corrected)
    assert _Recurrent._blocks_elements(SimpleNamespace(dtype=torch.float32), heads, dim, vdim, corrected) == 0
    if first == 0:
        assert reserve == 0
        return
    space, sizes = Workspace(most, torch.device("meta")), set()
    for tokens in range(first, most + 1, 64):
        records = kernels.scan_records(space, tokens, heads, dim, first, corrected)
        assert records.shape[0] >= tokens // kernels.SCAN_BLOCK + tokens // first      # whole blocks and a remainder an entry
        sizes.add(space.nbytes())
    assert not space._retired and len(sizes) == 1
    assert sizes.pop() <= most * 2 * reserve      # what a mixer reserves a token, in bytes
