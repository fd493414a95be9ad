"""How many CTAs and launches a step's recurrence asks for, by the lengths of its entries (no GPU: the library is a stand-in)."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from rapid_llm_b200.engine.batch import Workspace
from rapid_llm_b200.ops import kernels

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
