"""What a recurrence that walks prompts in pieces asks its workspace for (no GPU)."""

import pytest
import torch

from rapid_llm_b200.engine.batch import Workspace
from rapid_llm_b200.ops import kernels


@pytest.mark.parametrize("heads,dim,vdim", [(32, 128, 128), (16, 64, 64), (4, 100, 132)])
def test_growing_prompts_allocate_once_and_within_the_reserve(heads, dim, vdim):
    most, piece, first = 8192, kernels.scan_piece(heads, vdim), kernels.scan_pieces_from(heads, dim, vdim)
    space = Workspace(most, torch.device("meta"))
    sizes = set()
    for tokens in range(first, most + 1, 64):
        buffers = kernels.scan_buffers(space, tokens, heads, dim, vdim)
        # every entry that is cut keeps whole pieces and a remainder
        assert all(b.shape[0] >= tokens // piece + tokens // first for b in buffers)
        sizes.add(space.nbytes())
    assert not space._retired and len(sizes) == 1
    assert sizes.pop() <= most * 4 * 2 * -(-heads * dim * (vdim + 1) // piece)      # what a mixer reserves a token (`_pieces_elements`, in bytes)
