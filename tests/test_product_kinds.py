"""Which product kernels the routed experts of a step run on (no GPU)."""

import pytest
import torch

from rapid_llm_b200.ops import kernels


@pytest.mark.parametrize("tokens,experts,hidden,inter,kind", [
    (1, 16, 2048, 512, "few"), (8, 16, 2048, 512, "few"), (16, 16, 2048, 512, "few"), (32, 16, 2048, 512, "tensor"), (64, 16, 2048, 512, "tensor"), (1, 1, 2048, 512, "few"),
    (32, 8, 2048, 512, "few"), (64, 8, 2048, 512, "tensor"), (8, 64, 2048, 512, "few"), (16, 64, 2048, 512, "tensor"),
    (2, 8, 4096, 1024, "few"), (8, 8, 4096, 1024, "tensor"), (32, 8, 1024, 256, "few"), (256, 8, 1024, 256, True),
    (8, 32, 1024, 256, "few"), (32, 32, 1024, 256, True), (2048, 16, 2048, 512, "tensor"), (4, 16, 2048, 500, False)])
def test_the_kernel_for_few_pairs_stops_where_the_others_are_ahead(tokens, experts, hidden, inter, kind):
    """Two choices a token; each line of the table beside the rule, from both of its sides."""
    assert kernels.moe_kind(torch.bfloat16, 2 * tokens, experts, hidden, inter) == kind
    assert kernels.moe_kind(torch.float32, 2 * tokens, experts, hidden, inter) is False
