"""What a 32-bit product by a large weight asks of the host: launches and scratch (no GPU: the library is a stand-in)."""

from types import SimpleNamespace

import pytest
import torch

from rapid_llm_b200 import Qwen3Config
from rapid_llm_b200.engine.batch import Workspace
from rapid_llm_b200.models.causal_lm import CausalLM
from rapid_llm_b200.ops import kernels


def stand_in(monkeypatch, scratch):
    seen = []
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_stream", lambda: None)
    monkeypatch.setattr(kernels, "core", lambda: SimpleNamespace(rl_gemm_f32=lambda *args: seen.append(args) or 0, rl_gemm_f32_scratch=scratch))
    return seen


@pytest.mark.parametrize("rows,off,launches", [(33, 0, 2), (1024, 0, 2), (1025, 0, 3), (1056, 0, 3), (1057, 0, 4), (1025, 1, 4), (2048, 0, 4),
                                               (2049, 0, 5), (20, 1, 2), (20, 0, 1)])
def test_launches_of_a_product(monkeypatch, rows, off, launches):
    inner, width = 1024, 8
    wanted = 0 if rows <= 32 and off == 0 else 3 * min(rows, 1024) * inner      # as `rl_gemm_f32_scratch` has it
    stand_in(monkeypatch, lambda *args: wanted)
    a = torch.zeros(rows, inner + 4)[:, off : off + inner]
    before = kernels.LAUNCHES.count
    kernels.gemm_f32(a, torch.zeros(width, inner), torch.empty(rows, width))
    assert kernels.LAUNCHES.count - before == launches


@pytest.mark.parametrize("tokens", [200, 8192])
def test_scratch_is_the_workspaces_and_within_the_reserve(monkeypatch, tokens):
    """Steps of growing size allocate a buffer once for each width of rows, and no more than the cache pool leaves."""
    config = Qwen3Config(vocab_size=64, hidden_size=1024, intermediate_size=2052, num_hidden_layers=1, num_attention_heads=10,
                         num_key_value_heads=2, head_dim=128, max_position_embeddings=64, rms_norm_eps=1e-6)
    model = CausalLM(config.to_spec(), torch.float32, "cpu")
    kp = lambda inner: -(-inner // 8) * 8      # noqa: E731
    seen = stand_in(monkeypatch, lambda a, w, m, n, inner, stride: 3 * min(m, 1024) * kp(inner))
    space, sizes = Workspace(tokens, torch.device("cpu")), set()
    for rows in (33, 64, 129, tokens):
        for inner in (1024, 1280, 2052):       # the layer's and the head's; the attention's output; the feed-forward's way back
            kernels.gemm_f32(torch.empty(rows, inner), torch.empty(8, inner), torch.empty(rows, 8), space=space)
            held = [b for (name, cols, _), b in space._buffers.items() if name == "product_parts" and cols == 3 * kp(inner)]
            assert len(held) == 1 and seen[-1][-3] == held[0].data_ptr() and held[0].numel() >= 3 * min(rows, 1024) * kp(inner)
        sizes.add(space.nbytes())
    assert len(sizes) == 1 and not space._retired
    assert sizes.pop() <= model.product_scratch_bytes(tokens)
    assert CausalLM(config.to_spec(), torch.bfloat16, "cpu").product_scratch_bytes(tokens) == 0
