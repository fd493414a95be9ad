"""How many launches a 32-bit product by a large weight is counted as (no GPU: the library is a stand-in)."""

from types import SimpleNamespace

import pytest
import torch

from rapid_llm_b200.ops import kernels


@pytest.mark.parametrize("rows,off,launches", [(33, 0, 2), (1024, 0, 2), (1025, 0, 3), (1056, 0, 3), (1057, 0, 4), (1025, 1, 4), (2048, 0, 4),
                                               (2049, 0, 5), (20, 1, 2), (20, 0, 1)])
def test_launches_of_a_product(monkeypatch, rows, off, launches):
    inner, width = 1024, 8
    wanted = 0 if rows <= 32 and off == 0 else 3 * min(rows, 1024) * inner      # as `rl_gemm_f32_scratch` has it
    monkeypatch.setattr(kernels, "_need_cuda", lambda *tensors: None)
    monkeypatch.setattr(kernels, "_stream", lambda: None)
    monkeypatch.setattr(kernels, "core", lambda: SimpleNamespace(rl_gemm_f32=lambda *args: 0, rl_gemm_f32_scratch=lambda *args: wanted))
    a = torch.zeros(rows, inner + 4)[:, off : off + inner]
    before = kernels.LAUNCHES.count
    kernels.gemm_f32(a, torch.zeros(width, inner), torch.empty(rows, width))
    assert kernels.LAUNCHES.count - before == launches
