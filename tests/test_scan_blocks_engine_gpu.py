"""An engine's step over prompts long enough for blocks of tokens, beside a short one, and the tokens that follow."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
TOKENS = 1024      # a step's


def engine(kind):
    from rapid_llm_b200 import EngineConfig
    from rapid_llm_b200.config.model_spec import LayerSpec, ModelSpec, PartSpec, ScheduleEntry
    from rapid_llm_b200.engine.runner import ModelRunner
    from rapid_llm_b200.models.causal_lm import CausalLM
    from rapid_llm_b200.weights import fill_random_on_device

    hidden, norm = 256, PartSpec("rmsnorm", {"size": 256, "eps": 1e-6, "name": ""})
    if kind == "delta":
        mixer = PartSpec("gated_delta_rule", {"hidden_size": hidden, "num_heads": 2, "num_kv_heads": 2, "key_dim": 128, "value_dim": 128,
                                              "conv_width": 4, "decay_rank": 16, "gate_rank": 16, "norm_eps": 1e-6})
    else:
        mixer = PartSpec("lightning", {"hidden_size": hidden, "num_heads": 32, "key_dim": 128, "value_dim": 128,
                                       "decay": tuple(1 - 2.0 ** (-3 - h / 8) for h in range(32)), "norm_eps": 1e-6})
    names = {"mixer_norm": "norm1", "mixer": "mix.", "feed_forward_norm": "norm2", "feed_forward": "mlp."}
    spec = ModelSpec(
        architecture="Two layers", vocab_size=64, hidden_size=hidden, max_positions=1 << 12,
        embedding=PartSpec("token_embedding", {"vocab_size": 64, "hidden_size": hidden, "name": ""}),
        layers=tuple(LayerSpec(arrangement="prenorm", mixer=mixer, feed_forward=None, norm=norm, prefix=f"l{i}.", names=names) for i in range(2)),
        schedule=(ScheduleEntry(0), ScheduleEntry(1)), final_norm=norm,
        head=PartSpec("lm_head", {"vocab_size": 64, "hidden_size": hidden, "tied": True}),
        final_norm_prefix="final.norm", embedding_prefix="embed", head_prefix="head.")
    model = CausalLM(spec, torch.bfloat16, DEV)
    fill_random_on_device(model, 3, std=0.05, norm_std=0.1)
    return ModelRunner(model, EngineConfig(dtype=torch.bfloat16, max_seq_len=2048, num_pages=300, max_num_seqs=3, max_num_batched_tokens=TOKENS,
                                           max_chunk_size=TOKENS, use_cuda_graph=False))


@pytest.mark.parametrize("kind,long", [("delta", 700), ("lightning", 300)])
def test_a_step_in_blocks_and_the_tokens_behind_it(monkeypatch, kind, long):
    from rapid_llm_b200.engine.runner import StepEntry
    from rapid_llm_b200.ops import kernels

    rule, asked = kernels.scan_blocks_from, []
    results = []
    for blocks in (True, False):
        def taken(*args):
            asked.append(rule(*args))
            return asked[-1] if blocks else 0

        monkeypatch.setattr(kernels, "scan_blocks_from", taken)
        runner = engine(kind)
        generator = torch.Generator().manual_seed(1)
        prompts = [torch.randint(64, (n,), generator=generator).tolist() for n in (long, 9, long + 20)]
        for i in range(3):
            runner.admit(i)
        rows = [runner.step([StepEntry(i, prompts[i], [len(prompts[i]) - 1]) for i in group]).float().clone() for group in ((0, 1), (2,))]
        rows.append(runner.step([StepEntry(i, [7 + i], [0]) for i in range(3)]).float().clone())
        assert int(runner.fault.item()) == 0
        results.append(torch.cat(rows))
    assert 0 < asked[-1] <= long      # the rule of this engine's steps takes these prompts
    blocks, walked = results
    # orders of float32 sums, which bfloat16 rows round off once in a while: a few roundings of 2^-9 in what two layers add up to
    assert float((blocks - walked).norm() / walked.norm()) <= 4 * 2.0 ** -9
    assert bool(torch.isfinite(blocks).all()) and float(walked.abs().max()) > 0
