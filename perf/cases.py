"""What the engine is asked to do in earnest, as calls that can be timed and checked.

Whole calls: a decode step of the Qwen3 decoder replayed from its captured graph, a step over prompts, and the same in the
true 32-bit path (sizes of the 8B, 14B and tiny configurations of the benchmark and the tests, fewer layers).  Single parts
of the other architectures, at the widths of their benchmarks: the recurrent mixers, the routed feed-forward and the
attention over a cached latent, each on prompts and on single tokens.  A decode step of a part is replayed from a graph
captured with dependent launches, as the engine replays its own; prompts are launched one kernel after the other, as the
engine does.  Weights and inputs are random (matrices of variance 1 / inputs unless the model's own convention says
otherwise, decays between about 0.9 and 1), drawn on the GPU from the seed.
"""

from __future__ import annotations

import math

import torch

from rapid_llm_b200 import EngineConfig, Qwen3Config
from rapid_llm_b200.config.model_spec import LayerSpec, ModelSpec, PartSpec, ScheduleEntry
from rapid_llm_b200.engine.runner import ModelRunner, StepEntry
from rapid_llm_b200.models.causal_lm import CausalLM
from rapid_llm_b200.ops import kernels

DEV = "cuda:0"
F32, F64 = torch.float32, torch.float64
EPS = 1e-6
PAGE = 16
ROOM = 3072             # positions a decoding request may grow by before its case starts over

# -- the cases --------------------------------------------------------------------------------------------------------------

QWEN_8B = {"hidden": 4096, "heads": 32, "kv_heads": 8, "inter": 12288, "vocab": 151936}
QWEN_14B = {"hidden": 5120, "heads": 40, "kv_heads": 8, "inter": 17408, "vocab": 151936}


def listed() -> list[dict]:
    return [
        # one user's next token: the smallest step, bound by the weights' stream and the launches between
        {"name": "decode_1", "kind": "decode", "dtype": "bf16", "layers": 8, "batch": 1, "context": 1024, **QWEN_8B},
        # a full serving batch's next tokens
        {"name": "decode_64", "kind": "decode", "dtype": "bf16", "layers": 8, "batch": 64, "context": 1024, **QWEN_8B},
        # the benchmark's prompt, one step of 2,048 tokens
        {"name": "prompt_2048", "kind": "prompt", "dtype": "bf16", "layers": 4, "lengths": "2048", **QWEN_8B},
        # the 32-bit path over the ragged prompts of the second tiny configuration's workload, at real widths
        {"name": "prompts_32_bit", "kind": "prompt", "dtype": "f32", "layers": 1, "lengths": "1,7,31,64,100", **QWEN_8B},
        # Kopatar's delta rule over one prompt
        {"name": "delta_prompt", "kind": "delta", "width": 2048, "dim": 128, "lengths": "2048", "context": 0},
        # Mezadra's linear attention over a packed step of ragged prompts, the larger width
        {"name": "lightning_prompts", "kind": "lightning", "width": 4096, "dim": 128, "lengths": "700,333,1015", "context": 0},
        # Danalorn's gated linear attention over one prompt
        {"name": "gla_prompt", "kind": "gla", "width": 2048, "dim": 64, "lengths": "2048", "context": 0},
        # Basitar's recurrence at 64 single tokens of a serving batch
        {"name": "wkv_decode_64", "kind": "wkv", "width": 4096, "dim": 64, "lengths": ",".join(["1"] * 64), "context": 1024},
        # Mezadra's routed feed-forward (shared expert and gate) over a prompt
        {"name": "experts_prompt", "kind": "experts", "width": 2048, "inter": 512, "experts": 16, "top": 2, "shared": 1024,
         "tokens": 2048},
        # Basitar's routed feed-forward for a small decoding batch
        {"name": "experts_decode_8", "kind": "experts", "width": 2048, "inter": 512, "experts": 16, "top": 2, "shared": 0,
         "tokens": 8},
        # Basitar's latent attention over one prompt
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "lengths": "2048", "context": 0},
        # the same for a batch of single tokens behind 1,024 cached rows
        {"name": "latent_decode_64", "kind": "latent", "width": 2048, "lengths": ",".join(["1"] * 64), "context": 1024},
    ]


def _spread(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _ragged(rng, total: int) -> str:
    """``total`` tokens as one prompt or a few of uneven lengths."""
    parts, left = [], total
    for _ in range(rng.choice((0, 0, 1, 2, 4))):
        if left > 2:
            parts.append(rng.randint(1, left // 2))
            left -= parts[-1]
    return ",".join(str(n) for n in parts + [left])


def draw(rng) -> dict:
    kind = rng.choice(("decode", "prompt", "prompt", "f32", "delta", "lightning", "gla", "wkv", "experts", "experts", "latent", "latent"))
    if kind == "decode":
        model = rng.choice((QWEN_8B, QWEN_14B))
        return {"kind": "decode", "dtype": "bf16", "layers": rng.randint(4, 8), "batch": _spread(rng, 1, 64),
                "context": _spread(rng, 64, 2048), **model}
    if kind == "prompt":
        model = rng.choice((QWEN_8B, QWEN_14B))
        return {"kind": "prompt", "dtype": "bf16", "layers": 2, "lengths": _ragged(rng, _spread(rng, 65, 2048)), **model}
    if kind == "f32":
        return {"kind": "prompt", "dtype": "f32", "layers": 1, "lengths": _ragged(rng, _spread(rng, 1, 400)), **QWEN_8B}
    width = rng.choice((1024, 1536, 2048, 3072, 4096))
    if kind == "experts":
        return {"kind": "experts", "width": width, "inter": width // 4, "experts": rng.choice((8, 16, 32)), "top": rng.choice((1, 2, 4)),
                "shared": rng.choice((0, width // 2)), "tokens": _spread(rng, 1, 4096 if width <= 2048 else 2048)}
    single = rng.random() < 0.4
    lengths = ",".join(["1"] * _spread(rng, 1, 64)) if single else _ragged(rng, _spread(rng, 16, 2048))
    context = _spread(rng, 16, 4096) if single else 0
    if kind == "latent":
        return {"kind": "latent", "width": width, "lengths": lengths, "context": context}
    return {"kind": kind, "width": width, "dim": rng.choice((64, 128)), "lengths": lengths, "context": context}


def _lengths(case) -> list[int]:
    return [int(n) for n in case["lengths"].split(",")]


# -- tensors from a seed -----------------------------------------------------------------------------------------------------

def _random(seed: int, label: str, shape, std: float = 1.0, low: float | None = None, high: float | None = None) -> torch.Tensor:
    """Float32 numbers on the GPU that depend on the seed and the label alone."""
    key = (int(seed) * 1000003 + sum((i + 1) * 131 ** (i % 5) * ord(c) for i, c in enumerate(label))) % (1 << 62)
    generator = torch.Generator(device=DEV).manual_seed(key)
    out = torch.empty(shape, dtype=F32, device=DEV)
    if low is not None:
        return out.uniform_(low, high, generator=generator)
    return out.normal_(0.0, std, generator=generator)


def _dtype(case):
    return F32 if case.get("dtype") == "f32" else torch.bfloat16


def _matrix(seed, label, shape, dtype, std=None):
    return _random(seed, label, shape, shape[-1] ** -0.5 if std is None else std).to(dtype)


def _qwen_tensor(case, seed, name: str) -> torch.Tensor:
    h, d, i, v = case["hidden"], 128, case["inter"], case["vocab"]
    cq, ckv = case["heads"] * d, case["kv_heads"] * d
    tail = name.rsplit("layers.", 1)[-1].split(".", 1)[-1] if "layers." in name else name
    matrices = {"self_attn.q_proj.weight": (cq, h), "self_attn.k_proj.weight": (ckv, h), "self_attn.v_proj.weight": (ckv, h),
                "self_attn.o_proj.weight": (h, cq), "mlp.gate_proj.weight": (i, h), "mlp.up_proj.weight": (i, h),
                "mlp.down_proj.weight": (h, i), "model.embed_tokens.weight": (v, h), "lm_head.weight": (v, h)}
    if tail in matrices:
        return _matrix(seed, name, matrices[tail], _dtype(case), std=0.02)
    return 1.0 + _random(seed, name, (d,) if "self_attn" in name else (h,), 0.1)


def _heads(case) -> int:
    return case["width"] // case["dim"]


def _mixer_tensors(case, seed) -> dict[str, torch.Tensor]:
    """The part's checkpoint tensors by name: matrices in bfloat16, vectors in float32."""
    w, kind, bf = case["width"], case["kind"], torch.bfloat16
    m = lambda name, *shape, std=None: _matrix(seed, name, shape, bf, std)      # noqa: E731
    if kind == "latent":
        heads, plain, rot, vdim, rank, q_rank = _latent_sizes(case)
        return {"dq": m("dq", q_rank, w), "dq.norm": 1.0 + _random(seed, "dq.norm", (q_rank,), 0.1),
                "uq": m("uq", heads * (plain + rot), q_rank, std=2.0 * q_rank ** -0.5), "dkv": m("dkv", rank + rot, w),
                "dkv.norm": 1.0 + _random(seed, "dkv.norm", (rank,), 0.1), "uk": m("uk", heads * plain, rank),
                "uv": m("uv", heads * vdim, rank), "o": m("o", w, heads * vdim)}
    if kind == "experts":
        e, f, s = case["experts"], case["inter"], case["shared"]
        out = {}
        for index in range(e):
            out.update({f"e{index}.gate": m(f"e{index}.gate", f, w), f"e{index}.up": m(f"e{index}.up", f, w),
                        f"e{index}.down": m(f"e{index}.down", w, f)})
        out["router"] = _random(seed, "router", (e, w), w ** -0.5)
        if s:
            out.update({"shared.gate": m("shared.gate", s, w), "shared.up": m("shared.up", s, w),
                        "shared.down": m("shared.down", w, s), "shared.sg": _random(seed, "shared.sg", (1, w), w ** -0.5)})
        else:
            out["router.b"] = _random(seed, "router.b", (e,), 0.3)
        return out
    heads, dim = _heads(case), case["dim"]
    c = heads * dim
    out = {name: m(name, c, w) for name in (("r", "k", "v", "g") if kind == "wkv" else ("q", "k", "v"))}
    out["o"] = m("o", w, c)
    if kind == "lightning":
        out.update({"g": m("g", c, w), "norm": 1.0 + _random(seed, "norm", (c,), 0.1)})
    elif kind == "gla":
        out.update({"g": m("g", c, w), "norm": 1.0 + _random(seed, "norm", (dim,), 0.1), "a1": m("a1", 16, w), "a2": m("a2", c, 16),
                    "a2.b": _random(seed, "a2.b", (c,), low=0.0, high=4.0)})
    elif kind == "wkv":
        out.update({f"mu.{which}": _random(seed, f"mu.{which}", (w,), low=0.0, high=1.0) for which in ("r", "k", "v", "g", "w")})
        out.update({"w1": m("w1", 64, w), "w2": m("w2", c, 64, std=0.5 * 64 ** -0.5), "w0": _random(seed, "w0", (c,), low=-6.0, high=-2.0),
                    "u": _random(seed, "u", (heads, dim), 0.5), "norm": 1.0 + _random(seed, "norm", (c,), 0.1)})
    else:
        rank = w // 16
        out.update({f"{which}.conv": _random(seed, f"{which}.conv", (c, 4), 0.5) for which in ("q", "k", "v")})
        out.update({"b": m("b", heads, w), "a1": m("a1", rank, w), "a2": m("a2", c, rank), "g1": m("g1", rank, w), "g2": m("g2", c, rank),
                    "A_log": _random(seed, "A_log", (heads,), low=-5.0, high=-2.0), "dt_bias": _random(seed, "dt_bias", (c,), 0.5),
                    "norm": 1.0 + _random(seed, "norm", (dim,), 0.1)})
    return out


def _latent_sizes(case):
    w = case["width"]
    return w // 128, 128, 64, 128, 192, 3 * w // 8      # heads, plain, rotated, values, latent, query latent


def _decays(heads: int) -> tuple:
    return tuple(1.0 - 2.0 ** (-3 - 7 * h / max(heads - 1, 1)) for h in range(heads))


def _part(case) -> PartSpec:
    w, kind = case["width"], case["kind"]
    if kind == "latent":
        heads, plain, rot, vdim, rank, q_rank = _latent_sizes(case)
        return PartSpec("latent_attention", {
            "hidden_size": w, "num_heads": heads, "head_dim": plain, "rot_dim": rot, "value_dim": vdim, "kv_rank": rank,
            "q_rank": q_rank, "scale": (plain + rot) ** -0.5, "norm_eps": EPS, "rotation": "halves",
            "position": PartSpec("rotary_frequencies", {"rotary_dim": rot, "theta": 10000.0, "max_positions": 1 << 15})})
    if kind == "experts":
        options = ({"shared_size": case["shared"], "shared_gate": True, "scale_input": True} if case["shared"] else
                   {"scale_input": False, "router_bias": True, "weighting": "softmax_chosen"})
        return PartSpec("routed_experts", {"hidden_size": w, "num_experts": case["experts"], "top_k": case["top"],
                                           "expert_size": case["inter"], **options})
    heads, dim = _heads(case), case["dim"]
    if kind == "lightning":
        return PartSpec("lightning", {"hidden_size": w, "num_heads": heads, "key_dim": dim, "value_dim": dim, "decay": _decays(heads),
                                      "norm_eps": EPS})
    if kind == "gla":
        return PartSpec("gated_linear", {"hidden_size": w, "num_heads": heads, "key_dim": dim, "value_dim": dim, "decay_rank": 16,
                                         "tau": 16.0, "norm_eps": EPS})
    if kind == "wkv":
        return PartSpec("wkv", {"hidden_size": w, "num_heads": heads, "key_dim": dim, "decay_rank": 64, "norm_eps": EPS})
    return PartSpec("gated_delta_rule", {"hidden_size": w, "num_heads": heads, "num_kv_heads": heads, "key_dim": dim, "value_dim": dim,
                                         "conv_width": 4, "decay_rank": w // 16, "gate_rank": w // 16, "norm_eps": EPS})


def _state_rows(case, seed) -> torch.Tensor:
    """What the requests of a decoding recurrence carry: ``[requests, heads, value channel, key channel]`` (the row before
    and the convolutions' last inputs are zeros)."""
    return _random(seed, "state", (len(_lengths(case)), _heads(case), case["dim"], case["dim"]), 0.3)


def _latent_rows(case, seed) -> torch.Tensor:
    return _random(seed, "rows", (len(_lengths(case)), case["context"], 256)).to(torch.bfloat16)


def _inputs(case, seed) -> torch.Tensor:
    tokens = case["tokens"] if case["kind"] == "experts" else sum(_lengths(case))
    return _random(seed, "x", (tokens, case["width"])).to(torch.bfloat16)


def _token_ids(case, seed, count: int, label: str) -> list[int]:
    return _random(seed, label, (count,), low=0.0, high=float(case["vocab"])).long().clamp_(max=case["vocab"] - 1).tolist()


# -- what a program has in hand, and one pass --------------------------------------------------------------------------------

def _qwen_runner(case, seed, **sizes) -> ModelRunner:
    config = Qwen3Config.from_dict({
        "architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "vocab_size": case["vocab"], "hidden_size": case["hidden"],
        "intermediate_size": case["inter"], "num_hidden_layers": case["layers"], "num_attention_heads": case["heads"],
        "num_key_value_heads": case["kv_heads"], "head_dim": 128, "max_position_embeddings": 40960, "rms_norm_eps": EPS,
        "rope_theta": 1000000.0, "tie_word_embeddings": False})
    model = CausalLM(config.to_spec(), _dtype(case), DEV)
    names = list(model.tensor_specs())
    for name in names:
        model.load_tensor(name, _qwen_tensor(case, seed, name))
    model.finalize(set(names))
    return ModelRunner(model, EngineConfig(dtype=_dtype(case), page_size=PAGE, use_cuda_graph=True, **sizes))


def _prepare_decode(case, seed):
    batch, context = case["batch"], case["context"]
    most = context + ROOM
    runner = _qwen_runner(case, seed, max_seq_len=most, num_pages=batch * (-(-most // PAGE)), max_num_seqs=batch,
                          max_num_batched_tokens=4096, max_chunk_size=4096)
    ids = _token_ids(case, seed, batch * (context + 1), "ids")
    prompts = [ids[i * (context + 1) : (i + 1) * (context + 1)] for i in range(batch)]
    state = {"runner": runner, "prompts": prompts, "left": 0,
             "entries": [StepEntry(i, [prompt[-1]], [0]) for i, prompt in enumerate(prompts)]}
    _start_requests(state)
    return state


def _start_requests(state) -> None:
    runner, context = state["runner"], len(state["prompts"][0]) - 1
    for i in range(len(state["prompts"])):
        if runner.cache.has(i):
            runner.release(i)
    together = max(1, 4096 // context)
    for first in range(0, len(state["prompts"]), together):
        group = list(range(first, min(first + together, len(state["prompts"]))))
        for i in group:
            runner.admit(i)
        runner.step([StepEntry(i, state["prompts"][i][:-1]) for i in group])
    state["left"] = ROOM


def _prepare_prompt(case, seed):
    lengths = _lengths(case)
    total = sum(lengths)
    runner = _qwen_runner(case, seed, max_seq_len=max(lengths) + 16, num_pages=sum(-(-n // PAGE) for n in lengths) + len(lengths),
                          max_num_seqs=len(lengths), max_num_batched_tokens=total, max_chunk_size=total)
    ids, entries, at = _token_ids(case, seed, total, "ids"), [], 0
    for i, n in enumerate(lengths):
        entries.append(StepEntry(i, ids[at : at + n], [n - 1]))
        at += n
    return {"runner": runner, "entries": entries}


def _one_layer_runner(case, seed, lengths, context) -> ModelRunner:
    """An engine around one layer that holds the part (a feed-forward stands behind a small mixer)."""
    w, norm = case["width"], PartSpec("rmsnorm", {"size": case["width"], "eps": EPS, "name": ""})
    if case["kind"] == "experts":
        mixer = PartSpec("lightning", {"hidden_size": w, "num_heads": 1, "key_dim": 16, "value_dim": 16, "decay": (0.9,), "norm_eps": EPS})
        feed_forward = _part(case)
    else:
        mixer, feed_forward = _part(case), None
    names = {"mixer_norm": "norm1", "mixer": "mix.", "feed_forward_norm": "norm2", "feed_forward": "mlp."}
    spec = ModelSpec(
        architecture="One layer", vocab_size=64, hidden_size=w, max_positions=1 << 15,
        embedding=PartSpec("token_embedding", {"vocab_size": 64, "hidden_size": w, "name": ""}),
        layers=(LayerSpec(arrangement="prenorm", mixer=mixer, feed_forward=feed_forward, norm=norm, prefix="l0.", names=names),),
        schedule=(ScheduleEntry(0),), final_norm=norm, head=PartSpec("lm_head", {"vocab_size": 64, "hidden_size": w, "tied": True}),
        final_norm_prefix="final.norm", embedding_prefix="embed", head_prefix="head.")
    model = CausalLM(spec, torch.bfloat16, DEV)
    part = model.layers[0].feed_forward if case["kind"] == "experts" else model.layers[0].mixer
    tensors = _mixer_tensors(case, seed)
    for name, tensor in tensors.items():
        part.load_tensor(name, tensor)
    part.finalize(set(tensors))
    most = context + max(lengths)
    return ModelRunner(model, EngineConfig(
        dtype=torch.bfloat16, max_seq_len=max(most, 2), page_size=PAGE, num_pages=sum(-(-(context + n) // PAGE) for n in lengths),
        max_num_seqs=len(lengths), max_num_batched_tokens=max(sum(lengths), 1), max_chunk_size=max(lengths)))


def _prepare_part(case, seed):
    experts = case["kind"] == "experts"
    lengths, context = ([case["tokens"]], 0) if experts else (_lengths(case), case["context"])
    runner = _one_layer_runner(case, seed, lengths, context)
    for i in range(len(lengths)):
        runner.admit(i)
        if context:
            runner.cache.reserve(i, context)
    batch = runner.prepare([StepEntry(i, [0] * n) for i, n in enumerate(lengths)])
    cache = runner.layer_caches()[0]
    layer = runner.model.layers[0]
    x = _inputs(case, seed)
    outputs = {}
    if experts:
        forward = lambda: layer.feed_forward.forward(x, batch)                  # noqa: E731
    else:
        forward = lambda: layer.mixer.forward(x, batch, cache)                  # noqa: E731
        if case["kind"] == "latent":
            if context:
                rows = _latent_rows(case, seed)
                for i in range(len(lengths)):
                    places = torch.from_numpy(runner.cache.kv_destinations(0, runner.cache.slot_of(i), 0, context)).to(DEV).long()
                    cache.pages.view(-1, 256)[places] = rows[i]
        else:
            carried = _heads(case) * case["dim"] ** 2
            slots = [runner.cache.slot_of(i) for i in range(len(lengths))]
            if context:
                rows = _state_rows(case, seed).view(len(lengths), carried)
                for i, slot in enumerate(slots):
                    cache.state[slot, :carried] = rows[i]
            if slots != list(range(len(slots))):
                raise RuntimeError("the requests did not get the first slots in order")
            outputs["state"] = cache.state[: len(slots), :carried]
    state = {"forward": forward, "outputs": outputs, "runner": runner, "graph": None}
    tokens = x.shape[0]
    if (context or experts) and tokens <= 64:        # single tokens are replayed from a graph, as the engine does
        kept = None if cache.state is None else cache.state.clone()
        for _ in range(2):
            out = _as_a_step(forward)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _as_a_step(forward)
        if kept is not None:
            cache.state.copy_(kept)
        state["graph"], state["result"] = graph, {"y": out, **outputs}
    return state


def _as_a_step(forward):
    """The part's kernels chained by dependent launches, as the engine chains those of a step."""
    before = kernels.PDL
    kernels.PDL = True
    try:
        return forward()
    finally:
        kernels.PDL = before


@torch.no_grad()
def prepare(case, seed):
    if case["kind"] == "decode":
        state = _prepare_decode(case, seed)
    elif case["kind"] == "prompt":
        state = _prepare_prompt(case, seed)
    else:
        state = _prepare_part(case, seed)
    state["kind"] = case["kind"]
    return state


@torch.no_grad()
def run(state):
    if state["kind"] == "decode":
        if state["left"] == 0:
            _start_requests(state)
        state["left"] -= 1
        return state["runner"].step_decode(state["entries"])
    if state["kind"] == "prompt":
        runner = state["runner"]
        for entry in state["entries"]:
            runner.admit(entry.request_id)
        logits = runner.step(state["entries"])
        for entry in state["entries"]:
            runner.release(entry.request_id)
        return logits
    if state["graph"] is not None:
        state["graph"].replay()
        return state["result"]
    return {"y": _as_a_step(state["forward"]), **state["outputs"]}


# -- the work that cannot be left out ----------------------------------------------------------------------------------------

def work(case) -> dict:
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        size = 4 if case["dtype"] == "f32" else 2
        h, d = case["hidden"], 128
        cq, ckv = case["heads"] * d, case["kv_heads"] * d
        per_layer = (cq + 2 * ckv) * h + h * cq + 3 * case["inter"] * h
        lengths = [1] * case["batch"] if kind == "decode" else _lengths(case)
        context = case["context"] if kind == "decode" else 0
        tokens, rows = sum(lengths), len(lengths)
        keys = sum((context + n) * (context + n + 1) // 2 - context * (context + 1) // 2 for n in lengths)
        cached = sum(context + n for n in lengths)
        return {"bytes": case["layers"] * (per_layer * size + (cached + tokens) * 2 * ckv * size) + case["vocab"] * h * size
                + tokens * h * size + rows * case["vocab"] * size,
                "flops": case["layers"] * (2.0 * tokens * per_layer + 4.0 * keys * cq) + 2.0 * rows * case["vocab"] * h}
    w = case["width"]
    if kind == "experts":
        t, e, top, f, s = case["tokens"], case["experts"], case["top"], case["inter"], case["shared"]
        touched = e * (1.0 - (1.0 - top / e) ** t)
        weights = (touched * 3 * f * w + 3 * s * w) * 2 + (e + 1) * w * 4
        return {"bytes": weights + t * w * 4, "flops": 6.0 * t * top * f * w + 6.0 * t * s * w + 2.0 * t * e * w}
    lengths, context = _lengths(case), case["context"]
    t = sum(lengths)
    if kind == "latent":
        heads, plain, rot, vdim, rank, q_rank = _latent_sizes(case)
        weights = w * (q_rank + rank + rot) + heads * (plain + rot) * q_rank + heads * rank * (plain + vdim) + w * heads * vdim
        keys = sum((context + n) * (context + n + 1) // 2 - context * (context + 1) // 2 for n in lengths)
        expanded = 2.0 * heads * (plain + rot + vdim) * keys         # per key when keys and values are laid out per head
        absorbed = 2.0 * heads * (2 * rank + rot) * keys             # per key when the latent itself is attended
        return {"bytes": weights * 2 + t * w * 4 + sum(context + 2 * n for n in lengths) * (rank + rot) * 2,
                "flops": 2.0 * t * weights + (absorbed if context else min(expanded, absorbed))}
    heads, dim = _heads(case), case["dim"]
    c = heads * dim
    products = {"lightning": 5 * c * w, "gla": 5 * c * w + 16 * (w + c), "wkv": 5 * c * w + 64 * (w + c),
                "delta": 4 * c * w + heads * w + 2 * (w // 16) * (w + c)}[kind]
    states = len(lengths) * c * dim * 4 * (2 if context else 1)
    return {"bytes": products * 2 + t * w * 4 + states, "flops": 2.0 * t * products + (6.0 if kind == "delta" else 4.0) * t * c * dim}


# -- how far another correct implementation may be --------------------------------------------------------------------------

def tolerance(case) -> dict:
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        return {"rel": 2e-5, "max": 2e-4} if case["dtype"] == "f32" else {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.3}


# -- the same in 64 bits, plain ----------------------------------------------------------------------------------------------

def _norm64(x, weight=None, eps=EPS):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _rotate64(x, positions, theta):
    """Entry ``i`` paired with ``i + half``; ``x [T, heads, D]``."""
    half = x.shape[-1] // 2
    angle = positions.to(F64).view(-1, 1, 1) * theta ** (-torch.arange(half, dtype=F64, device=x.device) / half)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def _softmax64(scores, first_position):
    rows, keys = scores.shape[-2:]
    at = first_position + torch.arange(rows, device=scores.device)
    hidden = torch.arange(keys, device=scores.device)[None, :] > at[:, None]
    return torch.softmax(scores.masked_fill(hidden, -math.inf), dim=-1)


def _exact_qwen(case, seed):
    lengths = [case["context"] + 1] * case["batch"] if case["kind"] == "decode" else _lengths(case)
    tokens, layers = sum(lengths), case["layers"]
    if tokens * layers * (case["hidden"] + case["inter"]) > 3.0e9:
        return None
    tensor = lambda name: _qwen_tensor(case, seed, name).to(F64)      # noqa: E731
    ids = torch.tensor(_token_ids(case, seed, tokens, "ids"), device=DEV)
    x = _qwen_tensor(case, seed, "model.embed_tokens.weight")[ids].to(F64)
    ends = torch.tensor(lengths, device=DEV).cumsum(0).tolist()
    heads, kv, d = case["heads"], case["kv_heads"], 128
    positions = torch.cat([torch.arange(n, device=DEV) for n in lengths])
    for layer in range(layers):
        p = f"model.layers.{layer}."
        h = _norm64(x, tensor(p + "input_layernorm.weight"))
        q = (h @ tensor(p + "self_attn.q_proj.weight").T).view(tokens, heads, d)
        k = (h @ tensor(p + "self_attn.k_proj.weight").T).view(tokens, kv, d)
        v = (h @ tensor(p + "self_attn.v_proj.weight").T).view(tokens, kv, d)
        q = _rotate64(_norm64(q, tensor(p + "self_attn.q_norm.weight")), positions, 1.0e6)
        k = _rotate64(_norm64(k, tensor(p + "self_attn.k_norm.weight")), positions, 1.0e6)
        mixed = torch.empty(tokens, heads, d, dtype=F64, device=DEV)
        for end, n in zip(ends, lengths):
            rows = slice(end - n, end)
            for g in range(kv):
                mine = slice(g * heads // kv, (g + 1) * heads // kv)
                weights = _softmax64(torch.einsum("ihd,jd->hij", q[rows, mine], k[rows, g]) * d ** -0.5, 0)
                mixed[rows, mine] = torch.einsum("hij,jd->ihd", weights, v[rows, g])
        x = x + mixed.view(tokens, heads * d) @ tensor(p + "self_attn.o_proj.weight").T
        h = _norm64(x, tensor(p + "post_attention_layernorm.weight"))
        gate = h @ tensor(p + "mlp.gate_proj.weight").T
        gate = gate * torch.sigmoid(gate) * (h @ tensor(p + "mlp.up_proj.weight").T)
        x = x + gate @ tensor(p + "mlp.down_proj.weight").T
    x = _norm64(x[[end - 1 for end in ends]], tensor("model.norm.weight"))
    return x @ tensor("lm_head.weight").T


def _exact_experts(case, seed, w, x):
    logits = x @ w["router"].T + (w["router.b"] if "router.b" in w else 0.0)
    best, chosen = logits.topk(case["top"], dim=-1)
    weights = torch.sigmoid(best) if case["shared"] else torch.softmax(best, dim=-1)
    y = torch.zeros_like(x)
    for e in range(case["experts"]):
        at, place = (chosen == e).nonzero(as_tuple=True)
        if not at.numel():
            continue
        s = weights[at, place][:, None]
        given = x[at] * s if case["shared"] else x[at]
        gate = given @ w[f"e{e}.gate"].T
        one = (gate * torch.sigmoid(gate) * (given @ w[f"e{e}.up"].T)) @ w[f"e{e}.down"].T
        y[at] += one if case["shared"] else one * s
    if case["shared"]:
        gate = x @ w["shared.gate"].T
        y += (gate * torch.sigmoid(gate) * (x @ w["shared.up"].T)) @ w["shared.down"].T * torch.sigmoid(x @ w["shared.sg"].T)
    return {"y": y}


def _exact_latent(case, seed, w, x):
    heads, plain, rot, vdim, rank, _ = _latent_sizes(case)
    lengths, context = _lengths(case), case["context"]
    positions = torch.cat([context + torch.arange(n, device=DEV) for n in lengths])
    q = (_norm64(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(-1, heads, plain + rot)
    q_rot = _rotate64(q[..., plain:], positions, 1.0e4)
    down = x @ w["dkv"].T
    c, k_rot = _norm64(down[:, :rank], w["dkv.norm"]), _rotate64(down[:, None, rank:], positions, 1.0e4)[:, 0]
    old = _latent_rows(case, seed).to(F64) if context else None
    uk, uv = w["uk"].view(heads, plain, rank), w["uv"].view(heads, vdim, rank)
    mixed = torch.empty(x.shape[0], heads, vdim, dtype=F64, device=DEV)
    at = 0
    for i, n in enumerate(lengths):
        rows = slice(at, at + n)
        keys_c = c[rows] if old is None else torch.cat([old[i, :, :rank], c[rows]])
        keys_r = k_rot[rows] if old is None else torch.cat([old[i, :, rank:], k_rot[rows]])
        for h in range(heads):
            scores = (q[rows, h, :plain] @ uk[h]) @ keys_c.T + q_rot[rows, h] @ keys_r.T
            mixed[rows, h] = (_softmax64(scores * (plain + rot) ** -0.5, context) @ keys_c) @ uv[h].T
        at += n
    return {"y": mixed.view(-1, heads * vdim) @ w["o"].T}


def _exact_recurrence(case, seed, w, x):
    kind, heads, dim, lengths = case["kind"], _heads(case), case["dim"], _lengths(case)
    c, t = heads * dim, x.shape[0]
    silu = lambda z: z * torch.sigmoid(z)      # noqa: E731
    beta = bonus = None
    if kind == "lightning":
        q, k, v = (silu(x @ w[name].T).view(t, heads, dim) for name in "qkv")
        decay = torch.tensor(_decays(heads), dtype=F32, device=DEV).to(F64).view(1, heads, 1).expand(t, heads, dim)
    elif kind == "gla":
        q, k, v = ((x @ w[name].T).view(t, heads, dim) for name in "qkv")
        q = q * dim ** -0.5
        decay = torch.sigmoid(x @ w["a1"].T @ w["a2"].T + w["a2.b"]).pow(1.0 / 16.0).view(t, heads, dim)
    elif kind == "wkv":
        before = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
        before[torch.tensor([0] + lengths, device=DEV).cumsum(0)[:-1]] = 0.0
        blend = lambda name: x + (before - x) * w["mu." + name]      # noqa: E731
        q, k, v = ((blend(name) @ w[name].T).view(t, heads, dim) for name in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(blend("w") @ w["w1"].T) @ w["w2"].T + w["w0"])).view(t, heads, dim)
        bonus = w["u"].view(heads, dim, 1)
    else:
        def convolved(name):
            z, out = x @ w[name].T, torch.zeros(t, c, dtype=F64, device=DEV)
            local = torch.cat([torch.arange(n, device=DEV) for n in lengths])[:, None]
            for back in range(4):
                shifted = torch.cat([torch.zeros_like(z[:back]), z[: t - back]])
                out += torch.where(local >= back, shifted, torch.zeros_like(z)) * w[name + ".conv"][:, 3 - back]
            return silu(out).view(t, heads, dim)

        q, k, v = convolved("q"), convolved("k"), convolved("v")
        q = q / torch.sqrt(q.square().sum(-1, keepdim=True) + 1e-6) * dim ** -0.5
        k = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        beta = torch.sigmoid(x @ w["b"].T)
        step = torch.nn.functional.softplus(x @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(t, heads, dim)
        decay = torch.exp(-torch.exp(w["A_log"]).view(1, heads, 1) * step)
    read = torch.empty(t, heads, dim, dtype=F64, device=DEV)
    carried = _state_rows(case, seed).to(F64).transpose(2, 3) if case["context"] else None
    states, at = [], 0
    for i, n in enumerate(lengths):
        S = carried[i].clone() if carried is not None else torch.zeros(heads, dim, dim, dtype=F64, device=DEV)
        for row in range(at, at + n):
            kk, vv, dd = k[row][:, :, None], v[row][:, None, :], decay[row][:, :, None]
            if bonus is not None:
                read[row] = torch.einsum("hkv,hk->hv", S + bonus * kk * vv, q[row])
                S = dd * S + kk * vv
                continue
            S = dd * S
            S = S + kk * (vv if beta is None else beta[row][:, None, None] * (vv - torch.einsum("hkv,hk->hv", S, k[row])[:, None, :]))
            read[row] = torch.einsum("hkv,hk->hv", S, q[row])
        states.append(S.transpose(1, 2).reshape(-1))
        at += n
    if kind == "lightning":
        y = _norm64(read.reshape(t, c), w["norm"]) * torch.sigmoid(x @ w["g"].T)
    elif kind == "gla":
        y = (_norm64(read, w["norm"])).reshape(t, c) * silu(x @ w["g"].T)
    elif kind == "wkv":
        y = _norm64(read).reshape(t, c) * w["norm"] * silu(blend("g") @ w["g"].T)
    else:
        y = (_norm64(read) * w["norm"]).reshape(t, c) * torch.sigmoid(x @ w["g1"].T @ w["g2"].T)
    return {"y": y @ w["o"].T, "state": torch.stack(states)}


@torch.no_grad()
def exact(case, seed):
    if case["kind"] in ("decode", "prompt"):
        return _exact_qwen(case, seed)
    w = {name: tensor.to(F64) for name, tensor in _mixer_tensors(case, seed).items()}
    x = _inputs(case, seed).to(F64)
    if case["kind"] == "experts":
        return _exact_experts(case, seed, w, x)
    if case["kind"] == "latent":
        return _exact_latent(case, seed, w, x)
    return _exact_recurrence(case, seed, w, x)
