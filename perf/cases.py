"""What generation spends its time on, as cases that can be timed and compared.

Whole steps of a Qwen3 decoder of 4B layer sizes (a few of its layers, its whole head) and single
layers of the other designs, each built from its part's specification as a decoder builds it and
called through the part's ``forward`` over a cache with slots and pages.  Single-token steps run as
a recorded CUDA graph, as the generation loop runs them; prompts are launched one by one.

* ``qwen3_decode``: a single-token step of ``seqs`` sequences that hold up to ``context`` tokens;
* ``qwen3_prompt``: a step of prompts, opened and closed again as a program does per batch;
* ``delta``, ``mlstm``, ``linear``, ``scan``, ``state_space``, ``latent``, ``experts``: a layer of
  ``width`` over prompts of up to ``tokens`` tokens (``tokens`` 1: a single-token step).

``ragged``: the lengths of the sequences fall from the stated one to about an eighth of it.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

DTYPE = torch.bfloat16
PAGE = 64
EPS = 1e-6
QWEN = {"vocab": 151936, "hidden": 2560, "inter": 9728, "heads": 32, "kv_heads": 8, "dim": 128, "theta": 5000000.0}
PROMPT_KINDS = ("delta", "mlstm", "linear", "scan", "state_space", "latent", "experts")
DECODE_KINDS = ("delta", "mlstm", "linear", "state_space")


def listed():
    return [
        # one user's chat turn: the latency of a token
        {"name": "qwen3_decode_1", "kind": "qwen3_decode", "layers": 4, "seqs": 1, "context": 640, "ragged": False},
        # the benchmark's batch of eight after 512-token prompts
        {"name": "qwen3_decode_8", "kind": "qwen3_decode", "layers": 4, "seqs": 8, "context": 526, "ragged": False},
        # a full batch of conversations of all lengths
        {"name": "qwen3_decode_64", "kind": "qwen3_decode", "layers": 4, "seqs": 64, "context": 2047, "ragged": True},
        # time to the first token of a long prompt
        {"name": "qwen3_prompt_2048", "kind": "qwen3_prompt", "layers": 4, "seqs": 1, "tokens": 2048, "ragged": False},
        # Lanilix: most of its layers, on one prompt and on a batch's next token
        {"name": "delta_prompt_2048", "kind": "delta", "width": 2048, "seqs": 1, "tokens": 2048, "ragged": False},
        {"name": "delta_decode_8", "kind": "delta", "width": 2048, "seqs": 8, "tokens": 1, "ragged": False},
        # Bunudra: several requests of odd lengths admitted as one batch
        {"name": "mlstm_prompts_4", "kind": "mlstm", "width": 2048, "seqs": 4, "tokens": 1000, "ragged": True},
        # Dubazen: gated linear attention of the wide configuration, an odd length; the scan
        {"name": "linear_prompt_1531", "kind": "linear", "width": 4096, "seqs": 1, "tokens": 1531, "ragged": False},
        {"name": "scan_prompt_2048", "kind": "scan", "width": 2048, "seqs": 1, "tokens": 2048, "ragged": False},
        # Futepel: eight short prompts at once; its experts on one long prompt
        {"name": "state_space_prompts_8", "kind": "state_space", "width": 4096, "seqs": 8, "tokens": 512, "ragged": False},
        {"name": "experts_prompt_2048", "kind": "experts", "width": 2048, "seqs": 1, "tokens": 2048, "ragged": False},
        # latent attention of Bunudra, Futepel and Turutar, windowed, over ragged prompts
        {"name": "latent_prompts_3", "kind": "latent", "width": 4096, "seqs": 3, "tokens": 1500, "ragged": True},
    ]


def _between(rng, low, high):
    """A whole number, spread evenly over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))))


def draw(rng):
    what = rng.random()
    if what < 0.25:
        return {"kind": "qwen3_decode", "layers": rng.randint(2, 4), "seqs": _between(rng, 1, 64),
                "context": _between(rng, 64, 2047), "ragged": rng.random() < 0.5}
    if what < 0.35:
        seqs = _between(rng, 1, 4)
        return {"kind": "qwen3_prompt", "layers": rng.randint(2, 4), "seqs": seqs, "tokens": _between(rng, 64, 2048 // seqs),
                "ragged": rng.random() < 0.5}
    width = rng.choice((2048, 4096))
    if what < 0.5:
        return {"kind": rng.choice(DECODE_KINDS), "width": width, "seqs": _between(rng, 1, 64), "tokens": 1, "ragged": False}
    seqs = _between(rng, 1, 8)
    return {"kind": rng.choice(PROMPT_KINDS), "width": width, "seqs": seqs, "tokens": _between(rng, 64, min(2048, 4096 // seqs)),
            "ragged": rng.random() < 0.5}


def lengths(case):
    """Tokens that each sequence brings (a prompt) or holds (a single-token step of qwen3_decode)."""
    top, n = int(case.get("context") or case["tokens"]), int(case["seqs"])
    if not case["ragged"] or n == 1:
        return [top] * n
    return [max(1, top - (top * 7 * i) // (8 * (n - 1))) for i in range(n)]


# ---------------------------------------------------------------------------- weights and inputs


class _Draw:
    """Tensors in a fixed order from one seed, on the GPU; ``salt`` separates weights from inputs."""

    def __init__(self, seed, salt):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + salt)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, std, generator=self.g)

    def matrix(self, *shape):
        return self.normal(*shape, std=0.02, dtype=DTYPE)

    def gain(self, *shape):
        return self.normal(*shape, std=0.02, mean=1.0)

    def uniform(self, low, high, *shape):
        return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(low, high, generator=self.g)


def _heads(case):
    return case["width"] // 128


def layer_weights(case, seed):
    """The tensors of the case's layer, by the names its part gives them."""
    d, w, kind = _Draw(seed, 1), case["width"], case["kind"]
    h = _heads(case)
    if kind == "delta":
        kv = h // 4
        t = {"q": d.matrix(kv * 128, w), "k": d.matrix(kv * 128, w), "v": d.matrix(w, w), "g": d.matrix(w, w),
             "b": d.matrix(h, w), "a": d.matrix(h, w), "norm": d.gain(128), "o": d.matrix(w, w),
             "A_log": d.uniform(-0.69, 2.08, h), "dt_bias": d.normal(h)}
        for name, n in (("q", kv * 128), ("k", kv * 128), ("v", w)):
            t[name + ".conv"] = d.normal(n, 4, std=0.5)
        return t
    if kind == "mlstm":
        t = {name: d.matrix(w, w) for name in ("q", "k", "v", "g", "o")}
        t.update(i=d.matrix(h, w), f=d.matrix(h, w), i_bias=d.uniform(-2, 5, h), f_bias=d.uniform(-2, 5, h), norm=d.gain(w))
        return t
    if kind == "linear":
        t = {name: d.matrix(w, w) for name in ("q", "k", "v", "g", "o")}
        t.update(a1=d.matrix(64, w), a2=d.normal(w, 64, dtype=DTYPE), a2_bias=d.uniform(-2, 5, w), norm=d.gain(128))
        return t
    if kind == "scan":
        n, rank = 2 * w, w // 16
        return {"in": d.matrix(2 * n, w), "conv": d.normal(n, 4, std=0.5), "conv_bias": d.normal(n, std=0.02),
                "x": d.matrix(rank + 32, n), "dt": d.normal(n, rank, dtype=DTYPE), "dt_bias": d.normal(n, std=0.02),
                "A_log": d.normal(n, 16, std=0.02) + torch.arange(1, 17, device="cuda").float().log(), "D": d.gain(n),
                "o": d.matrix(w, n)}
    if kind == "state_space":
        sh, inner, groups = 4 * h, 2 * w, 8
        channels = inner + 2 * groups * 128
        return {"in": d.matrix(inner + channels + sh, w), "conv": d.normal(channels, 4, std=0.5),
                "conv_bias": d.normal(channels, std=0.02), "dt_bias": d.uniform(-4.6, 0, sh), "A_log": d.uniform(-0.69, 2.08, sh),
                "D": d.gain(sh), "norm": d.gain(inner), "o": d.matrix(w, inner)}
    if kind == "latent":
        return {"q_proj": d.matrix(h * 128, w), "down_proj": d.matrix(512 + 64, w), "latent_norm": d.gain(512),
                "up_k": d.matrix(h * 64, 512), "up_v": d.matrix(h * 128, 512), "g_proj": d.matrix(h * 128, w),
                "o_proj": d.matrix(w, h * 128)}
    if kind == "experts":
        ff = w // 2
        t = {"router": d.matrix(8, w)}
        for e in range(8):
            t.update({f"gate.{e}": d.matrix(ff, w), f"up.{e}": d.matrix(ff, w), f"down.{e}": d.matrix(w, ff)})
        t.update(shared_gate_proj=d.matrix(ff, w), shared_up=d.matrix(ff, w), shared_down=d.matrix(w, ff))
        return t
    raise ValueError(kind)


def layer_spec(case):
    """(family, kind, parameters) of the case's part, as the designs' configurations spell them."""
    w, h, kind = case["width"], _heads(case), case["kind"]
    if kind == "delta":
        return "mixer", "gated_delta", {"hidden_size": w, "n_heads": h, "n_kv_heads": h // 4, "key_dim": 128, "value_dim": 128,
                                        "conv_taps": 4, "norm_eps": EPS, "unit_norm_eps": EPS}
    if kind == "mlstm":
        return "mixer", "mlstm", {"hidden_size": w, "n_heads": h, "key_dim": 128, "value_dim": 128, "gate_cap": 15.0,
                                  "norm_eps": EPS, "denominator_floor": 1e-6}
    if kind == "linear":
        return "mixer", "linear_attention", {"hidden_size": w, "n_heads": h, "key_dim": 128, "value_dim": 128,
                                             "decay": {"kind": "gated", "rank": 64, "tau": 16.0}, "q_scale": 128 ** -0.5,
                                             "silu_inputs": False, "norm_scope": "head", "norm_eps": EPS, "gate": "silu"}
    if kind == "scan":
        return "mixer", "selective_scan", {"hidden_size": w, "inner": 2 * w, "state": 16, "dt_rank": w // 16, "conv_taps": 4}
    if kind == "state_space":
        return "mixer", "state_space", {"hidden_size": w, "n_heads": 4 * h, "value_dim": 64, "state": 128, "groups": 8,
                                        "conv_taps": 4, "norm_groups": 8, "norm_eps": EPS}
    if kind == "latent":
        from thing_htn_2026_b200.config.base import PartSpec
        rope = PartSpec("rope", {"head_dim": 64, "rotary_dim": 64, "theta": 500000.0, "layout": "interleaved",
                                 "frequency_precision": "float64", "angle_precision": "float64"})
        return "mixer", "latent_attention", {"hidden_size": w, "n_heads": h, "plain_dim": 64, "rot_dim": 64, "value_dim": 128,
                                             "latent_rank": 512, "scale": 128 ** -0.5, "window": 1024, "norm_eps": EPS,
                                             "gated": True, "softmax_weights": "float32", "position": rope}
    return "ffn", "routed_glu_experts", {"hidden_size": w, "n_experts": 8, "expert_ff": w // 2, "top": 2, "shared_ff": w // 2}


def layer_inputs(case, seed):
    """The layer's input rows, and the state that a single-token step finds (by part of the state)."""
    d, w, h, kind, n = _Draw(seed, 2), case["width"], _heads(case), case["kind"], int(case["seqs"])
    x = d.normal(sum(lengths(case)), w, dtype=DTYPE)
    if case["tokens"] > 1:
        return x, []
    if kind == "delta":
        return x, [d.normal(n, h, 128, 128, std=0.1), d.normal(n, 4, (h // 4) * 256 + w, dtype=DTYPE)]
    if kind == "mlstm":
        m = d.uniform(0, 4, n, h, 1, 1)
        keys = d.normal(n, h, 1, 128)
        return x, [d.normal(n, h, 128, 128), torch.cat([keys, m], dim=-1)]
    if kind == "linear":
        return x, [d.normal(n, h, 128, 128)]
    return x, [d.normal(n, 4 * h, 64, 128, std=0.1), d.normal(n, 4, 2 * w + 2048, dtype=DTYPE)]


HELD = 640      # tokens that the sequences of a layer's single-token step hold


def qwen_weights(case, seed):
    d, q = _Draw(seed, 1), QWEN
    t = {"model.embed_tokens.weight": d.matrix(q["vocab"], q["hidden"]), "model.norm.weight": d.gain(q["hidden"]).to(DTYPE)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        t[p + "input_layernorm.weight"] = d.gain(q["hidden"]).to(DTYPE)
        t[p + "post_attention_layernorm.weight"] = d.gain(q["hidden"]).to(DTYPE)
        for name, n in (("q", q["heads"]), ("k", q["kv_heads"]), ("v", q["kv_heads"])):
            t[p + f"self_attn.{name}_proj.weight"] = d.matrix(n * q["dim"], q["hidden"])
        t[p + "self_attn.o_proj.weight"] = d.matrix(q["hidden"], q["heads"] * q["dim"])
        t[p + "self_attn.q_norm.weight"] = d.gain(q["dim"]).to(DTYPE)
        t[p + "self_attn.k_norm.weight"] = d.gain(q["dim"]).to(DTYPE)
        t[p + "mlp.gate_proj.weight"] = d.matrix(q["inter"], q["hidden"])
        t[p + "mlp.up_proj.weight"] = d.matrix(q["inter"], q["hidden"])
        t[p + "mlp.down_proj.weight"] = d.matrix(q["hidden"], q["inter"])
    return t


def qwen_inputs(case, seed):
    """Tokens per sequence, and for single-token steps the cached keys and values of the positions
    ahead: per layer, K and V ``[sequences, positions, kv_heads, dim]``."""
    d, n = _Draw(seed, 2), int(case["seqs"])
    counts = [1] * n if case["kind"] == "qwen3_decode" else lengths(case)
    tokens = torch.randint(0, QWEN["vocab"], (sum(counts),), device="cuda", generator=d.g)
    held = []
    if case["kind"] == "qwen3_decode":
        for _ in range(case["layers"]):
            shape = (n, max(lengths(case)), QWEN["kv_heads"], QWEN["dim"])
            held.append((d.normal(*shape, dtype=DTYPE), d.normal(*shape, dtype=DTYPE)))
    return tokens.to(torch.int32), counts, held


# ---------------------------------------------------------------------------- prepare and run


def _record(call, restore):
    """``call`` as a CUDA graph: two runs ahead on a side stream, then the recording; what they changed
    is put back.  Returns the graph and the recorded call's result."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            call()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        result = call()
    restore()
    return graph, result


def _int32(values):
    return torch.tensor(list(values), dtype=torch.int32, device="cuda")


def _starts(counts):
    cu = [0]
    for c in counts:
        cu.append(cu[-1] + c)
    return cu


def _prepare_layer(case, seed):
    from thing_htn_2026_b200 import ops, parts
    from thing_htn_2026_b200.cache.sequence_cache import SequenceCache, StateSpec
    from thing_htn_2026_b200.config.base import PartSpec, ScheduleEntry
    device = torch.device("cuda", torch.cuda.current_device())
    family, kind, params = layer_spec(case)
    tensors = layer_weights(case, seed)
    runtime = parts.Runtime(DTYPE, device, dict(tensors))
    layer = parts.part_class(family, kind)(PartSpec(kind, params, {name: name for name in tensors}), runtime)
    runtime.tensors = {}
    x, held = layer_inputs(case, seed)
    counts, n = lengths(case), int(case["seqs"])
    at = HELD if case["tokens"] == 1 else 0
    need = layer.cache_need() if family == "mixer" else None
    pages = sum(-(-(at + c) // PAGE) for c in counts)
    cache = SequenceCache([need], max_tokens=pages * PAGE, dtype=DTYPE, device=device, max_slots=n)
    slots = sorted(cache.open(n))        # all of them: a state's rows stand in the sequences' order
    cache.prepare(slots, [at + c for c in counts])
    cache.seq_lens.fill_(at)
    kept = [one for one in (need if isinstance(need, tuple) else (need,)) if isinstance(one, StateSpec)]
    states = [cache.state_view(0, i) for i in range(len(kept))]
    for view, value in zip(states, held):
        view.copy_(value.expand(view.shape))
    for shared in runtime.shared.values():
        if hasattr(shared, "ensure"):
            shared.ensure(cache.max_pages_per_seq * PAGE)
    asked = {}
    if hasattr(layer, "step_inputs"):
        layer.step_inputs(parts.HostBatch(slots, counts, [at] * n, PAGE), asked)
    rows = ops.step_rows(_int32(_starts(counts)), _int32(slots), cache.seq_lens, sum(counts), max(counts),
                         max_context=at + max(counts), lengths_differ=ops.lengths_differ([at + c for c in counts]))
    ctx = parts.StepContext(rows=rows, cache=cache, err=ops.new_error_word(device), inputs={k: _int32(v) for k, v in asked.items()})
    entry = ScheduleEntry(layer=0, cache=0)

    def call():
        y = layer.forward(x, ctx) if family == "ffn" else layer.forward(x, ctx, entry)
        return {"y": y, "state": states}

    state = SimpleNamespace(call=call, graph=None, result=None, keep=(layer, cache, x))
    if case["tokens"] == 1:
        before = [s.clone() for s in states]

        def restore():
            for s, b in zip(states, before):
                s.copy_(b)
        state.graph, state.result = _record(call, restore)
    return state


def _prepare_qwen(case, seed):
    from thing_htn_2026_b200.cache.sequence_cache import SequenceCache
    from thing_htn_2026_b200.config import config_from_dict
    from thing_htn_2026_b200.engine.step import StepEntry, StepRunner
    from thing_htn_2026_b200.models.decoder import DecoderModel
    device = torch.device("cuda", torch.cuda.current_device())
    q = QWEN
    config = config_from_dict({
        "architectures": ["Qwen3ForCausalLM"], "hidden_act": "silu", "attention_bias": False, "vocab_size": q["vocab"],
        "hidden_size": q["hidden"], "intermediate_size": q["inter"], "num_hidden_layers": case["layers"],
        "num_attention_heads": q["heads"], "num_key_value_heads": q["kv_heads"], "head_dim": q["dim"], "rms_norm_eps": EPS,
        "rope_theta": q["theta"], "tie_word_embeddings": True, "max_position_embeddings": 4096})
    model = DecoderModel(config, qwen_weights(case, seed), DTYPE, device)
    tokens, counts, held = qwen_inputs(case, seed)
    n = int(case["seqs"])
    ahead = lengths(case) if held else [0] * n
    pages = sum(-(-(a + c) // PAGE) for a, c in zip(ahead, counts))
    cache = SequenceCache(model.cache_needs(), max_tokens=pages * PAGE, dtype=DTYPE, device=device, max_slots=n)
    runner = StepRunner(model, cache)
    if case["kind"] == "qwen3_prompt":
        texts, cu = tokens.tolist(), _starts(counts)
        prompts = [texts[cu[i]:cu[i + 1]] for i in range(n)]

        def call():
            slots = cache.open(n)
            logits = runner.step([StepEntry(s, p, (len(p) - 1,)) for s, p in zip(slots, prompts)], check=False)
            cache.close(slots)
            return {"logits": logits}
        return SimpleNamespace(call=call, graph=None, result=None, keep=(model, cache))

    from thing_htn_2026_b200 import ops
    slots = cache.open(n)
    cache.prepare(slots, [a + 1 for a in ahead])
    table = cache.block_tables[0]
    for i, (slot, a) in enumerate(zip(slots, ahead)):
        place = torch.arange(a, device=device)
        page = table[slot][place // PAGE].long()
        for layer, kv in enumerate(held):
            for part in (0, 1):
                cache.kv_storage[0][layer][page, part, :, place % PAGE] = kv[part][i, :a]
    lens = torch.zeros(n, dtype=torch.int32, device=device)
    lens[torch.tensor(slots, device=device)] = _int32(ahead)
    cu, slot_list = _int32(range(n + 1)), _int32(slots)
    # a program records its steps per class of context length, so that one recording serves many steps
    bound = ops.context_class(max(ahead) + 1)[1]
    differ = ops.lengths_differ([a + 1 for a in ahead])

    def call():
        cache.seq_lens.copy_(lens)
        return {"logits": runner.run_rows(tokens, cu, slot_list, n, 1, bound, None, lengths_differ=differ)}

    graph, result = _record(call, lambda: None)
    return SimpleNamespace(call=call, graph=graph, result=result, keep=(model, cache, tokens, cu, slot_list, lens, runner))


def prepare(case, seed):
    with torch.inference_mode():
        return _prepare_qwen(case, seed) if case["kind"].startswith("qwen3") else _prepare_layer(case, seed)


def run(state):
    if state.graph is not None:
        state.graph.replay()
        return state.result
    with torch.inference_mode():
        return state.call()


# ---------------------------------------------------------------------------- work and tolerance


def work(case):
    lens, n = lengths(case), int(case["seqs"])
    if case["kind"].startswith("qwen3"):
        q = QWEN
        layer = q["hidden"] * q["dim"] * (2 * q["heads"] + 2 * q["kv_heads"]) + 3 * q["hidden"] * q["inter"]
        head = q["vocab"] * q["hidden"]
        decode = case["kind"] == "qwen3_decode"
        rows = n if decode else sum(lens)
        pairs = sum(a + 1 for a in lens) if decode else sum(a * (a + 1) // 2 for a in lens)
        positions = sum(lens) + (n if decode else 0)
        token = 4 * q["kv_heads"] * q["dim"]      # bytes of a position's keys and values in one layer
        return {"bytes": 2 * (case["layers"] * layer + head) + case["layers"] * token * positions + 4 * n * q["vocab"],
                "flops": 2 * case["layers"] * layer * rows + 2 * head * n + 4 * case["layers"] * q["heads"] * q["dim"] * pairs}
    w, h, kind, rows = case["width"], _heads(case), case["kind"], sum(lens)
    at = 1 if case["tokens"] == 1 else 0
    # entries of the layer's matrices, float32 entries of a sequence's state, operations of a row outside the matrices
    if kind == "delta":
        entries, state, own = w * (3 * w + w // 2 + 2 * h), h * 128 * 128, 7 * h * 128 * 128
    elif kind == "mlstm":
        entries, state, own = w * (5 * w + 2 * h), h * (128 * 128 + 129), 5 * h * 128 * 128
    elif kind == "linear":
        entries, state, own = w * (5 * w + 128), h * 128 * 128, 5 * h * 128 * 128
    elif kind == "scan":
        inner = 2 * w
        entries, state, own = 3 * w * inner + inner * (2 * (w // 16) + 32), inner * 16, 6 * inner * 16
    elif kind == "state_space":
        inner = 2 * w
        entries, state, own = w * (3 * inner + 2048 + 4 * h), 4 * h * 64 * 128, 5 * 4 * h * 64 * 128
    elif kind == "latent":
        pairs = sum(sum(min(i + 1, 1024) for i in range(a)) for a in lens)
        entries, state, own = w * (3 * w + 576) + 512 * h * 192, 0, 4 * h * 128 * pairs / rows
    else:       # two of eight experts and the shared one per row; every expert's weights are read
        ff = w // 2
        return {"bytes": 2 * (9 * 3 * w * ff + 8 * w) + 4 * rows * w, "flops": 2 * rows * (3 * 3 * w * ff + 8 * w)}
    kept = 2 * rows * h * 256 if kind == "latent" else 4 * n * state * (1 + at)
    return {"bytes": 2 * entries + 4 * rows * w + kept, "flops": 2 * entries * rows + own * rows}


def tolerance(case):
    """About four times what a layer's outputs were seen to differ by from the same in 64 bits (0.004 to
    0.007: bfloat16 activations, rounded a few times); two correct whole steps of four layers, each 0.02
    from 64 bits, differ by up to the root of two of that."""
    if case["kind"].startswith("qwen3"):
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.3}


# ---------------------------------------------------------------------------- the same in 64 bits


def _rms(x, gain):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _turn(x, angle, layout):
    """Rotation of the last axis by ``angle`` [positions, half], ``x`` [positions, heads, 2 half]."""
    c, s = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    half = x.shape[-1] // 2
    if layout == "half":
        a, b = x[..., :half], x[..., half:]
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)


def _angles(positions, dim, theta):
    i = torch.arange(dim // 2, dtype=torch.float64, device="cuda")
    return positions.double()[:, None] * theta ** (-2.0 * i / dim)


def _padded(case, x):
    """Packed rows as [sequences, longest, ...] and which of them are there."""
    lens = lengths(case)
    out = x.new_zeros((len(lens), max(lens), *x.shape[1:]))
    there = torch.zeros(out.shape[:2], dtype=torch.bool, device=x.device)
    for i, (a, b) in enumerate(zip(_starts(lens), lens)):
        out[i, :b], there[i, :b] = x[a:a + b], True
    return out, there


def _convolved(case, z, taps, bias, ring):
    """silu of a causal convolution over time ``[rows, channels]``, and the ring of the last raw inputs
    (position p at p mod taps) as it stands afterwards."""
    n, at = taps.shape[1], HELD if case["tokens"] == 1 else 0
    wide, there = _padded(case, z)
    new = z.new_zeros((wide.shape[0], n, z.shape[1])) if ring is None else ring.double().clone()
    ahead = [new[:, (at - n + 1 + j) % n] for j in range(n - 1)]
    long = torch.cat([torch.stack(ahead, dim=1), wide], dim=1)
    y = sum(long[:, j:j + wide.shape[1]] * taps[:, j] for j in range(n))
    y = _silu(y if bias is None else y + bias)
    for i, length in enumerate(lengths(case)):
        for p in range(at + max(0, length - n), at + length):
            new[i, p % n] = wide[i, p - at]
    return y[there], new


def _recur(case, S, step, *rows):
    """Runs ``step(S, row...) -> (S, out)`` over the tokens of all sequences at once; S a tuple."""
    wide = [_padded(case, r)[0] for r in rows]
    there = _padded(case, rows[0])[1]
    outs = []
    for t in range(there.shape[1]):
        new, out = step(S, *(r[:, t] for r in wide))
        on = there[:, t]
        S = tuple(torch.where(on.view(-1, *[1] * (a.dim() - 1)), a, b) for a, b in zip(new, S))
        outs.append(out)
    return S, torch.stack(outs, dim=1)[there]


def _exact_layer(case, seed):
    t = {k: v.double() for k, v in layer_weights(case, seed).items()}
    x, held = layer_inputs(case, seed)
    x, held = x.double(), [a.double() for a in held]
    w, h, kind, n, rows = case["width"], _heads(case), case["kind"], int(case["seqs"]), x.shape[0]
    zeros = lambda *shape: torch.zeros(shape, dtype=torch.float64, device="cuda")  # noqa: E731
    if kind == "delta":
        kv = h // 4
        raw = torch.cat([x @ t[m].t() for m in "qkv"], dim=-1)
        mixed, ring = _convolved(case, raw, torch.cat([t[m + ".conv"] for m in "qkv"]), None, held[1] if held else None)
        q, k, v = mixed.split([kv * 128, kv * 128, w], dim=-1)
        unit = lambda a: a / torch.sqrt((a * a).sum(-1, keepdim=True) + EPS)  # noqa: E731
        q = (unit(q.view(rows, kv, 128)) * 128 ** -0.5).repeat_interleave(4, dim=1)
        k = unit(k.view(rows, kv, 128)).repeat_interleave(4, dim=1)
        beta = torch.sigmoid(x @ t["b"].t())
        decay = torch.exp(-torch.exp(t["A_log"]) * _softplus(x @ t["a"].t() + t["dt_bias"]))

        def step(S, q, k, v, beta, decay):
            s = S[0] * decay[..., None, None]
            u = beta[..., None] * (v - torch.einsum("shek,shk->she", s, k))
            s = s + u[..., :, None] * k[..., None, :]
            return (s,), torch.einsum("shek,shk->she", s, q)
        (S,), o = _recur(case, (held[0] if held else zeros(n, h, 128, 128),), step, q, k, v.view(rows, h, 128), beta, decay)
        y = _rms(o, t["norm"]).reshape(rows, w) * _silu(x @ t["g"].t())
        # a prompt leaves in the ring only what a later token reads
        return {"y": y @ t["o"].t(), "state": [S, ring if held else None]}
    if kind == "mlstm":
        q, k, v = ((x @ t[m].t()).view(rows, h, 128) for m in "qkv")
        cap = lambda z: 15.0 * torch.tanh(z / 15.0)  # noqa: E731
        gi = cap(x @ t["i"].t() + t["i_bias"])
        gf = -_softplus(-cap(x @ t["f"].t() + t["f_bias"]))
        start = (held[0], held[1][:, :, 0, :128], held[1][:, :, 0, 128]) if held else (zeros(n, h, 128, 128), zeros(n, h, 128), zeros(n, h))

        def step(S, q, k, v, gi, gf):
            s, sums, m = S
            top = torch.maximum(gf + m, gi)
            keep, take = torch.exp(gf + m - top), torch.exp(gi - top)
            s = keep[..., None, None] * s + take[..., None, None] * v[..., :, None] * k[..., None, :]
            sums = keep[..., None] * sums + take[..., None] * k
            below = torch.maximum((sums * q).sum(-1).abs(), torch.exp(-top)) + 1e-6
            return (s, sums, top), torch.einsum("shek,shk->she", s, q) / below[..., None]
        (S, sums, m), o = _recur(case, start, step, q * 128 ** -0.5, k, v, gi, gf)
        y = _rms(o, 1.0).reshape(rows, w) * t["norm"] * torch.sigmoid(x @ t["g"].t())
        # the second state tensor holds n and m once per block of columns
        return {"y": y @ t["o"].t(), "state": [S, None]}
    if kind == "linear":
        q, k, v = ((x @ t[m].t()).view(rows, h, 128) for m in "qkv")
        z = (x @ t["a1"].t()) @ t["a2"].t() + t["a2_bias"]
        decay = torch.exp(-_softplus(-z) / 16.0).view(rows, h, 128)

        def step(S, q, k, v, decay):
            s = S[0] * decay[..., None, :] + v[..., :, None] * k[..., None, :]
            return (s,), torch.einsum("shek,shk->she", s, q)
        (S,), o = _recur(case, (held[0] if held else zeros(n, h, 128, 128),), step, q * 128 ** -0.5, k, v, decay)
        y = _rms(o, t["norm"]).reshape(rows, w) * _silu(x @ t["g"].t())
        return {"y": y @ t["o"].t(), "state": [S]}
    if kind == "scan":
        inner, rank = 2 * w, w // 16
        u, z = (x @ t["in"].t()).split(inner, dim=-1)
        u, ring = _convolved(case, u, t["conv"], t["conv_bias"], None)
        dt, B, C = (u @ t["x"].t()).split([rank, 16, 16], dim=-1)
        dt = _softplus(dt @ t["dt"].t() + t["dt_bias"])
        A = -torch.exp(t["A_log"])

        def step(S, dt, u, B, C):
            s = torch.exp(dt[..., None] * A) * S[0] + (dt * u)[..., None] * B[:, None, :]
            return (s,), torch.einsum("scn,sn->sc", s, C)
        (S,), o = _recur(case, (zeros(n, inner, 16),), step, dt, u, B, C)
        return {"y": ((o + t["D"] * u) * _silu(z)) @ t["o"].t(), "state": [S, ring]}
    if kind == "state_space":
        sh, inner = 4 * h, 2 * w
        z, xbc, dt = (x @ t["in"].t()).split([inner, inner + 2048, sh], dim=-1)
        xbc, ring = _convolved(case, xbc, t["conv"], t["conv_bias"], held[1] if held else None)
        u, B, C = xbc.split([inner, 1024, 1024], dim=-1)
        u = u.view(rows, sh, 64)
        B, C = (a.view(rows, 8, 128).repeat_interleave(sh // 8, dim=1) for a in (B, C))
        dt = _softplus(dt + t["dt_bias"])
        decay = torch.exp(-torch.exp(t["A_log"]) * dt)

        def step(S, u, B, C, dt, decay):
            s = decay[..., None, None] * S[0] + (dt[..., None] * u)[..., :, None] * B[..., None, :]
            return (s,), torch.einsum("shek,shk->she", s, C)
        (S,), o = _recur(case, (held[0] if held else zeros(n, sh, 64, 128),), step, u, B, C, dt, decay)
        y = (o + t["D"][:, None] * u).reshape(rows, inner) * _silu(z)
        y = _rms(y.view(rows, 8, inner // 8), 1.0).reshape(rows, inner) * t["norm"]
        return {"y": y @ t["o"].t(), "state": [S, ring]}
    if kind == "latent":
        q = (x @ t["q_proj"].t()).view(rows, h, 128)
        low, shared = (x @ t["down_proj"].t()).split([512, 64], dim=-1)
        c = _rms(low, t["latent_norm"])
        k, v = (c @ t["up_k"].t()).view(rows, h, 64), (c @ t["up_v"].t()).view(rows, h, 128)
        out = []
        for a, length in zip(_starts(lengths(case)), lengths(case)):
            p = torch.arange(length, device="cuda")
            turn = _angles(p, 64, 500000.0)
            one = slice(a, a + length)
            qs = torch.cat([q[one, :, :64], _turn(q[one, :, 64:], turn, "interleaved")], dim=-1)
            ks = torch.cat([k[one], _turn(shared[one, None, :], turn, "interleaved").expand(-1, h, -1)], dim=-1)
            s = torch.einsum("qhd,khd->hqk", qs, ks) * 128 ** -0.5
            back = p[:, None] - p[None, :]
            s = s.masked_fill((back < 0) | (back >= 1024), -math.inf)
            out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, dim=-1), v[one]))
        y = torch.cat(out).reshape(rows, h * 128) * torch.sigmoid(x @ t["g_proj"].t())
        return {"y": y @ t["o_proj"].t(), "state": []}
    z = x @ t["router"].t()
    best, chosen = z.topk(2, dim=-1)
    weight = torch.zeros_like(z).scatter_(1, chosen, torch.softmax(best, dim=-1))
    y = (_silu(x @ t["shared_gate_proj"].t()) * (x @ t["shared_up"].t())) @ t["shared_down"].t()
    for e in range(8):
        y += weight[:, e:e + 1] * ((_silu(x @ t[f"gate.{e}"].t()) * (x @ t[f"up.{e}"].t())) @ t[f"down.{e}"].t())
    return {"y": y, "state": []}


def _exact_qwen(case, seed):
    t, q = qwen_weights(case, seed), QWEN
    tokens, counts, held = qwen_inputs(case, seed)
    ahead = lengths(case) if held else [0] * len(counts)
    starts = _starts(counts)
    W = lambda name: t[name].double()  # noqa: E731
    group = q["heads"] // q["kv_heads"]
    x = W("model.embed_tokens.weight")[tokens.long()]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        a = _rms(x, W(p + "input_layernorm.weight"))
        Q, K, V = (a @ W(p + f"self_attn.{m}_proj.weight").t() for m in "qkv")
        Q = _rms(Q.view(-1, q["heads"], q["dim"]), W(p + "self_attn.q_norm.weight"))
        K = _rms(K.view(-1, q["kv_heads"], q["dim"]), W(p + "self_attn.k_norm.weight"))
        V = V.view(-1, q["kv_heads"], q["dim"])
        out = []
        for j, (start, count, before) in enumerate(zip(starts, counts, ahead)):
            one = slice(start, start + count)
            place = torch.arange(before, before + count, device="cuda")
            turn = _angles(place, q["dim"], q["theta"])
            qs, ks, vs = _turn(Q[one], turn, "half"), _turn(K[one], turn, "half"), V[one]
            if before:
                ks = torch.cat([held[i][0][j, :before].double(), ks])
                vs = torch.cat([held[i][1][j, :before].double(), vs])
            ks, vs = ks.repeat_interleave(group, dim=1), vs.repeat_interleave(group, dim=1)
            s = torch.einsum("qhd,khd->hqk", qs, ks) * q["dim"] ** -0.5
            s = s.masked_fill(torch.arange(before + count, device="cuda")[None, :] > place[:, None], -math.inf)
            out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, dim=-1), vs).reshape(count, -1))
        x = x + torch.cat(out) @ W(p + "self_attn.o_proj.weight").t()
        a = _rms(x, W(p + "post_attention_layernorm.weight"))
        x = x + (_silu(a @ W(p + "mlp.gate_proj.weight").t()) * (a @ W(p + "mlp.up_proj.weight").t())) @ W(p + "mlp.down_proj.weight").t()
    last = torch.tensor([s - 1 for s in starts[1:]], device="cuda")
    return {"logits": _rms(x[last], W("model.norm.weight")) @ W("model.embed_tokens.weight").t()}


def exact(case, seed):
    with torch.inference_mode():
        return _exact_qwen(case, seed) if case["kind"].startswith("qwen3") else _exact_layer(case, seed)
