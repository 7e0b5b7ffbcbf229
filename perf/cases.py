"""The work that users of this package have it do, as cases that can be timed and compared.

A case is a dict of plain values; `kind` says which calls of the public API it makes:

  step      one blocking `forward` with the logits copied back: what a host loop pays per token
  generate  `generate_greedy`: the greedy run loop kept on the device, prompt included
  chat      a greedy host loop of a few tokens behind a long context
  sample    `forward` + `sample` per token: temperature / top-p choice on the device, the command line's default
  prefill   `prefill` of a prompt (or of the next turn of a conversation) and the first token's logits behind it
  batch     `batch_forward`: one decode step of several sequences, each at a position of its own
  quantise  `quant_encode` of host floats: the first load of a checkpoint

Shapes are those of `llama2j_b200.synthetic.SHAPES`; `kv_heads` makes them grouped-query, `own_classifier`
gives the small ones a classifier of their own, `layers` stacks fewer layers of the same widths, which cost the
same per layer and take less time to load.  Weights are drawn from the seed, N(0, 0.02^2) with RMSNorm
weights 1.0, and quantised on the device.
"""
from __future__ import annotations

import math

import numpy as np

from llama2j_b200 import lib
from llama2j_b200 import synthetic as syn
from llama2j_b200.model_files import GROUP_BYTES, ModelConfig, quant_bytes
from llama2j_b200.transformer import Transformer, argmax

RMS_TENSORS = (lib.T_RMS_ATT, lib.T_RMS_FFN, lib.T_RMS_FINAL)
LAYER_SHIFT = 7            # groups by which the weights of a layer are shifted against the layer below


def listed():
    return [
        # the smallest model, one token: launches, copies and the host call are all there is
        {"name": "step-15m", "kind": "step", "shape": "stories15M", "pos": 100},
        # a short story on the small model that is still quantised in whole groups
        {"name": "generate-110m", "kind": "generate", "shape": "stories110M", "prompt": 32, "steps": 128},
        # the headline workload: 32 prompt tokens and an answer
        {"name": "generate-7b", "kind": "generate", "shape": "llama2-7b", "prompt": 32, "steps": 48},
        # the end of a full context window, one blocking call per token
        {"name": "chat-7b-long", "kind": "chat", "shape": "llama2-7b", "pos": 3840, "steps": 8},
        # the larger model
        {"name": "generate-13b", "kind": "generate", "shape": "llama2-13b", "prompt": 16, "steps": 24},
        # sampled text with the command line's defaults (--temp 0.9 --topp 0.9)
        {"name": "sample-110m", "kind": "sample", "shape": "stories110M", "own_classifier": True, "pos": 48, "steps": 16,
         "temp": 0.9, "topp": 0.9},
        # the next turn of a conversation: a short question behind 900 positions
        {"name": "prefill-7b-turn", "kind": "prefill", "shape": "llama2-7b", "pos": 900, "prompt": 37, "layers": 16},
        # a document as the prompt
        {"name": "prefill-7b-document", "kind": "prefill", "shape": "llama2-7b", "pos": 0, "prompt": 3840, "layers": 16},
        # grouped-query heads, head size 64, a length that is no multiple of anything
        {"name": "prefill-110m-grouped", "kind": "prefill", "shape": "stories110M", "kv_heads": 4, "pos": 0, "prompt": 333},
        # serving: a full batch of short conversations, and a few long ones
        {"name": "batch-7b-64", "kind": "batch", "shape": "llama2-7b", "sequences": 64, "first": 10, "last": 200, "layers": 16},
        {"name": "batch-7b-4-long", "kind": "batch", "shape": "llama2-7b", "sequences": 4, "first": 600, "last": 1500, "layers": 16},
        # one W1 matrix of the 7B checkpoint, host floats to host bytes
        {"name": "quantise-w1", "kind": "quantise", "floats": 4096 * 11008},
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: every kind over the sizes between (and around) the listed ones."""
    kind = rng.choice(["step", "generate", "generate", "chat", "sample", "prefill", "prefill", "batch", "batch", "quantise"])
    if kind == "quantise":
        return {"kind": kind, "floats": _between(rng, 288 * 288 + 1, 4096 * 11008)}
    if kind == "step":
        shape = rng.choice(["stories15M", "stories110M", "llama2-7b"])
        return {"kind": kind, "shape": shape, "pos": _between(rng, 1, 250)}
    if kind == "generate":
        shape = rng.choice(["stories15M", "stories110M", "llama2-7b", "llama2-7b", "llama2-13b"])
        most = {"stories15M": 128, "stories110M": 200, "llama2-7b": 48, "llama2-13b": 24}[shape]
        steps = _between(rng, 8, most)
        case = {"kind": kind, "shape": shape, "prompt": rng.randint(0, steps - 1), "steps": steps}
        if shape == "llama2-13b":
            case["layers"] = 20
        return case
    if kind == "chat":
        pos = _between(rng, 300, 4000)
        return {"kind": kind, "shape": "llama2-7b", "pos": pos, "steps": rng.randint(2, 8)}
    if kind == "sample":
        shape = rng.choice(["stories15M", "stories110M", "llama2-7b"])
        return {"kind": kind, "shape": shape, "own_classifier": True, "pos": rng.randint(2, 200), "steps": rng.randint(4, 16),
                "temp": rng.choice([0.7, 0.9, 1.0]), "topp": rng.choice([0.8, 0.9, 0.95, 1.0])}
    if kind == "prefill":
        if rng.random() < 0.4:
            n = _between(rng, 5, 700)
            return {"kind": kind, "shape": "stories110M", "kv_heads": rng.choice([12, 4, 2]), "pos": rng.randint(0, 300),
                    "prompt": n}
        n = _between(rng, 5, 2500)
        return {"kind": kind, "shape": "llama2-7b", "pos": rng.choice([0, rng.randint(1, 1500)]), "prompt": n, "layers": 16}
    shape = rng.choice(["stories110M", "llama2-7b", "llama2-7b"])
    n = _between(rng, 2, 64)
    last = _between(rng, 30, min(900, 8000 // n))
    case = {"kind": "batch", "shape": shape, "sequences": n, "first": rng.randint(1, last), "last": last}
    if shape == "llama2-7b":
        case["layers"] = 16
    return case


def _config(case) -> ModelConfig:
    s = syn.SHAPES[case["shape"]]
    shared = s.shared_classifier and not case.get("own_classifier", False)
    return ModelConfig(s.dim, s.hidden_dim, case.get("layers", s.n_layers), s.n_heads, case.get("kv_heads", s.n_kv_heads),
                       s.vocab_size, s.seq_len, shared)


def _model(cfg: ModelConfig, seed: int, classifier_scale: float = syn.WEIGHT_SCALE) -> Transformer:
    """A loaded model.  A layer's matrices are slices of one generated stream, shifted by LAYER_SHIFT groups from
    layer to layer: all layers differ, and only little more than one of them has to be generated."""
    model = Transformer(cfg)
    for t in lib.QUANT_TENSORS:
        n = cfg.tensor_floats(t)
        if t in RMS_TENSORS:
            model.upload_quant(t, syn.quant_encode(np.ones(n, dtype=np.float32)))
            continue
        per_layer = n // cfg.n_layers
        groups = per_layer // 256
        data = syn.synth_quant((groups + LAYER_SHIFT * cfg.n_layers) * 256, seed, t)
        for layer in range(cfg.n_layers):
            first = LAYER_SHIFT * layer * GROUP_BYTES
            model.upload_quant(t, data[first: first + groups * GROUP_BYTES], per_layer, layer * per_layer)
    _upload_table(model, lib.T_TOKEN_EMBEDDING, seed, syn.WEIGHT_SCALE)
    if not cfg.shared_classifier:
        _upload_table(model, lib.T_WCLS, seed, classifier_scale)
    model.finalize()
    return model


def _upload_table(model: Transformer, tensor: int, seed: int, scale: float) -> None:
    """An FP32 table (vocabulary x dim) in four pieces, again shifted slices of one stream: no two rows are alike."""
    piece = model.cfg.tensor_floats(tensor) // 4
    values = syn.synth_f32(piece + 4 * LAYER_SHIFT, seed, tensor, scale=scale)
    for i in range(4):
        model.upload_f32(tensor, values[LAYER_SHIFT * i: LAYER_SHIFT * i + piece], i * piece)


def _fill_batch(model: Transformer, lengths, tokens) -> None:
    """The earlier positions of every sequence, 64 entries per call (entries of one sequence in slices)."""
    entries = [(s, p) for s, n in enumerate(lengths) for p in range(n)]
    for i in range(0, len(entries), 64):
        part = entries[i: i + 64]
        seq = [s for s, _ in part]
        model.batch_forward(seq, [p for _, p in part], [int(tokens[s][p]) for s, p in part], want_logits=False)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "quantise":
        return {"case": case, "values": syn.synth_f32(case["floats"], seed, lib.T_W1)}
    cfg = _config(case)
    # a trained model's next-token distribution is peaked (logits spread over about 6), which decides how many
    # candidates the sampler has; elsewhere the values of the logits do not matter
    scale = 6.0 / math.sqrt(cfg.dim) if kind == "sample" else syn.WEIGHT_SCALE
    model = _model(cfg, seed, scale)

    def ids(n):
        return rng.integers(3, cfg.vocab_size, n).astype(np.int32)

    state = {"case": case, "model": model}
    if kind in ("step", "chat", "sample"):
        model.prefill(ids(case["pos"]), 0)
        state["tokens"] = ids(case.get("steps", 1))
    elif kind == "generate":
        state["prompt"] = ids(case["prompt"])
    elif kind == "prefill":
        if case["pos"]:
            model.prefill(ids(case["pos"]), 0)
        state["prompt"] = ids(case["prompt"])
        state["next"] = int(ids(1)[0])
    else:
        n = case["sequences"]
        lengths = rng.integers(case["first"], case["last"] + 1, n)
        lengths[0] = case["last"]
        model.batch_create(n, case["last"] + 1)
        _fill_batch(model, lengths, [ids(int(m)) for m in lengths])
        state.update(seq=np.arange(n, dtype=np.int32), pos=lengths.astype(np.int32), tokens=ids(n))
    if kind == "sample":
        state["seed"] = int(rng.integers(1, 1 << 31))
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "quantise":
        return syn.quant_encode(state["values"])
    model = state["model"]
    vocab = model.cfg.vocab_size
    if kind == "step":
        logits, token = model.forward(state["tokens"][0], case["pos"])
        return {"logits": logits, "token": token}
    if kind == "generate":
        tokens = model.generate_greedy(state["prompt"], case["steps"])
        return {"tokens": tokens, "logits": model.read_buffer(4, vocab)}
    if kind == "chat":
        token, out = int(state["tokens"][0]), []
        for i in range(case["steps"]):
            logits, _ = model.forward(token, case["pos"] + i)
            token = argmax(logits)
            out.append(token)
        return {"tokens": np.asarray(out, dtype=np.int32), "logits": logits}
    if kind == "sample":
        # the inputs are a given text, so that a draw that falls on the other side of a tie does not change what follows
        model.sampler_seed(state["seed"])
        out = []
        for i, token in enumerate(state["tokens"]):
            model.forward(token, case["pos"] + i, want_logits=False)
            out.append(model.sample(case["temp"], case["topp"]))
        return {"tokens": np.asarray(out, dtype=np.int32), "probabilities": model.read_buffer(4, vocab)}
    if kind == "prefill":
        model.prefill(state["prompt"], case["pos"])
        logits, token = model.forward(state["next"], case["pos"] + case["prompt"])
        return {"logits": logits, "token": token}
    logits, tokens = model.batch_forward(state["seq"], state["pos"], state["tokens"])
    return {"logits": logits, "tokens": tokens}


def _matrix_floats(cfg: ModelConfig) -> int:
    """Elements of the quantised matrices of all layers."""
    return cfg.n_layers * (2 * cfg.dim * cfg.dim + 2 * cfg.kv_dim * cfg.dim + 3 * cfg.dim * cfg.hidden_dim)


def _sweep(cfg: ModelConfig) -> int:
    """Bytes of all quantised matrices and RMSNorm weights."""
    return quant_bytes(_matrix_floats(cfg)) + 2 * cfg.n_layers * quant_bytes(cfg.dim)


def _tail(cfg: ModelConfig) -> int:
    """Bytes of the FP32 classifier and the final RMSNorm weights."""
    return 4 * cfg.vocab_size * cfg.dim + quant_bytes(cfg.dim)


def _cache_row(cfg: ModelConfig) -> int:
    """Bytes of one position's keys and values in all layers."""
    return 8 * cfg.n_layers * cfg.kv_dim


def _decode(cfg: ModelConfig, pos: int):
    """Bytes and operations of one decode step at position pos."""
    nbytes = _sweep(cfg) + _tail(cfg) + 4 * cfg.dim + _cache_row(cfg) * (pos + 2) + 4 * cfg.vocab_size
    flops = 2 * _matrix_floats(cfg) + 2 * cfg.vocab_size * cfg.dim + 4 * cfg.n_layers * cfg.dim * (pos + 1)
    return nbytes, flops


def work(case):
    kind = case["kind"]
    if kind == "quantise":
        return {"bytes": 4 * case["floats"] + quant_bytes(case["floats"]), "flops": 6 * case["floats"]}
    cfg = _config(case)
    if kind == "prefill":
        pos, n = case["pos"], case["prompt"]
        keys = n * pos + n * (n + 1) // 2
        nbytes = _sweep(cfg) + 4 * cfg.dim * n + _cache_row(cfg) * (pos + n)
        flops = 2 * _matrix_floats(cfg) * n + 4 * cfg.n_layers * cfg.dim * keys
        last = _decode(cfg, pos + n)
        return {"bytes": nbytes + last[0], "flops": flops + last[1]}
    if kind == "batch":
        n, mean = case["sequences"], (case["first"] + case["last"]) / 2
        nbytes = _sweep(cfg) + _tail(cfg) + n * (4 * cfg.dim + _cache_row(cfg) * (mean + 2) + 4 * cfg.vocab_size)
        flops = n * (2 * _matrix_floats(cfg) + 2 * cfg.vocab_size * cfg.dim + 4 * cfg.n_layers * cfg.dim * (mean + 1))
        return {"bytes": nbytes, "flops": flops}
    first = 0 if kind == "generate" else case["pos"]
    steps = [_decode(cfg, first + i) for i in range(case.get("steps", 1))]
    return {"bytes": sum(b for b, _ in steps), "flops": sum(f for _, f in steps)}


def tolerance(case):
    """Four times the difference between two of the package's own paths that add the row sums in another order
    (persistent and per-step kernels, prompt path and decode path): 1.5e-6 at the small shapes, 1.3e-5 at 7B,
    2e-5 at 13B.  A probability is as far off as its logit, whose spread the sampled cases make about 6."""
    kind = case["kind"]
    if kind == "quantise":
        return "exact"
    rel = {"stories15M": 6e-6, "stories110M": 8e-6, "llama2-7b": 6e-5, "llama2-13b": 8e-5}[case["shape"]]
    if kind == "sample":
        return {"rel": 6 * rel, "differ": 0.1}       # a draw may fall on the other side of a tie
    if kind == "batch":
        return {"rel": rel, "differ": 0.02}          # as may an arg-max among 64
    return {"rel": rel}
