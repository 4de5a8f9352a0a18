"""Performance cases of the engine: one pass of each is one step of the step function (or one ``generate`` call), as a
server, a trace replay or a test makes it.

The kinds of pass:

* ``decode``    one token for each of ``batch`` requests whose caches hold ``context`` tokens at the first pass and one
                more after every pass; logits of every request.
* ``prefill``   ``prompts`` new prompts of ``tokens`` tokens in all, whole, in one step; logits at each last token.
* ``mixed``     a portion of ``tokens`` tokens of a new prompt beside ``batch`` decoding requests (a tick of the
                continuous-batching scheduler); logits of every request and at the portion's last token.
* ``generate``  ``Engine.generate`` on ``prompts`` short prompts, greedy, from token lists to token lists.

Weights are random (drawn on the device from the seed), token ids uniform, caches filled by real prefill.  Sizes are
those of the engine's benchmark: the Qwen3-4B/8B/14B shapes, two tiny Qwen3 models, and the Vopepel and Fikerax models
of the designs workload.  The large shapes have 8 layers, as the designs workload has: with random weights the rounding errors of
bfloat16 grow with the depth (under 2 % of the logits at 8 layers, 2 to 4 % at 36 and 40), and two correct implementations of the
whole depth are further apart than outputs can usefully be compared.  Models with a mixture of experts are not among the cases: in bfloat16 a rounding that differs
in the last digit can choose another expert, so that two correct implementations differ by more than any tolerance.

``exact`` states the models in float64 with plain torch operations; logits are compared with it for as many of a
case's requests as it can compute in some seconds.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

PAGE = 256
CHUNK = 2_048

QWEN3 = {
    "qwen3-4b": dict(vocab_size=151_936, hidden_size=2_560, num_hidden_layers=8, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                     intermediate_size=9_728, max_position_embeddings=262_144, rope_theta=5_000_000.0, rms_norm_eps=1e-6, tie_word_embeddings=True),
    "qwen3-8b": dict(vocab_size=151_936, hidden_size=4_096, num_hidden_layers=8, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                     intermediate_size=12_288, max_position_embeddings=40_960, rope_theta=1_000_000.0, rms_norm_eps=1e-6, tie_word_embeddings=False),
    "qwen3-14b": dict(vocab_size=151_936, hidden_size=5_120, num_hidden_layers=8, num_attention_heads=40, num_key_value_heads=8, head_dim=128,
                      intermediate_size=17_408, max_position_embeddings=40_960, rope_theta=1_000_000.0, rms_norm_eps=1e-6, tie_word_embeddings=False),
    "tiny-a": dict(vocab_size=256, hidden_size=64, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=16,
                   intermediate_size=128, max_position_embeddings=512, rope_theta=10_000.0, rms_norm_eps=1e-6, tie_word_embeddings=True),
    "tiny-b": dict(vocab_size=320, hidden_size=96, num_hidden_layers=3, num_attention_heads=6, num_key_value_heads=3, head_dim=32,
                   intermediate_size=224, max_position_embeddings=512, rope_theta=1_000_000.0, rms_norm_eps=1e-5, tie_word_embeddings=False),
}
DESIGN_SIZES = {
    "2k": dict(width=2_048, layers=8, heads=16, kv_heads=4, dim=128, ff=8_192, vocab=32_768),
    "4k": dict(width=4_096, layers=8, heads=32, kv_heads=8, dim=128, ff=12_288, vocab=32_768),
}


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the tiny model of the first correctness configuration, end to end: scheduler, sampling and launches, hardly any work on the device
        {"name": "tiny_generate", "kind": "generate", "model": "tiny-a", "dtype": "float32", "prompts": 3, "tokens": 55, "new": 8},
        # one user waiting for the next token
        {"name": "4b_decode_b1", "kind": "decode", "model": "qwen3-4b", "dtype": "bfloat16", "batch": 1, "context": 512, "ragged": False},
        # the benchmark's headline: eight requests in a long conversation
        {"name": "4b_decode_b8_ctx4096", "kind": "decode", "model": "qwen3-4b", "dtype": "bfloat16", "batch": 8, "context": 4_000, "ragged": False},
        # the decode-heavy workload at its largest batch: short contexts, every slot taken
        {"name": "4b_decode_b64", "kind": "decode", "model": "qwen3-4b", "dtype": "bfloat16", "batch": 64, "context": 384, "ragged": False},
        # the first token of a short prompt of an odd length
        {"name": "4b_prefill_137", "kind": "prefill", "model": "qwen3-4b", "dtype": "bfloat16", "prompts": 1, "tokens": 137},
        # the benchmark's prompt
        {"name": "4b_prefill_2048", "kind": "prefill", "model": "qwen3-4b", "dtype": "bfloat16", "prompts": 1, "tokens": 2_048},
        # continuous batching: a full portion of a prompt beside running requests
        {"name": "8b_mixed_31_2048", "kind": "mixed", "model": "qwen3-8b", "dtype": "bfloat16", "batch": 31, "context": 1_500, "ragged": True, "tokens": 2_048},
        # the sampled serving workload's decode step: prompts of any length up to 4,096
        {"name": "14b_decode_b16_ragged", "kind": "decode", "model": "qwen3-14b", "dtype": "bfloat16", "batch": 16, "context": 4_096, "ragged": True},
        # the 32-bit check run: decode steps of a few requests ...
        {"name": "4b_f32_decode_b16", "kind": "decode", "model": "qwen3-4b", "dtype": "float32", "batch": 16, "context": 72, "ragged": False},
        # ... and their prompts, of ragged lengths
        {"name": "4b_f32_prefill_193", "kind": "prefill", "model": "qwen3-4b", "dtype": "float32", "prompts": 3, "tokens": 193},
        # the other designs: a delta rule, chunked attention and several residual streams over a prompt ...
        {"name": "vopepel_prefill_2048", "kind": "prefill", "model": "vopepel-2k", "dtype": "bfloat16", "prompts": 1, "tokens": 2_048},
        # ... and lightning, windowed and latent attention in decode steps
        {"name": "fikerax_decode_b8", "kind": "decode", "model": "fikerax-4k", "dtype": "bfloat16", "batch": 8, "context": 2_000, "ragged": False},
    ]


def _between(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["4b-decode", "4b-decode", "4b-prefill", "4b-prefill", "8b-mixed", "14b-decode", "f32-decode", "f32-prefill", "design", "design", "tiny"])
    bf16, f32 = {"dtype": "bfloat16"}, {"dtype": "float32"}
    if kind == "4b-decode":
        batch = _between(rng, 1, 64)
        return {"kind": "decode", "model": "qwen3-4b", **bf16, "batch": batch, "context": _between(rng, 64, min(4_096, 49_152 // batch)), "ragged": rng.random() < 0.5}
    if kind == "4b-prefill":
        tokens = _between(rng, 24, 3_000)
        return {"kind": "prefill", "model": "qwen3-4b", **bf16, "prompts": rng.randint(1, min(4, tokens // 8)), "tokens": tokens}
    if kind == "8b-mixed":
        return {"kind": "mixed", "model": "qwen3-8b", **bf16, "batch": _between(rng, 1, 31), "context": _between(rng, 64, 1_500), "ragged": True, "tokens": _between(rng, 32, 2_048)}
    if kind == "14b-decode":
        return {"kind": "decode", "model": "qwen3-14b", **bf16, "batch": _between(rng, 1, 16), "context": _between(rng, 64, 4_096), "ragged": True}
    if kind == "f32-decode":
        return {"kind": "decode", "model": "qwen3-4b", **f32, "batch": _between(rng, 1, 16), "context": _between(rng, 16, 512), "ragged": rng.random() < 0.5}
    if kind == "f32-prefill":
        tokens = _between(rng, 17, 320)
        return {"kind": "prefill", "model": "qwen3-4b", **f32, "prompts": rng.randint(1, 4), "tokens": tokens}
    if kind == "design":
        model = rng.choice(["vopepel", "fikerax"]) + "-" + rng.choice(["2k", "4k"])
        if rng.random() < 0.5:
            return {"kind": "prefill", "model": model, **bf16, "prompts": rng.randint(1, 3), "tokens": _between(rng, 64, 2_048)}
        return {"kind": "decode", "model": model, **bf16, "batch": _between(rng, 1, 16), "context": _between(rng, 64, 2_048), "ragged": rng.random() < 0.5}
    prompts = rng.randint(1, 4)
    return {"kind": "generate", "model": rng.choice(["tiny-a", "tiny-b"]), **f32, "prompts": prompts, "tokens": rng.randint(prompts * 8, prompts * 30), "new": rng.randint(2, 12)}


def _fractions(count):
    """``count`` numbers in (0, 1), spread evenly, in no order."""
    return [(0.5 + index * 0.6180339887498949) % 1.0 for index in range(count)]


def _contexts(case):
    """Tokens each decoding request holds before the first pass."""
    batch, longest = case["batch"], case["context"]
    if not case["ragged"]:
        return [longest] * batch
    shortest = min(64, longest)
    return [shortest + int((longest - shortest) * share) for share in _fractions(batch)]


def _prompt_lengths(case):
    """``tokens`` tokens cut into ``prompts`` prompts of unequal lengths."""
    shares = [0.25 + share for share in _fractions(case["prompts"])]
    lengths = [max(1, int(case["tokens"] * share / sum(shares))) for share in shares]
    lengths[0] += case["tokens"] - sum(lengths)
    return lengths


def _room(case):
    """Tokens a decoding request may grow by before it is started again."""
    return 512 if case["model"] in ("qwen3-8b", "qwen3-14b") or case["batch"] > 32 else 1_024 if case["model"].startswith("qwen3") else 4_096


# ---------------------------------------------------------------------------------------
# the models
# ---------------------------------------------------------------------------------------
def _vopepel(size):
    """Of every four layers the first is a gated delta rule, the others attention in chunks of 1,024 positions with value
    mixing; four copies of the residual stream."""
    def layer(index):
        mlp = {"kind": "dense", "ff": size["ff"], "limit": 7.0}
        if index % 4 == 0:
            return {"type": "delta", "mlp": mlp, "mixer": {"heads": size["heads"], "kv_heads": size["heads"] // 2, "dim": size["dim"], "vdim": size["dim"], "conv": 4}}
        return {"type": "attention", "mlp": mlp, "mixer": {"heads": size["heads"], "kv_heads": size["kv_heads"], "dim": size["dim"], "vdim": size["dim"],
                                                           "scale": size["dim"] ** -0.5, "softcap": 30.0, "mask": {"size": 1_024}, "v_mix": True}}
    return {"architecture": "Vopepel", "vocab": size["vocab"], "width": size["width"], "norm": {"eps": 1e-5}, "residual_mult": 0.5, "streams": 4,
            "layers": [layer(index) for index in range(size["layers"])]}


def _fikerax(size):
    """Of every four layers the first is lightning attention, the third latent attention, the others grouped-query attention
    with biases; every attention inside a window of 1,024 tokens."""
    def layer(index):
        mlp, heads, dim = {"kind": "dense", "ff": size["ff"]}, size["heads"], size["dim"]
        if index % 4 == 0:
            decay = [1.0 - 2.0 ** (-5.0 - 3.0 * head / max(1, heads - 1)) for head in range(heads)]
            return {"type": "lightning", "mlp": mlp, "mixer": {"heads": heads, "dim": dim, "vdim": dim, "decay": decay}}
        if index % 4 == 2:
            return {"type": "latent_attention", "mlp": mlp, "mixer": {
                "heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "q_rank": size["width"] * 3 // 8, "kv_rank": 512, "scale": (dim + dim // 2) ** -0.5,
                "mask": {"size": 1_024}, "rot": {"dims": dim // 2, "base": 10_000.0, "scaling": {"factor": 8.0, "original": 4_096, "fast": 32.0, "slow": 1.0}}}}
        return {"type": "attention", "mlp": mlp, "mixer": {
            "heads": heads, "kv_heads": size["kv_heads"], "dim": dim, "vdim": dim, "scale": 12.0 / dim, "mask": {"size": 1_024},
            "rot": {"dims": dim, "base": 500_000.0, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8_192}}}}
    return {"architecture": "Fikerax", "vocab": size["vocab"], "width": size["width"], "embedding": {"scale": size["width"] ** 0.5}, "norm": {"eps": 1e-5},
            "loop": {"start": 0, "stop": 0, "times": 1}, "layers": [layer(index) for index in range(size["layers"])]}


def _fields(model):
    if model in QWEN3:
        return QWEN3[model]
    design, size = model.split("-")
    return (_vopepel if design == "vopepel" else _fikerax)(DESIGN_SIZES[size])


def _vocab(model):
    fields = _fields(model)
    return fields.get("vocab_size") or fields["vocab"]


def _tokens(case, seed):
    """Every token id the case uses, as lists: what each decoding request holds, the tokens it decodes next, the prompts."""
    rng, vocab = np.random.default_rng([int(seed), 1]), _vocab(case["model"])
    held, fed, prompts = [], [], []
    if case["kind"] in ("decode", "mixed"):
        held = [rng.integers(0, vocab, size=count).tolist() for count in _contexts(case)]
        fed = rng.integers(0, vocab, size=(_room(case), case["batch"])).tolist()
    if case["kind"] in ("prefill", "generate"):
        prompts = [rng.integers(0, vocab, size=count).tolist() for count in _prompt_lengths(case)]
    if case["kind"] == "mixed":
        prompts = [rng.integers(0, vocab, size=case["tokens"]).tolist()]
    return held, fed, prompts


# ---------------------------------------------------------------------------------------
# preparing and running
# ---------------------------------------------------------------------------------------
def _engine(case, seed):
    from pylon_b200.config import EngineConfig, Qwen3Config
    from pylon_b200.config.model_config import FikeraxConfig, VopepelConfig
    from pylon_b200.engine import Engine

    model, kind = case["model"], case["kind"]
    fields = _fields(model)
    if model in QWEN3:
        model_config = Qwen3Config(**fields)
    else:
        model_config = (VopepelConfig if model.startswith("vopepel") else FikeraxConfig).from_dict(fields)
    page = PAGE if not model.startswith("tiny") else 16
    lengths = []
    if kind in ("decode", "mixed"):
        lengths += [count + _room(case) for count in _contexts(case)]
    if kind == "mixed":
        lengths.append(case["tokens"])
    if kind in ("prefill", "generate"):
        lengths += [count + case.get("new", 0) for count in _prompt_lengths(case)]
    pages = sum(-(-count // page) for count in lengths)
    longest = -(-max(lengths) // page) * page
    if kind == "generate":
        pages, longest = 4 * pages, max(longest, 64)
    config = EngineConfig(dtype=case["dtype"], page_size=page, max_cache_tokens=max(pages + len(lengths), longest // page) * page, max_context=longest,
                          max_batch_size=len(lengths), max_queue_size=max(4, len(lengths)), prefill_chunk_size=max(CHUNK, case.get("tokens", 0)), cuda_graphs=True)
    return Engine(None, config, device="cuda:0", model_config=model_config, random_seed=int(seed))


def _start(state):
    """Opens the decoding requests and fills their caches, a portion of a few prompts at a time."""
    from pylon_b200.engine import StepEntry

    engine, held = state["engine"], state["held"]
    for request in state["requests"]:
        engine.close(request)
    state["starts"] += 1
    requests = [engine.open(("held", state["starts"], index), len(tokens) + state["room"]) for index, tokens in enumerate(held)]
    state["requests"], state["step"] = requests, 0
    graphs, engine.step_function.graphs = engine.step_function.graphs, None     # odd portions, once each: not worth a graph
    entries, used = [], 0
    for request, tokens in zip(requests, held):
        done = 0
        while done < len(tokens):
            count = min(CHUNK - used, len(tokens) - done)
            entries.append(StepEntry(request, tokens[done : done + count], ()))
            done, used = done + count, used + count
            if used == CHUNK:
                engine.step(entries)
                entries, used = [], 0
    if entries:
        engine.step(entries)
    engine.step_function.graphs = graphs


def prepare(case, seed):
    """An engine with its weights, the graphs of the steps that will come captured, and for decoding the requests with
    their caches filled; the tokens of every pass."""
    held, fed, prompts = _tokens(case, seed)
    engine = _engine(case, seed)
    state = {"engine": engine, "kind": case["kind"], "held": held, "fed": fed, "prompts": prompts, "requests": [], "starts": 0, "step": 0,
             "room": _room(case) if held else 0, "passes": 0, "checked": _checked(case)}
    if case["kind"] == "decode":
        engine.capture_decode_graphs([case["batch"]])
    elif case["kind"] == "prefill":
        engine.capture_padded_graphs([(0, case["prompts"], case["tokens"])])
    elif case["kind"] == "mixed":
        engine.capture_padded_graphs([(case["batch"], 1, case["tokens"])])
    else:
        from pylon_b200.sampling import SamplingParams

        state["sampling"] = SamplingParams(max_new_tokens=case["new"], temperature=0.0, ignore_eos=True)
    if held:
        _start(state)
    return state


def run(state):
    """One pass; the logits (of the requests that ``exact`` computes, and of the others), or the generated tokens."""
    from pylon_b200.engine import StepEntry

    engine, kind = state["engine"], state["kind"]
    if kind == "generate":
        return [torch.tensor(result.output_ids) for result in engine.generate(state["prompts"], state["sampling"])]
    entries, opened = [], []
    if state["requests"]:
        if state["step"] == state["room"]:
            _start(state)
        entries = [StepEntry(request, [token], (0,)) for request, token in zip(state["requests"], state["fed"][state["step"]])]
        state["step"] += 1
    for index, prompt in enumerate(state["prompts"]):
        state["passes"] += 1
        request = engine.open(("prompt", state["passes"]), len(prompt))
        opened.append(request)
        entries.append(StepEntry(request, prompt, (len(prompt) - 1,)))
    logits = engine.step(entries)
    for request in opened:
        engine.close(request)
    checked = state["checked"]
    return {"logits": logits} if checked == len(entries) else {"logits": logits[:checked], "others": logits[checked:]}


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _matrix_shapes(model):
    """(all matrices but the embedding and the head, as numbers of elements; attention layers as (heads, key width, value width, cached
    numbers per token, window); state numbers per request)."""
    fields = _fields(model)
    if model in QWEN3:
        h, q, kv, inter, layers = (fields["hidden_size"], fields["num_attention_heads"] * fields["head_dim"], fields["num_key_value_heads"] * fields["head_dim"],
                                   fields["intermediate_size"], fields["num_hidden_layers"])
        attention = (fields["num_attention_heads"], fields["head_dim"], fields["head_dim"], 2 * kv, None)
        return layers * (h * (q + 2 * kv) + q * h + 3 * h * inter), [attention] * layers, 0
    h, elements, attention, state = fields["width"], 0, [], 0
    for layer in fields["layers"]:
        m = layer["mixer"]
        if layer["type"] in ("delta", "lightning"):
            keys, values = m.get("kv_heads", m["heads"]) * m["dim"], m["heads"] * m["vdim"]
            elements += h * (2 * keys + 3 * values)
            state += m["heads"] * m["dim"] * m["vdim"]
        elif layer["type"] == "attention":
            elements += h * (m["heads"] * m["dim"] + m["kv_heads"] * (m["dim"] + m["vdim"]) + m["heads"] * m["vdim"])
            attention.append((m["heads"], m["dim"], m["vdim"], m["kv_heads"] * (m["dim"] + m["vdim"]), m["mask"]["size"]))
        else:
            rank, heads = m["kv_rank"], m["heads"]
            elements += h * (m["q_rank"] + rank + m["rot_dim"]) + m["q_rank"] * heads * (m["dim"] + m["rot_dim"]) + rank * heads * (m["dim"] + m["vdim"]) + heads * m["vdim"] * h
            attention.append((heads, m["dim"] + m["rot_dim"], m["vdim"], rank + m["rot_dim"], m["mask"]["size"]))
        elements += 3 * h * layer["mlp"]["ff"]
    return elements, attention, state


def work(case):
    """Bytes: every matrix once, the keys and values (and states) that are read and written, the logits.  Operations: the
    matrix products of every token, the visible scores and weighted sums, the head at the wanted places."""
    model, kind = case["model"], case["kind"]
    elements, attention, state = _matrix_shapes(model)
    fields = _fields(model)
    head = _vocab(model) * (fields.get("hidden_size") or fields["width"])
    size = 2 if case["dtype"] == "bfloat16" else 4
    rows = []   # (tokens held before, new tokens)
    if kind in ("decode", "mixed"):
        rows += [(count, 1) for count in _contexts(case)]
    if kind in ("prefill", "generate"):
        rows += [(0, count) for count in _prompt_lengths(case)]
    if kind == "mixed":
        rows.append((0, case["tokens"]))
    passes = case.get("new", 1)
    total = {"bytes": 0.0, "flops": 0.0}
    for turn in range(passes):
        if turn == 1:
            rows = [(count, 1) for _, count in rows]
        elif turn > 1:
            rows = [(before + 1, 1) for before, _ in rows]
        new, wanted = sum(count for _, count in rows), len(rows)
        bytes_, flops = (elements + head) * size + wanted * _vocab(model) * 4, 2.0 * elements * new + 2.0 * head * wanted
        for heads, keys, values, cached, window in attention:
            for before, count in rows:
                seen = count * before + count * (count + 1) / 2
                if window is not None:
                    seen = min(seen, float(count) * window)
                    before = min(before, window)
                flops += 2.0 * heads * (keys + values) * seen
                bytes_ += (before + count) * cached * size
        bytes_ += 2.0 * state * 4 * len(rows)
        total["bytes"] += bytes_
        total["flops"] += flops
    return total


def tolerance(case):
    """Float32: four times the 7e-6 that separates a pass from ``exact``.  bfloat16: passes are 0.8 to 1.9 % from it, and two that
    round at other places are up to the square root of two times that from each other."""
    if case["kind"] == "generate":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 3e-5, "max": 3e-4}
    return {"rel": 0.03, "max": 0.25}


# ---------------------------------------------------------------------------------------
# the same in float64, with plain torch operations
# ---------------------------------------------------------------------------------------
def _checked(case):
    """How many of the step's requests (the first ones) ``exact`` computes: as many as stay within some seconds."""
    counts = []
    if case["kind"] in ("decode", "mixed"):
        counts += [count + 1 for count in _contexts(case)]
    if case["kind"] in ("prefill", "generate"):
        counts += _prompt_lengths(case)
    if case["kind"] == "mixed":
        counts.append(case["tokens"])
    limit = 1.2e14 / (2.0 * _matrix_shapes(case["model"])[0])      # operations: some seconds of 64-bit products
    used, rows = 0, 0
    for count in counts:
        if rows and used + count > limit:
            break
        used, rows = used + count, rows + 1
    return rows


def exact(case, seed):
    if case["kind"] == "generate":
        return None
    held, fed, prompts = _tokens(case, seed)
    sequences = [tokens + [token] for tokens, token in zip(held, fed[0] if fed else [])] + prompts
    checked = _checked(case)
    model, dtype = case["model"], torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    forward = _qwen3_logits if model in QWEN3 else _vopepel_logits if model.startswith("vopepel") else _fikerax_logits
    with torch.no_grad():
        logits = forward(_fields(model), _Weights(seed, dtype), [torch.tensor(tokens, device="cuda") for tokens in sequences[:checked]])
    return {"logits": logits} if checked == len(sequences) else {"logits": logits, "others": None}


class _Weights:
    """The random weights of an engine made from a seed, in float64: each tensor from a generator seeded by (seed, name)."""

    def __init__(self, seed, dtype):
        self.seed, self.dtype, self.generator = int(seed), dtype, torch.Generator(device="cuda")

    def _drawn(self, name, shape, dtype, mean, deviation):
        self.generator.manual_seed((self.seed * 1_000_003 + zlib.crc32(name.encode())) % (2 ** 63 - 1))
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(mean, deviation, generator=self.generator)

    def matrix(self, name, *shape):
        return self._drawn(name, shape, self.dtype, 0.0, 0.02).double()

    def rows(self, name, ids, *shape):
        return self._drawn(name, shape, self.dtype, 0.0, 0.02)[ids].double()

    def around_one(self, name, *shape):
        return (self._drawn(name, shape, torch.float32, 0.0, 0.02) + 1.0).double()

    def vector(self, name, shape, mean, deviation):
        return self._drawn(name, shape, torch.float32, mean, deviation).double()


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _layer_norm(x, weight, eps):
    centred = x - x.mean(dim=-1, keepdim=True)
    return _unit(centred, eps) * weight


def _attention(q, k, v, scale, hidden=None, softcap=None, sink=None):
    """``q [T, heads, d]``, ``k``/``v [T, kv_heads, ...]`` of one sequence; ``hidden(i, j)``: which earlier positions j a position i does not see."""
    count, heads = q.shape[:2]
    group = heads // k.shape[1]
    k, v = (t.transpose(0, 1).repeat_interleave(group, dim=0) for t in (k, v))
    out = torch.empty(heads, count, v.shape[-1], dtype=q.dtype, device=q.device)
    j = torch.arange(count, device=q.device)[None, :]
    for begin in range(0, count, 1_024):
        end = min(count, begin + 1_024)
        scores = q[begin:end].transpose(0, 1) @ k.transpose(1, 2) * scale
        if softcap:
            scores = softcap * torch.tanh(scores / softcap)
        i = torch.arange(begin, end, device=q.device)[:, None]
        mask = j > i
        if hidden is not None:
            mask = mask | hidden(i, j)
        scores = scores.masked_fill(mask, -math.inf)
        if sink is not None:
            scores = torch.cat((scores, sink[:, None, None].expand(-1, end - begin, 1)), dim=-1)
        out[:, begin:end] = torch.softmax(scores, dim=-1)[..., :count] @ v
    return out.transpose(0, 1)


def _per_sequence(x, lengths, function):
    return torch.cat([function(part) for part in x.split(lengths)])


def _qwen3_logits(c, w, sequences):
    heads, groups, dim, h, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["hidden_size"], c["rms_norm_eps"]
    lengths, vocab = [len(tokens) for tokens in sequences], c["vocab_size"]
    x = w.rows("model.embed_tokens.weight", torch.cat(sequences), vocab, h)
    positions = torch.cat([torch.arange(count) for count in lengths])
    inverse = 1.0 / (c["rope_theta"] ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim))     # the angle is formed in 32 bits, as the model defines it
    angle = (positions.float()[:, None] * inverse[None, :]).double().cuda()
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]

    def turned(t):
        a, b = t[..., : dim // 2], t[..., dim // 2 :]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), dim=-1)

    for index in range(c["num_hidden_layers"]):
        p = f"model.layers.{index}."
        y = _unit(x, eps) * w.around_one(p + "input_layernorm.weight", h)
        q = (y @ w.matrix(p + "self_attn.q_proj.weight", heads * dim, h).T).view(-1, heads, dim)
        k = (y @ w.matrix(p + "self_attn.k_proj.weight", groups * dim, h).T).view(-1, groups, dim)
        v = (y @ w.matrix(p + "self_attn.v_proj.weight", groups * dim, h).T).view(-1, groups, dim)
        q = turned(_unit(q, eps) * w.around_one(p + "self_attn.q_norm.weight", dim))
        k = turned(_unit(k, eps) * w.around_one(p + "self_attn.k_norm.weight", dim))
        mixed = torch.cat([_attention(a, b, e, dim ** -0.5) for a, b, e in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        x = x + mixed.reshape(-1, heads * dim) @ w.matrix(p + "self_attn.o_proj.weight", h, heads * dim).T
        y = _unit(x, eps) * w.around_one(p + "post_attention_layernorm.weight", h)
        gate = y @ w.matrix(p + "mlp.gate_proj.weight", c["intermediate_size"], h).T
        up = y @ w.matrix(p + "mlp.up_proj.weight", c["intermediate_size"], h).T
        x = x + (gate * torch.sigmoid(gate) * up) @ w.matrix(p + "mlp.down_proj.weight", h, c["intermediate_size"]).T
    last = torch.tensor(lengths).cumsum(0).cuda() - 1
    x = _unit(x[last], eps) * w.around_one("model.norm.weight", h)
    return x @ w.matrix("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight", vocab, h).T


def _silu(x):
    return x * torch.sigmoid(x)


def _vopepel_logits(c, w, sequences):
    h, eps, mult, streams, vocab = c["width"], c["norm"]["eps"], c["residual_mult"], c["streams"], c["vocab"]
    lengths = [len(tokens) for tokens in sequences]
    x = w.rows("embed", torch.cat(sequences), vocab, h)
    xs = torch.stack([x] * streams)
    first_values = None

    def convolved(t, taps):
        padded = torch.cat((torch.zeros(taps.shape[1] - 1, t.shape[1], dtype=t.dtype, device=t.device), t))
        return _silu(sum(padded[j : j + t.shape[0]] * taps[:, j] for j in range(taps.shape[1])))

    def delta(y, p, m):
        heads, groups, dim, vdim = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        projected = {name: y @ w.matrix(p + name, width, h).T for name, width in
                     (("q", groups * dim), ("k", groups * dim), ("v", heads * vdim), ("g", heads * vdim), ("a", heads), ("b", heads))}
        for name in "qkv":
            taps = w.vector(p + name + ".conv", (projected[name].shape[1], m["conv"]), 0.0, 0.5)
            projected[name] = _per_sequence(projected[name], lengths, lambda t: convolved(t, taps))
        q, k = (projected[name].view(-1, groups, dim) for name in "qk")
        q = q / torch.sqrt((q * q).sum(dim=-1, keepdim=True) + 1e-6) * dim ** -0.5
        k = k / torch.sqrt((k * k).sum(dim=-1, keepdim=True) + 1e-6)
        q, k = (t.repeat_interleave(heads // groups, dim=1) for t in (q, k))
        v, beta = projected["v"].view(-1, heads, vdim), torch.sigmoid(projected["b"])
        dt = projected["a"] + w.vector(p + "dt_bias", (heads,), 0.0, 0.5)
        decay = torch.exp(-torch.exp(w.vector(p + "A_log", (heads,), -1.0, 0.5)) * torch.nn.functional.softplus(dt, threshold=1e9))
        out, begin = torch.empty_like(v), 0
        for count in lengths:
            state = torch.zeros(heads, dim, vdim, dtype=v.dtype, device=v.device)
            for t in range(begin, begin + count):
                state = state * decay[t, :, None, None]
                write = beta[t, :, None] * (v[t] - (k[t, :, None, :] @ state)[:, 0])
                state = torch.baddbmm(state, k[t, :, :, None], write[:, None, :])
                out[t] = (q[t, :, None, :] @ state)[:, 0]
            begin += count
        out = _unit(out, eps) * w.around_one(p + "norm", vdim) * _silu(projected["g"]).view(-1, heads, vdim)
        return out.reshape(-1, heads * vdim) @ w.matrix(p + "o", h, heads * vdim).T

    def attention(y, p, m):
        nonlocal first_values
        heads, groups, dim, vdim, chunk = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["mask"]["size"]
        q = _unit((y @ w.matrix(p + "q", heads * dim, h).T).view(-1, heads, dim), eps) * w.around_one(p + "q.norm", dim)
        k = _unit((y @ w.matrix(p + "k", groups * dim, h).T).view(-1, groups, dim), eps) * w.around_one(p + "k.norm", dim)
        v = (y @ w.matrix(p + "v", groups * vdim, h).T).view(-1, groups, vdim)
        if first_values is None:
            first_values = v
        else:
            share = w.vector(p + "vmix", (), 0.5, 0.1)
            v = (1 - share) * v + share * first_values
        out = torch.cat([_attention(a, b, e, m["scale"], lambda i, j: i // chunk != j // chunk, m["softcap"]) for a, b, e in
                         zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        return out.reshape(-1, heads * vdim) @ w.matrix(p + "o", h, heads * vdim).T

    def feed_forward(y, p, m):
        gate = torch.clamp(y @ w.matrix(p + "gate", m["ff"], h).T, max=m["limit"])
        up = torch.clamp(y @ w.matrix(p + "up", m["ff"], h).T, min=-m["limit"], max=m["limit"])
        return (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ w.matrix(p + "down", h, m["ff"]).T

    for index, layer in enumerate(c["layers"]):
        p = f"l{index}."
        for number in (1, 2):
            enter, leave = w.vector(f"{p}hc{number}.in", (streams,), 0.25, 0.1), w.vector(f"{p}hc{number}.out", (streams,), 1.0, 0.1)
            mix = w.vector(f"{p}hc{number}.mix", (streams, streams), 0.25, 0.1)
            y = _layer_norm(torch.einsum("s,sth->th", enter, xs), w.around_one(f"{p}norm{number}", h), eps)
            y = feed_forward(y, p + "mlp.", layer["mlp"]) if number == 2 else (delta if layer["type"] == "delta" else attention)(y, p + "mix.", layer["mixer"])
            xs = torch.einsum("sr,sth->rth", mix, xs) + mult * leave[:, None, None] * y
    last = torch.tensor(lengths).cumsum(0).cuda() - 1
    x = _layer_norm(xs.sum(dim=0)[last], w.around_one("final.norm", h), eps)
    return x @ w.matrix("head", vocab, h).T


def _fikerax_logits(c, w, sequences):
    h, eps, vocab = c["width"], c["norm"]["eps"], c["vocab"]
    lengths = [len(tokens) for tokens in sequences]
    positions = torch.cat([torch.arange(count) for count in lengths]).double().cuda()
    x = w.rows("embed", torch.cat(sequences), vocab, h) * c["embedding"]["scale"]

    def outside(window):
        return lambda i, j: i - j >= window

    def lightning(y, p, m):
        heads, dim, vdim = m["heads"], m["dim"], m["vdim"]
        q, k = (_silu(y @ w.matrix(p + name, heads * dim, h).T).view(-1, heads, dim) for name in "qk")
        v = _silu(y @ w.matrix(p + "v", heads * vdim, h).T).view(-1, heads, vdim)
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=y.device)[:, None, None]
        out, begin = torch.empty_like(v), 0
        for count in lengths:
            state = torch.zeros(heads, dim, vdim, dtype=v.dtype, device=v.device)
            for t in range(begin, begin + count):
                state = torch.baddbmm(state * decay, k[t, :, :, None], v[t, :, None, :])
                out[t] = (q[t, :, None, :] @ state)[:, 0]
            begin += count
        normed = _unit(out.reshape(-1, heads * vdim), eps) * w.around_one(p + "norm", heads * vdim)
        return (normed * torch.sigmoid(y @ w.matrix(p + "g", heads * vdim, h).T)) @ w.matrix(p + "o", h, heads * vdim).T

    def attention(y, p, m):
        heads, groups, dim, vdim, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
        q, k, v = ((y @ w.matrix(p + name, width, h).T + w.vector(p + name + ".b", (width,), 0.0, 0.02)).view(-1, count, width // count)
                   for name, count, width in (("q", heads, heads * dim), ("k", groups, groups * dim), ("v", groups, groups * vdim)))
        freq = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=torch.float64) / rot["dims"])
        s = rot["scaling"]
        wave = 2.0 * math.pi / freq
        blend = ((s["original"] / wave - s["low"]) / (s["high"] - s["low"])).clamp(0.0, 1.0)       # 1: a short wave, kept; 0: a long one, slowed
        angle = positions[:, None, None] * ((1.0 - blend) * freq / s["factor"] + blend * freq).cuda()
        cos, sin, half = torch.cos(angle), torch.sin(angle), rot["dims"] // 2

        def turned(t):
            a, b = t[..., :half], t[..., half : 2 * half]
            return torch.cat((a * cos - b * sin, b * cos + a * sin, t[..., 2 * half :]), dim=-1)

        q, k = _unit(turned(q), eps), _unit(turned(k), eps)
        out = torch.cat([_attention(a, b, e, m["scale"], outside(m["mask"]["size"])) for a, b, e in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        return out.reshape(-1, heads * vdim) @ w.matrix(p + "o", h, heads * vdim).T

    def latent(y, p, m):
        heads, dim, rot_dim, vdim, rank, rot = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["rot"]
        compressed = _unit(y @ w.matrix(p + "dq", m["q_rank"], h).T, eps) * w.around_one(p + "dq.norm", m["q_rank"])
        q = (compressed @ w.matrix(p + "uq", heads * (dim + rot_dim), m["q_rank"]).T).view(-1, heads, dim + rot_dim)
        down = y @ w.matrix(p + "dkv", rank + rot_dim, h).T
        row = _unit(down[:, :rank], eps) * w.around_one(p + "dkv.norm", rank)
        s, dims = rot["scaling"], rot["dims"]

        def pair_of(turns):
            return dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))

        low, high = max(math.floor(pair_of(s["fast"])), 0), min(math.ceil(pair_of(s["slow"])), dims - 1)
        pairs = torch.arange(dims // 2, dtype=torch.float64)
        freq, ramp = rot["base"] ** (-2.0 * pairs / dims), ((pairs - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        angle = positions[:, None, None] * (freq / s["factor"] * ramp + freq * (1.0 - ramp)).cuda()
        gain = 0.1 * math.log(s["factor"]) + 1.0
        cos, sin = torch.cos(angle) * gain, torch.sin(angle) * gain

        def turned(t):
            a, b = t[..., 0::2], t[..., 1::2]
            return torch.stack((a * cos - b * sin, b * cos + a * sin), dim=-1).flatten(-2)

        q = torch.cat((q[..., :dim], turned(q[..., dim:])), dim=-1)
        key_turn = turned(down[:, None, rank:]).expand(-1, heads, -1)
        k = torch.cat(((row @ w.matrix(p + "uk", heads * dim, rank).T).view(-1, heads, dim), key_turn), dim=-1)
        v = (row @ w.matrix(p + "uv", heads * vdim, rank).T).view(-1, heads, vdim)
        sink = w.vector(p + "sink", (heads,), 0.0, 1.0)
        out = torch.cat([_attention(a, b, e, m["scale"], outside(m["mask"]["size"]), sink=sink) for a, b, e in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        return out.reshape(-1, heads * vdim) @ w.matrix(p + "o", h, heads * vdim).T

    mixers = {"lightning": lightning, "attention": attention, "latent_attention": latent}
    for index, layer in enumerate(c["layers"]):
        p, ff = f"l{index}.", layer["mlp"]["ff"]
        x = x + mixers[layer["type"]](_unit(x, eps) * (1.0 + w.vector(p + "norm1", (h,), 0.0, 0.02)), p + "mix.", layer["mixer"])
        y = _unit(x, eps) * (1.0 + w.vector(p + "norm2", (h,), 0.0, 0.02))
        x = x + (_silu(y @ w.matrix(p + "mlp.gate", ff, h).T) * (y @ w.matrix(p + "mlp.up", ff, h).T)) @ w.matrix(p + "mlp.down", h, ff).T
    last = torch.tensor(lengths).cumsum(0).cuda() - 1
    x = _unit(x[last], eps) * (1.0 + w.vector("final.norm", (h,), 0.0, 0.02))
    return x @ w.matrix("head", vocab, h).T
