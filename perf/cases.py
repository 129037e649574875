"""Performance cases of the decoder hot path, run through the package's public entry points.

A case is one call a serving program makes with everything it keeps in hand: a planned and
bound decoder (``plan_decode`` / ``plan_prefill`` -> ``BoundDecoder``, what ``make_backend``
returns for a compiled model), called directly or replayed from a CUDA graph (``graphed``), or
a whole greedy generation (``GreedyGenerator``: compiled prefill, then a device-side loop).

* ``decode``    one token for every row of a batch whose KV cache already holds ``keys`` keys
                (``ragged``: a length of its own per row).  Every pass starts at the same lengths,
                as a program does that re-scores or re-samples from one cached prefix.
* ``prefill``   a whole prompt, logits at every position.
* ``generate``  prompt in, picked ids out: prefill that seeds the KV state, then one decode
                step and one greedy pick per token, with no host work in between.

Model shapes are the package's own presets (``megabake_b200.models.PRESETS``) with seeded
random weights; batch 1 to 8 (the 256-wide heads: to 4), 1 to 8,192 cached keys, 16 to 2,048
prompt tokens.
"""

from __future__ import annotations

import functools
import math

import torch

from megabake_b200 import BoundDecoder, GreedyGenerator, graphed, models
from megabake_b200.planner import plan_decode, plan_prefill

DECODE_MODELS = ("smollm-135m", "qwen2-0.5b", "llama-3.2-1b", "smollm-1.7b", "gemma-2b")
PREFILL_MODELS = ("smollm-135m", "qwen2-0.5b", "llama-3.2-1b", "gemma-2b")
MAX_KEYS, MAX_PROMPT_ROWS = 8192, 2048


def _decode(name, model, batch, keys, *, ragged=False, graph=False):
    return {"name": name, "kind": "decode", "model": model, "batch": batch, "keys": keys,
            "ragged": ragged, "graph": graph}


def _prefill(name, model, batch, tokens, *, graph=False):
    return {"name": name, "kind": "prefill", "model": model, "batch": batch, "tokens": tokens,
            "graph": graph}


def listed():
    return [
        # the smallest call: a chat turn on the smallest model, all latency
        _decode("decode-135m-b1-k33", "smollm-135m", 1, 33, graph=True),
        # interactive, one user with a document in the context; an odd context length
        _decode("decode-0.5b-b1-k1531", "qwen2-0.5b", 1, 1531),
        # the benchmark's default workload: a full batch over long contexts
        _decode("decode-0.5b-b8-k4096", "qwen2-0.5b", 8, 4096, graph=True),
        # one user on a 1B model, short context: bound by the weights
        _decode("decode-1b-b1-k512", "llama-3.2-1b", 1, 512, graph=True),
        # continuous batching: five requests at different depths of their conversations
        _decode("decode-1b-b5-ragged-k3001", "llama-3.2-1b", 5, 3001, ragged=True),
        # the largest decode: multi-head attention, full batch, bound by the KV cache
        _decode("decode-1.7b-b8-k8192", "smollm-1.7b", 8, 8192),
        # multi-query attention with 256-wide heads
        _decode("decode-gemma-b2-k777", "gemma-2b", 2, 777, graph=True),
        # a one-line prompt on the smallest model
        _prefill("prefill-135m-b1-t19", "smollm-135m", 1, 19, graph=True),
        # a few medium prompts at once, ragged tile edges everywhere
        _prefill("prefill-0.5b-b4-t333", "qwen2-0.5b", 4, 333),
        # short and long prompts of the benchmark's prefill workload
        _prefill("prefill-gemma-b1-t128", "gemma-2b", 1, 128, graph=True),
        _prefill("prefill-gemma-b1-t2048", "gemma-2b", 1, 2048),
        # a complete short answer, prompt to ids
        {"name": "generate-1b-b1-p64-n33", "kind": "generate", "model": "llama-3.2-1b", "batch": 1,
         "tokens": 64, "new": 33},
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choices(("decode", "prefill", "generate"), (60, 36, 4))[0]
    if kind == "decode":
        model = rng.choice(DECODE_MODELS)
        batch = rng.randint(1, 4 if model == "gemma-2b" else 8)
        case = _decode("", model, batch, _log_uniform(rng, 1, MAX_KEYS), ragged=rng.random() < 0.3,
                       graph=rng.random() < 0.5)
    elif kind == "prefill":
        batch, rows = rng.choice((1, 1, 2, 3, 4)), _log_uniform(rng, 16, MAX_PROMPT_ROWS)
        case = _prefill("", rng.choice(PREFILL_MODELS), batch, max(4, rows // batch),
                        graph=rng.random() < 0.5)
    else:
        case = {"name": "", "kind": kind, "model": "llama-3.2-1b", "batch": rng.randint(1, 4),
                "tokens": _log_uniform(rng, 16, 256), "new": rng.randint(8, 25)}
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
def _lengths(case):
    """Cached keys of every row; ragged rows are spread from ``keys`` down to a fraction of it."""
    batch, keys = case["batch"], case["keys"]
    if not case["ragged"]:
        return [keys] * batch
    return [max(1, keys - row * keys // (batch + 1)) for row in range(batch)]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _prepare_decode(case, seed):
    spec = models.get_spec(case["model"])
    batch, lengths = case["batch"], _lengths(case)
    capacity = case["keys"] + 33
    g = _generator(seed)
    weights = models.init_weights(spec, seed, "cuda", on_device=True)
    inv_freq = models.inv_freq_buffer(spec, "cuda")
    # keys and values of a normalised hidden state through N(0, 0.02) projections
    std = 0.02 * math.sqrt(spec.hidden)
    shape = (spec.layers, batch, capacity, spec.kv_heads, spec.head_dim)
    keys, values = (torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)
                    for _ in range(2))
    keys[:, :, case["keys"]:] = 0
    values[:, :, case["keys"]:] = 0
    count = batch if case["ragged"] else 1
    start = torch.zeros(spec.layers, (count + 3) // 4 * 4, dtype=torch.int32, device="cuda")
    start[:, :count] = torch.tensor(lengths[:count], dtype=torch.int32, device="cuda")
    length = start.clone()
    state = [t for layer in range(spec.layers)
             for t in (keys[layer], values[layer], length[layer, :count])]
    ids = torch.randint(0, spec.vocab, (batch, 1), generator=g, device="cuda")
    positions = torch.tensor(lengths, dtype=torch.int64, device="cuda")[:, None].contiguous()
    args = models.direct_arguments(spec, weights, inv_freq, ids, positions, state)
    program = models.direct_program(spec, batch, capacity, per_row_lengths=case["ragged"])
    step = BoundDecoder(plan_decode(program), args)
    if case["graph"]:
        step = graphed(step, *args)
    appended = [cache[:, row, lengths[row]] for row in range(batch) for cache in (keys, values)]
    return {"kind": "decode", "step": step, "args": args, "length": length, "start": start,
            "state": {"keys": keys, "values": values, "length": length, "appended": appended}}


def _prepare_prefill(case, seed):
    spec = models.get_spec(case["model"])
    weights = models.init_weights(spec, seed, "cuda", on_device=True)
    inv_freq = models.inv_freq_buffer(spec, "cuda")
    ids = torch.randint(0, spec.vocab, (case["batch"], case["tokens"]), generator=_generator(seed),
                        device="cuda")
    args = models.direct_prefill_arguments(spec, weights, inv_freq, ids)
    program = models.direct_prefill_program(spec, case["batch"], case["tokens"])
    step = BoundDecoder(plan_prefill(program), args)
    if case["graph"]:
        step = graphed(step, *args)
    return {"kind": "prefill", "step": step, "args": args}


@functools.lru_cache(maxsize=2)
def _served_model(model, batch, tokens, capacity):
    """The compiled generator a server keeps for one model and shape; requests only bring ids.
    The embedding rows are scaled up so that the picks have the margin of a trained model (with
    plain random weights the two best logits are often closer than one rounding step)."""
    spec = models.get_spec(model)
    weights = models.init_weights(spec, 0, "cuda", on_device=True)
    weights["model.embed_tokens.weight"] *= 50.0
    torch._dynamo.reset()
    return GreedyGenerator(models.build_hf_model(spec, 0, "cuda", weights), batch, tokens, capacity)


def _prepare_generate(case, seed):
    spec = models.get_spec(case["model"])
    generator = _served_model(case["model"], case["batch"], case["tokens"],
                              case["tokens"] + case["new"] + 15)
    ids = torch.randint(0, spec.vocab, (case["batch"], case["tokens"]), generator=_generator(seed),
                        device="cuda")
    return {"kind": "generate", "generator": generator, "ids": ids, "new": case["new"]}


def prepare(case, seed):
    return {"decode": _prepare_decode, "prefill": _prepare_prefill,
            "generate": _prepare_generate}[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "generate":
        generator, new = state["generator"], state["new"]
        ids = generator.on_device(state["ids"], new, steps_per_graph=_steps_per_graph(new))
        return {"ids": ids, "state": list(generator.state)}
    if state["kind"] == "prefill":
        return {"logits": state["step"](*state["args"])}
    state["length"].copy_(state["start"])
    return {"logits": state["step"](*state["args"]), **state["state"]}


def _steps_per_graph(new):
    """Decode steps per replayed graph: the largest divisor of ``new - 1`` up to 8."""
    return max(n for n in range(1, 9) if (new - 1) % n == 0)


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------
def _matmul_parameters(spec):
    """Weights of the layers' projections, and of the LM head."""
    q_dim, kv_dim = spec.heads * spec.head_dim, spec.kv_heads * spec.head_dim
    per_layer = 2 * q_dim * spec.hidden + 2 * kv_dim * spec.hidden + 3 * spec.hidden * spec.intermediate
    return spec.layers * per_layer, spec.vocab * spec.hidden


def _decode_work(spec, lengths):
    batch = len(lengths)
    kv_row = spec.layers * 2 * spec.kv_heads * spec.head_dim * 2
    layers, head = _matmul_parameters(spec)
    return {
        "bytes": 2 * spec.parameter_count() + kv_row * (sum(lengths) + batch) + 2 * batch * spec.vocab,
        "flops": 2 * batch * (layers + head)
        + 4 * (sum(lengths) + batch) * spec.heads * spec.head_dim * spec.layers,
    }


def _prefill_work(spec, batch, tokens, *, kv_rows=0):
    layers, head = _matmul_parameters(spec)
    attention = 2 * tokens * (tokens + 1) * spec.heads * spec.head_dim * spec.layers
    kv_row = spec.layers * 2 * spec.kv_heads * spec.head_dim * 2
    return {
        "bytes": 2 * spec.parameter_count() + 8 * batch * tokens + 2 * batch * tokens * spec.vocab
        + kv_row * kv_rows,
        "flops": batch * (2 * tokens * (layers + head) + attention),
    }


def work(case):
    spec = models.get_spec(case["model"])
    if case["kind"] == "decode":
        return _decode_work(spec, _lengths(case))
    if case["kind"] == "prefill":
        return _prefill_work(spec, case["batch"], case["tokens"])
    total = _prefill_work(spec, case["batch"], case["tokens"], kv_rows=case["batch"] * case["tokens"])
    for step in range(case["new"] - 1):
        one = _decode_work(spec, [case["tokens"] + step] * case["batch"])
        total = {key: total[key] + one[key] for key in total}
    return total


def tolerance(case):
    """bf16 activations rounded at some 200 points one after another: two forwards that differ
    only in the order of their fp32 sums end up about 2e-2 apart in the logits of a 16- to
    30-layer model (``tests/test_noise_floor.py`` measures it).  The largest single logit of a
    vocabulary of 50 to 256 thousand lies several standard deviations above that.  Ids and lengths
    are exact."""
    return {"rel": 0.03, "max": 0.3}
