"""Short prompts as one launch (``csrc/mb_prompt.cu``) against the same plan as one launch per phase.

Both round at the same points; what differs is the order of fp32 sums, so a few results land one bf16
step apart and travel on through the layers.  A one- or two-layer model rounds a value about 20 times
(2^-9 relative each, independent): 2^-9 x sqrt(20) ~ 0.9 % between two such forwards, taken twice.
"""

from dataclasses import replace

import pytest
import torch

from megabake_b200 import models
from megabake_b200.engine import BoundDecoder
from megabake_b200.planner import plan_prefill

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

REL = 0.018
SWITCH = "MEGABAKE_B200_PREFILL_ONE_LAUNCH"


def _program(spec, batch, tokens, capacity, q_scale, per_row):
    program = replace(models.direct_prefill_program(spec, batch, tokens), q_scale=q_scale)
    if capacity == 0:
        return program
    base = 2 + len(list(models.parameter_shapes(spec)))
    layers = tuple(replace(layer, key_cache=base + 3 * i, value_cache=base + 3 * i + 1, valid_length=base + 3 * i + 2)
                   for i, layer in enumerate(program.layers))
    return replace(program, capacity=capacity, layers=layers, length_count=batch if per_row else 1)


def _both(monkeypatch, spec, batch, tokens, *, capacity=0, q_scale=None, per_row=False):
    """(logits, state) of the one launch and of the launches of their own, and the plans' launch counts."""
    g = torch.Generator().manual_seed(tokens)
    weights = {k: v.cuda() for k, v in models.init_weights(spec, 5).items()}
    for name, value in weights.items():   # norm weights are 1.0 otherwise, and would not show a wrong index
        if "norm" in name:
            value += 0.25 * torch.randn(value.shape, generator=g).cuda().to(value.dtype)
    ids = torch.randint(0, spec.vocab, (batch, tokens), generator=g).cuda()
    layout = plan_prefill(_program(spec, batch, tokens, capacity, q_scale, per_row))
    results = []
    for switch in ("1", "0"):
        monkeypatch.setenv(SWITCH, switch)
        state = [torch.full_like(t, 7) for t in models.make_state(spec, batch, capacity, "cuda", per_row)] \
            if capacity else []
        args = models.direct_prefill_arguments(spec, weights, models.inv_freq_buffer(spec).cuda(), ids)
        args = [*args, *state]
        bound = BoundDecoder(layout, args)
        logits = bound(*args).clone()
        bound.check()
        assert torch.equal(bound(*args), logits)   # the counters are as the next launch wants them
        bound.check()
        results.append((logits.float(), state, bound.plan.launches))
    return results, len(layout.phases)


def _close(a, b):
    assert torch.isfinite(a).all()
    rel = float((a - b).norm() / b.norm())
    assert rel < REL, rel


@pytest.mark.parametrize("name,batch,tokens", [
    ("tiny-llama", 1, 1), ("tiny-llama", 1, 15), ("tiny-llama", 1, 16), ("tiny-llama", 1, 17),
    ("tiny-llama3", 3, 11), ("tiny-qwen2", 1, 64), ("tiny-qwen2", 1, 65), ("tiny-qwen2", 5, 31),
    ("tiny-mha", 1, 128), ("tiny-mha", 1, 129),      # one block of keys, two
    ("tiny-gemma", 1, 33), ("tiny-gemma", 1, 150),   # heads of 128; one row of tokens a CTA, then four
    ("tiny-gemma256", 2, 64), ("tiny-gemma256", 1, 128), ("tiny-gemma256", 1, 257),
    ("tiny-llama", 1, 640), ("tiny-qwen2", 2, 300),
])
def test_one_launch_matches_launches_of_their_own(monkeypatch, name, batch, tokens):
    (one, chain), phases = _both(monkeypatch, models.get_spec(name), batch, tokens)
    assert one[2] == 1 and chain[2] >= phases
    _close(one[0], chain[0])


@pytest.mark.parametrize("name,batch,tokens,capacity,per_row", [
    ("tiny-llama", 1, 19, 19, False), ("tiny-qwen2", 3, 5, 40, True), ("tiny-gemma", 2, 33, 70, False),
    ("tiny-mha", 7, 3, 9, True), ("tiny-gemma256", 1, 130, 131, False),
])
def test_one_launch_hands_over_the_state(monkeypatch, name, batch, tokens, capacity, per_row):
    spec = models.get_spec(name)
    (one, chain), _ = _both(monkeypatch, spec, batch, tokens, capacity=capacity, per_row=per_row)
    assert one[2] == 1 < chain[2]
    _close(one[0], chain[0])
    for index, (a, b) in enumerate(zip(one[1], chain[1])):
        if index % 3 == 2:
            assert torch.equal(a, b) and int(a.flatten()[0]) == tokens
        else:
            _close(a[:, :tokens].float(), b[:, :tokens].float())
            assert (a[:, tokens:] == 7).all()   # rows past the prompt are the caller's


@pytest.mark.parametrize("overrides", [
    dict(hidden=576, heads=9, kv_heads=3, intermediate=1536),        # features that are no multiple of a tile
    dict(hidden=2048, heads=8, kv_heads=8, head_dim=256, layers=1),   # the widest rows a thread per vector takes
    dict(vocab=1030, head_dim=128, heads=3, kv_heads=1),
    dict(intermediate=8192, layers=1),                                # slices of a long reduction
], ids=lambda o: ",".join(f"{k}={v}" for k, v in o.items()))
@pytest.mark.parametrize("tokens", [19, 150])
def test_shapes(monkeypatch, overrides, tokens):
    (one, chain), _ = _both(monkeypatch, models.get_spec("tiny-llama", **overrides), 1, tokens, q_scale=0.71)
    assert one[2] == 1 < chain[2]
    _close(one[0], chain[0])


@pytest.mark.parametrize("name,overrides,tokens", [
    ("tiny-llama", {}, 641),                    # more tokens than one launch pays for
    ("tiny-llama", dict(hidden=1024, intermediate=8192, layers=1), 161),   # 26 M weights a layer: 160 tokens
    ("tiny-llama", dict(hidden=264), 19),       # a reduction that is no multiple of 64
    ("tiny-llama", dict(intermediate=520), 19),
    ("tiny-llama", dict(vocab=513), 19),        # logit rows that start at odd addresses
    ("tiny-llama", dict(layers=31), 19),        # more layers than one launch has parameters for
    ("tiny-llama", dict(hidden=2112), 19),      # rows wider than 256 vectors
])
def test_other_plans_keep_their_launches(monkeypatch, name, overrides, tokens):
    (one, chain), phases = _both(monkeypatch, models.get_spec(name, **overrides), 1, tokens)
    assert one[2] == chain[2] >= phases
    assert torch.equal(one[0], chain[0])


def test_rebind_and_replay(monkeypatch):
    """A captured launch keeps the weights it was captured with; a plan follows its latest binding."""
    monkeypatch.setenv(SWITCH, "1")
    spec = models.get_spec("tiny-llama")
    layout = plan_prefill(models.direct_prefill_program(spec, 1, 24))
    ids = torch.arange(24, device="cuda")[None] % spec.vocab
    args = [models.direct_prefill_arguments(spec, {k: v.cuda() for k, v in models.init_weights(spec, seed).items()},
                                            models.inv_freq_buffer(spec).cuda(), ids) for seed in (1, 2)]
    bound = BoundDecoder(layout, args[0])
    expect = [bound(*a).clone() for a in args]
    assert not torch.equal(*expect)
    bound(*args[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = bound(*args[0])
    assert torch.equal(bound(*args[1]), expect[1])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, expect[0])
    bound.check()
