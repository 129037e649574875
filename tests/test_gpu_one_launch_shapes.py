"""Short prompts as one launch against the oracle: several attention units a CTA, logits in units of more than 128
features, biases of every projection that may have one.  What each shape reaches is asserted, from the host's
planning, in ``test_one_launch_rule.py``."""

from dataclasses import replace

import pytest
import torch

from megabake_b200 import models
from megabake_b200.engine import BoundDecoder
from megabake_b200.planner import plan_prefill
from oracle import decoder_oracle as oracle
from oracle.adapters import oracle_config, oracle_weights
from tests.helpers import ONE_LAUNCH_SHAPES, cosine, logits_close

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

SWITCH = "MEGABAKE_B200_PREFILL_ONE_LAUNCH"


def _run(monkeypatch, layout, args, switch):
    monkeypatch.setenv(SWITCH, switch)
    bound = BoundDecoder(layout, args)
    logits = bound(*args)
    bound.check()
    assert (bound.plan.launches == 1) == (switch == "1")
    return logits


@pytest.mark.parametrize("key", ONE_LAUNCH_SHAPES)
def test_every_position_matches_the_oracle(monkeypatch, key):
    overrides, batch, tokens, _ = ONE_LAUNCH_SHAPES[key]
    spec = models.get_spec(overrides.get("name", "tiny-llama"),
                           **{k: v for k, v in overrides.items() if k != "name"})
    weights, inv_freq = models.init_weights(spec, 3), models.inv_freq_buffer(spec)
    ids = torch.randint(0, spec.vocab, (batch, tokens), generator=torch.Generator().manual_seed(tokens))
    args = models.direct_prefill_arguments(spec, {k: v.cuda() for k, v in weights.items()}, inv_freq.cuda(),
                                           ids.cuda())
    layout = plan_prefill(models.direct_prefill_program(spec, batch, tokens))
    logits = _run(monkeypatch, layout, args, "1").cpu()
    reference = oracle.prefill(oracle_config(spec), oracle_weights(weights, inv_freq), ids)
    ok, worst = logits_close(logits, reference)   # the bar of the whole-model tests
    assert ok, worst
    for b in range(batch):
        for t in range(tokens):
            assert cosine(logits[b, t], reference[b, t]) > 0.9999


@pytest.mark.parametrize("tokens,vocab", [(1, 512), (19, 50000), (150, 512)])
def test_biases_of_o_down_and_head(monkeypatch, tokens, vocab):
    """Against a forward in 64 bits of the same weights: a two-layer model rounds a value to bf16 about 20 times,
    2^-9 sqrt(20) ~ 0.9 %, taken twice."""
    spec = models.get_spec("tiny-llama", vocab=vocab)
    g = torch.Generator().manual_seed(tokens)
    weights = models.init_weights(spec, 3)
    inv_freq = models.inv_freq_buffer(spec)
    ids = torch.randint(0, spec.vocab, (1, tokens), generator=g)
    program = models.direct_prefill_program(spec, 1, tokens)
    args = models.direct_prefill_arguments(spec, {k: v.cuda() for k, v in weights.items()}, inv_freq.cuda(),
                                           ids.cuda())
    biases = {}

    def bias(name, size):
        biases[name] = (0.2 * torch.randn(size, generator=g)).to(torch.bfloat16)
        args.append(biases[name].cuda())
        return len(args) - 1

    layers = tuple(replace(layer, o_bias=bias(f"o{i}", spec.hidden), down_bias=bias(f"down{i}", spec.hidden))
                   for i, layer in enumerate(program.layers))
    program = replace(program, layers=layers, lm_head_bias=bias("head", spec.vocab))
    logits = _run(monkeypatch, plan_prefill(program), args, "1").cpu().double()[0]

    w = {k: v.double() for k, v in weights.items()}
    b = {k: v.double() for k, v in biases.items()}
    dim, heads, group = spec.head_dim, spec.heads, spec.heads // spec.kv_heads
    angle = torch.arange(tokens).double()[:, None] * inv_freq.double()[None]
    cos, sin = angle.cos().repeat(1, 2), angle.sin().repeat(1, 2)
    turn = lambda t: t * cos + torch.cat([-t[..., dim // 2:], t[..., :dim // 2]], -1) * sin
    norm = lambda t, name: t * torch.rsqrt((t * t).mean(-1, keepdim=True) + spec.eps) * w[name]
    x = w["model.embed_tokens.weight"][ids[0]]
    for i in range(spec.layers):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        q, k, v = ((h @ w[p + f"self_attn.{n}_proj.weight"].T).view(tokens, -1, dim).transpose(0, 1) for n in "qkv")
        k, v = turn(k).repeat_interleave(group, 0), v.repeat_interleave(group, 0)
        scores = turn(q) @ k.transpose(1, 2) * dim ** -0.5
        scores += torch.full((tokens, tokens), float("-inf"), dtype=torch.float64).triu(1)
        a = (torch.softmax(scores, -1) @ v).transpose(0, 1).reshape(tokens, heads * dim)
        x = x + a @ w[p + "self_attn.o_proj.weight"].T + b[f"o{i}"]
        h = norm(x, p + "post_attention_layernorm.weight")
        gate = torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T)
        x = x + (gate * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T + b[f"down{i}"]
    ref = norm(x, "model.norm.weight") @ w["model.embed_tokens.weight"].T + b["head"]
    rel = ((logits - ref).norm(dim=-1) / ref.norm(dim=-1)).max()
    assert float(rel) < 0.018, float(rel)


def test_a_poisoned_prompt_stays_in_its_row(monkeypatch):
    """Three prompts in one launch, a NaN in the middle one's token 5: the others keep their bits, and every later
    position of the middle one is NaN.  (Positions before it may be: a masked probability of zero times NaN.)"""
    spec = models.get_spec("tiny-llama")
    weights = {k: v.cuda() for k, v in models.init_weights(spec, 3).items()}
    ids = torch.randint(0, spec.vocab - 1, (3, 37), generator=torch.Generator().manual_seed(1)).cuda()
    layout = plan_prefill(models.direct_prefill_program(spec, 3, 37))
    for switch in ("1", "0"):
        args = models.direct_prefill_arguments(spec, weights, models.inv_freq_buffer(spec).cuda(), ids)
        clean = _run(monkeypatch, layout, args, switch)
        for poison in (float("nan"), float("inf")):
            bad = dict(weights)
            bad["model.embed_tokens.weight"] = weights["model.embed_tokens.weight"].clone()
            bad["model.embed_tokens.weight"][spec.vocab - 1, 7] = poison
            poisoned = ids.clone()
            poisoned[1, 5] = spec.vocab - 1
            args = models.direct_prefill_arguments(spec, bad, models.inv_freq_buffer(spec).cuda(), poisoned)
            logits = _run(monkeypatch, layout, args, switch)
            keep = slice(0, spec.vocab - 1)   # the head shares the poisoned row
            assert torch.equal(logits[0, :, keep], clean[0, :, keep])
            assert torch.equal(logits[2, :, keep], clean[2, :, keep])
            assert torch.isnan(logits[1, 5:]).all()
