"""Which prompts run as one launch and how their projections are cut, from the host's own planning (no device).

The second half says what the shapes of ``test_gpu_one_launch_shapes.py`` reach in the kernel, so that another cost
model cannot take them off it unnoticed.
"""

import pytest

from megabake_b200 import models
from megabake_b200 import runtime as rt
from megabake_b200.planner import plan_prefill
from tests.helpers import ONE_LAUNCH_SHAPES

SMS = 148


def _cuts(spec, batch, tokens):
    return rt.prefill_cuts(plan_prefill(models.direct_prefill_program(spec, batch, tokens)).phases, 3, SMS)


def _weights(spec):
    q, kv = spec.heads * spec.head_dim, spec.kv_heads * spec.head_dim
    return spec.hidden * (2 * q + 2 * kv + 3 * spec.intermediate)


def _most_tokens(spec):
    low, high = 1, 1025
    while high - low > 1:
        middle = (low + high) // 2
        low, high = (middle, high) if _cuts(spec, 1, middle)[0] else (low, middle)
    return low


# layers between the presets: (hidden, heads, kv_heads, head_dim, intermediate)
LAYERS = [(256, 4, 2, 64, 512), (512, 8, 2, 64, 1152), (576, 9, 3, 64, 1536), (640, 10, 2, 64, 1600),
          (640, 10, 2, 64, 2560), (768, 6, 2, 128, 2560), (768, 12, 12, 64, 3072), (1024, 8, 2, 128, 3072),
          (896, 14, 2, 64, 4864), (1024, 16, 8, 64, 4096), (1024, 16, 4, 64, 5632), (1280, 20, 20, 64, 4352),
          (1536, 12, 2, 128, 8960), (2048, 32, 8, 64, 8192), (2048, 32, 8, 64, 9728), (2048, 8, 1, 256, 16384),
          (2048, 32, 8, 64, 32768)]


def test_the_limit_falls_with_the_weights_of_a_layer_and_without_steps():
    found = []
    for hidden, heads, kv_heads, head_dim, intermediate in LAYERS:
        spec = models.get_spec("tiny-llama", hidden=hidden, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                               intermediate=intermediate, layers=1)
        found.append((_weights(spec), _most_tokens(spec)))
    assert found == sorted(found, key=lambda x: (x[0], -x[1]))
    assert found[0][1] == 640 and found[-1][1] == 128
    limits = [limit for _, limit in found]
    assert limits == sorted(limits, reverse=True)
    # 5 % more weights take at most 15 % off the limit, between any two points of the table as well
    for intermediate in range(512, 12288, 128):
        pair = [models.get_spec("tiny-llama", hidden=1024, heads=8, kv_heads=2, intermediate=i, layers=1)
                for i in (intermediate, intermediate + 64)]
        if _weights(pair[1]) < 1.05 * _weights(pair[0]):
            a, b = map(_most_tokens, pair)
            assert b <= a and b >= 0.85 * a, (intermediate, a, b)


@pytest.mark.parametrize("name,batch,tokens,one", [
    ("smollm-135m", 1, 512, True), ("smollm-135m", 16, 32, True), ("smollm-135m", 1, 640, False),
    ("qwen2-0.5b", 1, 384, True), ("qwen2-0.5b", 4, 333, False), ("llama-3.2-1b", 1, 160, True),
    ("llama-3.2-1b", 1, 176, False), ("gemma-2b", 1, 128, True), ("gemma-2b", 1, 144, False),
])
def test_presets(name, batch, tokens, one):
    assert (_cuts(models.get_spec(name), batch, tokens)[0] > 0) == one


def test_many_heads_keep_their_launches():
    """Three waves of attention units over five blocks of keys."""
    spec = models.get_spec("tiny-llama", heads=16, kv_heads=16)
    assert _cuts(spec, 1, 576)[0] and not _cuts(spec, 1, 608)[0]


def test_bad_arguments_are_refused():
    phases = plan_prefill(models.direct_prefill_program(models.get_spec("tiny-llama"), 1, 19)).phases
    with pytest.raises(Exception):
        rt.prefill_cuts(phases, 3, 0)
    with pytest.raises(Exception):
        rt.prefill_cuts([], 3, SMS)


@pytest.mark.parametrize("key", ONE_LAUNCH_SHAPES)
def test_shapes_reach_what_they_are_for(key):
    overrides, batch, tokens, reach = ONE_LAUNCH_SHAPES[key]
    name = overrides.get("name", "tiny-llama")
    spec = models.get_spec(name, **{k: v for k, v in overrides.items() if k != "name"})
    form, cuts = _cuts(spec, batch, tokens)
    units = batch * spec.heads * ((tokens + 31) // 32)
    assert form == reach["form"]
    if "attention" in reach:   # some CTA has more than one unit, and o's units start past the last whole wave
        assert units > SMS and cuts[1].first_cta == units % SMS != 0
    if "logits" in reach:      # two accumulators of an unpaired product, several units a CTA
        assert cuts[4].accumulators == 2 and cuts[4].features > 128 and cuts[4].units > SMS
