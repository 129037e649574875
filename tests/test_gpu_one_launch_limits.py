"""Short prompts as one launch: its limits, its SMs and the tensors it leaves behind."""

from dataclasses import replace

import pytest
import torch

from megabake_b200 import models
from megabake_b200 import runtime as rt
from megabake_b200.diagnostics import CompilerError
from megabake_b200.engine import BoundDecoder
from megabake_b200.planner import plan_prefill

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

SWITCH = "MEGABAKE_B200_PREFILL_ONE_LAUNCH"


def _arguments(spec, tokens, batch=1, seed=1, weights=None):
    if weights is None:
        weights = {k: v.cuda() for k, v in models.init_weights(spec, seed).items()}
    ids = torch.randint(0, spec.vocab, (batch, tokens), generator=torch.Generator().manual_seed(tokens)).cuda()
    return models.direct_prefill_arguments(spec, weights, models.inv_freq_buffer(spec).cuda(), ids)


def test_a_hand_over_that_takes_longer_than_the_limit_ends_the_launch():
    """A gated projection of eight million features and the sum over them keep the device busy for milliseconds, and
    whoever waits for either does so for one (CTAs without work there), or for two (inside their own
    pipeline): the launch ends with a status and leaves the device and the plan usable."""
    spec = models.get_spec("tiny-llama", hidden=64, layers=1, heads=1, kv_heads=1, intermediate=1 << 23, vocab=20000)
    weights = {name: torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
               for name, shape in models.parameter_shapes(spec)}
    args = _arguments(spec, 128, weights=weights)
    layout = plan_prefill(models.direct_prefill_program(spec, 1, 128))
    short = BoundDecoder(layout, args, wait_limit_ms=1)
    assert short.plan.launches == 1
    for _ in range(2):
        short(*args)
        torch.cuda.synchronize()
        assert short.plan.status().code in (2, 7)   # MB_ST_PIPE_TIMEOUT, MB_ST_HANDOFF_TIMEOUT: whose limit was first
        with pytest.raises(CompilerError):
            short.check()                      # and makes it usable again
    patient = BoundDecoder(layout, args)
    assert not patient(*args).any()
    patient.check()


@pytest.mark.parametrize("name,batch,tokens,sms", [
    ("tiny-llama", 1, 24, 72), ("tiny-qwen2", 1, 100, 72), ("tiny-gemma256", 1, 257, 40), ("tiny-mha", 5, 9, 16),
])
def test_fewer_sms_give_the_same_bits(name, batch, tokens, sms):
    """Under a context that has a part of the device's SMs the launch takes that many CTAs."""
    from torch.cuda.green_contexts import GreenContext

    spec = models.get_spec(name)
    args = _arguments(spec, tokens, batch)
    bound = BoundDecoder(plan_prefill(models.direct_prefill_program(spec, batch, tokens)), args)
    assert bound.plan.launches == 1
    expect = bound(*args)
    bound.check()
    part = GreenContext.create(num_sms=sms, device_id=0)
    part.set_context()
    try:
        got = bound(*args)
        bound.check()
    finally:
        part.pop_context()
    assert torch.equal(got, expect)
    assert torch.equal(bound(*args), expect)
    bound.check()


@pytest.mark.parametrize("name,batch,tokens", [("tiny-qwen2", 3, 31), ("tiny-gemma256", 1, 150)])
def test_queries_keys_and_values_are_left_behind(monkeypatch, name, batch, tokens):
    """The tensors that the records name are written, as by the launches of their own: bf16 results of sums in another
    order, a few of them one step (2^-8) apart, and in the last layer of two what that step grew to."""
    spec = models.get_spec(name)
    args = _arguments(spec, tokens, batch)
    layout = plan_prefill(models.direct_prefill_program(spec, batch, tokens))
    names = {"q": spec.heads, "k": spec.kv_heads, "v": spec.kv_heads, "attention": spec.heads}
    left = []
    for switch in ("1", "0"):
        monkeypatch.setenv(SWITCH, switch)
        bound = BoundDecoder(layout, args)
        bound.workspace.fill_(0)
        bound(*args)
        bound.check()
        at = {s.name: s.offset for s in layout.slots if s.kind == "workspace"}
        left.append({n: bound.workspace[at[n]:at[n] + 2 * batch * tokens * heads * spec.head_dim]
                     .view(torch.bfloat16).float() for n, heads in names.items()})
    assert bound.plan.launches > 1
    for n in names:
        one, chain = left[0][n], left[1][n]
        assert chain.any() and float((one - chain).norm() / chain.norm()) < 0.018, n


def test_without_room_for_transposed_values_the_launches_stay(monkeypatch):
    """That record's attention computes with expf and exact division; it is not for the one launch to change that."""
    spec = models.get_spec("tiny-llama")
    args = _arguments(spec, 40)
    layout = plan_prefill(models.direct_prefill_program(spec, 1, 40))
    for phase in layout.phases:
        if phase.body == rt.BODY_ATTN_PREFILL:
            phase.slot[rt.AP_S_VT] = -1
    results = []
    for switch in ("1", "0"):
        monkeypatch.setenv(SWITCH, switch)
        bound = BoundDecoder(layout, args)
        assert bound.plan.launches >= len(layout.phases)
        results.append(bound(*args))
        bound.check()
    assert torch.equal(*results)
