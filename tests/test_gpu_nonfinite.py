"""Infinities and NaNs stay where they belong: in the outputs that attend to them, and in no others."""

import pytest
import torch

from megabake_b200 import planner as pl
from megabake_b200 import runtime as rt
from oracle import decoder_oracle as oracle
from tests.helpers import PhaseRunner
from tests.test_gpu_bodies import _attention_case

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]


@pytest.mark.parametrize("heads,dim", [(7, 64), (8, 256)])
@pytest.mark.parametrize("parts", [1, 5, 8, 9, 11, 13, 16, 17, 31, 32])
def test_infinite_cached_values_reach_the_output_as_infinities(heads, dim, parts):
    """One context cut into up to 32 parts, with infinite values in the last cached key: a sum of finite
    terms and one infinity is that infinity, whichever parts are added up beside it."""
    cached, capacity = 32000, 32002
    q, k, v, kc, vc, inv_freq, pos, length = _attention_case(1, heads, 1, dim, cached, capacity, seed=parts)
    vc[0, cached - 1, 0, 3] = float("inf")
    vc[0, cached - 1, 0, 6] = float("-inf")
    vc[0, cached - 1, 0, 40] = float("nan")
    cos, sin = oracle.rotary_tables(inv_freq, pos, 1.0)
    q_r = oracle.apply_rope(q.view(1, 1, heads, dim), cos, sin).view(heads, dim).double()
    k_r = oracle.apply_rope(k.view(1, 1, 1, dim), cos, sin).view(1, dim).double()
    keys = torch.cat([kc[0, :cached, 0].double(), k_r])
    values = torch.cat([vc[0, :cached, 0].double(), v.view(1, dim).double()])
    ref = torch.softmax(q_r @ keys.T * dim ** -0.5, dim=1) @ values

    qd, kd, vd, kcd, vcd, invd, posd, lend = [t.cuda() for t in (q, k, v, kc, vc, inv_freq, pos, length)]
    out = torch.zeros(1, heads * dim, dtype=torch.bfloat16, device="cuda")
    max_chunks = 2 * parts   # a context is cut into at most half as many
    partial = torch.zeros(max_chunks * heads * (dim + 2), dtype=torch.float32, device="cuda")
    counters = torch.zeros(4, dtype=torch.int32, device="cuda")
    runner = PhaseRunner()
    ph = rt.Phase.blank(rt.BODY_ATTN_DECODE, rt.FLAG_BARRIER | rt.FLAG_BUMP_LENGTH)
    ph.i[rt.AT_I_BATCH], ph.i[rt.AT_I_HEADS], ph.i[rt.AT_I_KV_HEADS] = 1, heads, 1
    ph.i[rt.AT_I_HEAD_DIM], ph.i[rt.AT_I_CAPACITY] = dim, capacity
    ph.i[rt.AT_I_INVFREQ_BF16], ph.i[rt.AT_I_MAX_CHUNKS] = 1, max_chunks
    merge_slots = pl.attention_merge_slots(dim, heads)
    ph.i[rt.AT_I_MERGE_SLOTS] = merge_slots
    ph.f[rt.AT_F_SCALE], ph.f[rt.AT_F_ROPE_SCALE] = dim ** -0.5, 1.0
    for index, (name, tensor) in enumerate([
        ("q", qd), ("k", kd), ("v", vd), ("kc", kcd), ("vc", vcd), ("len", lend), ("pos", posd),
        ("invf", invd), ("out", out), ("partial", partial), ("cnt", counters),
    ]):
        ph.slot[index] = runner.slot(name, tensor)
    plan = runner.run([ph], pl.attention_scratch_bytes(dim, heads, merge_slots))
    assert plan.status().code == 0
    got = out.cpu().double().view(heads, dim)
    finite = torch.ones(dim, dtype=torch.bool)
    finite[[3, 6, 40]] = False
    assert torch.equal(torch.isposinf(got), torch.isposinf(ref)) and torch.equal(torch.isneginf(got), torch.isneginf(ref))
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    # finite outputs: rounded scores, probabilities and results over thousands of keys, as in the test of the fold
    rel = float((got - ref)[:, finite].norm() / ref[:, finite].norm())
    assert rel < 0.01, rel
