"""Decode attention with one context cut into 1 to 32 parts: the fold takes up to eight parts a thread, and
four threads an output from nine on.

Against the same attention in 64 bits.  A score is rounded to bf16 once (2^-9 of a score of deviation 8 before
the scale 1/8: 0.2 % of its probability), a probability once (2^-9) and the result once (2^-9); over
thousands of keys of random sign these errors stay relative to the sum: about 0.3 % together, taken
three times.
"""

import pytest
import torch

from megabake_b200 import planner as pl
from megabake_b200 import runtime as rt
from oracle import decoder_oracle as oracle
from tests.helpers import PhaseRunner
from tests.test_gpu_bodies import _attention_case

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]


@pytest.mark.parametrize("heads,dim", [(7, 64), (8, 256)])
@pytest.mark.parametrize("parts", [1, 2, 7, 8, 9, 16, 17, 32])
def test_parts_meet_in_the_fold(heads, dim, parts):
    cached = 32000   # long enough that one pair is cut into as many parts as it may be, and 32 into more than 16
    batch, kv_heads, capacity = 1, 1, cached + 2
    q, k, v, kc, vc, inv_freq, pos, length = _attention_case(batch, heads, kv_heads, dim, cached, capacity, seed=parts)
    cos, sin = oracle.rotary_tables(inv_freq, pos, 1.0)
    q_r = oracle.apply_rope(q.view(batch, 1, heads, dim), cos, sin).view(heads, dim).double()
    k_r = oracle.apply_rope(k.view(batch, 1, kv_heads, dim), cos, sin).view(1, dim).double()
    keys = torch.cat([kc[0, :cached, 0].double(), k_r])
    values = torch.cat([vc[0, :cached, 0].double(), v.view(1, dim).double()])
    ref = torch.softmax(q_r @ keys.T * dim ** -0.5, dim=1) @ values

    dev = [t.cuda() for t in (q, k, v, kc, vc, inv_freq, pos, length)]
    qd, kd, vd, kcd, vcd, invd, posd, lend = dev
    out = torch.zeros(batch, heads * dim, dtype=torch.bfloat16, device="cuda")
    max_chunks = 2 * parts   # a context is cut into at most half as many
    partial = torch.zeros(batch * max_chunks * heads * (dim + 2), dtype=torch.float32, device="cuda")
    counters = torch.zeros(4, dtype=torch.int32, device="cuda")
    runner = PhaseRunner()
    ph = rt.Phase.blank(rt.BODY_ATTN_DECODE, rt.FLAG_BARRIER | rt.FLAG_BUMP_LENGTH)
    ph.i[rt.AT_I_BATCH], ph.i[rt.AT_I_HEADS], ph.i[rt.AT_I_KV_HEADS] = batch, heads, kv_heads
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
    rel = float((out.cpu().double().view(heads, dim) - ref).norm() / ref.norm())
    assert rel < 0.01, rel
    # cells of this many parts carry the launch's number, and no others
    tags = partial.view(torch.int32).view(-1, heads, dim + 2, 2)[:, 0, 0, 1] if parts > 1 else torch.zeros(1)
    count = int((tags != 0).sum())
    assert count == (parts if parts > 1 else 0) or parts == 32 and 16 < count <= 32
