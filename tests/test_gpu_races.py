"""Race, reuse and wait-limit evidence that needs no sanitizer.

* Poisoned workspace: every byte of the plan's workspace and the logits buffer are filled with 0xE5
  before a launch; the results must not change (the reference poisons its workspace the same way,
  ``src/megabake/compiler.py:1972-1973``, ``tests/gpu/test_task29_transformer_block.py:116-124``).
  Short contexts, and contexts that are cut over several CTAs.
* Distinct buffers: the same model planned with activation buffers of its own for every layer
  against the normal plan that reuses one set: bit-identical logits and KV state (reference
  ``src/megabake/compiler.py:227-241``).  A phase that read a buffer too early or wrote it too
  late shows up as a difference.  (In plans that hand over through the workspace; in the relay arena
  no place is used twice in a launch.)
* Wait limit: a consumer whose producer never stores (a flag nothing sets) gives up after the
  plan's limit, the kernel RETURNS ``MB_ST_HANDOFF_TIMEOUT`` through the status word, the context
  stays usable and the next plan runs.
"""

import math
import time

import pytest
import torch

from megabake_b200 import models
from megabake_b200 import runtime as rt
from megabake_b200.engine import BoundDecoder
from megabake_b200.planner import PlannerOptions, attention_scratch_bytes, plan_decode
from tests.helpers import PhaseRunner
from tests.test_gpu_bodies import _bf16, _gemv_phase, _ref_linear

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


def _decoder(name, batch, capacity, options, seed=3):
    spec = models.get_spec(name)
    weights = {k: v.cuda() for k, v in models.init_weights(spec, seed).items()}
    state = models.make_state(spec, batch, capacity, "cuda")
    ids = torch.zeros(batch, 1, dtype=torch.int64, device="cuda")
    pos = torch.zeros(batch, 1, dtype=torch.int64, device="cuda")
    args = models.direct_arguments(spec, weights, models.inv_freq_buffer(spec).cuda(), ids, pos,
                                   state)
    layout = plan_decode(models.direct_program(spec, batch, capacity), options)
    return spec, BoundDecoder(layout, args), args, ids, pos, state


def _fill_caches(spec, state, cached, seed=9):
    """``cached`` random keys and values in every row."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    for layer in range(spec.layers):
        for cache in state[3 * layer: 3 * layer + 2]:
            cache[:, :cached].normal_(0.0, 0.3, generator=g)
        state[3 * layer + 2].fill_(cached)


def _run_steps(decoder, args, ids, pos, tokens, poison=None, first=0):
    outputs = []
    for step in range(tokens.shape[1]):
        ids.copy_(tokens[:, step:step + 1])
        pos.fill_(first + step)
        if poison is not None:
            poison(decoder)
        logits = torch.empty(decoder.program.batch, 1, decoder.program.vocab, dtype=torch.bfloat16,
                             device="cuda")
        if poison is not None:
            logits.view(torch.uint8).fill_(0xE5)
        decoder.launch_into(ids, pos, logits)
        decoder.check()
        outputs.append(logits.clone())
    return outputs


# Hand-offs through the relay arena (the default), through plain tensors behind counters with q, k and
# v as cells or plain too, and everything as cells: only the last three work in the workspace.
HAND_OFFS = {
    "relay": {},
    "plain": {"relay": False},
    "all-plain": {"relay": False, "qkv_cells": False},
    "cells": {"relay": False, "cell_limit": 1 << 20},
}


@pytest.mark.parametrize("hand_offs", HAND_OFFS)
@pytest.mark.parametrize("name,batch,cached", [
    ("tiny-llama", 3, 0), ("tiny-qwen2", 8, 0), ("tiny-gemma", 2, 0), ("tiny-qwen2", 4, 300),
])
def test_poisoned_workspace_changes_nothing(name, batch, cached, hand_offs):
    options = PlannerOptions(**HAND_OFFS[hand_offs])
    spec, clean, args, ids, pos, state = _decoder(name, batch, cached + 16, options)
    tokens = torch.randint(0, spec.vocab, (batch, 5), generator=torch.Generator().manual_seed(2)).cuda()
    _fill_caches(spec, state, cached)
    expected = _run_steps(clean, args, ids, pos, tokens, first=cached)
    expected_state = [t.clone() for t in state]
    spec, dirty, args, ids, pos, state = _decoder(name, batch, cached + 16, options)
    _fill_caches(spec, state, cached)
    # cells and partials start zeroed; later on their sequence numbers decide, so poison is harmless
    assert dirty.layout.zero_ranges

    got = _run_steps(dirty, args, ids, pos, tokens, first=cached,
                     poison=lambda decoder: decoder.workspace.fill_(0xE5))
    for a, b in zip(expected, got):
        assert torch.equal(a, b)
    for a, b in zip(expected_state, state):
        assert torch.equal(a, b)


@pytest.mark.parametrize("name,batch,hand_offs", [
    ("tiny-llama", 2, "plain"), ("tiny-qwen2", 8, "all-plain"), ("tiny-mha", 4, "cells"),
    ("tiny-qwen2", 8, "relay"),
])
def test_distinct_buffers_give_identical_results(name, batch, hand_offs):
    shared = _decoder(name, batch, 16, PlannerOptions(**HAND_OFFS[hand_offs]))
    own = _decoder(name, batch, 16, PlannerOptions(**HAND_OFFS[hand_offs], distinct_buffers=True))
    assert own[1].layout.workspace_bytes > shared[1].layout.workspace_bytes
    spec = shared[0]
    tokens = torch.randint(0, spec.vocab, (batch, 6), generator=torch.Generator().manual_seed(4)).cuda()
    a = _run_steps(*shared[1:5], tokens)
    b = _run_steps(*own[1:5], tokens)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    for x, y in zip(shared[5], own[5]):
        assert torch.equal(x, y)


def _split_context(decoder_parts, seed):
    """Puts 300 cached keys into the state: contexts that are cut over several CTAs."""
    spec, decoder, args, ids, pos, state = decoder_parts
    _fill_caches(spec, state, 300, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    tokens = torch.randint(0, spec.vocab, (decoder.program.batch, 3), generator=g, device="cuda")
    outputs = []
    for step in range(3):
        ids.copy_(tokens[:, step:step + 1])
        pos.fill_(300 + step)
        outputs.append(decoder(*args).clone())
        decoder.check()
    return outputs + [t.clone() for t in state]


def test_a_workspace_of_a_plan_of_the_same_shape(monkeypatch):
    """A second decoder in the bytes the first one left: its launches wait for the very tags the first
    one's partials carry, so none of them may still be there."""
    clean = _split_context(_decoder("tiny-llama", 2, 320, PlannerOptions(), seed=5), seed=7)
    first = _decoder("tiny-llama", 2, 320, PlannerOptions(), seed=4)
    _split_context(first, seed=6)
    left = first[1].workspace.clone()
    partials, = [s for s in first[1].layout.slots if s.name == "attention_partials"]
    assert int(left[partials.offset:].view(torch.int32).count_nonzero()) > 0    # contexts were cut
    empty = torch.empty
    with monkeypatch.context() as m:
        m.setattr(torch, "empty", lambda *a, **k: left.clone() if k.get("dtype") == torch.uint8
                  else empty(*a, **k))
        second = _decoder("tiny-llama", 2, 320, PlannerOptions(), seed=5)
    phase = next(p for p in second[1].layout.phases if p.body == rt.BODY_ATTN_DECODE)
    size = 2 * second[0].heads * phase.i[rt.AT_I_MAX_CHUNKS] * (second[0].head_dim + 2) * 4
    assert int(second[1].workspace[partials.offset: partials.offset + size].count_nonzero()) == 0
    for a, b in zip(clean, _split_context(second, seed=7)):
        assert torch.equal(a, b)


def test_binding_clears_partials_of_another_owner():
    """The same through the C interface: a buffer that is new to the plan is cleared by the bind, one
    that it already works in is left alone."""
    from tests.test_gpu_bodies import _attention_case

    batch, heads, kv_heads, dim, cached, capacity = 1, 4, 2, 64, 300, 320
    dev = [t.cuda() for t in _attention_case(batch, heads, kv_heads, dim, cached, capacity)]
    out = torch.zeros(batch, heads * dim, dtype=torch.bfloat16, device="cuda")
    chunks = 20
    partial = torch.full((batch * heads * chunks * (dim + 2),), 1.0, device="cuda")
    phase = rt.Phase.blank(rt.BODY_ATTN_DECODE, 0)
    for i, value in ((rt.AT_I_BATCH, batch), (rt.AT_I_HEADS, heads), (rt.AT_I_KV_HEADS, kv_heads),
                     (rt.AT_I_HEAD_DIM, dim), (rt.AT_I_CAPACITY, capacity),
                     (rt.AT_I_INVFREQ_BF16, 1), (rt.AT_I_MAX_CHUNKS, chunks), (rt.AT_I_MERGE_SLOTS, 8),
                     (rt.AT_I_EXACT_KEYS, 128)):
        phase.i[i] = value
    phase.f[rt.AT_F_SCALE] = dim ** -0.5
    phase.f[rt.AT_F_ROPE_SCALE] = 1.0
    q, k, v, kc, vc, inv_freq, pos, length = dev
    tensors = [q, k, v, kc, vc, length, pos, inv_freq, out, partial,
               torch.zeros(4, dtype=torch.int32, device="cuda")]
    for index in range(len(tensors)):
        phase.slot[index] = index
    scratch = (attention_scratch_bytes(dim, heads // kv_heads, 8) + 127) // 128 * 128
    plan = rt.Plan([phase], n_slots=len(tensors), n_dynamic=0, activation_bytes=scratch, device=0)
    plan.bind([t.data_ptr() for t in tensors])
    torch.cuda.synchronize()
    assert int(partial.count_nonzero()) == 0
    partial.fill_(2.0)
    plan.bind([t.data_ptr() for t in tensors])
    torch.cuda.synchronize()
    assert bool((partial == 2.0).all())


def test_tensor_maps_follow_every_bind():
    """The tensor maps live in device memory that a bind rewrites, and that a new plan may get from a
    destroyed one: every launch reads the weights and caches of the latest bind."""
    rows, k, n = 3, 576, 1536
    x = _bf16(rows, k, seed=1)
    weights = [_bf16(n, k, scale=k ** -0.5, seed=10 + i) for i in range(3)]
    expected = [_ref_linear(x, w) for w in weights]
    out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    plan = None
    for step in range(12):
        which = step % 3
        runner = PhaseRunner()
        phase = _gemv_phase(runner, x=x, segs=[(weights[which], None, out)], k=k, rows=rows)
        out.zero_()
        if plan is None or step % 4 == 0:
            plan = None     # destroyed here: the next one may work at its addresses
            plan = runner.run([phase], (rows + 1) * (k + 32) * 2)
        else:
            plan.bind([t.data_ptr() for t in runner.tensors])
            plan.launch([], torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        assert plan.status().code == 0
        assert (out != expected[which]).float().mean() < 0.02, step
        assert float((out.float() - expected[which].float()).abs().max()) <= 0.06


def test_a_plain_residual_is_read_after_the_wait():
    """CTA 0 gathers and stores 8 x 8192 rows in phase 0 while the other CTAs, which own no output row of
    it, are long through to phase 2, where these rows are the residual: plain memory, ordered by
    nothing but the wait for phase 1."""
    rows, k, n = 8, 8192, 8192
    table, ids = _bf16(16, k, seed=1), torch.arange(3, 3 + rows, dtype=torch.int64, device="cuda")
    w0, other = _bf16(2, k, scale=k ** -0.5, seed=2), _bf16(rows, 64, seed=3)
    w1, w2 = _bf16(64, 64, scale=0.125, seed=4), _bf16(n, 64, scale=0.125, seed=5)
    stored = torch.zeros(rows, k, dtype=torch.bfloat16, device="cuda")
    o0, o1, out = (torch.zeros(rows, m, dtype=torch.bfloat16, device="cuda") for m in (2, 64, n))
    runner = PhaseRunner()
    gather = _gemv_phase(runner, x=table, segs=[(w0, None, o0)], k=k, rows=rows)
    gather.flags |= rt.FLAG_FENCE
    gather.i[rt.GV_I_GATHER], gather.i[rt.GV_I_VOCAB], gather.i[rt.GV_I_STORE_X] = 1, 16, 1
    gather.slot[rt.GV_S_IDS] = runner.slot("ids", ids)
    gather.slot[rt.GV_S_XSTORE] = runner.slot("stored", stored)
    runner.names = {}
    between = _gemv_phase(runner, x=other, segs=[(w1, None, o1)], k=64, rows=rows)
    between.flags |= rt.FLAG_FENCE
    runner.names = {}
    last = _gemv_phase(runner, x=o1, segs=[(w2, None, out)], k=64, rows=rows, residual=stored,
                       epilogue=rt.EPI_RESIDUAL)
    last.i[rt.GV_I_CELLS], last.i[rt.GV_I_X_SOURCE] = rt.CELLS_X_WAIT, 1
    plan = runner.run([gather, between, last], (rows + 1) * (k + 32) * 2)
    y = _ref_linear(other, w1)
    expected = table[ids] + _ref_linear(y, w2)
    for _ in range(5):
        assert plan.status().code == 0
        assert torch.equal(stored, table[ids])
        assert float((out.float() - expected.float()).abs().max()) <= 0.05
        for t in (stored, o1, out):
            t.zero_()
        plan.launch([], torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()


@pytest.mark.parametrize("name,batch", [("tiny-llama", 1), ("tiny-qwen2", 8), ("tiny-gemma256", 2)])
@pytest.mark.parametrize("qkv_cells,cell_limit", [(True, 0), (False, 0), (True, 1 << 20), (False, 2048)])
def test_hand_offs_through_the_workspace_give_the_same_results(name, batch, qkv_cells, cell_limit):
    """Plain tensors behind fenced counters, flagged cells and mixes of the two against the relay arena:
    the arithmetic is the same, so are the bits.  One short row: most CTAs have no attention to do."""
    relayed = _decoder(name, batch, 24, PlannerOptions())
    plain = _decoder(name, batch, 24, PlannerOptions(relay=False, qkv_cells=qkv_cells,
                                                     cell_limit=cell_limit))
    assert any(p.flags & rt.FLAG_RELAY for p in relayed[1].layout.phases)
    assert not any(p.flags & rt.FLAG_RELAY for p in plain[1].layout.phases)
    spec = relayed[0]
    tokens = torch.randint(0, spec.vocab, (batch, 20), generator=torch.Generator().manual_seed(4)).cuda()
    for a, b in zip(_run_steps(*relayed[1:5], tokens), _run_steps(*plain[1:5], tokens)):
        assert torch.equal(a, b)
    for a, b in zip(relayed[5], plain[5]):
        assert torch.equal(a, b)


def test_weights_of_a_captured_launch_stay_its_own():
    """Weights and caches given per launch are read through tensor maps made for that launch.  A captured
    launch replays with its own, whatever later launches of the plan were given."""
    from tests.test_gpu_bodies import _attention_case

    rows, k, n, heads, kv_heads, dim, cached, capacity = 2, 256, 512, 4, 2, 64, 200, 220
    x = _bf16(rows, k, seed=1)
    weights = [_bf16(n, k, scale=k ** -0.5, seed=10 + i) for i in range(3)]
    q, key, value, kc, vc, inv_freq, pos, length = (
        t.cuda() for t in _attention_case(rows, heads, kv_heads, dim, cached, capacity))
    caches = [(kc, vc), (kc.flip(1).contiguous(), vc.flip(1).contiguous()), (kc * 0.5, vc * 2)]
    linear = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    mixed = torch.zeros(rows, heads * dim, dtype=torch.bfloat16, device="cuda")
    chunks = math.ceil(capacity / 16)
    runner = PhaseRunner()
    for name, tensor in (("w0", weights[0]), ("kc", kc), ("vc", vc)):
        runner.slot(name, tensor)                       # slots 0 .. 2 come with the launch
    gemv = _gemv_phase(runner, x=x, segs=[(weights[0], None, linear)], k=k, rows=rows)
    attention = rt.Phase.blank(rt.BODY_ATTN_DECODE, 0)  # (the lengths stay: every launch sees the same keys)
    for i, v in ((rt.AT_I_BATCH, rows), (rt.AT_I_HEADS, heads), (rt.AT_I_KV_HEADS, kv_heads),
                 (rt.AT_I_HEAD_DIM, dim), (rt.AT_I_CAPACITY, capacity), (rt.AT_I_INVFREQ_BF16, 1),
                 (rt.AT_I_MAX_CHUNKS, chunks), (rt.AT_I_MERGE_SLOTS, 8), (rt.AT_I_EXACT_KEYS, 128)):
        attention.i[i] = v
    attention.f[rt.AT_F_SCALE], attention.f[rt.AT_F_ROPE_SCALE] = dim ** -0.5, 1.0
    for index, (name, tensor) in enumerate([
        ("q", q), ("k", key), ("v", value), ("kc", kc), ("vc", vc), ("len", length), ("pos", pos),
        ("invf", inv_freq), ("out", mixed),
        ("partial", torch.zeros(rows * heads * chunks * (dim + 2), device="cuda")),
        ("cnt", torch.zeros(8, dtype=torch.int32, device="cuda")),
    ]):
        attention.slot[index] = runner.slot(name, tensor)
    scratch = max((rows + 1) * (k + 32) * 2, attention_scratch_bytes(dim, heads // kv_heads, 8))
    plan = rt.Plan([gemv, attention], n_slots=len(runner.tensors), n_dynamic=3,
                   activation_bytes=(scratch + 127) // 128 * 128, device=0)
    plan.bind([t.data_ptr() for t in runner.tensors])

    def launch(which):
        plan.launch([weights[which].data_ptr(), *(t.data_ptr() for t in caches[which])],
                    torch.cuda.current_stream().cuda_stream)

    def results(run):
        linear.zero_(), mixed.zero_()
        run()
        torch.cuda.synchronize()
        assert plan.status().code == 0
        return linear.clone(), mixed.clone()

    alone = [results(lambda: launch(which)) for which in range(3)]
    for which, (product, _) in enumerate(alone):
        assert (product != _ref_linear(x, weights[which])).float().mean() < 0.02
    assert not torch.equal(alone[0][1], alone[1][1])
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        launch(0)
        launch(1)
    for which in (2, 1, 0):
        for a, b in zip(results(lambda: launch(which)), alone[which]):
            assert torch.equal(a, b)
        for a, b in zip(results(graph.replay), alone[1]):
            assert torch.equal(a, b)


def test_a_wait_that_runs_out_returns_a_status():
    """Phase 1 polls cells that phase 0 (a no-op) never writes.  With a 40 ms limit the kernel
    must come back by itself with MB_ST_HANDOFF_TIMEOUT; afterwards another plan runs normally."""
    rows, k, n = 2, 256, 512
    x_cells = torch.zeros(rows * k // 2, dtype=torch.int64, device="cuda")   # sequence numbers: 0
    w = _bf16(n, k, scale=0.05, seed=2)
    out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    runner = PhaseRunner()
    nop = rt.Phase.blank(rt.BODY_NOP, 0)
    phase = _gemv_phase(runner, x=x_cells, segs=[(w, None, out)], k=k, rows=rows)
    phase.i[rt.GV_I_CELLS] = rt.CELLS_X
    phase.i[rt.GV_I_X_SOURCE] = 0
    started = time.perf_counter()
    plan = runner.run([nop, phase], rows * (k + 32) * 2, wait_limit_ms=40)
    elapsed = time.perf_counter() - started
    status = plan.status()
    assert status.code == 7 and status.phase == 1        # MB_ST_HANDOFF_TIMEOUT in the GEMV phase
    assert status.calls == 0                              # the launch did not complete
    assert elapsed < 5.0
    plan.reset()
    assert plan.status().code == 0
    # the context is healthy: an ordinary plan computes the right thing
    x = _bf16(rows, k, seed=1)
    good = PhaseRunner()
    plan = good.run([_gemv_phase(good, x=x, segs=[(w, None, out)], k=k, rows=rows)],
                    rows * (k + 32) * 2)
    assert plan.status().code == 0
    ref = _ref_linear(x, w)
    assert (out != ref).float().mean() < 0.05


def test_a_fault_ends_the_walk_through_the_phases():
    """Every CTA's wait in phase 1 runs out; it leaves the launch at the end of phase 2 at the latest, so
    the phases behind never run and their outputs stay as they were.  Then the plan runs again."""
    rows, k, n = 2, 256, 512
    x_cells = torch.zeros(rows * k // 2, dtype=torch.int64, device="cuda")
    x, w = _bf16(rows, k, seed=1), _bf16(n, k, scale=0.05, seed=2)
    runner = PhaseRunner()
    waits = _gemv_phase(runner, x=x_cells, segs=[(w, None, torch.zeros(rows, n, dtype=torch.bfloat16,
                                                                       device="cuda"))], k=k, rows=rows)
    waits.i[rt.GV_I_CELLS], waits.i[rt.GV_I_X_SOURCE] = rt.CELLS_X, 0
    phases, outputs = [rt.Phase.blank(rt.BODY_NOP, 0), waits], []
    for _ in range(6):
        runner.names = {}
        outputs.append(torch.full((rows, n), 7.0, dtype=torch.bfloat16, device="cuda"))
        phases.append(_gemv_phase(runner, x=x, segs=[(w, None, outputs[-1])], k=k, rows=rows))
    phases[4].flags |= rt.FLAG_BARRIER
    plan = runner.run(phases, rows * (k + 32) * 2, wait_limit_ms=40)
    status = plan.status()
    assert status.code == 7 and status.phase == 1 and status.calls == 0
    for out in outputs[1:]:
        assert bool((out == 7.0).all())
    plan.reset()
    # the same records with the wait satisfied: cells of the epoch after the reset
    tag = 1 * len(phases) + 0 + 1
    x_cells.copy_((x.view(torch.int32).to(torch.int64).flatten() & 0xFFFFFFFF) | (tag << 32))
    plan.launch([], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.status().code == 0
    for out in outputs:
        assert (out != _ref_linear(x, w)).float().mean() < 0.05


def test_an_embedding_row_of_all_ones():
    """bf16 0xffff is a NaN, and a pair of them the pattern of a word nobody has written yet: such a row
    gives NaN logits for its batch row, no fault, and leaves the other row alone."""
    spec, decoder, args, ids, pos, state = _decoder("tiny-llama", 2, 8, PlannerOptions())
    table = next(a for a in args if isinstance(a, torch.Tensor) and a.shape == (spec.vocab, spec.hidden))
    ids.copy_(torch.tensor([[3], [5]]))
    clean = decoder(*args).clone()
    decoder.check()
    table[5].view(torch.int16).fill_(-1)
    for layer in range(spec.layers):
        state[3 * layer + 2].zero_()
    got = decoder(*args)
    decoder.check()
    assert bool(got[1].isnan().all())
    changed = torch.tensor([5])                  # the table is the LM head too: only logit 5 of row 0
    keep = torch.ones(spec.vocab, dtype=torch.bool)
    keep[changed] = False
    assert torch.equal(got[0, 0].cpu()[keep], clean[0, 0].cpu()[keep])


def test_a_faulted_launch_leaves_the_state_alone():
    """A token outside the embedding table is recorded in phase 0.  Waits that are still spinning
    see the status and drain; CTAs that get through reach the end of the launch, where the valid
    lengths are advanced only if no fault was recorded: the KV state still describes the step
    before, and after ``check()`` has reset the plan the corrected call runs from there."""
    from megabake_b200 import CompilerError

    spec, decoder, args, ids, pos, state = _decoder("tiny-llama", 2, 8, PlannerOptions())
    ids.fill_(spec.vocab + 5)
    started = time.perf_counter()
    logits = torch.empty(2, 1, spec.vocab, dtype=torch.bfloat16, device="cuda")
    decoder.launch_into(ids, pos, logits)
    with pytest.raises(CompilerError):
        decoder.check()
    assert time.perf_counter() - started < 3.0
    ids.fill_(1)
    decoder.launch_into(ids, pos, logits)                 # recovered by check(): runs again
    decoder.check()
    assert int(state[2]) == 1
