"""Hand-offs inside a decode launch and reductions shared by a cluster, at the sizes where their
tilings can go wrong: one row and eight, reductions of less than one stage and of several slices of
shared memory, outputs that fill no block, tiles with one live row and with one row too many."""

import pytest
import torch

from megabake_b200 import runtime as rt
from oracle import decoder_oracle as oracle
from tests import test_gpu_bodies as decode
from tests import test_gpu_prefill_bodies as prefill
from tests.helpers import PhaseRunner, cosine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 8])
@pytest.mark.parametrize("k,mid,n", [
    (64, 32, 2),            # less than a stage of either shape, one pair of rows in all
    (576, 1536, 576),       # blocks of eight rows
    (896, 4864, 896),       # 20 slots of a slice from five rows on: the wide slices
    (896, 6016, 896),       # more than a wide slice from five rows on: two chunks
    (2048, 8192, 2560),     # blocks of sixteen rows, several per CTA
])
def test_results_handed_over_inside_the_launch(rows, k, mid, n):
    """norm + gated pair -> residual projection: the second phase polls what the first one stores.
    Two launches: each leaves the other half of the arena blank."""
    x = decode._bf16(rows, k, seed=1)
    nw = decode._bf16(k, scale=0.3, seed=2)
    wg, wu = decode._bf16(mid, k, scale=k ** -0.5, seed=3), decode._bf16(mid, k, scale=k ** -0.5, seed=4)
    wd = decode._bf16(n, mid, scale=mid ** -0.5, seed=5)
    base = decode._bf16(rows, n, seed=6)
    glu = torch.zeros(rows, mid, dtype=torch.bfloat16, device="cuda")
    out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    runner = PhaseRunner()
    first = decode._gemv_phase(runner, x=x, segs=[(wg, None, glu)], k=k, rows=rows, pair=wu,
                               prologue=rt.PRO_RMS_LLAMA, norm_w=nw, epilogue=rt.EPI_SILU_MUL)
    first.flags |= rt.FLAG_RELAY
    names, runner.names = runner.names, {"x": runner.names["o0"]}  # x of the second is the first's result
    second = decode._gemv_phase(runner, x=glu, segs=[(wd, None, out)], k=mid, rows=rows,
                                epilogue=rt.EPI_RESIDUAL, residual=base)
    assert names["o0"] == second.slot[rt.GV_S_X]
    plan = runner.run([first, second], (rows + 1) * (max(k, mid) + 32) * 2)
    assert plan.status().code == 0
    once = out.clone()
    out.zero_()
    plan.launch([], torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert plan.status().code == 0 and torch.equal(out, once)
    normed = oracle.rms_norm(x.cpu(), nw.cpu(), 1e-5, "llama").cuda()
    act = oracle._activation(decode._ref_linear(normed, wg).cpu(), "silu").cuda()
    ref = base + decode._ref_linear(act * decode._ref_linear(normed, wu), wd)
    assert cosine(out, ref) > 0.9999
    assert float((out.float() - ref.float()).abs().max()) <= 0.06


@pytest.mark.parametrize("rows", [1, 19, 127, 129])
@pytest.mark.parametrize("n,k", [(72, 2048), (576, 1536), (1004, 4096)])
def test_reduction_shared_by_a_cluster(rows, n, k):
    """Few output tiles and a long reduction; plain with bias, in-place residual, gated pair."""
    x = prefill._bf16(rows, k, seed=1)
    w, b = prefill._bf16(n, k, scale=k ** -0.5, seed=2), prefill._bf16(n, seed=3)
    out = torch.zeros(rows, n, dtype=torch.bfloat16, device="cuda")
    runner = PhaseRunner()
    prefill._run(runner, [prefill._gemm_phase(runner, x=x.cuda(), segs=[(w.cuda(), b.cuda(), out)])])
    prefill._check_gemm(out, prefill._ref_linear(x, w, b))

    hidden0 = prefill._bf16(rows, n, seed=4)
    hidden = hidden0.clone().cuda()
    runner = PhaseRunner()
    prefill._run(runner, [prefill._gemm_phase(runner, x=x.cuda(), segs=[(w.cuda(), None, hidden)],
                                              residual=hidden, epilogue=rt.EPI_RESIDUAL)])
    ref = hidden0 + prefill._ref_linear(x, w)
    assert prefill._mismatch(hidden, ref) < 0.02 and cosine(hidden, ref) > 0.99999

    up = prefill._bf16(n, k, scale=k ** -0.5, seed=5)
    runner = PhaseRunner()
    prefill._run(runner, [prefill._gemm_phase(runner, x=x.cuda(), segs=[(w.cuda(), None, out)], pair=up.cuda(),
                                              epilogue=rt.EPI_SILU_MUL)])
    ref = oracle._activation(prefill._ref_linear(x, w), "silu") * prefill._ref_linear(x, up)
    assert prefill._mismatch(out, ref) < 0.03 and cosine(out, ref) > 0.99999
