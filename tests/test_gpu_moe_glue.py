"""GPU: the mixture-of-experts steps around the grouped GEMMs (gate, permutation,
gather / weighted scatter, SwiGLU, and the forms fused with the 1 x 128 quantizer)
through the C ABI against the oracle's restatement of the reference's torch checks
(benchmarks/bench.py:957-958, 1555-1557, 2546-2548, 2570-2579).

Bars: indices, permutations, gathered rows and every fp8 code / scale of the fused
forms bit-exact; routing weights within 2e-6 relative; sums and activations within one
rounding of the output type of the fp32 value."""
import os
import subprocess
import sys
import threading

import pytest
import torch

import ks_oracle as orc
from _util import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,top_k,dtype,renorm", [
    (4096, 256, 8, torch.float32, True),      # the MoE configuration of the benchmark
    (4096, 256, 8, torch.bfloat16, True),
    (33, 8, 2, torch.float16, False),
    (5, 1000, 32, torch.float32, True),       # the limits: 1000 experts, top-32
    (1, 4, 4, torch.float32, True),           # every expert chosen
])
def test_gate_softmax_topk(ks, cuda, tokens, experts, top_k, dtype, renorm):
    logits = torch.randn(tokens, experts, generator=gen(tokens + experts)).to(dtype)
    w = torch.empty(tokens, top_k, dtype=torch.float32, device=cuda)
    idx = torch.empty(tokens, top_k, dtype=torch.int32, device=cuda)
    ks.moe.gate_softmax_topk(w, idx, logits.to(cuda), tokens, experts, top_k, renormalize=renorm)
    torch.cuda.synchronize()
    probs = torch.softmax(logits.float(), dim=-1)
    ref_w, ref_i = torch.topk(probs, top_k, dim=-1)
    if renorm:
        ref_w = ref_w / ref_w.sum(-1, keepdim=True)
    w, idx = w.cpu(), idx.cpu().to(torch.int64)
    assert torch.allclose(w, ref_w, rtol=2e-6, atol=1e-9)
    # the same experts in the same order, except between experts of equal probability (16-bit
    # logits repeat values; which of two equal ones is taken at the cut is not specified)
    assert bool((idx >= 0).all()) and bool((idx < experts).all())
    assert all(len(set(row)) == top_k for row in idx.tolist()), "an expert was chosen twice"
    differs = idx != ref_i
    assert torch.equal(probs.gather(1, idx)[differs], probs.gather(1, ref_i)[differs])
    if dtype == torch.float32:
        assert not bool(differs.any())
    assert bool((w[:, :-1] >= w[:, 1:]).all()), "weights are not in descending order"


def test_gate_ties_go_to_the_lowest_expert(ks, cuda):
    logits = torch.zeros(3, 16)
    logits[1, 5] = 1.0
    logits[2, 9:12] = 2.0
    w = torch.empty(3, 4, dtype=torch.float32, device=cuda)
    idx = torch.empty(3, 4, dtype=torch.int32, device=cuda)
    ks.moe.gate_softmax_topk(w, idx, logits.to(cuda), 3, 16, 4, renormalize=True)
    assert idx.cpu().tolist() == [[0, 1, 2, 3], [5, 0, 1, 2], [9, 10, 11, 0]]
    assert torch.allclose(w.cpu().sum(1), torch.ones(3))


def _route(tokens, experts, top_k, seed):
    _, ids = orc.moe_route(torch.randn(tokens, experts, generator=gen(seed)), top_k)
    return ids.to(torch.int32)


@pytest.mark.parametrize("tokens,experts,top_k", [
    (4096, 256, 8),      # 32768 pairs: 1024 per warp
    (3, 4, 2),
    (1000, 7, 3),        # pair count not a multiple of 32, experts not a multiple of anything
    (257, 1000, 5),
])
def test_compute_permutation_is_the_stable_sort(ks, cuda, tokens, experts, top_k):
    ids = _route(tokens, experts, top_k, 3)
    sorted_ids = torch.full((tokens * top_k,), -7, dtype=torch.int32, device=cuda)
    offsets = torch.full((experts + 1,), -7, dtype=torch.int32, device=cuda)
    ks.moe.compute_permutation(sorted_ids, offsets, ids.to(cuda), tokens, experts, top_k)
    torch.cuda.synchronize()
    order, ref_off = orc.sort_by_expert(ids.to(torch.int64), experts)
    assert torch.equal(offsets.cpu(), ref_off)
    assert torch.equal(sorted_ids.cpu().to(torch.int64), order)


def test_compute_permutation_drops_ids_out_of_range(ks, cuda):
    ids = torch.tensor([[0, 3], [9, 1], [-1, 3], [2, 2]], dtype=torch.int32)   # 9 and -1 are not experts (E = 4)
    sorted_ids = torch.empty(8, dtype=torch.int32, device=cuda)
    offsets = torch.empty(5, dtype=torch.int32, device=cuda)
    ks.moe.compute_permutation(sorted_ids, offsets, ids.to(cuda), 4, 4, 2)
    assert offsets.cpu().tolist() == [0, 1, 2, 4, 6]
    assert sorted_ids.cpu().tolist() == [0, 3, 6, 7, 1, 5, -1, -1]


@pytest.mark.parametrize("tokens,hidden,experts,top_k,dtype", [
    (4096, 7168, 256, 8, torch.bfloat16),
    (100, 200, 8, 2, torch.float32),
    (77, 129, 8, 3, torch.float16),          # rows that are not 16-byte multiples: element-wise path
    (64, 256, 16, 4, torch.float8_e4m3fn),
])
def test_permute_gathers_rows(ks, cuda, tokens, hidden, experts, top_k, dtype):
    ids = _route(tokens, experts, top_k, 11)
    order, _ = orc.sort_by_expert(ids.to(torch.int64), experts)
    x = torch.randn(tokens, hidden, generator=gen(5)).to(dtype)
    out = torch.empty(tokens * top_k, hidden, dtype=dtype, device=cuda)
    ks.moe.permute(out, x.to(cuda), order.to(torch.int32).to(cuda), tokens, top_k, hidden)
    torch.cuda.synchronize()
    ref = orc.moe_permute(x.view(torch.uint8) if dtype == torch.float8_e4m3fn else x, order, top_k)
    got = out.cpu()
    assert torch.equal(got.view(torch.uint8) if dtype == torch.float8_e4m3fn else got, ref)


def test_permute_zero_fills_dropped_rows(ks, cuda):
    x = torch.randn(4, 64, generator=gen(1)).to(torch.bfloat16)
    ids = torch.tensor([3, -1, 0, 99], dtype=torch.int32)
    out = torch.empty(4, 64, dtype=torch.bfloat16, device=cuda)
    ks.moe.permute(out, x.to(cuda), ids.to(cuda), 4, 1, 64)
    got = out.cpu()
    assert torch.equal(got[0], x[3]) and torch.equal(got[2], x[0])
    assert not got[1].any() and not got[3].any()


@pytest.mark.parametrize("tokens,hidden,experts,top_k,dtype", [
    (4096, 7168, 256, 8, torch.bfloat16),
    (50, 384, 8, 2, torch.float16),
    (9, 128, 4, 1, torch.float32),
])
def test_permute_quant_equals_permute_then_quantize(ks, cuda, tokens, hidden, experts, top_k, dtype):
    ids = _route(tokens, experts, top_k, 12)
    order, _ = orc.sort_by_expert(ids.to(torch.int64), experts)
    x = torch.randn(tokens, hidden, generator=gen(6)).to(dtype)
    q = torch.empty(tokens * top_k, hidden, dtype=torch.float8_e4m3fn, device=cuda)
    s = torch.empty(tokens * top_k, hidden // 128, dtype=torch.float32, device=cuda)
    ks.moe.permute_quant_fp8(q, s, x.to(cuda), order.to(torch.int32).to(cuda), tokens, top_k, hidden)
    torch.cuda.synchronize()
    rows = 4096 if tokens * top_k > 4096 else tokens * top_k      # the oracle affords a window of the big case
    q_ref, s_ref = orc.quantize_fp8_group(orc.moe_permute(x, order[:rows], top_k), 128)
    assert torch.equal(q.cpu()[:rows].view(torch.uint8), q_ref.view(torch.uint8))
    assert torch.equal(s.cpu()[:rows], s_ref)
    # and the whole output against the two library calls run one after the other
    p = torch.empty(tokens * top_k, hidden, dtype=dtype, device=cuda)
    ks.moe.permute(p, x.to(cuda), order.to(torch.int32).to(cuda), tokens, top_k, hidden)
    q2, s2 = ks.dispatch.per_token_group_quant(p)
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)


@pytest.mark.parametrize("tokens,hidden,experts,top_k,dtype", [
    (4096, 7168, 256, 8, torch.bfloat16),
    (40, 264, 8, 2, torch.float16),
    (21, 100, 4, 3, torch.float32),
    (16, 99, 4, 2, torch.bfloat16),          # element-wise path
])
def test_unpermute_weighted_sum(ks, cuda, tokens, hidden, experts, top_k, dtype):
    g = gen(13)
    w, ids = orc.moe_route(torch.randn(tokens, experts, generator=g), top_k)
    order, _ = orc.sort_by_expert(ids, experts)
    y = torch.randn(tokens * top_k, hidden, generator=g).to(dtype)
    out = torch.empty(tokens, hidden, dtype=dtype, device=cuda)
    sid = order.to(torch.int32).to(cuda)
    ks.moe.unpermute(out, y.to(cuda), sid, w.to(cuda), tokens, top_k, hidden)
    out2 = torch.empty_like(out)
    ks.moe.unpermute(out2, y.to(cuda), sid, w.to(cuda), tokens, top_k, hidden)   # workspace reused
    torch.cuda.synchronize()
    ref32 = orc.moe_unpermute(y, order, w, tokens, top_k, out_dtype=None)
    got = out.cpu().float()
    tol = {torch.float32: 2e-6, torch.float16: 1.2e-3, torch.bfloat16: 9e-3}[dtype]
    assert float(((got - ref32).abs() / (ref32.abs() + 0.05)).max()) < tol
    assert orc.rel_frobenius(got, ref32) < (1e-6 if dtype == torch.float32 else 3e-3)
    assert torch.equal(out, out2)


def test_unpermute_skips_dropped_pairs(ks, cuda):
    y = torch.ones(4, 32, dtype=torch.bfloat16)
    ids = torch.tensor([0, 3, -1, -1], dtype=torch.int32)        # pairs 1 and 2 were dropped
    w = torch.tensor([[0.25, 0.75], [0.5, 0.5]])
    out = torch.empty(2, 32, dtype=torch.bfloat16, device=cuda)
    ks.moe.unpermute(out, y.to(cuda), ids.to(cuda), w.to(cuda), 2, 2, 32)
    assert out.cpu().float()[:, 0].tolist() == [0.25, 0.5]


@pytest.mark.parametrize("rows,inter,dtype", [
    (4096, 2048, torch.bfloat16),     # between the expert GEMMs of the MoE configuration (per 4096 rows)
    (33, 144, torch.float16),
    (7, 50, torch.float32),           # element-wise path
    (1, 14336, torch.bfloat16),       # a decode row
])
def test_swiglu(ks, cuda, rows, inter, dtype):
    g = gen(rows + inter)
    x = (torch.randn(rows, 2 * inter, generator=g) * 2).to(dtype)
    out = torch.empty(rows, inter, dtype=dtype, device=cuda)
    ks.activation.swiglu_packed(out, x.to(cuda))
    gate, up = x[:, :inter].contiguous(), x[:, inter:].contiguous()
    out2 = torch.empty(rows, inter, dtype=dtype, device=cuda)
    ks.activation.swiglu(out2, gate.to(cuda), up.to(cuda))
    torch.cuda.synchronize()
    assert torch.equal(out, out2)
    ref32 = orc.swiglu_packed(x, out_dtype=None)
    got = out.cpu().float()
    tol = {torch.float32: 2e-6, torch.float16: 1.2e-3, torch.bfloat16: 9e-3}[dtype]
    assert float(((got - ref32).abs() / (ref32.abs() + 1e-3)).max()) < tol
    assert orc.rel_err_max(got, ref32) < tol


@pytest.mark.parametrize("rows,inter,dtype", [(4096, 2048, torch.bfloat16), (37, 256, torch.float16)])
def test_swiglu_quant_equals_swiglu_then_quantize(ks, cuda, rows, inter, dtype):
    x = (torch.randn(rows, 2 * inter, generator=gen(rows)) * 2).to(dtype).to(cuda)
    q = torch.empty(rows, inter, dtype=torch.float8_e4m3fn, device=cuda)
    s = torch.empty(rows, inter // 128, dtype=torch.float32, device=cuda)
    ks.activation.swiglu_packed_quant_fp8(q, s, x)
    act = torch.empty(rows, inter, dtype=dtype, device=cuda)
    ks.activation.swiglu_packed(act, x)
    q2, s2 = ks.dispatch.per_token_group_quant(act)
    torch.cuda.synchronize()
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)
    # against the oracle: the quantizer is exact, so the codes differ only where the
    # activation itself fell on the other side of a rounding boundary
    q_ref, s_ref = orc.quantize_fp8_group(orc.swiglu_packed(x.cpu()), 128)
    mismatch = (q.cpu().view(torch.uint8) != q_ref.view(torch.uint8)).float().mean().item()
    assert mismatch < 2e-3
    assert torch.allclose(s.cpu(), s_ref, rtol=1e-2)


def test_peer_dispatch_and_combine_on_one_device(ks, cuda):
    """The three steps of the peer-memory dispatch / combine with both "ranks" on one GPU (the
    destination pointers are local tensors): every row must land, bit for bit, where the plan
    says, and come back to the position of the source's sorted order."""
    world, experts, per, tokens, k, hidden = 2, 6, 3, 40, 2, 256
    g = gen(31)
    pairs = tokens * k
    cap = pairs * world
    xs, sorted_ids, offsets, q_loc, s_loc = [], [], [], [], []
    for r in range(world):
        x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16).to(cuda)
        ids = torch.stack([torch.randperm(experts, generator=g)[:k] for _ in range(tokens)]).to(torch.int32).to(cuda)
        sid = torch.empty(pairs, dtype=torch.int32, device=cuda)
        off = torch.empty(experts + 1, dtype=torch.int32, device=cuda)
        ks.moe.compute_permutation(sid, off, ids, tokens, experts, k)
        q = torch.empty(pairs, hidden, dtype=torch.float8_e4m3fn, device=cuda)
        s = torch.empty(pairs, hidden // 128, dtype=torch.float32, device=cuda)
        ks.moe.permute_quant_fp8(q, s, x, sid, tokens, k, hidden)
        xs.append(x); sorted_ids.append(sid); offsets.append(off); q_loc.append(q); s_loc.append(s)
    counts = torch.stack([o[1:] - o[:-1] for o in offsets]).contiguous()        # [world, experts]
    recv_q = [torch.full((cap, hidden), 0xAA, dtype=torch.uint8, device=cuda) for _ in range(world)]
    recv_s = [torch.full((cap, hidden // 128), -1.0, device=cuda) for _ in range(world)]
    plans = []
    for r in range(world):
        dst_base = torch.empty(experts, dtype=torch.int32, device=cuda)
        local_off = torch.empty(per + 1, dtype=torch.int32, device=cuda)
        seg_start = torch.empty(per * world + 1, dtype=torch.int32, device=cuda)
        ret_base = torch.empty(per * world, dtype=torch.int32, device=cuda)
        ks.moe.dispatch_plan(dst_base, local_off, seg_start, ret_base, counts, world, r, per)
        plans.append((dst_base, local_off, seg_start, ret_base))
        ks.moe.permute_quant_fp8_scatter(recv_q, recv_s, cap, dst_base, offsets[r], experts, per, xs[r], sorted_ids[r],
                                         tokens, k, hidden)
    torch.cuda.synchronize()
    c = counts.cpu()
    offs_h = [o.cpu() for o in offsets]
    for d in range(world):
        local_off = plans[d][1].cpu()
        row = 0
        for el in range(per):
            e = d * per + el
            assert int(local_off[el]) == row
            for s in range(world):
                n = int(c[s, e])
                lo = int(offs_h[s][e])
                assert torch.equal(recv_q[d][row:row + n], q_loc[s][lo:lo + n].view(torch.uint8)), (d, el, s)
                assert torch.equal(recv_s[d][row:row + n], s_loc[s][lo:lo + n]), (d, el, s)
                row += n
        assert int(local_off[per]) == row
        assert bool((recv_q[d][row:] == 0xAA).all()), "rows beyond the received ones were written"
    # the way back
    back = [torch.zeros(pairs, hidden, dtype=torch.bfloat16, device=cuda) for _ in range(world)]
    ys = [torch.randn(cap, hidden, generator=g).to(torch.bfloat16).to(cuda) for _ in range(world)]
    for d in range(world):
        ks.moe.scatter_rows(back, pairs, ys[d], cap, plans[d][2], plans[d][3], per * world, hidden)
    torch.cuda.synchronize()
    for d in range(world):
        row = 0
        for el in range(per):
            e = d * per + el
            for s in range(world):
                n = int(c[s, e])
                lo = int(offs_h[s][e])
                assert torch.equal(back[s][lo:lo + n], ys[d][row:row + n]), (d, el, s)
                row += n


@pytest.mark.parametrize("top_k,dtype", [(2, torch.bfloat16), (4, torch.float32)])
def test_permute_quant_of_large_problems_takes_any_ids(ks, cuda, top_k, dtype):
    """From 64 M elements on (32 M with four pairs a token), tokens are quantized once and written to all their rows; ids out of range and
    repeated ids are rows that no token writes. Bit for bit what gather + quantizer give."""
    tokens, hidden = ((64 if top_k < 4 else 32) << 20) // 4096 // top_k + 3, 4096
    pairs = tokens * top_k
    g = gen(31)
    ids = torch.randperm(pairs, generator=g).to(torch.int32)
    ids[5::97] = ids[4::97][:ids[5::97].numel()]     # repeated
    ids[7::101] = -1                                 # dropped
    ids[9::103] = pairs + 9                          # out of range
    x = torch.randn(tokens, hidden, generator=g).to(dtype).to(cuda)
    ids = ids.to(cuda)
    q = torch.full((pairs, hidden), 7, dtype=torch.uint8, device=cuda).view(torch.float8_e4m3fn)
    s = torch.full((pairs, hidden // 128), float("nan"), dtype=torch.float32, device=cuda)
    ks.moe.permute_quant_fp8(q, s, x, ids, tokens, top_k, hidden)
    p = torch.empty(pairs, hidden, dtype=dtype, device=cuda)
    ks.moe.permute(p, x, ids, tokens, top_k, hidden)
    q2, s2 = ks.dispatch.per_token_group_quant(p)
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)


@pytest.mark.parametrize("top_k,hidden,fp8", [(2, 4096, "e4m3"), (3, 1152, "e5m2"), (4, 4096, "e4m3"), (6, 640, "e4m3"), (8, 2048, "e5m2")])
@pytest.mark.parametrize("drop", [0.6, 1.0])
def test_permute_quant_of_large_problems_drops_tokens(ks, cuda, top_k, hidden, fp8, drop):
    """Just above the sizes from which tokens are quantized once, with whole tokens dropped (hidden widths
    where a warp holds segments of two tokens among them): bit for bit what gather + quantizer give."""
    from_m = 24 if top_k >= 6 else 32 if top_k >= 4 else 64
    tokens = (from_m << 20) // (hidden * top_k) + 5
    pairs = tokens * top_k
    g = torch.Generator(device=cuda).manual_seed(top_k)
    ids = torch.randperm(pairs, generator=g, device=cuda).to(torch.int32)
    gone = torch.rand(tokens, generator=g, device=cuda) < drop
    ids[gone[(ids // top_k).long()]] = -1
    ids[::7] = torch.where(ids[::7] % 5 == 0, -1, ids[::7])
    x = torch.randn(tokens, hidden, generator=g, device=cuda).to(torch.bfloat16)
    dt = {"e4m3": torch.float8_e4m3fn, "e5m2": torch.float8_e5m2}[fp8]
    kw = dict(fp8_dtype=ks.DType.F8E5M2 if fp8 == "e5m2" else ks.DType.F8E4M3)
    q = torch.full((pairs, hidden), 7, dtype=torch.uint8, device=cuda).view(dt)
    s = torch.full((pairs, hidden // 128), float("nan"), dtype=torch.float32, device=cuda)
    ks.moe.permute_quant_fp8(q, s, x, ids, tokens, top_k, hidden, **kw)
    p = torch.empty(pairs, hidden, dtype=torch.bfloat16, device=cuda)
    ks.moe.permute(p, x, ids, tokens, top_k, hidden)
    q2, s2 = ks.dispatch.per_token_group_quant(p, **kw)
    assert torch.equal(q.view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s, s2)


@pytest.mark.parametrize("hidden,dtype", [(64, torch.bfloat16), (33, torch.float16), (64, torch.float32)])
def test_unpermute_does_not_see_an_earlier_permutation(ks, cuda, hidden, dtype):
    """The inverse map outlives a call. A permutation that names every pair, then one on the same stream that drops
    most of them (ids -1 and out of range): the dropped pairs add nothing, whatever row the map still has for them."""
    tokens, top_k = 300, 4
    pairs = tokens * top_k
    g = gen(8)
    w = torch.rand(tokens, top_k, generator=g).to(cuda)
    for drop in (0.0, 0.7, 0.0, 1.0):
        ids = torch.randperm(pairs, generator=g).to(torch.int32)
        cut = torch.rand(pairs, generator=g) < drop
        ids[cut] = torch.where(torch.rand(int(cut.sum()), generator=g) < 0.5, -1, pairs + 3).to(torch.int32)
        y = torch.randint(-8, 9, (pairs, hidden), generator=g).to(dtype)
        out = torch.full((tokens, hidden), float("nan"), dtype=dtype, device=cuda)
        ks.moe.unpermute(out, y.to(cuda), ids.to(cuda), w, tokens, top_k, hidden)
        ref = torch.zeros(pairs, hidden, dtype=torch.float64)
        ref[ids[~cut].long()] = y[~cut].double()
        ref = (ref.view(tokens, top_k, hidden) * w.cpu().double()[:, :, None]).sum(1)
        # four fp32 additions and one rounding to the output type
        eps = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -22}[dtype]
        assert torch.allclose(out.cpu().double(), ref, rtol=2 * eps, atol=32 * 2.0 ** -22), drop


@pytest.mark.parametrize("experts", [360, 361, 362, 372])
def test_compute_permutation_around_48_kb(ks, cuda, experts):
    """34 counters an expert are 48 KB of dynamic shared memory at 361 experts, with the static part just over it. In
    a process of its own: a call with more experts before it would have raised the limit for the rest."""
    code = f"""
import torch, kernel_set_b200 as ks
ids = torch.randint(0, {experts}, (50, 4), dtype=torch.int32, device="cuda")
so = torch.empty(200, dtype=torch.int32, device="cuda"); off = torch.empty({experts} + 1, dtype=torch.int32, device="cuda")
ks.moe.compute_permutation(so, off, ids, 50, {experts}, 4)
assert torch.equal(so.long(), torch.sort(ids.view(-1), stable=True).indices)
assert int(off[-1]) == 200
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=root, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("tokens,experts,top_k", [
    (25000, 64, 8),        # 200000 pairs, more than a pair per thread of 148 CTAs: a warp's piece has several steps
    (50001, 7, 3),         # ... 150003 pairs, not a multiple of 32
    (4001, 40, 5),         # several CTAs of one step, the last one partial
])
def test_compute_permutation_of_many_pairs_with_dropped_ones(ks, cuda, tokens, experts, top_k):
    """Many CTAs, running counters carried from step to step, ids out of range in every CTA."""
    g = gen(tokens)
    ids = torch.randint(0, experts, (tokens, top_k), generator=g).to(torch.int32)
    ids[torch.rand(tokens, top_k, generator=g) < 0.1] = -1
    ids[torch.rand(tokens, top_k, generator=g) < 0.05] = experts + 2
    pairs = tokens * top_k
    sorted_ids = torch.full((pairs,), -7, dtype=torch.int32, device=cuda)
    offsets = torch.full((experts + 1,), -7, dtype=torch.int32, device=cuda)
    ks.moe.compute_permutation(sorted_ids, offsets, ids.to(cuda), tokens, experts, top_k)
    flat = ids.view(-1).long()
    valid = ((flat >= 0) & (flat < experts)).nonzero().view(-1)
    order = valid[torch.sort(flat[valid], stable=True).indices]
    assert torch.equal(sorted_ids.cpu()[:order.numel()].long(), order)
    assert bool((sorted_ids.cpu()[order.numel():] == -1).all())
    assert torch.equal(offsets.cpu().long()[1:], torch.bincount(flat[valid], minlength=experts).cumsum(0)) and int(offsets[0]) == 0


def test_host_threads_share_a_stream(ks, cuda):
    """Two host threads on one stream, each with problems of its own and growing sizes: the inverse map that a call
    writes is the one that it reads. (Values are small integers and weights powers of two: sums are exact.)"""
    stream = torch.cuda.Stream(cuda)
    hidden, top_k, calls = 64, 4, 60

    def problem(seed, tokens):
        g = gen(seed)
        pairs = tokens * top_k
        ids = torch.randperm(pairs, generator=g).to(torch.int32)
        ids[torch.rand(pairs, generator=g) < 0.3] = -1
        y = torch.randint(-8, 9, (pairs, hidden), generator=g)
        ref = torch.zeros(pairs, hidden, dtype=torch.int64)
        keep = ids >= 0
        ref[ids[keep].long()] = y[keep]
        return ids.to(cuda), y.to(torch.float32).to(cuda), ref.view(tokens, top_k, hidden).sum(1), tokens

    problems = [[problem(100 * t + i, 50 + (7 + 3 * t) * i * i) for i in range(calls)] for t in range(2)]
    weights = torch.ones(max(p[3] for ps in problems for p in ps), top_k, device=cuda)
    outs = [[torch.empty(p[3], hidden, dtype=torch.bfloat16 if i % 2 else torch.float32, device=cuda)
             for i, p in enumerate(ps)] for ps in problems]
    ys = [[p[1].to(o.dtype) for p, o in zip(ps, os_)] for ps, os_ in zip(problems, outs)]
    torch.cuda.synchronize()
    errors = []

    def run(t):
        try:
            for p, y, o in zip(problems[t], ys[t], outs[t]):
                ks.moe.unpermute(o, y, p[0], weights, p[3], top_k, hidden, stream=stream)
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stream.synchronize()
    assert not errors
    for t in range(2):
        for i, (p, o) in enumerate(zip(problems[t], outs[t])):
            assert torch.equal(o.cpu().long(), p[2]), (t, i)


@pytest.mark.parametrize("tokens", [1, 40, 700])
def test_kernels_that_begin_early_wait_for_each_other(ks, cuda, tokens):
    """A layer's steps on buffers that every pass overwrites, queued back to back, against the same steps with the
    device drained after each: a kernel that read or wrote before the one before it was done would show."""
    hidden, inter, experts, top_k = 1024, 512, 16, 4
    rows = tokens * top_k
    g = torch.Generator(device=cuda).manual_seed(tokens)
    e = lambda *shape, **kw: torch.empty(*shape, device=cuda, **kw)
    w1 = torch.randint(0, 120, (experts, 2 * inter, hidden), generator=g, device=cuda, dtype=torch.uint8).view(torch.float8_e4m3fn)
    w2 = torch.randint(0, 120, (experts, hidden, inter), generator=g, device=cuda, dtype=torch.uint8).view(torch.float8_e4m3fn)
    s1 = torch.rand(experts, 2 * inter // 128, hidden // 128, generator=g, device=cuda) * 1e-3
    s2 = torch.rand(experts, hidden // 128, inter // 128, generator=g, device=cuda) * 1e-3
    codes = torch.randint(0, 256, (hidden // 2, hidden), generator=g, device=cuda, dtype=torch.uint8)
    scales = (torch.rand(hidden // 128, hidden, generator=g, device=cuda) * 0.02).bfloat16()
    perm = torch.randperm(hidden, generator=g, device=cuda).to(torch.int32)
    gamma = torch.ones(hidden, device=cuda, dtype=torch.bfloat16)
    inputs = [(torch.randn(tokens, hidden, generator=g, device=cuda).bfloat16(),
               torch.randn(tokens, experts, generator=g, device=cuda)) for _ in range(6)]
    x8, xs = e(tokens, hidden, dtype=torch.float8_e4m3fn), e(tokens, hidden // 128)
    wts, ids = e(tokens, top_k), e(tokens, top_k, dtype=torch.int32)
    order, off = e(rows, dtype=torch.int32), e(experts + 1, dtype=torch.int32)
    p8, ps = e(rows, hidden, dtype=torch.float8_e4m3fn), e(rows, hidden // 128)
    h, y = e(rows, 2 * inter, dtype=torch.bfloat16), e(rows, hidden, dtype=torch.bfloat16)
    a8, as_ = e(rows, inter, dtype=torch.float8_e4m3fn), e(rows, inter // 128)
    z, gx, o = (e(tokens, hidden, dtype=torch.bfloat16) for _ in range(3))

    def layer(x, logits, after):
        outs = []
        steps = [
            lambda: ks.int4.gather_columns(gx, x, perm, tokens, hidden),
            lambda: ks.gemm.gemm_w4a16(z, gx, codes, scales, None, tokens, hidden, hidden, group_size=128),
            lambda: ks.norm.rms_norm_quant_fp8(x8, xs, z, gamma),
            lambda: ks.gemm.gemm_fp8_blockwise(z, x8, w1[0, :, :].view(2 * inter, hidden), xs, s1[0], tokens, 2 * inter, hidden,
                                               b_layout="nk"),
            lambda: ks.moe.gate_softmax_topk(wts, ids, logits, tokens, experts, top_k),
            lambda: ks.moe.compute_permutation(order, off, ids, tokens, experts, top_k),
            lambda: ks.moe.permute_quant_fp8(p8, ps, z, order, tokens, top_k, hidden),
            lambda: ks.moe.grouped_gemm_fp8_blockwise(h, p8, w1, ps, s1, off, experts, rows, 2 * inter, hidden),
            lambda: ks.activation.swiglu_packed_quant_fp8(a8, as_, h, rows, inter),
            lambda: ks.moe.grouped_gemm_fp8_blockwise(y, a8, w2, as_, s2, off, experts, rows, hidden, inter),
            lambda: ks.moe.unpermute(o, y, order, wts, tokens, top_k, hidden),
        ]
        for step in steps:
            step()
            after()
        outs.append(o.clone())
        return outs

    drained = [layer(x, lg, torch.cuda.synchronize)[0] for x, lg in inputs]
    torch.cuda.synchronize()
    for _ in range(3):
        queued = [layer(x, lg, lambda: None)[0] for x, lg in inputs]
        torch.cuda.synchronize()
        for a, b in zip(queued, drained):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("tokens", [2, 24])     # the decode kernel and the tcgen05 kernel
def test_w4a16_behind_a_quantizer_reads_scales_written_just_before(ks, cuda, tokens):
    """New scales and zero-points by another library's kernels, a quantizer, then W4A16, queued back to back: W4A16 reads
    them ahead of its own wait, so the quantizer must not have let it begin before they were there."""
    k, n = 2048, 11008
    g = torch.Generator(device=cuda).manual_seed(tokens)
    x = torch.randn(tokens, k, generator=g, device=cuda).bfloat16()
    codes = torch.randint(0, 256, (k // 2, n), generator=g, device=cuda, dtype=torch.uint8)
    versions = [(torch.rand(k // 128, n, generator=g, device=cuda).mul(0.02).bfloat16(),
                 torch.randint(0, 16, (k // 128, n), generator=g, device=cuda).bfloat16()) for _ in range(4)]
    scales, zeros = torch.empty_like(versions[0][0]), torch.empty_like(versions[0][1])
    x8 = torch.empty(tokens, k, dtype=torch.float8_e4m3fn, device=cuda)
    xs = torch.empty(tokens, k // 128, device=cuda)

    def layer(version, after):
        out = torch.empty(tokens, n, dtype=torch.bfloat16, device=cuda)
        for step in (lambda: scales.copy_(version[0]), lambda: zeros.copy_(version[1]),
                     lambda: ks.quant.quantize_fp8_group(x8, xs, x, tokens, k),
                     lambda: ks.gemm.gemm_w4a16(out, x, codes, scales, zeros, tokens, n, k, group_size=128)):
            step()
            after()
        return out

    drained = [layer(v, torch.cuda.synchronize) for v in versions]
    for _ in range(10):
        queued = [layer(v, lambda: None) for v in versions]
        torch.cuda.synchronize()
        for a, b in zip(queued, drained):
            assert torch.equal(a, b)


def _swiglu_both_ways(ks, x, inter):
    """SwiGLU of packed x by the kernel that corrects an approximate reciprocal, and by the one that divides (rows at
    an odd address)."""
    out = torch.empty(x.shape[0], inter, dtype=x.dtype, device=x.device)
    ks.activation.swiglu_packed(out, x)
    odd = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(x.shape).copy_(x)
    ref = torch.empty(out.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(out.shape)
    ks.activation.swiglu_packed(ref, odd)
    return out, ref


@pytest.mark.parametrize("up", [1.0, -3.25])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_quotient_over_every_gate(ks, cuda, dtype, up):
    """Every bit pattern as the gate times an up of every significand: the corrected quotient is the rounded one, so the two
    kernels agree to the bit, and no result depends on its neighbours or on the address of its row."""
    bits = 7 if dtype == torch.bfloat16 else 10
    gate = torch.arange(-32768, 32768, dtype=torch.int32, device=cuda).to(torch.int16).view(dtype)
    ups = (torch.arange(2 ** bits, device=cuda).float() / 2 ** bits + 1).mul(up).to(dtype)
    x = torch.empty(2 ** bits, 2 * 65536, dtype=dtype, device=cuda)
    x[:, :65536], x[:, 65536:] = gate, ups[:, None]
    a, b = _swiglu_both_ways(ks, x, 65536)
    nan = torch.isnan(b)
    assert torch.equal(torch.isnan(a), nan)
    assert torch.equal(a.view(torch.int16).masked_fill(nan, 0), b.view(torch.int16).masked_fill(nan, 0))
    # mixed rows: one value beyond the range sends its neighbours through the division too
    mixed = torch.randn(64, 256, generator=gen(1)).to(dtype)
    mixed[::3, 5] = 100.0
    mixed[1::3, 77] = float("inf")
    mixed[2::3, 130] = float("nan")
    m = torch.cat([mixed, torch.full_like(mixed, up)], 1).to(cuda)
    om = torch.empty(64, 256, dtype=dtype, device=cuda)
    ks.activation.swiglu_packed(om, m)
    want = orc.swiglu_packed(m.cpu())
    ok = ~torch.isnan(want)
    assert torch.equal(torch.isnan(om.cpu()), ~ok)
    assert (om.cpu().view(torch.int16).int() - want.view(torch.int16).int())[ok].abs().max() <= 1
    divided = _swiglu_both_ways(ks, m, 256)[1].cpu()
    assert torch.equal(om.cpu().view(torch.int16)[ok], divided.view(torch.int16)[ok])
