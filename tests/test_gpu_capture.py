"""GPU: calls that use the library's scratch memory, captured into CUDA graphs: on a stream that has no scratch yet, on
one that has, and with calls on the same stream between replays that need more of it."""
import ctypes

import pytest
import torch

from _util import gen

pytestmark = pytest.mark.gpu


def _w4a16(ks, cuda, m, k, n, gs):
    g = torch.Generator(device=cuda).manual_seed(m + k + n)
    x = torch.randn(m, k, generator=g, device=cuda).to(torch.bfloat16)
    codes = torch.randint(0, 256, (k // 2, n), generator=g, device=cuda, dtype=torch.uint8)
    scales = (torch.randn(k // gs, n, generator=g, device=cuda).mul(0.02).abs() + 1e-3).to(torch.bfloat16)
    zeros = torch.randint(0, 16, (k // gs, n), generator=g, device=cuda).to(torch.bfloat16)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=cuda)
    return x, out, lambda: ks.gemm.gemm_w4a16(out, x, codes, scales, zeros, m, n, k, gs)


def _unpermute(ks, cuda, tokens, hidden, dtype):
    top_k = 4
    pairs = tokens * top_k
    ids = torch.randperm(pairs, generator=gen(3)).to(torch.int32).to(cuda)
    ids[::5] = -1
    y = torch.randn(pairs, hidden, generator=gen(4)).to(dtype).to(cuda)
    w = torch.rand(tokens, top_k, generator=gen(5)).to(cuda)
    out = torch.empty(tokens, hidden, dtype=dtype, device=cuda)
    return y, out, lambda: ks.moe.unpermute(out, y, ids, w, tokens, top_k, hidden)


def _permute_quant(ks, cuda, tokens, hidden):
    top_k = 8
    pairs = tokens * top_k
    ids = torch.randperm(pairs, generator=gen(6)).to(torch.int32).to(cuda)
    x = torch.randn(tokens, hidden, generator=gen(7)).to(torch.bfloat16).to(cuda)
    out = torch.empty(pairs, hidden, dtype=torch.float8_e4m3fn, device=cuda)
    scale = torch.empty(pairs, hidden // 128, device=cuda)
    return x, out.view(torch.uint8), lambda: ks.moe.permute_quant_fp8(out, scale, x, ids, tokens, top_k, hidden)


def _fp8(ks, cuda, m, k, n):
    x = torch.randn(m, k, generator=gen(8)).to(torch.bfloat16).to(cuda)
    a8, a_s = ks.dispatch.per_token_group_quant(x)
    b8 = torch.randn(n, k, generator=gen(9)).to(torch.float8_e4m3fn).to(cuda)
    b_s = torch.rand(-(-n // 128), k // 128, generator=gen(10)).to(cuda)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=cuda)
    return a_s, out, lambda: ks.gemm.gemm_fp8_blockwise(out, a8, b8, a_s, b_s, m, n, k, b_layout="nk")


def _grouped(ks, cuda, kind, sizes=(300, 0, 129, 17), n=1024, k=4096):
    e, rows = len(sizes), sum(sizes)
    off = torch.tensor([0] + torch.tensor(sizes).cumsum(0).tolist(), dtype=torch.int32, device=cuda)
    g = torch.Generator(device=cuda).manual_seed(rows + n + k)
    x = torch.randn(rows, k, generator=g, device=cuda).bfloat16()
    out = torch.empty(rows, n, dtype=torch.bfloat16, device=cuda)
    if kind == "16":
        w = torch.randn(e, k, n, generator=g, device=cuda).mul_(0.05).bfloat16()
        return x, out, lambda: ks.moe.grouped_gemm(out, x, w, off, e, rows, n, k)
    x8, xs = ks.dispatch.per_token_group_quant(x)
    w = torch.randint(0, 120, (e, n, k), generator=g, device=cuda, dtype=torch.uint8).view(torch.float8_e4m3fn)
    ws = torch.rand(e, n // 128, k // 128, generator=g, device=cuda) * 1e-3
    if kind == "fp8":
        return xs, out, lambda: ks.moe.grouped_gemm_fp8_blockwise(out, x8, w, xs, ws, off, e, rows, n, k)
    top = max(sizes)
    m8 = torch.zeros(e, top, k, dtype=torch.uint8, device=cuda)
    ms = torch.ones(e, top, k // 128, device=cuda)
    for i, s in enumerate(sizes):
        m8[i, :s], ms[i, :s] = x8.view(torch.uint8)[int(off[i]):int(off[i]) + s], xs[int(off[i]):int(off[i]) + s]
    m8, out = m8.view(torch.float8_e4m3fn), torch.zeros(e, top, n, dtype=torch.bfloat16, device=cuda)
    counts = torch.tensor(sizes, dtype=torch.int32, device=cuda)
    return ms, out, lambda: ks.moe.grouped_gemm_fp8_blockwise_masked(out, m8, w, ms, ws, counts, e, top, n, k)


CALLS = {
    "w4a16 equal runs": lambda ks, d: _w4a16(ks, d, 24, 8192, 28688, 128),
    "w4a16 decode kernel": lambda ks, d: _w4a16(ks, d, 8, 4096, 11008, 128),
    "w4a16 above 128 rows": lambda ks, d: _w4a16(ks, d, 150, 8192, 11008, 128),
    "w4a16 narrow groups": lambda ks, d: _w4a16(ks, d, 24, 8192, 28688, 64),
    "w4a16 narrow groups, decode kernel": lambda ks, d: _w4a16(ks, d, 8, 8192, 11008, 64),
    "unpermute": lambda ks, d: _unpermute(ks, d, 500, 256, torch.bfloat16),
    "unpermute f32": lambda ks, d: _unpermute(ks, d, 500, 256, torch.float32),
    "permute + quantize": lambda ks, d: _permute_quant(ks, d, 800, 4096),
    "fp8 with a split last round": lambda ks, d: _fp8(ks, d, 2500, 4096, 2000),
    "grouped fp8": lambda ks, d: _grouped(ks, d, "fp8"),
    "grouped fp8, masked": lambda ks, d: _grouped(ks, d, "masked"),
    "grouped 16-bit": lambda ks, d: _grouped(ks, d, "16"),
}


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("name", list(CALLS))
def test_scratch_in_a_graph(ks, cuda, name, warm):
    stream = torch.cuda.Stream(cuda)
    x, out, call = CALLS[name](ks, cuda)
    eager, exact = [], "w4a16" not in name   # without scratch W4A16 may deal otherwise: sums in another order
    x0 = x.clone()

    def check(what):
        torch.cuda.synchronize()
        a, b = out, eager[what]
        if exact or warm:
            assert torch.equal(a, b), what
        else:
            assert float((a.double() - b.double()).norm() / b.double().norm()) < 2e-3, what

    for factor in (1.0, 0.5):     # reference results, on the default stream
        x.copy_(x0 * factor)
        call()
        torch.cuda.synchronize()
        eager.append(out.clone())
    stream.wait_stream(torch.cuda.current_stream())
    if warm:
        with torch.cuda.stream(stream):
            call()
        stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    # an ordinary call on the stream before the graph has ever run: no address of the graph's may serve it
    with torch.cuda.stream(stream):
        x.copy_(x0)
        out.zero_()
        call()
    stream.synchronize()
    assert torch.equal(out, eager[0])
    big = {"w4a16": lambda: _w4a16(ks, cuda, 128, 4096, 28672, 128)[2], "unpermute": lambda: _unpermute(ks, cuda, 70000, 64, torch.bfloat16)[2],
           "permute": lambda: _unpermute(ks, cuda, 70000, 64, torch.float32)[2], "fp8": lambda: _fp8(ks, cuda, 5000, 4096, 4096)[2],
           "grouped": lambda: _fp8(ks, cuda, 5000, 4096, 4096)[2]}
    grow = big[name.split()[0]]()
    for turn in range(3):
        for what, factor in enumerate((1.0, 0.5)):
            x.copy_(x0 * factor)
            out.zero_()
            graph.replay()
            check(what)
        if turn < 2:
            with torch.cuda.stream(stream):
                grow()                # needs more of the same scratch
                filler = torch.full((1 << 24,), 7, dtype=torch.int32, device=cuda)   # what a freed buffer might become
            torch.cuda.synchronize()
            del filler
    torch.cuda.synchronize()
    ks.runtime.stream_synchronize(0)


@pytest.mark.parametrize("kind", ["fp8", "masked", "16"])
def test_grouped_call_is_one_kernel_in_a_graph(ks, cuda, kind):
    """A grouped GEMM neither allocates nor clears nor shares scratch: captured on a stream that has none, it is one
    kernel node and no other."""
    driver = ctypes.CDLL("libcuda.so.1")
    _, out, call = _grouped(ks, cuda, kind)
    call()
    torch.cuda.synchronize()
    eager = out.clone()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream(cuda)):
        call()
    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert driver.cuGraphGetNodes(handle, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert driver.cuGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0
    kinds = []
    for node in nodes:
        t = ctypes.c_int(-1)
        assert driver.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(t)) == 0
        kinds.append(t.value)
    assert kinds == [0], kinds     # CU_GRAPH_NODE_TYPE_KERNEL
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


def test_forked_streams_in_a_graph(ks, cuda):
    """Programmatic launches behind event waits: a quantizer forks into two streams, each runs a layer's GEMM on its codes,
    and the kernel behind the join depends on both."""
    m, k, n = 200, 1024, 1024
    g = torch.Generator(device=cuda).manual_seed(2)
    x = torch.randn(m, k, generator=g, device=cuda).bfloat16()
    w = [torch.randint(0, 120, (n, k), generator=g, device=cuda, dtype=torch.uint8).view(torch.float8_e4m3fn) for _ in range(2)]
    ws = [torch.rand(n // 128, k // 128, generator=g, device=cuda) * 1e-3 for _ in range(2)]
    x8, xs = torch.empty(m, k, dtype=torch.float8_e4m3fn, device=cuda), torch.empty(m, k // 128, device=cuda)
    gate_up = torch.empty(2, m, n, dtype=torch.bfloat16, device=cuda)
    out = torch.empty(m, n, dtype=torch.bfloat16, device=cuda)
    a, b = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)

    def layer():
        ks.quant.quantize_fp8_group(x8, xs, x, m, k)
        b.wait_stream(a)
        ks.gemm.gemm_fp8_blockwise(gate_up[0], x8, w[0], xs, ws[0], m, n, k, b_layout="nk")
        with torch.cuda.stream(b):
            ks.gemm.gemm_fp8_blockwise(gate_up[1], x8, w[1], xs, ws[1], m, n, k, b_layout="nk")
        a.wait_stream(b)
        ks.activation.swiglu(out, gate_up[0], gate_up[1], m, n)

    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        layer()
    torch.cuda.synchronize()
    eager = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a):
        layer()
    for _ in range(5):
        out.zero_()
        gate_up.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, eager)
