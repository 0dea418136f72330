"""Kernels that start while the one in front of them still runs: same results as with every launch waited for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(x, w13, w2, wait):
    """Quantise -> e4m3 product -> SwiGLU -> bf16 product: four launches, each reading what the last one wrote."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.fused import swiglu
    from torchcomms_b200.ops.tp import gemm_e4m3_nt, quantize_rows

    q, scale = quantize_rows(x)
    wait()
    gate_up = gemm_e4m3_nt(q, w13[0], scale, w13[1])
    wait()
    h = swiglu(gate_up)
    wait()
    y, status = _comms.ops.gemm_bf16_nt(h, w2)
    wait()
    return y, status


# One row; one tile of each product; several K shares; more tiles than SMs; row counts off the tiles.
@pytest.mark.parametrize("rows,hidden,ffn", [(1, 256, 128), (67, 4096, 1792), (128, 2048, 1024), (300, 1040, 520), (2050, 512, 4096)])
@pytest.mark.parametrize("graph", [False, True])
def test_chain_is_ordered(rows, hidden, ffn, graph):
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(rows)
    w13 = quantize_rows((torch.randn(2 * ffn, hidden, generator=g, device="cuda") * 0.02).to(torch.bfloat16))
    w2 = (torch.randn(hidden, ffn, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    xs = [torch.randn(rows, hidden, generator=g, device="cuda").to(torch.bfloat16) for _ in range(8)]
    want = [_chain(x, w13, w2, torch.cuda.synchronize)[0] for x in xs]
    # Two streams at a time, nothing waited for, memory handed from call to call by the allocator.
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    if graph:
        src, graphs = xs[0].clone(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs):
            y, status = _chain(src, w13, w2, lambda: None)
        for x, ref in zip(xs, want):
            src.copy_(x)
            graphs.replay()
            assert torch.equal(y, ref) and not status.any()
        return
    for _ in range(5):
        got = []
        for i, x in enumerate(xs):
            with torch.cuda.stream(streams[i % 2]):
                got.append(_chain(x, w13, w2, lambda: None))
        torch.cuda.synchronize()
        for (y, status), ref in zip(got, want):
            assert torch.equal(y, ref) and not status.any()


def test_status_words_are_each_call_s_own():
    from torchcomms_b200 import _comms

    a = torch.ones(8, 64, device="cuda", dtype=torch.bfloat16)
    seen = [_comms.ops.gemm_bf16_nt(a, a)[1] for _ in range(1100)]  # more than one block of words
    assert len({s.data_ptr() for s in seen}) == len(seen) and all(s.shape == (2,) for s in seen)
    seen[0].fill_(7)
    assert not torch.stack(seen[1:]).any()


# The split kernel; pairs of 128 and of 256 columns; single CTAs (in bf16).
@pytest.mark.parametrize("m,n,k", [(5, 1024, 2048), (300, 6144, 1024), (2050, 4096, 512), (700, 6144, 256)])
@pytest.mark.parametrize("fp8", [False, True])
def test_a_product_is_one_launch_and_clears_its_status(m, n, k, fp8):
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    if fp8:
        (a, sa), (b, sb) = quantize_rows(a), quantize_rows(b)
        run = lambda: _comms.ops.gemm_e4m3_nt(a, b, sa, sb)
    else:
        run = lambda: _comms.ops.gemm_bf16_nt(a, b)
    want, _ = run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    before = _comms.ops.kernel_launch_count()
    with torch.cuda.graph(graph):
        c, captured = run()
    assert _comms.ops.kernel_launch_count() - before == 1
    for _ in range(2):
        captured.fill_(7)
        c.zero_()
        graph.replay()
        assert torch.equal(c, want) and not captured.any()
    # Outside a graph, on memory that others have written.
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    seen = []
    for i in range(40):
        with torch.cuda.stream(streams[i % 2]):
            dirty = [torch.full((2,), 7, device="cuda", dtype=torch.int32) for _ in range(4)]
            del dirty
            seen.append(run()[1])
    torch.cuda.synchronize()
    assert not torch.stack(seen).any()
    seen[0].fill_(7)
    assert seen[1]._version == 0 and not torch.stack(seen[1:]).any()


@pytest.mark.parametrize("rows,n,k", [(5, 1024, 2048), (128, 3584, 1024), (1000, 6144, 512)])
def test_an_event_between_holds_the_product_back(rows, n, k):
    """A product behind an event record, and one whose operand another stream still writes while the product in front of
    it already lets it start."""
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(rows)
    ws = [(torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16) for _ in range(2)]
    xs = [torch.randn(rows, k, generator=g, device="cuda").to(torch.bfloat16) for _ in range(6)]
    want = [_comms.ops.gemm_bf16_nt(x, ws[1])[0] for x in xs]
    front = _comms.ops.gemm_bf16_nt(xs[0], ws[0])[0]
    busy = torch.zeros(64 << 20, device="cuda")
    torch.cuda.synchronize()
    writer, reader = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros_like(xs[0])
    written, read = torch.cuda.Event(), torch.cuda.Event()
    got = []
    for src in xs:
        with torch.cuda.stream(writer):
            busy.add_(1.0)  # some 80 us, so that the operand comes late
            x.copy_(src)
            written.record()
        with torch.cuda.stream(reader):
            first = _comms.ops.gemm_bf16_nt(xs[0], ws[0])[0]
            reader.wait_event(written)
            y = _comms.ops.gemm_bf16_nt(x, ws[1])[0]
            read.record()
            again = _comms.ops.gemm_bf16_nt(x, ws[1])[0]
            read.record()
        got.append((first, y, again))
        writer.wait_event(read)
    torch.cuda.synchronize()
    for (first, y, again), ref in zip(got, want):
        assert torch.equal(first, front) and torch.equal(y, ref) and torch.equal(again, ref)
