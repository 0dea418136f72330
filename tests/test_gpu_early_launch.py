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


def test_taking_turns_between_streams_allocates_results_only():
    from torchcomms_b200 import _comms

    a = torch.ones(8, 64, device="cuda", dtype=torch.bfloat16)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()

    def turns(n):
        for i in range(n):
            with torch.cuda.stream(streams[i % 3]):
                seen.append(_comms.ops.gemm_bf16_nt(a, a))

    seen = []
    turns(6)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    turns(300)
    # One result per call; at most one new block of words per stream.
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before <= 300 + 3
    torch.cuda.synchronize()
    assert len({s.data_ptr() for _, s in seen}) == len(seen) and not torch.stack([s for _, s in seen]).any()


def test_status_words_have_versions_of_their_own():
    from torchcomms_b200 import _comms

    a = torch.ones(8, 64, device="cuda", dtype=torch.bfloat16)
    first, second = (_comms.ops.gemm_bf16_nt(a, a)[1] for _ in range(2))
    first.fill_(7)
    assert second._version == 0 and not second.any()
    with torch.inference_mode():
        third = _comms.ops.gemm_bf16_nt(a, a)[1]
    assert third.is_inference() and not first.is_inference() and not third.any()
