"""tcgen05 / TMEM GEMM against a PyTorch fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (128, 256, 256), (256, 512, 1024), (300, 384, 512), (300, 264, 200), (1024, 7168, 2048),
                                   (4096, 4096, 4096)])
def test_gemm_bf16_nt(m, n, k):
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    c, status = _comms.ops.gemm_bf16_nt(a, b)
    torch.cuda.synchronize()
    assert int(status[0]) == 0, "a bounded wait inside the kernel ran out"
    ref = a.float() @ b.float().t()
    torch.testing.assert_close(c.float(), ref, rtol=2e-2, atol=2e-2 * (k ** 0.5))


@pytest.mark.parametrize("kind", ["e4m3", "bf16", "pairs"])
@pytest.mark.parametrize("m,n,k", [(3332, 2160, 864), (2000, 4168, 432), (6500, 1032, 256)])
def test_gemm_partial_last_column_tiles(m, n, k, kind):
    """Column tiles of which only the first 64-column chunks exist, followed by further tiles of the same CTA: a chunk
    that is not stored must not overwrite one that still is."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(m)
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    if kind == "e4m3":
        (qa, sa), (qb, sb) = quantize_rows(a), quantize_rows(b)
        ref = (qa.double() * sa.double().unsqueeze(1)) @ (qb.double() * sb.double().unsqueeze(1)).t()
        run = lambda: _comms.ops.gemm_e4m3_nt(qa, qb, sa, sb)
    else:
        ref = a.double() @ b.double().t()
        run = lambda: (_comms.ops.gemm_bf16_nt if kind == "bf16" else _comms.ops.gemm_bf16_nt_pair)(a, b)
    for _ in range(5):
        c, status = run()
        assert int(status[0]) == 0
        # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 1/4 before it.
        torch.testing.assert_close(c.double(), ref, rtol=2**-8, atol=1e-6 * k)


@pytest.mark.parametrize("m", [1, 32, 33, 67, 128, 129, 300])
@pytest.mark.parametrize("n,k", [(8, 8), (136, 72), (128, 256), (136, 264), (520, 704), (520, 712), (264, 896), (264, 904),
                                 (3584, 4096), (6144, 1928), (10248, 1032)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gemm_split_over_clusters(m, n, k, fp8):
    """Products of fewer tiles than SMs: every number of K shares, ragged edges in all three sizes, both sides of the
    lines below which the persistent kernel takes them."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    if fp8:
        if k % 16:
            a, b = torch.nn.functional.pad(a, (0, 8)), torch.nn.functional.pad(b, (0, 8))
        (qa, sa), (qb, sb) = quantize_rows(a), quantize_rows(b)
        c, status = _comms.ops.gemm_e4m3_nt(qa, qb, sa, sb)
        ref = (qa.double() * sa.double().unsqueeze(1)) @ (qb.double() * sb.double().unsqueeze(1)).t()
    else:
        c, status = _comms.ops.gemm_bf16_nt(a, b)
        ref = a.double() @ b.double().t()
    assert int(status[0]) == 0
    # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 1/4 before it.
    torch.testing.assert_close(c.double(), ref, rtol=2**-8, atol=1e-6 * k)


@pytest.mark.parametrize("m,n,k", [(128, 3584, 4096), (128, 4096, 1792), (5, 4096, 4096), (100, 1032, 2056)])
def test_gemm_split_repeats_and_rounds_no_worse(m, n, k):
    """The same bits at every call; no more results away from the exact product's bf16 value than the kernel that adds
    up K in one chain has (sums are closer, so the reverse holds by a wide margin), and each next to it."""
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    c = _comms.ops.gemm_bf16_nt(a, b)[0]
    for _ in range(20):
        assert torch.equal(_comms.ops.gemm_bf16_nt(a, b)[0], c)
    exact = a.double() @ b.double().t()
    rounded = exact.to(torch.bfloat16)
    chain = _comms.ops.gemm_bf16_nt_pair(a, b)[0]
    assert int((c != rounded).sum()) <= int((chain != rounded).sum())
    # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 0.02 before it.
    torch.testing.assert_close(c.double(), exact, rtol=2**-8, atol=2e-8 * k)


@pytest.mark.parametrize("m,n,k", [(5, 1024, 2048), (700, 4096, 256)])
def test_gemm_in_a_graph_clears_its_status(m, n, k):
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(k)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    want, status = _comms.ops.gemm_bf16_nt(a, b)
    assert not status.any()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c, status = _comms.ops.gemm_bf16_nt(a, b)
    for _ in range(2):
        status.fill_(7)
        c.zero_()
        graph.replay()
        assert torch.equal(c, want) and not status.any()


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (512, 512, 1024), (300, 264, 200), (1024, 7168, 2048), (4096, 4096, 4096),
                                   (8192, 1792, 512)])
def test_gemm_bf16_nt_cta_pairs(m, n, k):
    """Same product on clusters of two CTAs (tcgen05 cta_group::2)."""
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    for _ in range(2):
        c, status = _comms.ops.gemm_bf16_nt_pair(a, b)
        torch.cuda.synchronize()
        assert int(status[0]) == 0, "a bounded wait inside the kernel ran out"
        ref = a.float() @ b.float().t()
        torch.testing.assert_close(c.float(), ref, rtol=2e-2, atol=2e-2 * (k ** 0.5))
