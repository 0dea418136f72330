"""Products whose K is shared by a cluster: every cluster size, row and column remainders, against a 64-bit product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# Column tiles of 128 that leave room for clusters of 8, 5, 4, 3, 2 and 1; the last tile whole, 8 or 104 columns wide; K in
# equal and unequal shares, on the 128-byte lines and off them.
@pytest.mark.parametrize("n", [128, 1928, 2560, 3432, 4096, 5640, 6144, 9096, 9472, 18824])
@pytest.mark.parametrize("k", [2048, 2072])
@pytest.mark.parametrize("m", [1, 33, 100, 128])
@pytest.mark.parametrize("fp8", [False, True])
def test_shared_product(m, n, k, fp8):
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    k = 2 * k if fp8 else k
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    if fp8:
        (qa, sa), (qb, sb) = quantize_rows(a), quantize_rows(b)
        ref = (qa.double() * sa.double().unsqueeze(1)) @ (qb.double() * sb.double().unsqueeze(1)).t()
        run = lambda: _comms.ops.gemm_e4m3_nt(qa, qb, sa, sb)
    else:
        ref = a.double() @ b.double().t()
        run = lambda: _comms.ops.gemm_bf16_nt(a, b)
    c, status = run()
    assert not status.any()
    # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 1/4 before it.
    torch.testing.assert_close(c.double(), ref, rtol=2**-8, atol=1e-6 * k)
    for _ in range(3):
        assert torch.equal(run()[0], c)
