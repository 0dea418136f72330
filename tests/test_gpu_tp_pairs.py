"""The fused tensor-parallel kernels on CTA pairs, with 1, 2 and 4 ranks in one launch, against 64-bit products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(rows, cols, seed, scale, fp8):
    """What the kernel reads, its row scales, and the values that the two stand for."""
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn(rows, cols, generator=g, device="cuda") * scale).to(torch.bfloat16)
    if not fp8:
        return x, None, x.double()
    q, s = quantize_rows(x)
    return q, s, q.double() * s.double().unsqueeze(1)


# One pair tile per rank; several source tiles and column tiles; more pair tiles than a rank has pairs.
@pytest.mark.parametrize("nranks,m_local,n,k", [(1, 256, 256, 128), (2, 256, 512, 1024), (2, 1280, 2304, 256), (4, 512, 768, 640), (4, 1024, 2560, 128)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gather_gemm(nranks, m_local, n, k, fp8):
    from torchcomms_b200 import _comms

    world = _comms.TpEmuWorld(nranks, "ag_gemm", m_local, k, 5000.0, fp8, pairs=True)
    for it in range(3):
        xs = [_operands(m_local, k, 100 * it + r, 1.0, fp8) for r in range(nranks)]
        ws = [_operands(n, k, 100 * it + 50 + r, 0.05, fp8) for r in range(nranks)]
        for r in range(nranks):
            world.input(r).copy_(xs[r][0])
            if fp8:
                world.input_scales(r).copy_(xs[r][1])
        ys = world.ag_gemm([w[0] for w in ws], [w[1] for w in ws] if fp8 else [])
        torch.cuda.synchronize()
        assert world.status()[0] == 0, world.status()
        full = torch.cat([x[2] for x in xs])
        for r in range(nranks):
            # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 0.05 before it.
            torch.testing.assert_close(ys[r].double(), full @ ws[r][2].t(), rtol=2**-8, atol=5e-8 * k)


@pytest.mark.parametrize("nranks,m_local,n,k", [(1, 256, 256, 128), (2, 256, 512, 1024), (2, 1280, 2304, 256), (4, 512, 768, 640), (4, 1024, 2560, 128)])
@pytest.mark.parametrize("fp8", [False, True])
def test_gemm_scatter(nranks, m_local, n, k, fp8):
    from torchcomms_b200 import _comms

    m = m_local * nranks
    world = _comms.TpEmuWorld(nranks, "gemm_rs", m, n, 5000.0, fp8, pairs=True)
    for it in range(3):
        hs = [_operands(m, k, 200 * it + r, 1.0, fp8) for r in range(nranks)]
        ws = [_operands(n, k, 200 * it + 50 + r, 0.05, fp8) for r in range(nranks)]
        scales = ([h[1] for h in hs], [w[1] for w in ws]) if fp8 else ([], [])
        outs = world.gemm_rs([h[0] for h in hs], [w[0] for w in ws], *scales)
        torch.cuda.synchronize()
        assert world.status()[0] == 0, world.status()
        parts = [h[2] @ w[2].t() for h, w in zip(hs, ws)]
        total = sum(parts)
        # Each rank's share travels in bf16 and the sum is rounded once more (2^-9 relative each), and the sums over k.
        bound = 2**-8 * (sum(p.abs() for p in parts) + total.abs()) + 5e-8 * k * nranks
        for r in range(nranks):
            rows = slice(r * m_local, (r + 1) * m_local)
            assert bool(((outs[r].double() - total[rows]).abs() <= bound[rows]).all())


def test_shards_off_the_pair_tiles_are_refused():
    from torchcomms_b200 import _comms

    world = _comms.TpEmuWorld(2, "gemm_rs", 256, 256, 100.0, pairs=True)
    h, w = (torch.zeros(256, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    with pytest.raises(RuntimeError):
        world.gemm_rs([h, h], [w, w])
