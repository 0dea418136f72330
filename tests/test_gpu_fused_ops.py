"""Numerics of the fused model kernels against plain PyTorch fp32 references,
and the training engine on one GPU."""
import os

import pytest
import torch
import torch.nn.functional as F
import torch.utils.checkpoint

pytestmark = pytest.mark.gpu


def _bf(*shape, seed=0, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("rows,cols", [(5, 64), (300, 4096), (17, 8192), (4, 16384)])
def test_rmsnorm_forward_backward(rows, cols):
    from torchcomms_b200.ops import fused

    x = _bf(rows, cols, seed=1).requires_grad_(True)
    w = (_bf(cols, seed=2, scale=0.1) + 1).detach().requires_grad_(True)
    y = fused.rms_norm(x, w, 1e-5)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + 1e-5) * wf
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    if cols <= 8192:
        dy = _bf(rows, cols, seed=3)
        y.backward(dy)
        ref.backward(dy.float())
        torch.testing.assert_close(x.grad.float(), xf.grad, rtol=3e-2, atol=3e-2)
        torch.testing.assert_close(w.grad.float(), wf.grad, rtol=3e-2, atol=3e-2 * max(1.0, rows ** 0.5))


@pytest.mark.parametrize("cols", [8, 256, 264, 512, 1000, 1024, 1032, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("rows", [1, 4, 9, 74, 75, 148, 149, 1200, 2377])
def test_rmsnorm_row_layouts(rows, cols):
    """Every split of a row over threads, at its edges, with fewer and more rows than row groups on the GPU."""
    from torchcomms_b200 import _comms

    x, dy, w = _bf(rows, cols, seed=1), _bf(rows, cols, seed=2), _bf(cols, seed=3, scale=0.1) + 1
    y, rstd = _comms.ops.rmsnorm_fwd(x, w, 1e-5)
    dx, dw = _comms.ops.rmsnorm_bwd(dy, x, w, rstd)
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    rdx, rdw = torch.autograd.grad(ref, (xd, wd), dy.double())
    # Half a bf16 ulp (2^-9 relative) and fp32 sums of up to 8192 (dx) or `rows` (dw) terms of unit size before it.
    torch.testing.assert_close(y.double(), ref.detach(), rtol=2**-8, atol=1e-6)
    torch.testing.assert_close(dx.double(), rdx, rtol=2**-8, atol=2e-5)
    torch.testing.assert_close(dw.double(), rdw, rtol=2**-8, atol=1e-6 * rows**0.5 + 2e-5)


@pytest.mark.parametrize("cols", [8200, 10240, 10248, 16384, 40008])
@pytest.mark.parametrize("rows", [1, 1300])
def test_rmsnorm_forward_wide_rows(rows, cols):
    """Rows that the registers do not hold, from one vector past them on, with fewer and more rows than blocks."""
    from torchcomms_b200 import _comms

    x, w = _bf(rows, cols, seed=77), _bf(cols, seed=78, scale=0.1) + 1
    y, rstd = _comms.ops.rmsnorm_fwd(x, w, 1e-5)
    ref = torch.rsqrt(x.double().pow(2).mean(-1) + 1e-5)
    # fp32 sums of up to 40008 squares; half a bf16 ulp (2^-9 relative) on the result.
    torch.testing.assert_close(rstd.double(), ref, rtol=5e-6, atol=0)
    torch.testing.assert_close(y.double(), x.double() * ref.unsqueeze(1) * w.double(), rtol=2**-8, atol=1e-6)


def test_swiglu_forward_backward():
    from torchcomms_b200.ops import fused

    gu = _bf(33, 2 * 1024, seed=4).requires_grad_(True)
    h = fused.swiglu(gu)
    guf = gu.detach().float().requires_grad_(True)
    g, u = guf.chunk(2, dim=-1)
    ref = F.silu(g) * u
    torch.testing.assert_close(h.float(), ref, rtol=2e-2, atol=2e-2)
    dh = _bf(33, 1024, seed=5)
    h.backward(dh)
    ref.backward(dh.float())
    torch.testing.assert_close(gu.grad.float(), guf.grad, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("rows,ffn", [(1, 8), (3, 264), (511, 8), (1025, 520), (7, 14336), (592, 4096), (593, 4096), (2500, 1000)])
def test_swiglu_every_vector(rows, ffn):
    """Row lengths that end anywhere in a block's span of vectors, one and two vectors per thread."""
    from torchcomms_b200 import _comms

    gu, dh = _bf(rows, 2 * ffn, seed=4, scale=3.0), _bf(rows, ffn, seed=5)
    gud = gu.double().requires_grad_(True)
    g, u = gud.chunk(2, dim=-1)
    ref = F.silu(g) * u
    (rdgu,) = torch.autograd.grad(ref, gud, dh.double())
    # Half a bf16 ulp (2^-9 relative); the derivative of silu crosses zero, where fp32 terms of size 30 cancel.
    torch.testing.assert_close(_comms.ops.swiglu_fwd(gu).double(), ref.detach(), rtol=2**-8, atol=1e-6)
    torch.testing.assert_close(_comms.ops.swiglu_bwd(dh, gu).double(), rdgu, rtol=2**-8, atol=2e-5)


def test_rope_matches_complex_rotation_and_inverts():
    from torchcomms_b200.ops import fused

    tokens, heads, hd = 50, 4, 128
    cos_t, sin_t = fused.rope_tables(64, hd, 500000.0, "cuda")
    pos = torch.arange(tokens, dtype=torch.int32, device="cuda") % 64
    x = _bf(tokens, heads, hd, seed=6).requires_grad_(True)
    y = fused.apply_rope(x, pos, cos_t, sin_t)
    xc = torch.view_as_complex(x.detach().float().reshape(tokens, heads, hd // 2, 2))
    rot = torch.polar(torch.ones_like(cos_t), torch.atan2(sin_t, cos_t))[pos.long()].unsqueeze(1)
    ref = torch.view_as_real(xc * rot).reshape(tokens, heads, hd)
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    # the backward is the inverse rotation: rotating the output gradient back
    y.backward(y.detach())
    torch.testing.assert_close(x.grad.float(), x.detach().float(), rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("tokens,heads,hd", [(1, 1, 8), (3, 5, 96), (31, 1, 256), (257, 8, 64), (1025, 4, 128)])
@pytest.mark.parametrize("layout", ["slice", "transposed", "expanded", "odd_offset"])
def test_rope_reads_strided_inputs(tokens, heads, hd, layout):
    from torchcomms_b200.ops import fused

    cos_t, sin_t = fused.rope_tables(2048, hd, 10000.0, "cuda")
    pos = torch.randint(0, 2048, (tokens,), dtype=torch.int32, device="cuda")
    if layout == "slice":
        x = _bf(tokens, (heads + 2) * hd, seed=6)[:, hd : (heads + 1) * hd].reshape(tokens, heads, hd)
    elif layout == "transposed":
        x = _bf(heads, tokens, hd, seed=6).transpose(0, 1)
    elif layout == "expanded":
        x = _bf(tokens, 1, hd, seed=6).expand(tokens, heads, hd)
    else:
        x = _bf(tokens * heads * hd + 1, seed=6)[1:].view(tokens, heads, hd)
    x = x.detach().requires_grad_(True)
    y = fused.apply_rope(x, pos, cos_t, sin_t)
    (dx,) = torch.autograd.grad(y, x, _bf(heads, tokens, hd, seed=7).transpose(0, 1))
    assert y.is_contiguous()

    def rotate(t, sign):
        a, b = t.float().unflatten(-1, (-1, 2)).unbind(-1)
        c, s = cos_t[pos.long()].unsqueeze(1), sign * sin_t[pos.long()].unsqueeze(1)
        return torch.stack((a * c - b * s, a * s + b * c), dim=-1).flatten(-2)

    # One rounding to bf16 of a two-term fp32 sum: half a unit in the last place (2^-9), plus cancellation noise.
    torch.testing.assert_close(y.float(), rotate(x.detach(), 1.0), rtol=2**-8, atol=2e-6)
    torch.testing.assert_close(dx.float(), rotate(_bf(heads, tokens, hd, seed=7).transpose(0, 1), -1.0), rtol=2**-8, atol=2e-6)


@pytest.mark.parametrize("rows,vocab", [(7, 1000), (64, 32003), (9, 128256)])
def test_cross_entropy_loss_and_gradient(rows, vocab):
    from torchcomms_b200 import _comms

    logits = _bf(rows, vocab, seed=7, scale=2.0)
    targets = torch.randint(0, vocab, (rows,), device="cuda")
    targets[0] = -1  # ignored row
    lf = logits.float().requires_grad_(True)
    ref = F.cross_entropy(lf, targets, reduction="none", ignore_index=-1)
    (ref.sum() * 0.25).backward()
    work = logits.clone()
    loss = _comms.ops.cross_entropy_fwd_bwd_(work, targets, 0.25)
    torch.testing.assert_close(loss, ref.detach(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(work.float(), lf.grad, rtol=3e-2, atol=2e-3)


@pytest.mark.parametrize("rows,vocab", [(r, v) for r in (1, 300, 1300) for v in (1, 7, 9, 16, 23, 4096, 4097, 16384, 16391, 40003)]
                         + [(r, v) for r in (1, 130) for v in (60007, 128256, 131071, 200001, 300007)])
def test_cross_entropy_row_layouts(rows, vocab):
    """Heads and tails of rows that start off a 16-byte boundary, every block size, targets at both ends, and rows with
    masked (-inf, lowest finite) logits."""
    from torchcomms_b200 import _comms

    logits = _bf(rows, vocab, seed=11, scale=3.0)
    targets = torch.randint(0, vocab, (rows,), device="cuda")
    targets[-1], targets[0] = vocab - 1, 0
    if rows > 8 and vocab > 8:
        logits[1, 1:] = float("-inf")                        # one allowed token
        targets[1] = 0
        logits[2, : vocab // 2] = float("-inf")
        targets[2] = vocab - 1
        logits[3] = torch.finfo(torch.bfloat16).min          # everything masked with the lowest value
        logits[4, : vocab // 2] = torch.finfo(torch.bfloat16).min
        targets[4] = vocab - 1
        logits[5] -= 30.0
        targets[6] = -1
        targets[7] = vocab
    ld = logits.double()
    keep = ((targets >= 0) & (targets < vocab)).double()
    logp = torch.log_softmax(ld, dim=-1)
    at = targets.clamp(0, vocab - 1).unsqueeze(1)
    ref_loss = -logp.gather(1, at).squeeze(1) * keep
    ref = (logp.exp() - torch.zeros_like(ld).scatter_(1, at, 1.0)) * (0.5 * keep).unsqueeze(1)
    loss = _comms.ops.cross_entropy_fwd_bwd_(logits, targets, 0.5)
    if rows > 8 and vocab > 8:  # a row without any allowed token has no meaningful value, but stays finite
        assert torch.isfinite(loss[3]) and torch.isfinite(logits[3].float()).all()
        loss, ref_loss, logits, ref, at, keep = (torch.cat((t[:3], t[4:])) for t in (loss, ref_loss, logits, ref, at, keep))
    # fp32 sums of up to 300007 exponentials
    torch.testing.assert_close(loss.double(), ref_loss, rtol=2e-6, atol=1e-5)
    # At the target p - 1 cancels to the error of the fp32 sum and exponential (1e-5); everywhere else the gradient is
    # p / 2, as small as 1e-9, with a relative error of an fp32 exponential of arguments up to 64 (64 x 2^-23 < 1e-5) and
    # of one bf16 rounding (2^-9). Rows without a target have none.
    torch.testing.assert_close(logits.gather(1, at).double(), ref.gather(1, at), rtol=2**-8, atol=1e-5)
    rest, rest_ref = logits.double().scatter_(1, at, 0.0), ref.scatter_(1, at, 0.0)
    torch.testing.assert_close(rest, rest_ref, rtol=2**-8, atol=1e-12)
    assert not rest[keep == 0].any()


@pytest.mark.parametrize("rows,dim,vocab", [(1, 64, 9), (130, 128, 5001), (70, 256, 40002), (130, 640, 40001), (257, 64, 1000),
                                            (2, 256, 98305), (512, 512, 13107), (512, 512, 13109), (3000, 256, 5365)])
def test_linear_cross_entropy_any_vocabulary(rows, dim, vocab):
    """Vocabularies off the 16-byte grid (from some sizes on with a padded weight, both sides of the line here) and on
    it, in one and in several chunks."""
    from torchcomms_b200.ops import fused

    x, w = _bf(rows, dim, seed=60).requires_grad_(True), _bf(vocab, dim, seed=61, scale=0.1).requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda")
    t[-1] = vocab - 1
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    ref = F.cross_entropy(xd @ wd.t(), t)
    rx, rw = torch.autograd.grad(ref, (xd, wd))
    for chunk in (4096, 100):
        loss = fused.linear_cross_entropy(x, w, t, chunk)
        dx, dw = torch.autograd.grad(loss, (x, w))
        # bf16 logits of size up to 5 (2^-9 x 5 absolute) enter the loss, bf16 logit gradients the sums.
        torch.testing.assert_close(loss.double(), ref.detach(), rtol=0, atol=1e-2)
        assert float((dx.double() - rx).norm() / rx.norm()) < 1e-2
        assert float((dw.double() - rw).norm() / rw.norm()) < 1e-2


@pytest.mark.parametrize("numel", [1, 8, 4099, 3_000_001])
def test_scale_by_matches_operators(numel):
    from torchcomms_b200 import _comms

    t = _bf(numel, seed=12)
    for value in (1.0, -0.3337, 0.0, float("inf")):
        f = torch.tensor(value, device="cuda")
        torch.testing.assert_close(_comms.ops.scale_by(t, f), t * f.to(t.dtype), rtol=0, atol=0, equal_nan=True)
    w = t[: numel // 2 * 2].view(-1, 2).t() if numel > 1 else t.view(1, 1)
    assert torch.equal(_comms.ops.scale_by(w, torch.tensor(2.0, device="cuda")), w * 2)
    assert _comms.ops.scale_by(w, torch.tensor(2.0, device="cuda")).stride() == (w * 2).stride()
    g = torch.tensor(3.0, device="cuda", requires_grad=True)
    assert _comms.ops.scale_by(t, g).requires_grad  # a gradient of the gradient keeps its graph


# Two tensors in one launch, the grid that of the larger: either one the larger, below a vector, empty.
@pytest.mark.parametrize("first,second", [(1, 3_000_001), (3_000_001, 7), (0, 4099), (4099, 0), (8, 8), (0, 0)])
@pytest.mark.parametrize("consume", [False, True])
def test_scale_both_by_matches_operators(first, second, consume):
    from torchcomms_b200 import _comms

    for value in (1.0, -0.3337, 0.0, float("inf")):
        t, u, f = _bf(first, seed=12), _bf(second, seed=13), torch.tensor(value, device="cuda")
        want = [v * f.to(v.dtype) for v in (t, u)]
        got = _comms.ops.scale_both_by(t, u, f, consume)
        for v, a, b in zip((t, u), got, want):
            torch.testing.assert_close(a, b, rtol=0, atol=0, equal_nan=True)
            assert v.numel() == 0 or (a.data_ptr() == v.data_ptr()) == consume
    # what the kernel does not take: strides of a transposed matrix it does, a view off the grid and a factor with a gradient it does not
    m, odd, f = _bf(6, 10, seed=14).t(), _bf(4100, seed=15)[1:], torch.tensor(-0.5, device="cuda")
    a, b = _comms.ops.scale_both_by(m, odd, f, False)
    assert torch.equal(a, m * -0.5) and a.stride() == (m * 1).stride() and torch.equal(b, odd * -0.5)
    g = torch.tensor(3.0, device="cuda", requires_grad=True)
    assert all(v.requires_grad for v in _comms.ops.scale_both_by(m, odd, g, consume))


def test_linear_cross_entropy_matches_unfused():
    from torchcomms_b200.ops import fused

    rows, dim, vocab = 300, 256, 5000
    x = _bf(rows, dim, seed=8).requires_grad_(True)
    w = _bf(vocab, dim, seed=9, scale=0.05).requires_grad_(True)
    t = torch.randint(0, vocab, (rows,), device="cuda")
    loss = fused.linear_cross_entropy(x, w, t, chunk_rows=128)
    loss.backward()
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    ref = F.cross_entropy(xf @ wf.t(), t)
    ref.backward()
    torch.testing.assert_close(loss, ref.detach(), rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(x.grad.float(), xf.grad, rtol=5e-2, atol=2e-4)
    torch.testing.assert_close(w.grad.float(), wf.grad, rtol=5e-2, atol=2e-4)


@pytest.mark.parametrize("n", [1, 100_003, 454_659, 454_660, 600_001])
def test_adamw_matches_torch(n):
    from torchcomms_b200.ops import fused

    p = torch.randn(n, device="cuda")
    g = torch.randn(n, device="cuda")
    ref_p = p.clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for step in range(1, 4):
        ref_p.grad = g.clone()
        opt.step()
        fused.adamw_step_(p, g, m, v, lr=1e-2, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=step)
    torch.testing.assert_close(p, ref_p.detach(), rtol=1e-4, atol=1e-5)


def test_adamw_refuses_shards_off_the_vector_grid():
    """Updated in place, so a shard at an odd offset cannot be copied: an error, and nothing is launched. Three elements
    use no vectors and go anywhere."""
    from torchcomms_b200.ops import fused

    ts = [torch.zeros(65, device="cuda") for _ in range(4)]
    for i in range(4):
        with pytest.raises(RuntimeError):
            fused.adamw_step_(*(t[1:] if k == i else t[:64] for k, t in enumerate(ts)), lr=0.1, step=1)
    before = [t.clone() for t in ts]
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(before, ts))
    ts[1].fill_(1.0)
    fused.adamw_step_(*(t[1:4] for t in ts), lr=0.1, step=1)
    assert bool((ts[0][1:4] < 0).all()) and not ts[0][0] and not ts[0][4:].any()


@pytest.mark.parametrize("rows,cols", [(1, 8), (9, 256), (40, 512), (80, 512), (140, 776), (700, 1000), (5, 2048), (601, 4096), (3, 8192), (300, 8192)])
def test_norm_with_residual_stream(rows, cols):
    """x + delta and its norm in one kernel: forward bit for bit what addition and norm give, backward with the
    residual's gradient added in fp32."""
    from torchcomms_b200.ops import fused

    w = (_bf(cols, seed=42, scale=0.1) + 1).detach().requires_grad_(True)
    x, d = _bf(rows, cols, seed=40).requires_grad_(True), _bf(rows, cols, seed=41).requires_grad_(True)
    s, y = fused.add_rms_norm(x, d, w, 1e-5)
    assert torch.equal(s, (x + d).detach()) and torch.equal(y, fused.rms_norm((x + d).detach(), w, 1e-5))
    gs, gy = _bf(rows, cols, seed=43), _bf(rows, cols, seed=44)
    sd, wd = s.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    ref = sd * torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd
    rs, rw = torch.autograd.grad(ref, (sd, wd), gy.double())
    # Half a bf16 ulp (2^-9 relative) on top of fp32 sums of up to 8192 (ds) or `rows` (dw) terms of unit size.
    for got, skip in ((torch.autograd.grad((s, y), (x, d, w), (gs, gy)), gs.double()),):
        torch.testing.assert_close(got[0].double(), rs + skip, rtol=2**-8, atol=2e-5)
        assert torch.equal(got[0], got[1])
        torch.testing.assert_close(got[2].double(), rw, rtol=2**-8, atol=1e-6 * rows**0.5 + 2e-5)
    x2 = s.detach().requires_grad_(True)
    skip, y2 = fused.rms_norm_skip(x2, w, 1e-5)
    assert torch.equal(skip, x2) and torch.equal(y2, y)
    (dx,) = torch.autograd.grad((skip, y2), x2, (gs, gy), retain_graph=True)
    assert torch.equal(dx, got[0])
    (dx,) = torch.autograd.grad(y2, x2, gy)                        # a result nobody used counts as zero
    torch.testing.assert_close(dx.double(), rs, rtol=2**-8, atol=2e-5)


@pytest.mark.parametrize("offset", [1, 4, 7])
def test_norm_and_swiglu_at_odd_offsets(offset):
    """Contiguous views that start off a 16-byte boundary (a narrow of a flat buffer, a slice of a gradient) give the
    bits that copies of them give, for every input and incoming gradient."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    def odd(*shape, seed):
        n = 1
        for d in shape:
            n *= d
        t = _bf(n + offset, seed=seed)[offset:].view(*shape)
        assert t.is_contiguous() and t.data_ptr() % 16 != 0
        return t

    rows, cols = 37, 1032
    x, d, w = odd(rows, cols, seed=70), odd(rows, cols, seed=71), odd(cols, seed=72)
    gs, gy = odd(rows, cols, seed=73), odd(rows, cols, seed=74)
    gu, dh = odd(rows, 2 * cols, seed=75), odd(rows, cols, seed=76)

    def passes(*ts):
        x, d, w, gs, gy, gu, dh = ts
        x, d, w, gu = (t.detach().requires_grad_(True) for t in (x, d, w, gu))
        s, y = fused.add_rms_norm(x, d, w)
        out = [s, y, *torch.autograd.grad((s, y), (x, d, w), (gs, gy))]
        s, y = fused.rms_norm_skip(x, w)
        out += [s, y, *torch.autograd.grad((s, y), (x, w), (gs, gy))]
        y = fused.rms_norm(x, w)
        out += [y, *torch.autograd.grad(y, (x, w), gy)]
        h = fused.swiglu(gu)
        out += [h, *torch.autograd.grad(h, gu, dh)]
        y, rstd = _comms.ops.rmsnorm_fwd(x, w, 1e-5)
        out += [y, rstd, *_comms.ops.rmsnorm_bwd(gy, x, w, rstd), _comms.ops.swiglu_fwd(gu), _comms.ops.swiglu_bwd(dh, gu)]
        return out

    aligned = passes(*(t.clone() for t in (x, d, w, gs, gy, gu, dh)))
    assert all(torch.equal(a, b) for a, b in zip(passes(x, d, w, gs, gy, gu, dh), aligned))
    for i in range(7):                                             # one at a time
        ts = [t if k == i else t.clone() for k, t in enumerate((x, d, w, gs, gy, gu, dh))]
        assert all(torch.equal(a, b) for a, b in zip(passes(*ts), aligned)), i


@pytest.mark.parametrize("tokens,heads,kv,hd", [(1, 1, 1, 8), (37, 6, 2, 96), (1000, 8, 8, 64), (513, 4, 1, 128)])
@pytest.mark.parametrize("layout", ["contiguous", "transposed", "odd"])
def test_split_rope_matches_split_and_rotate(tokens, heads, kv, hd, layout):
    """Same bits as splitting the projection and rotating the pieces, in both directions, for gradients of any layout."""
    from torchcomms_b200.ops import fused

    cos_t, sin_t = fused.rope_tables(2048, hd, 10000.0, "cuda")
    pos = torch.randint(0, 2048, (tokens,), dtype=torch.int32, device="cuda")
    qkv = _bf(tokens, (heads + 2 * kv) * hd, seed=50).requires_grad_(True)
    q, k, v = qkv.split([heads * hd, kv * hd, kv * hd], dim=-1)
    want = (fused.apply_rope(q.reshape(tokens, heads, hd), pos, cos_t, sin_t),
            fused.apply_rope(k.reshape(tokens, kv, hd), pos, cos_t, sin_t), v.reshape(tokens, kv, hd))
    got = fused.split_rope(qkv, pos, cos_t, sin_t, heads, kv)
    grads = []
    for i, n in enumerate((heads, kv, kv)):
        if layout == "contiguous":
            grads.append(_bf(tokens, n, hd, seed=51 + i))
        elif layout == "transposed":
            grads.append(_bf(n, tokens, hd, seed=51 + i).transpose(0, 1))
        else:
            grads.append(_bf(tokens, n, hd + 1, seed=51 + i)[:, :, 1:])
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    (da,), (db,) = torch.autograd.grad(got, qkv, grads), torch.autograd.grad(want, qkv, grads)
    assert torch.equal(da, db)


@pytest.mark.parametrize("factor", [1.0, 0.37])
def test_linear_cross_entropy_gradients_are_handed_out_once(factor):
    """The last backward gives its gradients away in place; retained graphs, hooks and later passes get copies."""
    from torchcomms_b200.ops import fused

    x, w = _bf(64, 128, seed=30).requires_grad_(True), _bf(1000, 128, seed=31, scale=0.05).requires_grad_(True)
    t = torch.randint(0, 1000, (64,), device="cuda")
    g = torch.tensor(factor, device="cuda")
    first = torch.autograd.grad(fused.linear_cross_entropy(x, w, t), (x, w), g)
    loss = fused.linear_cross_entropy(x, w, t)
    a = torch.autograd.grad(loss, (x, w), g, retain_graph=True)
    b = torch.autograd.grad(loss, (x, w), 2 * g, retain_graph=True)
    c = torch.autograd.grad(loss, (x, w), g)
    for f, p, q, r in zip(first, a, b, c):
        assert torch.equal(f, p) and torch.equal(p, r) and p.data_ptr() != r.data_ptr()
        torch.testing.assert_close(q.float(), 2 * p.float(), rtol=2**-7, atol=0)   # two bf16 roundings apart
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda s: kept.append(s) or s, lambda s: s):
        loss = fused.linear_cross_entropy(x, w, t)
    before = [k.clone() for k in kept]
    d = torch.autograd.grad(loss, (x, w), g)
    assert all(torch.equal(k, b) for k, b in zip(kept, before)) and all(torch.equal(p, q) for p, q in zip(d, first))
    loss = fused.linear_cross_entropy(x, w, t) * factor             # reaches .grad the same way
    loss.backward()
    assert torch.equal(x.grad, first[0]) and torch.equal(w.grad, first[1])


def _op_calls():
    from torchcomms_b200.ops import fused

    cos_t, sin_t = fused.rope_tables(64, 64, 10000.0, "cuda")
    pos = torch.arange(24, dtype=torch.int32, device="cuda")
    w = (_bf(256, seed=20, scale=0.1) + 1).detach().requires_grad_(True)
    return {
        "rms_norm": (lambda x: fused.rms_norm(x, w, 1e-5), (24, 256), fused._RmsNorm, (w, 1e-5)),
        "swiglu": (lambda x: fused.swiglu(x), (24, 512), fused._SwiGlu, ()),
        "apply_rope": (lambda x: fused.apply_rope(x, pos, cos_t, sin_t), (24, 4, 64), fused._Rope, (pos, cos_t, sin_t)),
    }


@pytest.mark.parametrize("name", ["rms_norm", "swiglu", "apply_rope"])
def test_native_autograd_nodes(name):
    """Same values and gradients as the autograd functions in Python, hooks and graph modes seen alike."""
    call, shape, function, rest = _op_calls()[name]
    x = _bf(*shape, seed=21).requires_grad_(True)
    y, ref = call(x), function.apply(x, *rest)
    assert y.grad_fn.name() != ref.grad_fn.name()
    assert torch.equal(y, ref)
    g = _bf(*y.shape, seed=22)
    leaves = (x,) + tuple(t for t in rest if isinstance(t, torch.Tensor) and t.requires_grad)
    for a, b in zip(torch.autograd.grad(y, leaves, g, retain_graph=True), torch.autograd.grad(ref, leaves, g)):
        assert torch.equal(a, b)
    for a, b in zip(torch.autograd.grad(y, leaves, g, retain_graph=True), torch.autograd.grad(y, leaves, g)):
        assert torch.equal(a, b)                                   # a second pass over a retained graph
    # saved tensors go through hooks (activation checkpointing and offloading rest on them)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.clone(), lambda t: t):
        z = call(x)
    (dx,) = torch.autograd.grad(z, x, g)
    assert packed and torch.equal(dx, torch.autograd.grad(call(x), x, g)[0])
    c = torch.utils.checkpoint.checkpoint(call, x, use_reentrant=False)
    assert torch.equal(torch.autograd.grad(c, x, g)[0], dx)
    with torch.no_grad():
        assert call(x).grad_fn is None
    # inputs of any layout, and calls on another stream
    xt = _bf(*shape[:-2], shape[-1], shape[-2], seed=23).transpose(-1, -2)
    assert torch.equal(call(xt), call(xt.contiguous()))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ys = call(x)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(ys, y)
    # forward mode and vmap are refused as by the autograd functions in Python
    import torch.autograd.forward_ad as fwad

    with fwad.dual_level():
        with pytest.raises(Exception):
            call(fwad.make_dual(x.detach(), torch.ones_like(x)))
    with pytest.raises(Exception):
        torch.func.vmap(call)(x.detach().unsqueeze(0).expand(2, *shape))


def test_engine_step_on_gpu_matches_reference_forward():
    os.environ.setdefault("RANK", "0")
    os.environ.setdefault("WORLD_SIZE", "1")
    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29541")
    import torchcomms_b200 as tc
    from torchcomms_b200.models.llama import LlamaConfig
    from torchcomms_b200.ops import fused
    from torchcomms_b200.parallel.engine import TrainEngine

    comm = tc.new_comm("b200", torch.device("cuda", 0), name="engine_gpu")
    cfg = LlamaConfig.tiny()
    engine = TrainEngine(cfg, comm, lr=3e-3, weight_decay=0.0, seed=1, recompute_blocks=1)
    before = fused.kernel_launch_count()
    tokens = torch.randint(0, cfg.vocab_size, (2, 129), device="cuda")
    losses = [float(engine.step(tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous())) for _ in range(5)]
    torch.cuda.synchronize()
    assert abs(losses[0] - torch.log(torch.tensor(float(cfg.vocab_size))).item()) < 0.5, losses
    assert losses[-1] < losses[0] - 0.05, losses
    assert fused.kernel_launch_count() - before > 50  # norms, rope, swiglu, loss, adamw, gathers, reductions
    comm.finalize()
