"""Loss and gradients of a head on the logits kernel: edges of its tiles and vectors, chunks, ignored rows."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _head(rows, dim, vocab, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(rows, dim, generator=g, device="cuda").bfloat16()
    w = (torch.randn(vocab, dim, generator=g, device="cuda") * 0.3).bfloat16()
    t = torch.randint(vocab, (rows,), generator=g, device="cuda")
    return x, w, t


def _reference(x, w, t):
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    loss = F.cross_entropy(xd @ wd.t(), t, reduction="none", ignore_index=-1).sum() / x.shape[0]
    return (loss.detach(), *torch.autograd.grad(loss, (xd, wd)))


@pytest.mark.parametrize("rows,dim,vocab", [(1, 8, 1), (3, 64, 7), (127, 72, 8), (128, 64, 9), (129, 136, 127), (257, 64, 129),
                                            (255, 64, 255), (256, 64, 257), (513, 200, 4095), (700, 64, 4097), (33, 264, 16385),
                                            (2049, 64, 1000), (20, 64, 40003), (1030, 128, 9475)])
def test_head_against_64_bits(rows, dim, vocab):
    from torchcomms_b200 import _comms

    x, w, t = _head(rows, dim, vocab, 5)
    t[-1], t[0] = vocab - 1, 0
    t[rows // 3] = -1
    ref = _reference(x, w, t)
    for chunk in (4096, 100):
        out = _comms.ops.head(x, w, t, chunk)
        # Sums of `dim` products in fp32: dim x 2^-24 of the products' magnitudes, which are below 0.3 sqrt(dim) x 5 here;
        # then fp32 exponentials and sums, 1e-5 as for the loss kernel that makes its own statistics.
        assert abs(float(out[0].double() - ref[0])) < 1e-5 + dim**1.5 * 1.5 * 2**-24
        # bf16 logits off by 2^-9 of up to 0.3 sqrt(dim) x 5 move a probability by as much; their gradients and the results
        # are rounded to 2^-9. One number in a row of one has nothing to average over, hence the maximum, not a norm.
        for a, b in zip(out[1:], ref[1:]):
            assert float((a.double() - b).norm()) <= (2**-8 + 2**-9 * 1.5 * dim**0.5) * float(b.norm()) + 1e-12
    again = _comms.ops.head(x, w, t, 4096)
    assert all(torch.equal(a, b) for a, b in zip(again, _comms.ops.head(x, w, t, 4096)))  # the same bits every time


# Large weights and few rows, or a last unit of 256 rows that is mostly empty: the logits of the tensor library's product; a chunk
# of each kind.
@pytest.mark.parametrize("rows,chunk,vocab", [(20, 4096, 65544), (556, 300, 65549)])
def test_head_of_few_rows_and_large_weights(rows, chunk, vocab):
    from torchcomms_b200 import _comms

    x, w, t = _head(rows, 2112, vocab, 8)
    w = w * 0.1
    t[-1], t[0], t[rows // 3] = vocab - 1, 0, -1
    ref = _reference(x, w, t)
    out = _comms.ops.head(x, w, t, chunk)
    # bf16 logits, of 0.03 sqrt(dim) x 5 at most, are 2^-9 of that off; gradients as above.
    assert abs(float(out[0].double() - ref[0])) < 2**-9 * 0.15 * 2112**0.5
    for a, b in zip(out[1:], ref[1:]):
        assert float((a.double() - b).norm()) <= (2**-8 + 2**-9 * 0.15 * 2112**0.5) * float(b.norm())
    loss = _comms.ops.head(x, w, torch.full_like(t, -1), chunk)[0]
    assert loss.shape == () and float(loss) == 0


@pytest.mark.parametrize("rows,vocab", [(40, 1), (1, 9)])
def test_head_of_single_rows_of_any_stride(rows, vocab):
    """A row by itself is contiguous whatever its stride says."""
    from torchcomms_b200 import _comms

    x, w, t = _head(rows, 64, vocab, 11)
    odd = [v.as_strided(v.shape, (1, 1)) if v.shape[0] == 1 else v for v in (x, w)]
    assert all(v.is_contiguous() for v in odd)
    for a, b in zip(_comms.ops.head(x, w, t, 4096), _comms.ops.head(*odd, t, 4096)):
        assert torch.equal(a, b)


def test_head_all_rows_ignored_and_infinities():
    from torchcomms_b200 import _comms

    x, w, t = _head(300, 64, 1003, 6)
    loss, dx, dw = _comms.ops.head(x, w, torch.full_like(t, -1), 4096)
    assert float(loss) == 0 and not dx.any() and not dw.any()
    loss, dx, dw = _comms.ops.head(x, w, torch.full_like(t, 1003), 4096)  # past the vocabulary, as in the loss kernel
    assert float(loss) == 0 and not dx.any() and not dw.any()
    x[7, 3] = float("inf")
    loss, dx, _ = _comms.ops.head(x, w, t, 4096)
    bad = torch.isnan(dx.float()).any(dim=1)
    assert torch.isnan(loss) and bool(bad[7]) and int(bad.sum()) == 1  # its own row, as with separate operators


def _by_operators(x, w, t):
    """Gradients by one product of logits, the loss kernel on them, and two products."""
    from torchcomms_b200 import _comms

    logits = x @ w.t()
    _comms.ops.cross_entropy_fwd_bwd_(logits, t, 1.0 / x.shape[0])
    return logits @ w, logits.t() @ x


# Targets that the model has learnt to a degree, up to rows whose gradient all but vanishes, and targets at random among logits of
# 12 to several hundred; by the logits kernel and by the tensor library's product.
@pytest.mark.parametrize("rows,dim,vocab,learnt,scale", [
    (200, 256, 8000, True, 0.05), (200, 256, 8000, True, 0.08), (128, 256, 8000, True, 0.06), (33, 512, 16385, True, 0.03),
    (200, 64, 2051, False, 1.0), (200, 64, 2051, False, 30.0), (200, 64, 2051, False, 100.0),
    (20, 2112, 65544, True, 0.008), (300, 2112, 65544, True, 0.01), (20, 2112, 65544, False, 10.0)])
def test_head_normalises_what_it_differentiates(rows, dim, vocab, learnt, scale):
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(9)
    w = torch.randn(vocab, dim, generator=g, device="cuda").bfloat16()
    t = torch.randint(vocab, (rows,), generator=g, device="cuda")
    if learnt:
        x = (w[t].float() * scale).bfloat16()
    else:
        x, w = (torch.randn(rows, dim, generator=g, device="cuda") * scale).bfloat16(), (w.float() * 0.3).bfloat16()
    ref = _reference(x, w, t)
    out = _comms.ops.head(x, w, t, 4096)
    # Both round the logits to bf16 and normalise what came out, so that a probability near one stays one and its gradient
    # small: the same error, but for sums in another order that fall to the other side of a tie.
    for a, b, r in zip(out[1:], _by_operators(x, w, t), ref[1:]):
        mine, theirs = float((a.double() - r).norm()), float((b.double() - r).norm())
        assert mine <= 2 * theirs + 1e-6 * float(r.norm())


@pytest.mark.parametrize("vocab", [2051, 8000, 1048600])
@pytest.mark.parametrize("scale", [0.02, 0.06, 1.0])
def test_probabilities_of_a_row_sum_to_one(vocab, scale):
    """Rows that are unit vectors in columns where the weight is zero have the gradient of their logits in those columns of dw."""
    from torchcomms_b200 import _comms

    rows, dim = 128, 512
    g = torch.Generator(device="cuda").manual_seed(10)
    w = torch.randn(vocab, dim, generator=g, device="cuda").bfloat16()
    w[:, :rows] = 0
    t = torch.randint(vocab, (rows,), generator=g, device="cuda")
    x = (w[t].float() * scale).bfloat16()
    x[:, :rows] = torch.eye(rows, device="cuda")
    dlogits = _comms.ops.head(x, w, t, 4096)[2][:, :rows].t().double() * rows
    # A gradient is rounded to bf16, half an ulp of 2^-8 at most; before that fp32 exponentials and sums.
    assert bool((dlogits.sum(dim=1).abs() <= 1e-3 + 2**-9 * dlogits.abs().sum(dim=1)).all())
    assert float(dlogits.abs().max()) <= 1 + 1e-3


def test_head_of_large_logits():
    """Logits whose exponentials overflow by themselves, and rows with one logit far above the rest."""
    from torchcomms_b200 import _comms

    x, w, t = _head(200, 64, 2051, 7)
    x *= 100
    ref = _reference(x, w, t)
    loss, _, _ = _comms.ops.head(x, w, t, 4096)
    # fp32 logits of up to 1500: 2^-24 of that, 64 times over in the worst order
    assert abs(float(loss.double() - ref[0])) < 1500 * 64 * 2**-24


@pytest.mark.parametrize("vocab", [99, 2051])
@pytest.mark.parametrize("scale", [0.3, 3.0, 30.0, 1e30])
def test_head_loss_of_unrounded_logits(vocab, scale):
    """Around the line at which the loss takes exponentials of what rounding took off, and with logits far below all others."""
    from torchcomms_b200 import _comms

    x, w, t = _head(130, 64, vocab, 12)
    x[:, 0], w[:, 0] = 1, 0
    w[::7, 0] = -scale if scale < 1e3 else -1e30  # lows: no exponential is left of them at the last scale
    t = t // 7 * 7 + 1 if scale > 1e3 else t
    t.clamp_(max=vocab - 2)
    if scale > 1e3:
        t[t % 7 == 0] += 1
    else:
        x[:, 1:] *= scale
    ref = _reference(x, w, t)
    out = _comms.ops.head(x, w, t, 4096)
    size = float((x.double().abs() @ w.double().abs().t())[:, 1::7].max()) if scale < 1e3 else 1.5 * 64**0.5
    # Products of that size in sum, 2^-24 of it per addition in the worst order; exponentials and sums as above.
    assert abs(float(out[0].double() - ref[0])) < 1e-5 + 64 * size * 2**-24
    for a, b in zip(out[1:], ref[1:]):
        assert bool(a.isfinite().all()) and float((a.double() - b).norm()) <= 0.1 * float(b.norm())
    # A logit of minus infinity has no probability.
    w[5], w[5, 0], t[t == 5] = 0, float("-inf"), 6
    assert abs(float(_comms.ops.head(x, w, t, 4096)[0].double() - _reference(x, w, t)[0])) < 1e-5 + 64 * size * 2**-24


def test_what_the_head_leaves_to_operators():
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    x, w, t = _head(40, 64, 99, 8)
    assert _comms.ops.head(x, w, t, 4096) is not None
    assert _comms.ops.head(x[:, :63], w[:, :63], t, 4096) is None                      # strides
    assert _comms.ops.head(x[:, :60].contiguous(), w[:, :60].contiguous(), t, 4096) is None  # no multiple of 8
    assert _comms.ops.head(x.float(), w.float(), t, 4096) is None
    assert _comms.ops.head(x, w, t.int(), 4096) is None
    with torch.autocast("cuda", torch.bfloat16):
        assert _comms.ops.head(x, w, t, 4096) is None
    for cols in (64, 60):  # both ways through the public entry point
        xs, ws = x[:, :cols].contiguous().requires_grad_(True), w[:, :cols].contiguous().requires_grad_(True)
        loss = fused.linear_cross_entropy(xs, ws, t)
        dx, dw = torch.autograd.grad(loss, (xs, ws))
        ref = _reference(xs.detach(), ws.detach(), t)
        assert abs(float(loss.detach().double() - ref[0])) < 2e-2  # the operators' logits are rounded first
        for a, b in zip((dx, dw), ref[1:]):
            assert float((a.double() - b).norm() / b.norm()) < 2**-8 + 2**-9 * 12
