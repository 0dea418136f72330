"""The two nodes of a decoder block against the separate operations in 64 bits: edges of the gated product's tiles, gradients
that nobody asks for, and what they leave to the separate nodes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()


def _norm64(x, w, eps=1e-5):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _off(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


# Row tiles of 256 and column tiles of 128 with and without a remainder, one column vector, depths below and above a K step; few
# rows of large weights, which take the activation kernel.
@pytest.mark.parametrize("rows,dim,ffn,width", [(1, 64, 8, 64), (127, 72, 120, 64), (256, 128, 128, 192), (257, 200, 136, 128),
                                                (300, 256, 1032, 256), (1000, 512, 2048, 512), (130, 1024, 9480, 1024),
                                                (40, 3200, 8192, 64)])
def test_block_out(rows, dim, ffn, width):
    from torchcomms_b200 import _comms

    ins = [_rand(rows, dim, seed=1), _rand(rows, width, seed=2), _rand(dim, width, seed=3, scale=width**-0.5),
           _rand(dim, seed=4, scale=0.1) + 1, _rand(2 * ffn, dim, seed=5, scale=dim**-0.5), _rand(dim, ffn, seed=6, scale=ffn**-0.5)]
    dy = _rand(rows, dim, seed=7)
    ins = [t.requires_grad_(True) for t in ins]
    y = _comms.ops.block_out(*ins, 1e-5)
    grads = torch.autograd.grad(y, ins, dy)
    wide = [t.detach().double().requires_grad_(True) for t in ins]
    x, o, wo, norm, w13, w2 = wide
    s = x + o @ wo.t()
    gate, up = (_norm64(s, norm) @ w13.t()).chunk(2, dim=-1)
    ref = s + (torch.nn.functional.silu(gate) * up) @ w2.t()
    ref_grads = torch.autograd.grad(ref, wide, dy.double())
    # Forward: seven roundings to bf16 (2^-9 each, of numbers of about the result's size); backward: three or four more on the way.
    assert _off(y.detach(), ref.detach()) < 7 * 2**-9
    for a, b in zip(grads, ref_grads):
        assert _off(a, b) < 12 * 2**-9


# The gradient of gate and up in its product's epilogue: narrow and wide tiles, their last columns and rows, a last wave in
# halves, K steps that end early; gates beyond where exponentials end, and those that are no numbers.
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (257, 136, 72), (1000, 520, 1000), (2049, 2312, 136), (300, 4808, 200)])
def test_gated_gradient(m, n, k):
    from torchcomms_b200 import _comms

    dy, w, gate_up = _rand(m, k, seed=1), _rand(k, n, seed=2, scale=k**-0.5), _rand(m, 2 * n, seed=3, scale=2.0)
    gate_up[:, 3], gate_up[:, 4], gate_up[0, 5], gate_up[0, 6] = 300.0, -300.0, float("nan"), float("-inf")
    out, status = _comms.ops.gemm_gated_grad(dy, w, gate_up)
    assert int(status[0]) == 0 and torch.equal(out.isnan(), _comms.ops.swiglu_bwd(_comms.ops.gemm_bf16_mn(dy, w)[0], gate_up).isnan())
    gate_up[0, 5] = gate_up[0, 6] = 1.0
    out, _ = _comms.ops.gemm_gated_grad(dy, w, gate_up)
    d = dy.double() @ w.double()
    g, u = gate_up.double().chunk(2, dim=1)
    sig = torch.sigmoid(g)
    ref = torch.cat([d * u * (sig + g * sig * (1 - sig)), d * g * sig], dim=1)
    # Half a bf16 ulp (2^-9 relative); before it k fp32 additions of terms of size k^-1/2 and a few operations, of which the
    # sum of sigmoid and silu x (1 - sigmoid) may cancel, scaled by gates and ups of up to 10, a column's by 300.
    big = torch.tensor([300.0 if c in (3, n + 3, n + 4) else 10.0 for c in range(2 * n)], device="cuda", dtype=torch.float64)
    assert bool(((out.double() - ref).abs() <= 2**-8 * ref.abs() + big * (k**0.5 * 2**-23 + 4e-6)).all())
    for wrong in ((dy[:, :-1].contiguous(), w), (dy, w[:, :-1].contiguous())):
        with pytest.raises(Exception):
            _comms.ops.gemm_gated_grad(*wrong, gate_up)


@pytest.mark.parametrize("m,n", [(257, 136), (1000, 9480)])
def test_gated_gradient_of_exact_products(m, n):
    """Where the product is a bf16 number, the activation's own backward kernel makes the same bits of it."""
    from torchcomms_b200 import _comms

    w, gate_up = _rand(64, n, seed=2), _rand(m, 2 * n, seed=3, scale=3.0)
    dy = torch.zeros(m, 64, device="cuda", dtype=torch.bfloat16)
    dy[torch.arange(m), torch.arange(m) % 64] = 1.0
    out, _ = _comms.ops.gemm_gated_grad(dy, w, gate_up)
    assert torch.equal(out, _comms.ops.swiglu_bwd(w[torch.arange(m) % 64], gate_up))


def test_activation_of_every_gate():
    """All bf16 gates: the activation and its gradients as the definition with a correctly rounded division has them."""
    from torchcomms_b200 import _comms

    gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    up = _rand(65536, seed=1)
    gate_up = torch.cat((gate.view(8, -1), up.view(8, -1)), dim=1)
    g, u = gate.double(), up.double()
    act, grads = _comms.ops.swiglu_fwd(gate_up).view(-1), _comms.ops.swiglu_bwd(torch.ones(8, 8192, device="cuda").bfloat16(), gate_up)
    finite = g.isfinite() & (g.abs() < 80)
    sig = torch.sigmoid(g)
    for out, ref in ((act, g * sig * u), (grads[:, 8192:].reshape(-1), g * sig), (grads[:, :8192].reshape(-1), u * (sig + g * sig * (1 - sig)))):
        # Half a bf16 ulp (2^-9, or 2^-134 where there are no more bits); in fp32 before it the exponential's 2 ulp and its argument's
        # half (of up to 80), a handful of roundings, and a sum that may cancel.
        assert bool(((out.double() - ref).abs() <= 2**-8 * ref.abs() + u.abs() * 2**-20 + 2**-133)[finite].all())
    # Exponentials that overflow end in a zero of the sign of the gate; infinities and NaN as in the expression itself.
    low = g < -89
    assert not act[low & g.isfinite()].any()
    assert torch.equal(act.isnan(), (g * sig * u).isnan())


@pytest.mark.parametrize("rows,dim,heads,kv_heads,hd", [(1, 64, 1, 1, 8), (129, 200, 4, 2, 32), (1000, 512, 8, 2, 64)])
def test_block_in(rows, dim, heads, kv_heads, hd):
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    x, norm = _rand(rows, dim, seed=1).requires_grad_(True), (_rand(dim, seed=2, scale=0.1) + 1).requires_grad_(True)
    w = _rand((heads + 2 * kv_heads) * hd, dim, seed=3, scale=dim**-0.5).requires_grad_(True)
    cos_t, sin_t = fused.rope_tables(64, hd, 10000.0, "cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda") % 64
    got = _comms.ops.block_in(x, norm, w, pos, cos_t, sin_t, heads, kv_heads, 1e-5)
    # The same kernels as the separate nodes, but for a product of sums in another order.
    x2, h = fused.rms_norm_skip(x, norm, 1e-5)
    want = (x2, *fused.split_rope(torch.nn.functional.linear(h, w), pos, cos_t, sin_t, heads, kv_heads))
    douts = [_rand(*t.shape, seed=10 + i) for i, t in enumerate(want)]
    assert torch.equal(got[0], want[0]) and got[0].data_ptr() == x.data_ptr()
    # Products that differ by the order of their fp32 sums are rounded to bf16 (2^-9) on one side of a tie or the other, rotated
    # and rounded again.
    for a, b in zip(got, want):
        assert a.shape == b.shape and _off(a.detach(), b.detach()) < 2**-8
    # Backward takes nothing from the forward product: the same bits.
    for a, b in zip(torch.autograd.grad(got, (x, norm, w), douts), torch.autograd.grad(want, (x, norm, w), douts)):
        assert torch.equal(a, b)


def test_single_rows_of_any_stride():
    """A row by itself is contiguous whatever its stride says: a column transposed, for one."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    def column(t):
        return t.detach().as_strided(t.shape, (1, 1))

    ins = [_rand(1, 64, seed=1), _rand(1, 128, seed=2), _rand(64, 128, seed=3, scale=0.1), _rand(64, seed=4, scale=0.1) + 1,
           _rand(400, 64, seed=5, scale=0.1), _rand(64, 200, seed=6, scale=0.1)]
    dy = _rand(1, 64, seed=7)
    assert column(dy).is_contiguous()
    plain = [t.clone().requires_grad_(True) for t in ins]
    odd = [(column(t) if i < 2 else t).requires_grad_(True) for i, t in enumerate(ins)]
    a, b = _comms.ops.block_out(*plain, 1e-5), _comms.ops.block_out(*odd, 1e-5)
    assert torch.equal(a, b)
    for p, q in zip(torch.autograd.grad(a, plain, dy), torch.autograd.grad(b, odd, column(dy))):
        assert torch.equal(p, q)

    cos_t, sin_t = fused.rope_tables(4, 16, 10000.0, "cuda")
    pos = torch.ones(1, dtype=torch.int32, device="cuda")
    wqkv = _rand(8 * 16, 64, seed=8, scale=0.1).requires_grad_(True)
    norm = ins[3].clone().requires_grad_(True)
    results = []
    for x in (ins[0].clone(), column(ins[0])):
        x.requires_grad_(True)
        out = _comms.ops.block_in(x, norm, wqkv, pos, cos_t, sin_t, 4, 2, 1e-5)
        douts = [dy if x.stride(0) == 64 else column(dy), *(_rand(*t.shape, seed=10 + i) for i, t in enumerate(out[1:]))]
        results.append((*out, *torch.autograd.grad(out, (x, norm, wqkv), douts)))
    assert all(torch.equal(p, q) for p, q in zip(*results))


def test_only_what_is_asked_for():
    """Frozen weights and partial gradients: the others come out the same."""
    from torchcomms_b200 import _comms

    ins = [_rand(64, 128, seed=1), _rand(64, 128, seed=2), _rand(128, 128, seed=3, scale=0.1), _rand(128, seed=4, scale=0.1) + 1,
           _rand(512, 128, seed=5, scale=0.1), _rand(128, 256, seed=6, scale=0.1)]
    dy = _rand(64, 128, seed=7)
    full = [t.clone().requires_grad_(True) for t in ins]
    grads = torch.autograd.grad(_comms.ops.block_out(*full, 1e-5), full, dy)
    frozen = [t.clone().requires_grad_(i in (0, 3)) for i, t in enumerate(ins)]
    a, b = torch.autograd.grad(_comms.ops.block_out(*frozen, 1e-5), (frozen[0], frozen[3]), dy)
    assert torch.equal(a, grads[0]) and torch.equal(b, grads[3])
    y = _comms.ops.block_out(*full, 1e-5)
    one = torch.autograd.grad(y, full[4], dy, retain_graph=True)[0]
    two = torch.autograd.grad(y, full[1], dy)[0]
    assert torch.equal(one, grads[4]) and torch.equal(two, grads[1])
    with torch.no_grad():
        assert not _comms.ops.block_out(*full, 1e-5).requires_grad


def _launches(call):
    from torchcomms_b200 import _comms

    before = _comms.ops.kernel_launch_count()
    call()
    return _comms.ops.kernel_launch_count() - before


def test_backward_makes_only_what_is_asked_for():
    """The last weight's gradient takes one product, the one before it the activation's too; the norm waits for whoever wants it."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    ins = [_rand(64, 128, seed=1), _rand(64, 128, seed=2), _rand(128, 128, seed=3, scale=0.1), _rand(128, seed=4, scale=0.1) + 1,
           _rand(512, 128, seed=5, scale=0.1), _rand(128, 256, seed=6, scale=0.1)]
    ins = [t.requires_grad_(True) for t in ins]
    dy = _rand(64, 128, seed=7)
    y = _comms.ops.block_out(*ins, 1e-5)
    full = torch.autograd.grad(y, ins, dy, retain_graph=True)
    # one launch each: a product, the activation's gradients with theirs; the norm's two
    for wanted, launches in (([5], 1), ([4], 2), ([4, 5], 3), ([3], 4), ([0], 4), ([2], 5), ([1], 5)):
        some = []
        assert _launches(lambda: some.extend(torch.autograd.grad(y, [ins[i] for i in wanted], dy, retain_graph=True))) == launches
        assert all(torch.equal(a, full[i]) for a, i in zip(some, wanted))

    cos_t, sin_t = fused.rope_tables(64, 16, 10000.0, "cuda")
    pos = torch.arange(64, dtype=torch.int32, device="cuda")
    wqkv = _rand(8 * 16, 128, seed=8, scale=0.1).requires_grad_(True)
    out = _comms.ops.block_in(ins[0], ins[3], wqkv, pos, cos_t, sin_t, 4, 2, 1e-5)
    douts = [_rand(*t.shape, seed=10 + i) for i, t in enumerate(out)]
    full = torch.autograd.grad(out, (ins[0], ins[3], wqkv), douts, retain_graph=True)
    for wanted, launches in (((2,), 2), ((1,), 4), ((0,), 4)):
        some = []
        assert _launches(lambda: some.extend(torch.autograd.grad(out, [(ins[0], ins[3], wqkv)[i] for i in wanted], douts, retain_graph=True))) == launches
        assert all(torch.equal(a, full[i]) for a, i in zip(some, wanted))


def test_frozen_weights_keep_nothing():
    """What a forward pass makes on the way is kept only for the gradients that take it, as separate operations keep it."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    rows, dim, width, ffn = 40, 128, 64, 256
    ins = [_rand(rows, dim, seed=1), _rand(rows, width, seed=2), _rand(dim, width, seed=3, scale=0.1), _rand(dim, seed=4, scale=0.1) + 1,
           _rand(2 * ffn, dim, seed=5, scale=0.1), _rand(dim, ffn, seed=6, scale=0.1)]
    dy = _rand(rows, dim, seed=7)

    def made(call, args):  # elements kept beside the arguments, and the norm's statistics
        kept, given = {}, {t.data_ptr() for t in args}

        def pack(t):
            if t.data_ptr() not in given:
                kept[t.data_ptr()] = t.numel()
            return t

        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            out = call()
        return sum(kept.values()) - rows, out

    full = [t.clone().requires_grad_(True) for t in ins]
    grads = torch.autograd.grad(_comms.ops.block_out(*full, 1e-5), full, dy)
    # sum and norm's output are rows x dim, gate and up rows x 2 ffn, the activation rows x ffn
    for wanted, cols in (((0, 1, 2, 3, 4, 5), 2 * dim + 3 * ffn), ((0,), dim + 2 * ffn), ((1, 4), 2 * dim + 2 * ffn), ((5,), ffn), ((4,), dim + 2 * ffn)):
        some = [t.clone().requires_grad_(i in wanted) for i, t in enumerate(ins)]
        elements, y = made(lambda: _comms.ops.block_out(*some, 1e-5), some)
        assert elements == rows * cols
        for i, g in zip(wanted, torch.autograd.grad(y, [some[i] for i in wanted], dy)):
            assert torch.equal(g, grads[i])

    cos_t, sin_t = fused.rope_tables(rows, 16, 10000.0, "cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    wqkv = _rand(8 * 16, dim, seed=8, scale=0.1)
    for wanted, cols in (((0, 1, 2), dim), ((0,), 0), ((2,), dim)):
        some = [t.clone().requires_grad_(i in wanted) for i, t in enumerate((ins[0], ins[3], wqkv))]
        elements, out = made(lambda: _comms.ops.block_in(*some, pos, cos_t, sin_t, 4, 2, 1e-5), (*some, pos, cos_t, sin_t))
        assert elements == rows * cols
        torch.autograd.grad(out[1:], [some[i] for i in wanted], [t.detach() for t in out[1:]])


def test_gradients_of_gradients():
    """Second-order gradients are those of the separate operations, also where attention makes one argument from another."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused

    rows, dim, ffn = 48, 128, 200
    ins = [_rand(rows, dim, seed=1), _rand(dim, dim, seed=3, scale=0.1), _rand(dim, seed=4, scale=0.1) + 1, _rand(2 * ffn, dim, seed=5, scale=0.1),
           _rand(dim, ffn, seed=6, scale=0.1)]
    dy = _rand(rows, dim, seed=7)

    def apart(x, o, wo, norm, w13, w2):
        s, h = fused.add_rms_norm(x, torch.nn.functional.linear(o, wo), norm, 1e-5)
        return s + torch.nn.functional.linear(fused.swiglu(torch.nn.functional.linear(h, w13)), w2)

    def orders(f, frozen):
        x, *weights = [t.clone().requires_grad_(i not in frozen) for i, t in enumerate(ins)]
        o = x * x  # made from another argument
        leaves = [t for t in (x, *weights) if t.requires_grad]
        first = torch.autograd.grad(f(x, o, *weights), leaves, dy, create_graph=True)
        with_history = [g for g in first if g.requires_grad]
        assert with_history
        second = torch.autograd.grad(sum(g.float().square().sum() for g in with_history), leaves, allow_unused=True)
        return [g.requires_grad for g in first], first, second

    for frozen in ((), (1, 4), (2, 3)):
        mine, theirs = orders(lambda *a: _comms.ops.block_out(*a, 1e-5), frozen), orders(apart, frozen)
        assert mine[0] == theirs[0]
        # The same kernels; the engine adds what meets in an argument, four terms in bf16 at most, in its own order.
        for a, b in zip(mine[1] + mine[2], theirs[1] + theirs[2]):
            assert (a is None and b is None) or _off(a.detach(), b.detach()) < 4 * 2**-9

    cos_t, sin_t = fused.rope_tables(rows, 16, 10000.0, "cuda")
    pos = torch.arange(rows, dtype=torch.int32, device="cuda")
    wqkv = _rand(8 * 16, dim, seed=8, scale=0.1)

    def apart_in(x, norm, w):
        x, h = fused.rms_norm_skip(x, norm, 1e-5)
        return (x, *fused.split_rope(torch.nn.functional.linear(h, w), pos, cos_t, sin_t, 4, 2))

    for frozen in ((), (0, 1), (2,), (1, 2)):
        results = []
        for f in (lambda *a: _comms.ops.block_in(*a, pos, cos_t, sin_t, 4, 2, 1e-5), apart_in):
            args = [t.clone().requires_grad_(i not in frozen) for i, t in enumerate((ins[0], ins[2], wqkv))]
            leaves = [t for t in args if t.requires_grad]
            out = f(*args)
            used = [(t, _rand(*t.shape, seed=10 + i)) for i, t in enumerate(out) if i > 0 or 0 not in frozen]
            first = torch.autograd.grad([t for t, _ in used], leaves, [d for _, d in used], create_graph=True)
            with_history = [g for g in first if g.requires_grad]
            second = torch.autograd.grad(sum(g.float().square().sum() for g in with_history), leaves, allow_unused=True) if with_history else ()
            results.append((*first, *second))
        assert len(results[0]) == len(results[1])
        for a, b in zip(*results):
            assert (a is None and b is None) or (_off(a.detach(), b.detach()) < 4 * 2**-9 and a.requires_grad == b.requires_grad)


def test_block_takes_and_leaves():
    """What the nodes do not take runs as before: other types, autocast, transforms."""
    from torchcomms_b200 import _comms
    from torchcomms_b200.models.llama import Block, LlamaConfig
    from torchcomms_b200.ops import fused

    cfg = LlamaConfig(dim=128, n_layers=1, n_heads=4, n_kv_heads=2, ffn_dim=200, vocab_size=64, max_seq_len=64)
    torch.manual_seed(0)
    block = Block(cfg).cuda().bfloat16()
    cos_t, sin_t = fused.rope_tables(64, cfg.head_dim, cfg.rope_theta, "cuda")
    pos = torch.arange(48, dtype=torch.int32, device="cuda")
    x = _rand(1, 48, 128, seed=1)
    y = block(x, pos, cos_t, sin_t)
    with torch.autocast("cuda", torch.bfloat16):
        assert _off(block(x, pos, cos_t, sin_t).detach(), y.detach()) < 2**-7
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t) or t, lambda t: t):
        (block(x, pos, cos_t, sin_t).float().sum()).backward()
    assert kept and all(p.grad is not None for p in block.parameters())
    n = block.ffn_norm
    assert _comms.ops.block_out(x[0], x[0], block.wo, n, block.w13, block.w2[:, :199], 1e-5) is None
    assert _comms.ops.block_out(x[0].float(), x[0], block.wo, n, block.w13, block.w2, 1e-5) is None
    assert _comms.ops.block_in(x[0, :, :64], n, block.wqkv, pos, cos_t, sin_t, 4, 2, 1e-5) is None
    out = torch.func.functional_call(block, dict(block.named_parameters()), (x, pos, cos_t, sin_t))
    assert torch.equal(out, y)
