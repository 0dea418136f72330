"""Every kernel that a plain product can take, at the edges of the rule that picks it, against a 64-bit product."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# Narrow pair tiles at most one wave, more than one; short sums on single CTAs, and one step more; rows off the 128-byte
# lines; row and column remainders of every tile.
@pytest.mark.parametrize("m,n,k", [(256, 9472, 256), (257, 9480, 256), (129, 136, 1024), (700, 6144, 1024), (700, 6144, 1088), (700, 6152, 1032),
                                   (4096, 2304, 128), (4096, 2320, 1040), (1000, 6144, 2048), (385, 264, 8)])
@pytest.mark.parametrize("fp8", [False, True])
def test_plain_product(m, n, k, fp8):
    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import quantize_rows

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    k = 2 * k if fp8 else k  # the rule counts bytes
    a = (torch.randn(m, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    b = (torch.randn(n, k, generator=g, device="cuda") * 0.5).to(torch.bfloat16)
    if fp8:
        (qa, sa), (qb, sb) = quantize_rows(a), quantize_rows(b)
        ref = (qa.double() * sa.double().unsqueeze(1)) @ (qb.double() * sb.double().unsqueeze(1)).t()
        run = lambda: _comms.ops.gemm_e4m3_nt(qa, qb, sa, sb)
    else:
        ref = a.double() @ b.double().t()
        run = lambda: _comms.ops.gemm_bf16_nt(a, b)
    first = None
    for _ in range(3):
        c, status = run()
        assert int(status[0]) == 0
        # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 1/4 before it.
        torch.testing.assert_close(c.double(), ref, rtol=2**-8, atol=1e-6 * k)
        assert first is None or torch.equal(c, first)
        first = c


# A wave less on single CTAs than on pairs: one wave, with rows off the lines and a long sum, and three; four, with a last
# column tile of eight columns and further tiles behind it; as many waves; more tiles than SMs for the split kernel, and
# fewer with unshared sums on and off the lines; boxes of 1, 5, 67 and all rows of A.
@pytest.mark.parametrize("m,n,k", [(3190, 5640, 64), (1, 28672, 256), (67, 28672, 576), (128, 22016, 1096), (640, 7168, 1152), (300, 10240, 1032), (384, 28672, 128),
                                   (384, 28672, 136), (5, 14336, 1088), (100, 14336, 1096), (128, 14336, 1032), (256, 9472, 2112), (5, 9472, 1032)])
@pytest.mark.parametrize("fp8", [False, True])
def test_plain_product_by_waves(m, n, k, fp8):
    test_plain_product(m, n, k, fp8)


# Pairs in tiles of 192, 192, 224, 224 and 192 columns, the last tile of a few columns, of a row and of a K step's part; narrow
# pairs where a shared sum would not pay, and where it does; unshared sums of few steps, and of few rows in many tiles.
@pytest.mark.parametrize("m,n,k", [(1000, 6144, 136), (1000, 6152, 1096), (1500, 5000, 200), (257, 14344, 1096), (300, 20488, 72),
                                   (256, 2816, 1280), (128, 4096, 1792), (3, 408, 376), (256, 1536, 192), (100, 6000, 320)])
@pytest.mark.parametrize("fp8", [False, True])
def test_plain_product_by_tile_width(m, n, k, fp8):
    test_plain_product(m, n, k, fp8)


# A last wave in halves of tiles of 256, of 224 and of 192 columns, one of them past the last column; no whole tile at all.
@pytest.mark.parametrize("m,n,k", [(4096, 2560, 200), (2049, 2312, 136), (1025, 3784, 520), (1793, 5344, 72), (4096, 1288, 1032)])
@pytest.mark.parametrize("fp8", [False, True])
def test_plain_product_with_half_tiles(m, n, k, fp8):
    test_plain_product(m, n, k, fp8)


# Tiles of 112, 96 and 128 columns of gate and of up, one of them in a row, ragged ends of rows, columns and K steps; a last wave in
# halves of tiles of 192 columns (1 x 8 to 1000 x 2568), of 224 and of 256.
@pytest.mark.parametrize("m,n,k", [(700, 5000, 768), (300, 4808, 72), (1000, 2056, 200), (1, 8, 8), (257, 120, 64), (2049, 232, 136),
                                   (1000, 2568, 136), (2048, 1160, 72), (512, 9480, 264), (512, 5288, 136), (768, 4728, 136)])
def test_gated_product(m, n, k):
    _gated_product(m, n, k, 0)


# Every width with whole tiles and with halves, some of which lie past the last column: one tile, 4 to 6, and 90 to 135 for 74
# pairs.
@pytest.mark.parametrize("columns", [192, 224, 256])
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (257, 200, 200), (2300, 1000, 72), (2300, 1192, 72), (1000, 2840, 136), (513, 4264, 72)])
def test_gated_product_of_every_width(m, n, k, columns):
    _gated_product(m, n, k, columns)


def _gated_product(m, n, k, columns):
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * n, k, generator=g, device="cuda") * k**-0.5).to(torch.bfloat16)
    gate_up, act, status = _comms.ops.gemm_gated(x, w, columns)
    assert int(status[0]) == 0
    torch.testing.assert_close(gate_up.double(), x.double() @ w.double().t(), rtol=2**-8, atol=1e-6 * k)
    assert torch.equal(act, _comms.ops.swiglu_fwd(gate_up))  # the activation kernel's bits
    # The activation from the rounded gate and up: an fp32 expression of five roundings, the exponential's and reciprocal's 2 ulp
    # among them, then one to bf16, which may fall either way.
    gate, up = gate_up.double().chunk(2, dim=-1)
    torch.testing.assert_close(act.double(), torch.nn.functional.silu(gate) * up, rtol=2**-8, atol=1e-12)
    again = _comms.ops.gemm_gated(x, w, columns)
    assert torch.equal(again[0], gate_up) and torch.equal(again[1], act)


def test_gated_product_of_extremes():
    """Gates whose exponential overflows or vanishes, zeros, infinities and NaN come out as from the activation kernel."""
    from torchcomms_b200 import _comms

    values = torch.tensor([0.0, -0.0, 1e-30, 87.0, -87.0, -89.0, -104.0, 300.0, -300.0, 1e38, -1e38, float("inf"), float("-inf"), float("nan")],
                          device="cuda").to(torch.bfloat16)
    x = torch.zeros(16, 8, device="cuda", dtype=torch.bfloat16)
    x[: len(values), 0] = values
    x[:, 1] = 1.0
    w = torch.zeros(16, 8, device="cuda", dtype=torch.bfloat16)
    w[:8, 0], w[8:, 1] = 1.0, 3.0
    gate_up, act, _ = _comms.ops.gemm_gated(x, w)
    torch.testing.assert_close(act, _comms.ops.swiglu_fwd(gate_up), rtol=2**-7, atol=0, equal_nan=True)


# K in the rows of both operands, or in the rows of b alone: one row, one column unit, K steps that end anywhere, narrow and wide
# tiles, a last wave in halves; rows of a that are apart.
@pytest.mark.parametrize("m,n,k", [(8, 8, 1), (1, 8, 8), (257, 136, 65), (1000, 520, 1003), (2049, 2312, 136), (4096, 2560, 200), (130, 9480, 77)])
@pytest.mark.parametrize("by_columns", [False, True])
def test_product_along_rows(m, n, k, by_columns):
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    rows, cols = (k, m) if by_columns else (m, k)
    wide = torch.randn(rows, (cols + 63) // 64 * 64, generator=g, device="cuda").to(torch.bfloat16)
    wide[:, cols:] = float("nan")  # between the rows, not read
    a = wide[:, :cols]
    b = torch.randn(k, n, generator=g, device="cuda").to(torch.bfloat16)
    c, status = _comms.ops.gemm_bf16_mn(a, b, by_columns)
    assert int(status[0]) == 0
    ref = (a.t() if by_columns else a).double() @ b.double()
    # Half a bf16 ulp (2^-9 relative), and k fp32 additions of terms of size 1 before it.
    torch.testing.assert_close(c.double(), ref, rtol=2**-8, atol=4e-6 * k)
    assert torch.equal(c, _comms.ops.gemm_bf16_mn(a, b, by_columns)[0])


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (128, 3584, 4096), (384, 512, 704), (512, 5120, 512)])
def test_gather_layer_leaves_its_input_behind(m, n, k):
    """A single rank's layer reads the activations where they are; its input buffer holds them afterwards all the same."""
    from torchcomms_b200.ops.tp import AllGatherGemm

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    layer = AllGatherGemm(None, m_local=m, k=k)
    layer.input.zero_()
    y = layer(w, x)
    assert torch.equal(layer.input, x) and torch.equal(layer(w), y)
    torch.testing.assert_close(y.double(), x.double() @ w.double().t(), rtol=2**-8, atol=2e-7 * k)
    # What cannot be read in place is copied first: other layouts and types, and the buffer itself.
    wide = torch.zeros(m, k + 8, device="cuda", dtype=torch.bfloat16)
    wide[:, :k] = x
    off = torch.zeros(m * k + 1, device="cuda", dtype=torch.bfloat16)[1:].view(m, k).copy_(x)
    for other in (wide[:, :k], off, x.t().contiguous().t(), x.float(), layer.input):
        if other is not layer.input and other.data_ptr() != layer.input.data_ptr():
            layer.input.zero_()
        assert torch.equal(layer(w, other), y) and torch.equal(layer.input, x)


# The kernel copies the activations on its way; a copy in front of it does.
@pytest.mark.parametrize("m,n,k", [(128, 3584, 1024), (512, 5120, 512)])
def test_gather_layer_in_a_graph(m, n, k):
    from torchcomms_b200.ops.tp import AllGatherGemm

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    xs = [torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.1).to(torch.bfloat16)
    layer = AllGatherGemm(None, m_local=m, k=k)
    want = [layer(w, x) for x in xs]
    src, graph = xs[0].clone(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        y = layer(w, src)
    for x, ref in zip(xs, want):
        src.copy_(x)
        layer.input.zero_()
        y.zero_()
        graph.replay()
        assert torch.equal(y, ref) and torch.equal(layer.input, x) and layer.status()[0] == 0


def test_products_in_threads_that_have_called_nothing_yet():
    """Every product as the first CUDA call of its thread, whose buffers the allocator has at hand."""
    import threading

    from torchcomms_b200 import _comms
    from torchcomms_b200.ops.tp import AllGatherGemm

    g = torch.Generator(device="cuda").manual_seed(1)
    x, w = (torch.randn(128, 256, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    big = torch.randn(4096, 256, generator=g, device="cuda").to(torch.bfloat16)
    gate_up = torch.randn(128, 512, generator=g, device="cuda").to(torch.bfloat16)
    square = torch.randn(256, 256, generator=g, device="cuda").to(torch.bfloat16)
    targets = torch.zeros(128, dtype=torch.long, device="cuda")
    layer = AllGatherGemm(None, m_local=128, k=256)
    calls = [lambda: _comms.ops.gemm_bf16_nt(x, w)[0], lambda: _comms.ops.gemm_bf16_nt(big, big)[0], lambda: _comms.ops.gemm_bf16_mn(x, square)[0],
             lambda: _comms.ops.gemm_gated(x, w)[1], lambda: _comms.ops.gemm_gated_grad(x, square, gate_up)[0],
             lambda: _comms.ops.head(x, w, targets, 4096)[1], lambda: layer(square, x)]
    for call in calls:
        first = call().clone()
        for _ in range(2):  # the cache then has what the thread asks for
            call()
        torch.cuda.synchronize()
        results = []

        def work():
            try:
                results.append(call())
            except Exception as e:
                results.append(e)

        thread = threading.Thread(target=work)
        thread.start()
        thread.join()
        if isinstance(results[0], Exception):
            raise results[0]
        torch.cuda.synchronize()
        assert torch.equal(results[0], first)


# Loads that are never complete and waits of 20 ms, on every kernel: split, single CTAs, pairs with more tiles than pairs and a last
# wave in halves, fewer and more K steps than stages; the gated epilogues.
@pytest.mark.parametrize("kind,m,n,k", [("nt", 128, 4096, 1792), ("nt", 640, 7168, 4096), ("pair", 4096, 2560, 200), ("pair", 300, 264, 1024),
                                        ("gated", 1000, 5136, 136), ("gated", 200, 272, 1024), ("gated_grad", 300, 4808, 200),
                                        ("gated_grad", 257, 136, 1024)])
def test_a_product_that_gives_up_says_so(kind, m, n, k):
    """Whoever drops the status words, as a decoder block does, finds NaN and not what the memory held."""
    from torchcomms_b200 import _comms

    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn(m, k, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(*((k, n) if kind == "gated_grad" else (n, k)), generator=g, device="cuda").to(torch.bfloat16)
    gate_up = torch.randn(m, 2 * n, generator=g, device="cuda").to(torch.bfloat16) if kind == "gated_grad" else None
    out, status = _comms.ops.gemm_giving_up(kind, a, w, gate_up, 20)
    torch.cuda.synchronize()
    assert int(status[0]) != 0 and bool(out.isnan().all())
    # The context goes on, and so does the same kernel.
    if kind == "gated_grad":
        c, status = _comms.ops.gemm_gated_grad(a, w, gate_up)
        assert not c.isnan().any()
    elif kind == "gated":
        c, _, status = _comms.ops.gemm_gated(a, w)
        torch.testing.assert_close(c.double(), a.double() @ w.double().t(), rtol=2**-8, atol=4e-6 * k)
    else:
        c, status = (_comms.ops.gemm_bf16_nt if kind == "nt" else _comms.ops.gemm_bf16_nt_pair)(a, w)
        torch.testing.assert_close(c.double(), a.double() @ w.double().t(), rtol=2**-8, atol=4e-6 * k)
    assert int(status[0]) == 0
