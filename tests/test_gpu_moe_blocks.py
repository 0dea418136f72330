"""Single-rank dispatch over every number of tokens that a block takes, bases on and off the 32-byte grid."""
import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu


# One token; blocks of 2, 4 and 8 tokens with a remainder; one, two and an odd number of pieces per row.
@pytest.mark.parametrize("tokens,hidden", [(1, 512), (5, 2560), (2559, 1024), (2561, 1536), (5119, 512), (5121, 1024)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("offset", [0, 8])
def test_dispatch(tokens, hidden, fp8, offset, monkeypatch):
    import torchcomms_b200 as tc
    from torchcomms_b200.ops.moe_ep import Buffer, per_token_cast_to_fp8

    for name, value in (("RANK", "0"), ("WORLD_SIZE", "1"), ("LOCAL_RANK", "0")):
        monkeypatch.setenv(name, value)
    comm = tc.new_comm("b200", torch.device("cuda", 0), name=f"blocks{tokens}_{hidden}_{fp8}_{offset}", store=dist.HashStore())
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    x = torch.randn(offset + tokens * hidden, generator=g, device="cuda").to(torch.bfloat16)[offset:].view(tokens, hidden)
    idx = torch.randint(-1, 16, (tokens, 4), generator=g, device="cuda", dtype=torch.int32)
    w = torch.rand(tokens, 4, generator=g, device="cuda")
    buf = Buffer(comm, tokens, hidden, 16, 4, fp8=fp8)
    for _ in range(2):
        d = buf.dispatch(x, idx, w)
        sent = (idx >= 0).any(dim=1).nonzero().squeeze(1)
        n = int(d.num_tokens)
        src = d.src[:n].long()
        assert n == sent.numel() and torch.equal(src.sort().values, sent) and d.tokens_per_src.tolist() == [n]
        assert torch.equal(d.topk_idx[:n], idx[src])
        if fp8:
            q, s = per_token_cast_to_fp8(x)
            # A division against a product with the rounded reciprocal of 448: two roundings apart at most.
            torch.testing.assert_close(d.scales[:n], s[src], rtol=2**-22, atol=0)
            # The kernel multiplies by the reciprocal of the scale: one rounding more, so a neighbouring e4m3 value at most.
            torch.testing.assert_close(d.x[:n].float(), q[src].float(), rtol=2**-3, atol=2**-9)
        else:
            assert torch.equal(d.x[:n], x[src])
    comm.finalize()


# Both sides of the lines between 2 and 4 and, for wide rows, between 4 and 8 tokens.
@pytest.mark.parametrize("tokens,hidden", [(1184, 512), (1185, 512), (5121, 4096), (7697, 4096)])
@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_at_the_lines_between_block_sizes(tokens, hidden, fp8, monkeypatch):
    test_dispatch(tokens, hidden, fp8, 0, monkeypatch)


# Both sides of the lines between shapes of blocks; rows of a quarter piece to three pieces and a bit.
@pytest.mark.parametrize("tokens,hidden", [(592, 512), (593, 2560), (1185, 1536), (1186, 1024), (2072, 2048), (2073, 2560),
                                           (2368, 1536), (2369, 4608), (2370, 6656)])
@pytest.mark.parametrize("fp8", [False, True])
def test_dispatch_at_the_lines_between_blocks(tokens, hidden, fp8, monkeypatch):
    test_dispatch(tokens, hidden, fp8, 0, monkeypatch)


@pytest.mark.parametrize("fp8", [False, True])
def test_low_latency_outputs_can_be_saved_together(fp8, tmp_path, monkeypatch):
    """torch.save refuses tensors of different types over one storage; outputs that share an allocation are of one type."""
    import torchcomms_b200 as tc
    from torchcomms_b200.ops.moe_ep import LowLatencyBuffer

    for name, value in (("RANK", "0"), ("WORLD_SIZE", "1"), ("LOCAL_RANK", "0")):
        monkeypatch.setenv(name, value)
    comm = tc.new_comm("b200", torch.device("cuda", 0), name=f"ll_saved{fp8}", store=dist.HashStore())
    buf = LowLatencyBuffer(comm, 16, 512, 8, 2, fp8=fp8)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(13, 512, generator=g, device="cuda").to(torch.bfloat16)
    r = buf.dispatch(x, torch.randint(0, 8, (13, 2), generator=g, device="cuda", dtype=torch.int32))
    outputs = {k: v for k, v in vars(r).items() if v is not None}
    small = ("count", "src_info", "layout_range", "send_slot", "begin")
    torch.save(outputs, tmp_path / "outputs.pt")
    back = torch.load(tmp_path / "outputs.pt")
    assert set(back) == set(outputs) and int(back["count"].sum()) == 26
    assert all(torch.equal(back[k], outputs[k]) for k in small)
    # Each keeps a version counter of its own.
    r.count.zero_()
    assert all(getattr(r, k)._version == 0 for k in small if k != "count")
    comm.finalize()
