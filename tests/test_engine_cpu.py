"""The sharded training engine on CPU ranks (gloo): sharding, gather /
reduce-scatter plumbing, optimizer, and equivalence between 1 and 2 ranks."""
from datetime import timedelta

import torch

from tests.mp_util import run_ranks


def _train(rank, world, out_path):
    import torchcomms_b200 as tc
    from torchcomms_b200.models.llama import LlamaConfig
    from torchcomms_b200.parallel.engine import TrainEngine

    torch.manual_seed(0)
    comm = tc.new_comm("gloo", torch.device("cpu"), name="engine", timeout=timedelta(seconds=120))
    cfg = LlamaConfig(dim=64, n_layers=2, n_heads=4, n_kv_heads=2, ffn_dim=128, vocab_size=97, max_seq_len=32)
    engine = TrainEngine(cfg, comm, lr=1e-2, weight_decay=0.0, seed=3, recompute_blocks=1)
    g = torch.Generator().manual_seed(11)
    tokens = torch.randint(0, cfg.vocab_size, (2, 17), generator=g)  # same batch on every rank
    losses = []
    for _ in range(4):
        loss = engine.step(tokens[:, :-1].contiguous(), tokens[:, 1:].contiguous())
        losses.append(float(loss))
    assert all(l == l for l in losses)
    assert losses[-1] < losses[0], losses
    # every unit's transient buffers are gone after the step
    for u in engine.units:
        assert u.flat_grad is None and u.grad_shard is None
        assert u.flat_param.untyped_storage().nbytes() == 0 or u is engine.units[-1]
    state = engine.state_dict()
    assert state["step"] == 4
    if rank == 0:
        torch.save({"losses": losses, "world": world}, out_path)
    comm.finalize()


def test_engine_trains_and_matches_across_world_sizes(tmp_path):
    p1, p2 = str(tmp_path / "w1.pt"), str(tmp_path / "w2.pt")
    run_ranks(_train, 1, args=(p1,), timeout=240)
    run_ranks(_train, 2, args=(p2,), timeout=240)
    a, b = torch.load(p1), torch.load(p2)
    # identical data on every rank: the averaged gradient equals the single-rank gradient
    for x, y in zip(a["losses"], b["losses"]):
        assert abs(x - y) < 5e-2, (a["losses"], b["losses"])


def test_block_pieces_on_cpu_tensors():
    """CPU tensors take the plain compositions of the fused block pieces, gradients included, and the kernels' entry
    points decline them."""
    import torch

    from torchcomms_b200 import _comms
    from torchcomms_b200.ops import fused
    from torchcomms_b200.ops.tp import quantize_rows

    torch.manual_seed(3)
    x, d, w = (torch.randn(6, 16, requires_grad=True) for _ in range(3))
    w = w[0].detach().requires_grad_(True)
    s, y = fused.add_rms_norm(x, d, w)
    torch.testing.assert_close(s, x + d)
    torch.testing.assert_close(y, fused.rms_norm(x + d, w))
    skip, y2 = fused.rms_norm_skip(x, w)
    assert skip is x
    (g,) = torch.autograd.grad((skip, y2), x, (torch.ones_like(x), torch.ones_like(x)))
    (ref,) = torch.autograd.grad(fused.rms_norm(x, w).sum() + x.sum(), x)
    torch.testing.assert_close(g, ref)

    cos_t, sin_t = fused.rope_tables(32, 8, 10000.0, "cpu")
    pos = torch.arange(6, dtype=torch.int32)
    qkv = torch.randn(6, (4 + 2 * 2) * 8, requires_grad=True)
    q, k, v = fused.split_rope(qkv, pos, cos_t, sin_t, 4, 2)
    parts = qkv.split([32, 16, 16], dim=-1)
    torch.testing.assert_close(q, fused.apply_rope(parts[0].reshape(6, 4, 8), pos, cos_t, sin_t))
    torch.testing.assert_close(k, fused.apply_rope(parts[1].reshape(6, 2, 8), pos, cos_t, sin_t))
    torch.testing.assert_close(v, parts[2].reshape(6, 2, 8))
    assert torch.autograd.grad(q.sum() + k.sum() + v.sum(), qkv)[0].shape == qkv.shape

    b = torch.randn(3, 32).to(torch.bfloat16)
    assert _comms.ops.quantize_rows(b) is None
    assert _comms.ops.rms_norm(b, b[0], 1e-5) is None and _comms.ops.swiglu(b) is None
    q8, scale = quantize_rows(b)
    assert q8.dtype == torch.float8_e4m3fn
    torch.testing.assert_close(scale, b.float().abs().amax(dim=1) / 448.0)
    # A loss and its gradients twice over a retained graph give the same on the device without kernels.
    xs, ws = torch.randn(5, 16, requires_grad=True), torch.randn(11, 16, requires_grad=True)
    t = torch.randint(0, 11, (5,))
    loss = fused.linear_cross_entropy(xs, ws, t, chunk_rows=2)
    a = torch.autograd.grad(loss, (xs, ws), retain_graph=True)
    c = torch.autograd.grad(loss, (xs, ws))
    ref = torch.autograd.grad(torch.nn.functional.cross_entropy(xs @ ws.t(), t), (xs, ws))
    for p, q_, r in zip(a, c, ref):
        assert torch.equal(p, q_)
        torch.testing.assert_close(p, r, rtol=1e-4, atol=1e-6)


def test_padded_head_follows_rows_and_weight():
    """The choice between a padded copy of the weight and none looks at the rows as well as at the weight."""
    from torchcomms_b200.ops.fused import _worth_padding

    m = 1 << 20
    assert _worth_padding(4096, 20 * m) and _worth_padding(4096, m) and _worth_padding(512, 25 * m)  # several times faster
    assert _worth_padding(1, 250 * m) and _worth_padding(2, 25 * m)
    # the GPU waits for the host either way: a copy only takes longer
    assert not _worth_padding(64, 2 * m) and not _worth_padding(1500, m) and not _worth_padding(2, 20 * m)
    assert not _worth_padding(0, 500 * m)
