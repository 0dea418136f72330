"""Timed cases of the framework's single-GPU work.

Each case is one pass through public entry points, at the sizes of the Llama-3-8B
training step and of the MoE workload that the benchmark runs (hidden 4096, 32 query
and 8 key/value heads of 128, FFN 14336, vocabulary 128256; 256 experts, top-8,
hidden 7168), plus small and ragged ones.  The kinds:

``ar_norm``   residual add + RMSNorm of a decode batch after a row-parallel projection
``norm``      RMSNorm of a training batch, forward and backward
``rope``      rotary embedding of queries and keys out of a fused QKV, forward and backward
``swiglu``    gated activation of a training batch, forward and backward
``head``      vocabulary projection + cross-entropy, loss and gradients
``block``     a whole decoder block, forward and backward
``adamw``     optimizer step on a flat fp32 shard
``mlp``       the tensor-parallel MLP (gather -> GEMM, SwiGLU, GEMM -> scatter), bf16 or fp8
``linear8``   fp8 linear layer on bf16 activations (row quantisation + GEMM)
``moe``       expert-parallel dispatch and combine of a prefill / training batch
``moe_ll``    low-latency dispatch and combine of a decode batch
"""
from __future__ import annotations

import math
import os

import torch

F64 = torch.float64
BF16 = torch.bfloat16
EPS = 1e-5


# ------------------------------------------------------------------- the cases


def listed():
    return [
        # One speculative-decode step: a handful of tokens after the attention output projection.
        {"name": "decode_norm", "kind": "ar_norm", "rows": 5, "hidden": 4096},
        # The two norms of every block in the benchmark's training step (sequence 4096, micro-batch 1).
        {"name": "train_norm", "kind": "norm", "rows": 4096, "hidden": 4096},
        # Rotary embedding of the same step, on a packed batch whose token count is odd.
        {"name": "train_rope", "kind": "rope", "tokens": 4093, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # The activation of the same step.
        {"name": "train_swiglu", "kind": "swiglu", "rows": 4096, "ffn": 14336},
        # The head of the same step: the largest single call of a training step.
        {"name": "train_head", "kind": "head", "rows": 4096, "hidden": 4096, "vocab": 128256},
        # One block at a short, uneven sequence, where launches and small grids weigh more.
        {"name": "train_block", "kind": "block", "tokens": 1000, "hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336},
        # AdamW on one block's parameters (the shard of a one-GPU job).
        {"name": "train_adamw", "kind": "adamw", "numel": 218112000},
        # MLP of a decode batch: weights are streamed once for 128 tokens; one rank of an 8-way split.
        {"name": "decode_mlp", "kind": "mlp", "tokens": 128, "hidden": 4096, "ffn": 1792, "fp8": False},
        # MLP of a prefill batch on fp8 operands, bf16 activations quantised on the way in.
        {"name": "prefill_mlp_fp8", "kind": "mlp", "tokens": 4096, "hidden": 4096, "ffn": 14336, "fp8": True},
        # Fused QKV projection of a decode batch with fp8 weights; the token count is not a tile multiple.
        {"name": "decode_qkv_fp8", "kind": "linear8", "rows": 67, "k": 4096, "n": 6144},
        # MoE prefill: the benchmark's dispatch (fp8) and combine.
        {"name": "prefill_moe", "kind": "moe", "tokens": 4096, "hidden": 7168, "experts": 256, "topk": 8, "fp8": True},
        # MoE decode: the benchmark's low-latency batch.
        {"name": "decode_moe", "kind": "moe_ll", "tokens": 128, "hidden": 7168, "experts": 256, "topk": 8, "fp8": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ar_norm", "norm", "rope", "swiglu", "head", "block", "adamw", "mlp", "linear8", "moe", "moe_ll"])
    case = {"kind": kind}
    if kind == "ar_norm":
        case.update(rows=_log(rng, 1, 128), hidden=8 * _log(rng, 32, 1024))
    elif kind == "norm":
        case.update(rows=_log(rng, 1, 16384), hidden=8 * _log(rng, 32, 1024))
    elif kind == "rope":
        kv = rng.choice([1, 2, 4, 8])
        case.update(tokens=_log(rng, 1, 8192), heads=kv * rng.choice([1, 2, 4]), kv_heads=kv, head_dim=rng.choice([32, 64, 96, 128]))
    elif kind == "swiglu":
        case.update(rows=_log(rng, 1, 8192), ffn=8 * _log(rng, 64, 1792))
    elif kind == "head":
        # Vocabularies that are no multiple of eight are ordinary (an added token or two).
        case.update(rows=_log(rng, 16, 4096), hidden=64 * _log(rng, 4, 64), vocab=_log(rng, 1000, 128256))
    elif kind == "block":
        kv = rng.choice([2, 4, 8])
        heads = kv * rng.choice([1, 2, 4])
        case.update(tokens=_log(rng, 16, 2048), hidden=heads * 64, heads=heads, kv_heads=kv, ffn=8 * _log(rng, 64, 1024))
    elif kind == "adamw":
        case.update(numel=_log(rng, 1000, 200000000))
    elif kind == "mlp":
        case.update(tokens=128 * _log(rng, 1, 32), hidden=256 * _log(rng, 2, 20), ffn=128 * _log(rng, 2, 112), fp8=rng.random() < 0.5)
    elif kind == "linear8":
        case.update(rows=_log(rng, 1, 4096), k=16 * _log(rng, 16, 512), n=8 * _log(rng, 32, 1792))
    elif kind == "moe":
        topk = rng.choice([1, 2, 4, 8])
        case.update(tokens=_log(rng, 16, 8192), hidden=512 * _log(rng, 2, 14), experts=rng.choice([8, 32, 64, 256]), topk=topk,
                    fp8=rng.random() < 0.5)
    else:
        case.update(tokens=_log(rng, 1, 128), hidden=512 * _log(rng, 2, 14), experts=rng.choice([8, 32, 64, 256]),
                    topk=rng.choice([1, 2, 4, 8]), fp8=rng.random() < 0.5)
    return case


# ------------------------------------------------------------- inputs and state


class _Rand:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.dev).manual_seed(1000003 * (seed % 1000003) + 17)

    def normal(self, *shape, std=1.0, dtype=BF16):
        return torch.empty(shape, dtype=dtype, device=self.dev).normal_(0.0, std, generator=self.g)

    def around_one(self, n):
        return (1.0 + 0.1 * torch.randn(n, generator=self.g, device=self.dev)).to(BF16)

    def ints(self, high, *shape):
        return torch.randint(high, shape, generator=self.g, device=self.dev)

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.g, device=self.dev)


_comms = []


def _comm():
    """The one-rank communicator of this process (a program makes it once, at start-up)."""
    if not _comms:
        import torch.distributed as dist

        import torchcomms_b200 as tc

        for name, value in (("RANK", "0"), ("WORLD_SIZE", "1"), ("LOCAL_RANK", "0")):
            os.environ.setdefault(name, value)
        _comms.append(tc.new_comm("b200", torch.device("cuda", torch.cuda.current_device()), name="perf", store=dist.HashStore()))
    return _comms[0]


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    r = _Rand(seed)
    kind = case["kind"]
    if kind == "ar_norm":
        m, h = case["rows"], case["hidden"]
        return {"x": r.normal(m, h), "w": r.around_one(h), "resid": r.normal(m, h, std=2.0)}
    if kind == "norm":
        m, h = case["rows"], case["hidden"]
        return {"x": r.normal(m, h, std=1.5), "w": r.around_one(h), "dy": r.normal(m, h)}
    if kind == "rope":
        t, nh, nkv, hd = case["tokens"], case["heads"], case["kv_heads"], case["head_dim"]
        # Queries and keys are slices of the fused projection's output, as in a block.
        qkv = r.normal(t, (nh + 2 * nkv) * hd)
        pos = torch.arange(t, dtype=torch.int32, device=r.dev) % 4096
        return {"qkv": qkv, "pos": pos, "dq": r.normal(t, nh, hd), "dk": r.normal(t, nkv, hd)}
    if kind == "swiglu":
        m, f = case["rows"], case["ffn"]
        return {"gate_up": r.normal(m, 2 * f), "dh": r.normal(m, f)}
    if kind == "head":
        m, h, v = case["rows"], case["hidden"], case["vocab"]
        targets = r.ints(v, m)
        targets[r.uniform(m) < 0.02] = -1  # padding rows
        return {"x": r.normal(m, h), "w": r.normal(v, h, std=0.02), "targets": targets}
    if kind == "block":
        t, d, f = case["tokens"], case["hidden"], case["ffn"]
        hd = d // case["heads"]
        return {
            "x": r.normal(1, t, d), "dy": r.normal(1, t, d),
            "attn_norm": r.around_one(d), "ffn_norm": r.around_one(d),
            "wqkv": r.normal((case["heads"] + 2 * case["kv_heads"]) * hd, d, std=0.02),
            "wo": r.normal(d, d, std=0.02), "w13": r.normal(2 * f, d, std=0.02), "w2": r.normal(d, f, std=0.02),
        }
    if kind == "adamw":
        n = case["numel"]
        f32 = torch.float32
        return {"p": r.normal(n, std=0.02, dtype=f32), "g": r.normal(n, std=1e-3, dtype=f32),
                "m": r.normal(n, std=1e-3, dtype=f32), "v": r.normal(n, std=1e-3, dtype=f32).square_()}
    if kind == "mlp":
        m, d, f = case["tokens"], case["hidden"], case["ffn"]
        return {"x": r.normal(m, d), "w13": r.normal(2 * f, d, std=0.02), "w2": r.normal(d, f, std=0.02)}
    if kind == "linear8":
        return {"x": r.normal(case["rows"], case["k"]), "w": r.normal(case["n"], case["k"], std=0.02)}
    t, h, e, k = case["tokens"], case["hidden"], case["experts"], case["topk"]
    scores = r.uniform(t, e)
    weights, idx = scores.topk(k, dim=-1)
    weights = weights / weights.sum(-1, keepdim=True)
    out = {"x": r.normal(t, h), "idx": idx.to(torch.int32).contiguous(), "weights": weights.contiguous()}
    if kind == "moe":
        out["expert_out"] = r.normal(t, h)
    else:
        out["expert_row"] = r.normal(e, h)  # what expert e returns for any of its rows
    return out


def prepare(case, seed):
    s = _inputs(case, seed)
    s["kind"] = kind = case["kind"]
    if kind == "ar_norm":
        from torchcomms_b200.ops.ar_norm import AllReduceRMSNorm

        s["layer"] = AllReduceRMSNorm(None, case["hidden"], EPS)
    elif kind == "norm":
        s["x"].requires_grad_(True)
        s["w"].requires_grad_(True)
    elif kind == "rope":
        from torchcomms_b200.ops.fused import rope_tables

        t, nh, nkv, hd = case["tokens"], case["heads"], case["kv_heads"], case["head_dim"]
        q, k, _ = s["qkv"].split([nh * hd, nkv * hd, nkv * hd], dim=-1)
        s["q"] = q.reshape(t, nh, hd).requires_grad_(True)
        s["k"] = k.reshape(t, nkv, hd).requires_grad_(True)
        s["cos"], s["sin"] = rope_tables(4096, hd, 500000.0, s["qkv"].device)
    elif kind == "swiglu":
        s["gate_up"].requires_grad_(True)
    elif kind == "head":
        s["x"].requires_grad_(True)
        s["w"].requires_grad_(True)
    elif kind == "block":
        from torchcomms_b200.models.llama import Block, LlamaConfig
        from torchcomms_b200.ops.fused import rope_tables

        cfg = LlamaConfig(dim=case["hidden"], n_layers=1, n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn_dim=case["ffn"],
                          vocab_size=1024, max_seq_len=4096)
        with torch.device("meta"):
            block = Block(cfg)
        s["names"] = [n for n, _ in block.named_parameters()]
        for n in s["names"]:
            setattr(block, n, torch.nn.Parameter(s[n]))
        s["block"] = block
        s["x"].requires_grad_(True)
        s["pos"] = torch.arange(case["tokens"], dtype=torch.int32, device=s["x"].device)
        s["cos"], s["sin"] = rope_tables(4096, cfg.head_dim, cfg.rope_theta, s["x"].device)
    elif kind == "mlp":
        from torchcomms_b200.ops.tp import AllGatherGemm, GemmReduceScatter, quantize_rows

        s["up"] = AllGatherGemm(None, m_local=case["tokens"], k=case["hidden"], fp8=case["fp8"])
        s["down"] = GemmReduceScatter(None, m=case["tokens"], n=case["hidden"], fp8=case["fp8"])
        if case["fp8"]:
            s["w13"], s["s13"] = quantize_rows(s["w13"])
            s["w2"], s["s2"] = quantize_rows(s["w2"])
    elif kind == "linear8":
        from torchcomms_b200.ops.tp import quantize_rows

        s["w"], s["sw"] = quantize_rows(s["w"])
    elif kind == "moe":
        from torchcomms_b200.ops.moe_ep import Buffer

        s["buf"] = Buffer(_comm(), case["tokens"], case["hidden"], case["experts"], case["topk"], fp8=case["fp8"])
    elif kind == "moe_ll":
        from torchcomms_b200.ops.moe_ep import LowLatencyBuffer

        s["buf"] = LowLatencyBuffer(_comm(), case["tokens"], case["hidden"], case["experts"], case["topk"], fp8=case["fp8"])
        rows = s["buf"].expert_output.shape[1]
        s["buf"].expert_output.copy_(s.pop("expert_row").unsqueeze(1).expand(-1, rows, -1))
        # First row of every (token, expert) pair's expert in the flattened [experts * rows] output.
        s["first_row"] = s["idx"].reshape(-1) * rows
    return s


# ------------------------------------------------------------------- one pass


def run(s):
    kind = s["kind"]
    if kind == "ar_norm":
        return {"out": s["layer"](s["x"], s["w"], residual=s["resid"]), "resid": s["resid"]}
    if kind == "norm":
        from torchcomms_b200.ops.fused import rms_norm

        y = rms_norm(s["x"], s["w"], EPS)
        dx, dw = torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])
        return {"y": y.detach(), "dx": dx, "dw": dw}
    if kind == "rope":
        from torchcomms_b200.ops.fused import apply_rope

        q = apply_rope(s["q"], s["pos"], s["cos"], s["sin"])
        k = apply_rope(s["k"], s["pos"], s["cos"], s["sin"])
        dq, dk = torch.autograd.grad((q, k), (s["q"], s["k"]), (s["dq"], s["dk"]))
        return {"q": q.detach(), "k": k.detach(), "dq": dq, "dk": dk}
    if kind == "swiglu":
        from torchcomms_b200.ops.fused import swiglu

        h = swiglu(s["gate_up"])
        (dgu,) = torch.autograd.grad(h, (s["gate_up"],), s["dh"])
        return {"h": h.detach(), "dgate_up": dgu}
    if kind == "head":
        from torchcomms_b200.ops.fused import linear_cross_entropy

        loss = linear_cross_entropy(s["x"], s["w"], s["targets"])
        dx, dw = torch.autograd.grad(loss, (s["x"], s["w"]))
        return {"loss": loss.detach(), "dx": dx, "dw": dw}
    if kind == "block":
        block = s["block"]
        y = block(s["x"], s["pos"], s["cos"], s["sin"])
        params = [getattr(block, n) for n in s["names"]]
        grads = torch.autograd.grad(y, [s["x"]] + params, s["dy"])
        return {"y": y.detach(), "dx": grads[0], **{"d" + n: g for n, g in zip(s["names"], grads[1:])}}
    if kind == "adamw":
        from torchcomms_b200.ops.fused import adamw_step_

        adamw_step_(s["p"], s["g"], s["m"], s["v"], lr=3e-4, weight_decay=0.1, step=100)
        return {"p": s["p"], "m": s["m"], "v": s["v"]}
    if kind == "mlp":
        from torchcomms_b200.ops.fused import swiglu

        gate_up = s["up"](s["w13"], s["x"], s.get("s13"))
        return {"y": s["down"](swiglu(gate_up), s["w2"], scale_w=s.get("s2"))}
    if kind == "linear8":
        from torchcomms_b200.ops.tp import gemm_e4m3_nt, quantize_rows

        q, scale = quantize_rows(s["x"])
        return {"q": q.view(torch.uint8), "scale": scale, "y": gemm_e4m3_nt(q, s["w"], scale, s["sw"])}
    if kind == "moe":
        buf, tokens = s["buf"], s["x"].shape[0]
        d = buf.dispatch(s["x"], s["idx"], s["weights"])
        src = d.src[:tokens]  # one rank: every token arrives, in an order of the kernel's choosing
        # The experts' last GEMM writes its rows next to the dispatched ones.
        torch.index_select(s["expert_out"], 0, src, out=buf.combine_input[:tokens])
        out = {"y": buf.combine()}
        at = torch.empty_like(src)
        at[src.long()] = torch.arange(tokens, dtype=src.dtype, device=src.device)
        out["rows"] = (d.x.view(torch.uint8) if d.scales is not None else d.x).index_select(0, at)
        if d.scales is not None:
            out["scales"] = d.scales.index_select(0, at)
        out["weights"] = d.topk_weights.index_select(0, at)
        return out
    buf = s["buf"]
    r = buf.dispatch(s["x"], s["idx"])
    # The rows of every (token, expert) pair, in the caller's order.
    at = s["first_row"] + r.send_slot.reshape(-1)
    rows = r.x.view(torch.uint8) if r.scales is not None else r.x
    out = {"rows": rows.view(-1, rows.shape[-1]).index_select(0, at), "count": r.count}
    if r.scales is not None:
        out["scales"] = r.scales.view(-1, r.scales.shape[-1]).index_select(0, at)
    out["y"] = buf.combine(s["idx"], s["weights"], r)
    return out


# ------------------------------------------------------- work and tolerance


def work(case):
    kind = case["kind"]
    if kind == "ar_norm":
        n = case["rows"] * case["hidden"]
        return {"bytes": 2 * (4 * n + case["hidden"]), "flops": 6 * n}
    if kind == "norm":
        n = case["rows"] * case["hidden"]
        return {"bytes": 2 * (4 * n + 2 * case["hidden"]), "flops": 14 * n}
    if kind == "rope":
        n = case["tokens"] * (case["heads"] + case["kv_heads"]) * case["head_dim"]
        return {"bytes": 2 * 4 * n + 4 * min(case["tokens"], 4096) * case["head_dim"], "flops": 6 * n}
    if kind == "swiglu":
        n = case["rows"] * case["ffn"]
        return {"bytes": 2 * 6 * n, "flops": 18 * n}
    if kind == "head":
        m, h, v = case["rows"], case["hidden"], case["vocab"]
        # x, dx, W and dW once; the logits are the path's own and need not reach memory.
        return {"bytes": 2 * (2 * m * h + 2 * v * h) + 8 * m, "flops": 6 * m * h * v}
    if kind == "block":
        t, d, f = case["tokens"], case["hidden"], case["ffn"]
        hd = d // case["heads"]
        weights = (case["heads"] + 2 * case["kv_heads"]) * hd * d + d * d + 3 * f * d
        return {"bytes": 2 * (2 * weights + 4 * d + 4 * t * d), "flops": 6 * t * weights + 7 * t * t * d}
    if kind == "adamw":
        return {"bytes": 28 * case["numel"], "flops": 14 * case["numel"]}
    if kind == "mlp":
        m, d, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * 2 * m * d + 3 * f * d * (1 if case["fp8"] else 2), "flops": 6 * m * d * f}
    if kind == "linear8":
        m, k, n = case["rows"], case["k"], case["n"]
        return {"bytes": 2 * m * k + m * k + n * k + 4 * (m + n) + 2 * m * n, "flops": 2 * m * k * n}
    t, h, k = case["tokens"], case["hidden"], case["topk"]
    row = h + h // 128 * 4 if case["fp8"] else 2 * h
    if kind == "moe":
        # Dispatch (read x, write rows), the experts' write (read, write), combine (read, write), the rows once more in token order.
        return {"bytes": t * (2 * h + 3 * row + 4 * h + 4 * h + 5 * 8 * k), "flops": 4 * t * h}
    # Dispatch (read x, write a row per pair), the rows once more in pair order, combine (a row per pair, one output).
    return {"bytes": t * (2 * h + k * 3 * row + k * 2 * h + 2 * h + 8 * k), "flops": 2 * t * k * h}


def tolerance(case):
    # About four times the distance from the 64-bit results that the paths show.
    kind = case["kind"]
    if kind in ("norm", "rope", "swiglu", "head", "moe", "moe_ll"):
        return {"rel": 0.008}  # results rounded to bf16
    if kind == "ar_norm":
        return {"rel": 0.01}  # two roundings in a row: the sum, then the normalised value
    if kind == "block":
        return {"rel": 0.035}  # a chain of bf16 intermediates
    if kind == "adamw":
        return {"rel": 3e-7}
    if kind == "mlp":
        # Activations that sit on an e4m3 rounding boundary fall either way.
        return {"rel": 0.06} if case["fp8"] else {"rel": 0.015}
    return {"rel": 0.008, "differ": 0.001}


# ------------------------------------------------------ the same in 64 bits


def _norm64(x, w):
    rstd = torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return x * rstd * w


def _rope64(x, pos, head_dim, inverse=False):
    inv = 1.0 / (500000.0 ** (torch.arange(0, head_dim, 2, dtype=torch.float32) / head_dim))
    ang = torch.outer(torch.arange(4096, dtype=torch.float32), inv)  # the tables are inputs: fp32 angles
    c = ang.cos().to(x.device)[pos.long()].to(F64).unsqueeze(1)
    s = ang.sin().to(x.device)[pos.long()].to(F64).unsqueeze(1)
    if inverse:
        s = -s
    a, b = x.reshape(*x.shape[:-1], -1, 2).unbind(-1)
    return torch.stack((a * c - b * s, a * s + b * c), -1).reshape(x.shape)


def _quant_rows(x):
    """e4m3 rows and fp32 row scales of a matrix, in plain torch."""
    x = x.float()
    scale = x.abs().amax(dim=1).clamp_min(1e-8) / 448.0
    return (x / scale.unsqueeze(1)).to(torch.float8_e4m3fn), scale


def _dequant_rows(x):
    q, scale = _quant_rows(x)
    return q.to(torch.float32).to(F64) * scale.to(F64).unsqueeze(1)


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "ar_norm":
        total = s["x"].to(F64) + s["resid"].to(F64)
        return {"out": _norm64(total, s["w"].to(F64)), "resid": total}
    if kind == "norm":
        x, w = s["x"].to(F64).requires_grad_(True), s["w"].to(F64).requires_grad_(True)
        y = _norm64(x, w)
        dx, dw = torch.autograd.grad(y, (x, w), s["dy"].to(F64))
        return {"y": y.detach(), "dx": dx, "dw": dw}
    if kind == "rope":
        t, nh, nkv, hd = case["tokens"], case["heads"], case["kv_heads"], case["head_dim"]
        q, k, _ = s["qkv"].to(F64).split([nh * hd, nkv * hd, nkv * hd], dim=-1)
        return {"q": _rope64(q.reshape(t, nh, hd), s["pos"], hd), "k": _rope64(k.reshape(t, nkv, hd), s["pos"], hd),
                "dq": _rope64(s["dq"].to(F64), s["pos"], hd, True), "dk": _rope64(s["dk"].to(F64), s["pos"], hd, True)}
    if kind == "swiglu":
        gu = s["gate_up"].to(F64).requires_grad_(True)
        gate, up = gu.chunk(2, dim=-1)
        h = torch.nn.functional.silu(gate) * up
        (dgu,) = torch.autograd.grad(h, (gu,), s["dh"].to(F64))
        return {"h": h.detach(), "dgate_up": dgu}
    if kind == "head":
        x, w, t = s["x"].to(F64), s["w"].to(F64), s["targets"]
        m, loss, dx, dw = x.shape[0], 0.0, torch.empty_like(x), torch.zeros_like(w)
        for a in range(0, m, 1024):
            xs, ts = x[a : a + 1024], t[a : a + 1024]
            keep = (ts >= 0).to(F64)
            logp = torch.log_softmax(xs @ w.t(), dim=-1)
            at = ts.clamp_min(0).unsqueeze(1)
            loss = loss - (logp.gather(1, at).squeeze(1) * keep).sum() / m
            g = logp.exp_()
            g.scatter_add_(1, at, torch.full_like(at, -1, dtype=F64))
            g.mul_((keep / m).unsqueeze(1))
            dx[a : a + 1024] = g @ w
            dw.addmm_(g.t(), xs)
        return {"loss": loss, "dx": dx, "dw": dw}
    if kind == "block":
        t, d, nh, nkv = case["tokens"], case["hidden"], case["heads"], case["kv_heads"]
        hd = d // nh
        names = ["attn_norm", "wqkv", "wo", "ffn_norm", "w13", "w2"]
        p = {n: s[n].to(F64).requires_grad_(True) for n in names}
        x = s["x"].to(F64).requires_grad_(True)
        pos = torch.arange(t, device=x.device)
        q, k, v = (_norm64(x[0], p["attn_norm"]) @ p["wqkv"].t()).split([nh * hd, nkv * hd, nkv * hd], dim=-1)
        q = _rope64(q.reshape(t, nh, hd), pos, hd).transpose(0, 1)
        k = _rope64(k.reshape(t, nkv, hd), pos, hd).repeat_interleave(nh // nkv, dim=1).transpose(0, 1)
        v = v.reshape(t, nkv, hd).repeat_interleave(nh // nkv, dim=1).transpose(0, 1)
        mask = torch.full((t, t), float("-inf"), dtype=F64, device=x.device).triu(1)
        o = torch.softmax(q @ k.transpose(1, 2) / math.sqrt(hd) + mask, dim=-1) @ v
        r = x[0] + o.transpose(0, 1).reshape(t, d) @ p["wo"].t()
        gate, up = (_norm64(r, p["ffn_norm"]) @ p["w13"].t()).chunk(2, dim=-1)
        y = (r + (torch.nn.functional.silu(gate) * up) @ p["w2"].t()).unsqueeze(0)
        grads = torch.autograd.grad(y, [x] + [p[n] for n in names], s["dy"].to(F64))
        return {"y": y.detach(), "dx": grads[0], **{"d" + n: g for n, g in zip(names, grads[1:])}}
    if kind == "adamw":
        p, g, m, v = (s[n].to(F64) for n in ("p", "g", "m", "v"))
        m = 0.9 * m + 0.1 * g
        v = 0.95 * v + 0.05 * g * g
        step = (m / (1 - 0.9**100)) / ((v / (1 - 0.95**100)).sqrt_() + 1e-8)
        return {"p": p * (1 - 3e-4 * 0.1) - 3e-4 * step, "m": m, "v": v}
    if kind == "mlp":
        cast = _dequant_rows if case["fp8"] else (lambda a: a.to(F64))
        gate, up = (cast(s["x"]) @ cast(s["w13"]).t()).chunk(2, dim=-1)
        h = torch.nn.functional.silu(gate) * up
        return {"y": cast(h) @ cast(s["w2"]).t()}
    if kind == "linear8":
        return {"q": None, "scale": s["x"].to(F64).abs().amax(dim=1) / 448.0, "y": _dequant_rows(s["x"]) @ _dequant_rows(s["w"]).t()}
    if kind == "moe":
        out = {"y": s["expert_out"].to(F64), "rows": None if case["fp8"] else s["x"].to(F64)}
        if case["fp8"]:
            out["scales"] = s["x"].to(F64).reshape(s["x"].shape[0], -1, 128).abs().amax(-1) / 448.0
        out["weights"] = s["weights"].to(F64)
        return out
    t, k = case["tokens"], case["topk"]
    pairs = s["x"].to(F64).repeat_interleave(k, dim=0)
    out = {"rows": None if case["fp8"] else pairs, "count": None}
    if case["fp8"]:
        out["scales"] = pairs.reshape(t * k, -1, 128).abs().amax(-1) / 448.0
    rows = s["expert_row"].to(F64)[s["idx"].long()]
    out["y"] = (rows * s["weights"].to(F64).unsqueeze(-1)).sum(1)
    return out
