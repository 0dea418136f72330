"""Autograd wrappers around the fused sm_100a model kernels.

CUDA tensors always take the hand-written kernels (``_comms.ops``); there is no
silent eager fallback on a GPU.  CPU tensors take a plain PyTorch restatement
of the same math so that the training engine can be exercised with the gloo
backend on machines without a GPU.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .. import _comms

_k = _comms.ops

__all__ = [
    "rms_norm",
    "swiglu",
    "apply_rope",
    "rope_tables",
    "linear_cross_entropy",
    "adamw_step_",
    "kernel_launch_count",
]


def kernel_launch_count() -> int:
    """Kernels launched by this library since process start."""
    return int(_k.kernel_launch_count())


_PLAIN = (torch.Tensor, torch.nn.Parameter)


def _native(*tensors: torch.Tensor) -> bool:
    """Whether the native autograd nodes may be asked (they look at the rest themselves): no tensor subclasses, no
    compilation, which traces the autograd functions below."""
    return all(type(t) in _PLAIN for t in tensors) and not torch.compiler.is_compiling()


# ------------------------------------------------------------------ RMSNorm


class _RmsNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        y, rstd = _k.rmsnorm_fwd(x, w, eps)
        ctx.save_for_backward(x, w, rstd)
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w, rstd = ctx.saved_tensors
        dx, dw = _k.rmsnorm_bwd(dy.contiguous(), x, w, rstd)
        return dx, dw, None


def rms_norm(x: torch.Tensor, w: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    if x.is_cuda:
        y = _k.rms_norm(x, w, eps) if _native(x, w) else None
        return _RmsNorm.apply(x.contiguous(), w, eps) if y is None else y
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()
    return y.to(x.dtype)


def rms_norm_skip(x: torch.Tensor, w: torch.Tensor, eps: float = 1e-5) -> tuple[torch.Tensor, torch.Tensor]:
    """``(x, rms_norm(x, w))``: the residual stream and its norm, whose gradients meet in one kernel."""
    out = _k.rms_norm_skip(x, w, eps) if x.is_cuda and _native(x, w) else None
    return (x, rms_norm(x, w, eps)) if out is None else (out[0], out[1])


def add_rms_norm(x: torch.Tensor, delta: torch.Tensor, w: torch.Tensor, eps: float = 1e-5) -> tuple[torch.Tensor, torch.Tensor]:
    """``(s, rms_norm(s, w))`` for ``s = x + delta``."""
    out = _k.add_rms_norm(x, delta, w, eps) if x.is_cuda and _native(x, delta, w) else None
    return rms_norm_skip(x + delta, w, eps) if out is None else (out[0], out[1])


# ------------------------------------------------------------------- SwiGLU


class _SwiGlu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate_up):
        ctx.save_for_backward(gate_up)
        return _k.swiglu_fwd(gate_up)

    @staticmethod
    def backward(ctx, dh):
        (gate_up,) = ctx.saved_tensors
        return _k.swiglu_bwd(dh.contiguous(), gate_up)


def swiglu(gate_up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` for ``gate_up = [..., 2*ffn]`` (gate first)."""
    if gate_up.is_cuda:
        h = _k.swiglu(gate_up) if _native(gate_up) else None
        return _SwiGlu.apply(gate_up.contiguous()) if h is None else h
    gate, up = gate_up.float().chunk(2, dim=-1)
    return (F.silu(gate) * up).to(gate_up.dtype)


# --------------------------------------------------------------------- RoPE


def rope_tables(max_pos: int, head_dim: int, theta: float, device) -> tuple[torch.Tensor, torch.Tensor]:
    inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, dtype=torch.float32) / head_dim))
    ang = torch.outer(torch.arange(max_pos, dtype=torch.float32), inv)
    return ang.cos().to(device).contiguous(), ang.sin().to(device).contiguous()


class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, pos, cos_t, sin_t):
        ctx.save_for_backward(pos, cos_t, sin_t)
        return _k.rope(x, pos, cos_t, sin_t, False)

    @staticmethod
    def backward(ctx, dy):
        pos, cos_t, sin_t = ctx.saved_tensors
        return _k.rope(dy, pos, cos_t, sin_t, True), None, None, None


def apply_rope(x: torch.Tensor, pos: torch.Tensor, cos_t: torch.Tensor, sin_t: torch.Tensor) -> torch.Tensor:
    """Rotates interleaved pairs of ``x = [tokens, heads, head_dim]`` by the angle of ``pos[token]``."""
    if x.is_cuda:
        y = _k.apply_rope(x, pos, cos_t, sin_t) if _native(x, pos, cos_t, sin_t) else None
        return _Rope.apply(x, pos, cos_t, sin_t) if y is None else y
    xf = x.float().reshape(*x.shape[:-1], -1, 2)
    c = cos_t[pos.long()].unsqueeze(-2)  # [tokens, 1, hd/2]
    s = sin_t[pos.long()].unsqueeze(-2)
    a, b = xf[..., 0], xf[..., 1]
    out = torch.stack((a * c - b * s, a * s + b * c), dim=-1)
    return out.reshape(x.shape).to(x.dtype)


def split_rope(qkv: torch.Tensor, pos: torch.Tensor, cos_t: torch.Tensor, sin_t: torch.Tensor, heads: int,
               kv_heads: int) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """Rotated queries, rotated keys and values, each ``[tokens, heads or kv_heads, head_dim]``, out of the fused
    projection ``qkv = [tokens, (heads + 2 * kv_heads) * head_dim]``."""
    if qkv.is_cuda and _native(qkv, pos, cos_t, sin_t):
        out = _k.split_rope(qkv, pos, cos_t, sin_t, heads, kv_heads)
        if out is not None:
            return out[0], out[1], out[2]
    t, hd = qkv.shape[0], qkv.shape[1] // (heads + 2 * kv_heads)
    q, k, v = qkv.split([heads * hd, kv_heads * hd, kv_heads * hd], dim=-1)
    return (apply_rope(q.reshape(t, heads, hd), pos, cos_t, sin_t), apply_rope(k.reshape(t, kv_heads, hd), pos, cos_t, sin_t),
            v.reshape(t, kv_heads, hd))


# ------------------------------------------------------- decoder block


def block_in(x: torch.Tensor, norm: torch.Tensor, wqkv: torch.Tensor, pos: torch.Tensor, cos_t: torch.Tensor, sin_t: torch.Tensor,
             heads: int, kv_heads: int, eps: float = 1e-5) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """What a decoder block does before attention: ``x = [tokens, dim]`` (for the residual), and queries, keys and values of
    ``split_rope(rms_norm(x) @ wqkv.T)``."""
    if x.is_cuda and _native(x, norm, wqkv, pos, cos_t, sin_t):
        out = _k.block_in(x, norm, wqkv, pos, cos_t, sin_t, heads, kv_heads, eps)
        if out is not None:
            return out[0], out[1], out[2], out[3]
    x, h = rms_norm_skip(x, norm, eps)
    return (x, *split_rope(F.linear(h, wqkv), pos, cos_t, sin_t, heads, kv_heads))


def block_out(x: torch.Tensor, o: torch.Tensor, wo: torch.Tensor, norm: torch.Tensor, w13: torch.Tensor, w2: torch.Tensor,
              eps: float = 1e-5) -> torch.Tensor:
    """What a decoder block does after attention (``o = [tokens, heads * head_dim]``): ``s + swiglu(rms_norm(s) @ w13.T) @ w2.T``
    with ``s = x + o @ wo.T``."""
    if x.is_cuda and _native(x, o, wo, norm, w13, w2):
        y = _k.block_out(x, o, wo, norm, w13, w2, eps)
        if y is not None:
            return y
    x, h = add_rms_norm(x, F.linear(o, wo), norm, eps)
    return x + F.linear(swiglu(F.linear(h, w13)), w2)


# ------------------------------------------------- linear + cross entropy


def _worth_padding(rows: int, weight: int) -> bool:
    """Whether a head off the 16-byte grid works on a zero-padded copy of its weight (``weight`` elements).

    The three products on two-element accesses take about 0.04 us longer per million weight elements and row, and as
    long again for reading the weight as for 128 rows. The copy costs a read and a write of the weight, which they win
    back, and 35 us of host time for its launches; a pass forward and backward has the GPU wait for the host (172 us)
    until the products are that much longer. Such a pass without and with the copy, in us: at 3844 M (200 rows, 11.7 M
    elements) 251 and 208, at 4097 M (128, 16 M) 236 and 205, at 4126 M (4096, 1 M) 304 and 206, at 4800 M (64, 25 M)
    245 and 212; below, at 2500 M (512, 3.9 M) 175 and 206; above, at 16 G (512, 25 M) 663 and 214, at 64 G (1, 501 M)
    1960 and 1485. From 24 M elements on, fewer rows take the copy as well (16 rows, 25 M: 189 and 208, even at 32
    rows): their products are as accurate as the others' that way (error of dx 0.0017, without it 0.0034).
    """
    return rows > 0 and (weight >= 24 << 20 or weight * (rows + 128) >= 4 << 30)


class _LinearCrossEntropy(torch.autograd.Function):
    """``mean(cross_entropy(x @ W^T, targets))`` without keeping the logits.

    Rows are processed in chunks: one GEMM makes a chunk of logits, a kernel
    turns it in place into its own gradient while emitting the per-row loss,
    and two more GEMMs fold that gradient into ``dx`` and ``dW``.  The
    gradients are therefore ready when forward returns; backward only scales
    them by the incoming gradient of the loss.  bf16 heads on the GPU take
    ``_comms.ops.head``, whose first GEMM leaves the statistics that the
    gradient needs; what it does not take goes operator by operator.
    """

    @staticmethod
    def forward(ctx, x, weight, targets, chunk_rows):
        out = _k.head(x, weight, targets, chunk_rows) if x.is_cuda and _native(x, weight, targets) else None
        if out is not None:
            ctx.save_for_backward(out[1], out[2])
            ctx.own = not _k.saved_tensor_hooks_active()
            return out[0]
        rows = x.shape[0]
        # Mean over all rows; rows with a negative target contribute zero.
        scale = 1.0 / max(rows, 1)
        dx = torch.empty_like(x)
        dw = torch.empty_like(weight) if x.is_cuda and rows else torch.zeros_like(weight)
        loss_sum = torch.zeros((), dtype=torch.float32, device=x.device)
        vocab = weight.shape[0]
        # Rows of a vocabulary that is no multiple of 8 start off 16-byte boundaries, which costs the three GEMMs their
        # tiled loads and stores. A copy of the weight with a few zero rows more puts logits and weight back on them:
        # their logits are zero, stay zero, and add nothing.
        pad = -vocab % 8 if x.is_cuda and x.dtype == weight.dtype == torch.bfloat16 and _worth_padding(rows, weight.numel()) else 0
        wide = F.pad(weight, (0, 0, 0, pad)) if pad else weight
        for r0 in range(0, rows, chunk_rows):
            r1 = min(rows, r0 + chunk_rows)
            logits = x[r0:r1] @ wide.t()
            if x.is_cuda:
                dlogits = logits[:, :vocab] if pad else logits
                loss = _k.cross_entropy_fwd_bwd_(dlogits, targets[r0:r1].contiguous(), scale)
            else:
                lf = logits.float()
                loss = F.cross_entropy(lf, targets[r0:r1], reduction="none", ignore_index=-1)
                p = torch.softmax(lf, dim=-1)
                onehot = F.one_hot(targets[r0:r1].clamp_min(0), lf.shape[-1]).float()
                dlogits = ((p - onehot) * (targets[r0:r1] >= 0).unsqueeze(-1) * scale).to(x.dtype)
            loss_sum += loss.sum()
            if x.is_cuda:
                torch.mm(logits, wide, out=dx[r0:r1])  # the kernel left the gradient in the logits
            else:
                dx[r0:r1] = dlogits @ weight
            if x.is_cuda and r0 == 0:
                torch.mm(dlogits.t(), x[r0:r1], out=dw)  # the first chunk needs no zeroed gradient to add to
            else:
                dw.addmm_(dlogits.t(), x[r0:r1])
        ctx.save_for_backward(dx, dw)
        # The gradients belong to this node alone unless a hook was handed them.
        ctx.own = x.is_cuda and not _k.saved_tensor_hooks_active()
        return loss_sum * scale

    @staticmethod
    def backward(ctx, dloss):
        dx, dw = ctx.saved_tensors
        if dx.is_cuda and _native(dx, dw, dloss):
            # A backward that frees the graph hands them out themselves; the gradient of the weight is the size of the
            # weight, and a copy of it would take longer than the loss kernel.
            last = ctx.own and not torch._C._autograd._get_current_graph_task_keep_graph()
            return *_k.scale_both_by(dx, dw, dloss, last), None, None
        return dx * dloss.to(dx.dtype), dw * dloss.to(dw.dtype), None, None


def linear_cross_entropy(x: torch.Tensor, weight: torch.Tensor, targets: torch.Tensor, chunk_rows: int = 4096) -> torch.Tensor:
    """Mean token cross-entropy of the logits ``x @ weight.T`` (``x``: [rows, dim]).

    The forward pass holds the logits of ``chunk_rows`` rows and the gradient of the weight; for a bf16 vocabulary that is
    no multiple of 8 also their ``dx`` in fp32, and where the width is no multiple of 8 either, from the sizes of
    ``_worth_padding`` on, a padded copy of the weight. A vocabulary padded by the caller needs neither.
    """
    return _LinearCrossEntropy.apply(x.contiguous(), weight, targets, chunk_rows)


# -------------------------------------------------------------------- AdamW


def adamw_step_(p, g, m, v, *, lr, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.0, step=1, grad_scale=1.0) -> None:
    """In-place AdamW on flat fp32 tensors (bias-corrected, decoupled weight decay)."""
    if p.is_cuda:
        _k.adamw_step_(p, g, m, v, lr, beta1, beta2, eps, weight_decay, step, grad_scale)
        return
    gr = g * grad_scale
    m.mul_(beta1).add_(gr, alpha=1 - beta1)
    v.mul_(beta2).addcmul_(gr, gr, value=1 - beta2)
    mhat = m / (1 - beta1**step)
    vhat = v / (1 - beta2**step)
    p.mul_(1 - lr * weight_decay).addcdiv_(mhat, vhat.sqrt() + eps, value=-lr)
