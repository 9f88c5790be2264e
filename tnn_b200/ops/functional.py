"""``torch.autograd`` bridges to the hand-written kernels, for code that lives in ordinary PyTorch modules.

The framework's own layers (``nn/layers.py``) call explicit forward / backward kernels and never touch autograd. These
functions expose the same kernels to a model written with ``torch.nn`` and trained with ``loss.backward()``: each is a
``torch.autograd.Function`` whose forward and backward are one or two kernel launches (tcgen05 GEMM with fused bias /
GELU epilogues, fused flash attention on the packed QKV matrix, layer norm with fused residual add, streaming softmax
cross-entropy). On CPU tensors the same calls run the plain-torch references in ``ops/raw.py``, so a module built on
them runs anywhere.

    y = F.linear(x, w, b)                       # x [..., K] @ w[N, K]^T + b, optional fused tanh-GELU
    h, s = F.add_layer_norm(x, delta, g, b)     # s = x + delta ; h = LN(s)
    o = F.causal_self_attention(qkv, heads)     # qkv [B, S, 3E] packed q | k | v
    l = F.cross_entropy(logits, labels)         # mean over rows

Gradients with respect to parameters are accumulated in fp32 and rounded once to the parameter's dtype, by autograd or, for
the weights of few rows, where they are computed.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import raw
from .gemm import gemm


def _flat2d(t: torch.Tensor) -> torch.Tensor:
    return t.reshape(-1, t.shape[-1])


def _is_plain(t: torch.Tensor) -> bool:
    """True for a tensor that is its memory and nothing more, which a kernel may take by address: no graph is recorded on it
    (``create_graph``), and it is no batch of gradients (``is_grads_batched``, ``vmap``) and no dual number."""
    f = torch._C._functorch
    return not ((t.requires_grad and torch.is_grad_enabled()) or f.is_legacy_batchedtensor(t) or f.is_functorch_wrapped_tensor(t)
                or torch.autograd.forward_ad._current_level >= 0)


def _in_one_launch(rows: int, m: int, n: int) -> bool:
    """Whether the gradient of an ``[m, n]`` weight is summed up (in fp32) by one CTA per tile and leaves the product as bf16, the type
    autograd would cast it to: one launch. Otherwise the rows are split over the SMs and added into fp32 zeros, which autograd
    then casts: three launches, but no CTA walks through more than a few K blocks.

    Us of both forms, split first. Eager, where the host pays for each launch: 1024 rows, 64 x 64 18.2 and 7.7; 2048 rows, 64 x 64
    17.7 and 12.2, 320 x 320 18.3 and 12.4, 2048 x 2048 33.5 and 15.8. Captured in a graph, where the launches saved are nearly
    free, the walk decides: 1024 rows, 64 x 64 8.5 and 8.4, 320 x 320 9.1 and 8.7; 2048 rows, 64 x 64 8.6 and 12.9, 320 x 320 9.3 and
    13.2, 768 x 768 (36 tiles of 128 x 128) 12.2 and 13.8, 1024 x 1024 (64) 16.2 and 14.6, 4096 x 1024 29.3 and 16.2. From 4096 rows the
    split is faster for small weights in either case (64 x 64 18.1 and 21.1). Relative error against fp64 in all of them: that of
    the rounding to bf16, 1.66e-3 (before it 2.4e-7 and, for 2048 rows in one walk, 2.1e-6)."""
    if rows <= 1024:
        return rows > 0
    tiles = (m + 127) // 128 * ((n + 127) // 128)
    return rows <= 2048 and (tiles >= 64 or not torch.cuda.is_current_stream_capturing())


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b, gelu):
        x2 = _flat2d(x).contiguous()
        z = torch.empty(x2.shape[0], w.shape[0], dtype=x2.dtype, device=x2.device) if gelu else None
        y = gemm(x2, w, bias=b, gelu=gelu, save_preact=z, split_k=1)  # a row's result does not depend on how many there are
        ctx.save_for_backward(x2, w, z)
        ctx.has_bias, ctx.gelu, ctx.in_shape = b is not None, gelu, x.shape
        return y.reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w, z = ctx.saved_tensors
        dy2 = _flat2d(dy).contiguous()
        if ctx.gelu:  # back through the activation first: dz = dy * gelu'(z) from the saved pre-activation
            dy2 = raw.act_bwd(z, dy2, "gelu")
        dx = gemm(dy2, w, b_t=True).reshape(ctx.in_shape) if ctx.needs_input_grad[0] else None
        dw = db = None
        if ctx.needs_input_grad[1]:
            if dy2.is_cuda and w.dtype == dy2.dtype == torch.bfloat16 and _in_one_launch(dy2.shape[0], *w.shape):
                dw = gemm(dy2, x2, a_t=True, b_t=True)
            else:
                dw = torch.zeros(w.shape, dtype=torch.float32, device=w.device)
                gemm(dy2, x2, a_t=True, b_t=True, out=dw, atomic=True)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = torch.zeros(w.shape[0], dtype=torch.float32, device=w.device)
            raw.colsum_accum(dy2, db)
        return dx, dw, db, None


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, gelu: bool = False) -> torch.Tensor:
    """``gelu(x @ weight.T + bias)`` with the bias and the tanh-GELU applied in the GEMM epilogue."""
    return _Linear.apply(x, weight, bias, gelu)


class _AddLayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, gamma, beta, eps):
        x2 = _flat2d(x).contiguous()
        d2 = _flat2d(delta).contiguous() if delta is not None else None
        s, h, mean, rstd = raw.layernorm_fwd(x2, d2, gamma, beta, eps)
        s = x2 if s is None else s
        ctx.save_for_backward(s, mean, rstd, gamma)
        ctx.has_delta, ctx.shape = delta is not None, x.shape
        ctx.mark_non_differentiable(mean, rstd)
        return h.reshape(x.shape), s.reshape(x.shape)

    @staticmethod
    def backward(ctx, dh, ds):
        s, mean, rstd, gamma = ctx.saved_tensors
        C = s.shape[1]
        dg = torch.zeros(C, dtype=torch.float32, device=s.device) if gamma is not None else None
        db = torch.zeros(C, dtype=torch.float32, device=s.device) if gamma is not None else None
        dres = _flat2d(ds).contiguous() if ds is not None else None
        dx, _ = raw.layernorm_bwd(_flat2d(dh).contiguous(), s, mean, rstd, gamma, dres, False, 0.0, 0, dg, db)
        dx = dx.reshape(ctx.shape)
        return dx, (dx if ctx.has_delta else None), dg, db, None


def add_layer_norm(x: torch.Tensor, delta: Optional[torch.Tensor], gamma: Optional[torch.Tensor],
                   beta: Optional[torch.Tensor], eps: float = 1e-5) -> Tuple[torch.Tensor, torch.Tensor]:
    """``s = x + delta`` (``delta`` may be None) and ``h = LayerNorm(s)`` over the last dimension in one pass.
    Returns ``(h, s)``: the pre-LN transformer block keeps ``s`` as its residual stream."""
    return _AddLayerNorm.apply(x, delta, gamma, beta, eps)


def layer_norm(x: torch.Tensor, gamma: Optional[torch.Tensor], beta: Optional[torch.Tensor], eps: float = 1e-5) -> torch.Tensor:
    return _AddLayerNorm.apply(x, None, gamma, beta, eps)[0]


class _CausalSelfAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, heads, causal, scale):
        B, S, E3 = qkv.shape
        E = E3 // 3
        D = E // heads
        q2 = qkv.reshape(B * S, E3).contiguous()
        out, lse = raw.attn_fwd(q2, B, S, heads, D, causal, scale)
        ctx.save_for_backward(q2, out, lse)
        ctx.dims = (B, S, heads, D, causal, scale)
        return out.reshape(B, S, E)

    @staticmethod
    def backward(ctx, dout):
        q2, out, lse = ctx.saved_tensors
        B, S, H, D, causal, scale = ctx.dims
        dqkv = raw.attn_bwd(q2, out, dout.reshape(B * S, H * D).contiguous(), lse, B, S, H, D, causal, scale)
        return dqkv.reshape(B, S, 3 * H * D), None, None, None


def causal_self_attention(qkv: torch.Tensor, heads: int, causal: bool = True, scale: Optional[float] = None) -> torch.Tensor:
    """Flash attention on the packed projection ``qkv [B, S, 3E]`` (``q | k | v``, heads contiguous inside each):
    no head transposes, no score matrix in memory. ``scale`` defaults to ``1 / sqrt(head size)``."""
    D = qkv.shape[-1] // 3 // heads
    if qkv.dim() != 3 or qkv.shape[-1] != 3 * heads * D or not D:
        raise ValueError(f"qkv {tuple(qkv.shape)} is not [B, S, 3 * {heads} heads * head size]")
    return _CausalSelfAttention.apply(qkv, heads, causal, float(scale) if scale is not None else D ** -0.5)


class _CrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, labels):
        l2 = _flat2d(logits)
        rows, vocab = l2.shape
        # the gradient of the mean loss is produced in the same pass and kept for backward
        loss, corrects, grad = raw.softmax_ce(l2, labels, vocab, 1.0 / rows, 1.0 / rows)
        ctx.save_for_backward(grad)
        ctx.shape = logits.shape
        ctx.mark_non_differentiable(corrects)
        return loss.reshape(()), corrects

    @staticmethod
    def backward(ctx, dloss, _):
        (grad,) = ctx.saved_tensors
        dlogits = raw.scale_by(grad, dloss) if _is_plain(dloss) else (grad.float() * dloss).to(grad.dtype)
        return dlogits.reshape(ctx.shape), None


def cross_entropy(logits: torch.Tensor, labels: torch.Tensor, return_corrects: bool = False):
    """Mean softmax cross-entropy over all rows of ``logits [..., V]`` with integer ``labels [...]``; with
    ``return_corrects`` also the number of rows whose arg-max equals the label (computed by the same kernel)."""
    loss, corrects = _CrossEntropy.apply(logits, labels)
    return (loss, corrects) if return_corrects else loss
