"""bf16 GEMM with fused epilogues (tcgen05 kernel on CUDA, torch math on CPU).

``gemm(a, b)`` computes ``op(a) @ op(b).T`` where each operand is either
``[rows, K]`` (K-major, the default) or ``[K, rows]`` (``a_t`` / ``b_t``).
That covers the forward, dgrad and wgrad products of a dense layer
(reference: src/nn/engines/cuda_engine.cu:1652-1707) without a transpose pass.
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib

EPI_BIAS, EPI_GELU, EPI_DGELU, EPI_RESID, EPI_RELU, EPI_ATOMIC, EPI_OUT_F32, EPI_ACCUM = 1, 2, 4, 8, 16, 32, 64, 128
EPI_RELU_LAST = 512

LAUNCHES = {"count": 0}


def gelu_tanh(x: torch.Tensor) -> torch.Tensor:
    return torch.nn.functional.gelu(x, approximate="tanh")


def gelu_tanh_grad(x: torch.Tensor) -> torch.Tensor:
    k0, k1 = 0.7978845608028654, 0.044715
    u = k0 * (x + k1 * x ** 3)
    t = torch.tanh(u)
    return 0.5 * (1 + t) + 0.5 * x * (1 - t * t) * k0 * (1 + 3 * k1 * x * x)


def _ld(t: torch.Tensor) -> int:
    assert t.dim() == 2 and t.stride(1) == 1, "operands must be 2-D with a unit inner stride"
    return t.stride(0) if t.shape[0] > 1 else max(t.stride(0), t.shape[1])


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """An operand the TMA descriptors accept: unit inner stride, row pitch and base address multiples of 16 bytes.
    Tensors produced by the layers already are (their buffers are allocated with padded pitches); anything else -
    a gradient handed in by user code, an odd-width slice - is copied once into a padded buffer."""
    per16 = 16 // t.element_size()
    if t.dim() == 2 and t.stride(1) == 1 and t.data_ptr() % 16 == 0 and _ld(t) % per16 == 0:
        return t
    pitch = (t.shape[1] + per16 - 1) // per16 * per16
    buf = torch.zeros((t.shape[0], pitch), dtype=t.dtype, device=t.device)
    buf[:, :t.shape[1]].copy_(t)
    return buf[:, :t.shape[1]]


def _operand(t: torch.Tensor):
    """``(tensor, row pitch, address)`` of an operand that the TMA descriptors accept (:func:`_tma_ready`)."""
    s0, s1 = t.stride()
    if s1 == 1:
        r, c = t.shape
        ld = s0 if r > 1 else max(s0, c)
        addr = t.data_ptr()
        if not (ld & 7) and not (addr & 15):  # bf16: eight elements are 16 bytes
            return t, ld, addr
    t = _tma_ready(t)
    return t, _ld(t), t.data_ptr()


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_t: bool = False, b_t: bool = False,
         bias: Optional[torch.Tensor] = None, gelu: bool = False, save_preact: Optional[torch.Tensor] = None,
         dgelu_of: Optional[torch.Tensor] = None, relu: bool = False, residual: Optional[torch.Tensor] = None,
         out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None, accumulate: bool = False,
         atomic: bool = False, split_k: int = 0, force_bn: int = 0) -> torch.Tensor:
    """``out = epilogue(op(a) @ op(b).T)``.

    a: ``[M,K]`` (or ``[K,M]`` with ``a_t``); b: ``[N,K]`` (or ``[K,N]`` with ``b_t``).
    ``atomic`` adds into an fp32 ``out`` with red.add and enables split-K (used by wgrad,
    whose reduction dimension is the batch). Without it ``split_k=1`` keeps each sum in one range of K, so that a row's result
    does not depend on M; 0 takes what is fastest, which for few tiles and a long K is two or four ranges, added in order.
    """
    if a.is_cuda:
        r = _lib.gemm(_lib.load().tnnb_gemm_bf16, a, b, a_t, b_t, bias, save_preact if gelu else None, dgelu_of, residual, out, out_dtype,
                      (EPI_GELU if gelu else 0) | (EPI_RELU if relu else 0) | (EPI_ATOMIC if atomic else 0)
                      | (EPI_ACCUM if accumulate else 0), split_k, force_bn, _lib.status_addr(a.device), _lib.raw_stream())
        if r is not None:
            LAUNCHES["count"] += 1
            return r
    M, K = a.shape
    if a_t:
        M, K = K, M
    N, Kb = b.shape
    if b_t:
        N, Kb = Kb, N
    assert K == Kb, f"inner dimensions differ: {K} vs {Kb}"
    if atomic:
        assert out is not None and out.dtype == torch.float32
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype or a.dtype, device=a.device)
    else:
        assert out.shape == (M, N)

    if not a.is_cuda:
        A = (a.t() if a_t else a).float()
        B = (b.t() if b_t else b).float()
        r = A @ B.t()
        if bias is not None:
            r = r + bias.float()
        if gelu:
            if save_preact is not None:
                save_preact.copy_(r.to(save_preact.dtype))
                r = save_preact.float()
            r = gelu_tanh(r)
        if dgelu_of is not None:
            r = r * gelu_tanh_grad(dgelu_of.float())
        if relu:
            r = torch.relu(r)
        if residual is not None:
            r = r + residual.float()
        if atomic or accumulate:
            out.add_(r.to(out.dtype))
        else:
            out.copy_(r.to(out.dtype))
        return out

    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16
    a, lda, pa = _operand(a)
    b, ldb, pb = _operand(b)
    flags = 0
    if bias is not None:
        flags |= EPI_BIAS
        assert bias.dtype == torch.bfloat16 and bias.numel() == N
    if gelu:
        flags |= EPI_GELU
    if dgelu_of is not None:
        flags |= EPI_DGELU
    if relu:
        flags |= EPI_RELU
    if residual is not None:
        flags |= EPI_RESID
        assert residual.dtype == torch.bfloat16
    if atomic:
        flags |= EPI_ATOMIC
    elif out.dtype == torch.float32:
        flags |= EPI_OUT_F32
    if accumulate and not atomic:
        flags |= EPI_ACCUM
    aux = save_preact if gelu else dgelu_of
    lib = _lib.load()
    rc = lib.tnnb_gemm_bf16(
        pa, pb, out, M, N, K, int(a_t), int(b_t), lda, ldb, _ld(out),
        bias, dgelu_of, save_preact if gelu else None,
        _ld(aux) if aux is not None else 0, residual, _ld(residual) if residual is not None else 0,
        flags, split_k, force_bn, _lib.status_addr(a.device), _lib.raw_stream())
    _lib.check_rc(rc, "tnnb_gemm_bf16")
    LAUNCHES["count"] += 1
    return out


_NORM_DECLARED = False


def gemm_norm(a, b, bias, gamma, beta, mean, var, eps: float, relu: int, residual, split_k: int = 0) -> torch.Tensor:
    """``relu?(norm(a @ b.T [+ bias]) [+ residual])`` on a GPU, where ``norm`` is a batch norm over the columns with running
    statistics (fp32 ``mean``, ``var``; ``gamma``, ``beta`` bf16 or None). ``relu``: 0 none, 1 before the residual is added,
    2 after."""
    global _NORM_DECLARED
    lib = _lib.load()
    if not _NORM_DECLARED:
        import ctypes
        vp, ll, i, f = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
        _lib.declare(lib, "tnnb_gemm_bf16_norm", [vp, vp, vp, i, i, i, ll, ll, ll, vp, vp, vp, vp, vp, f, vp, ll, i, i, vp, vp])
        _NORM_DECLARED = True
    (M, K), N = a.shape, b.shape[0]
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16 and b.shape[1] == K and mean.numel() == N and var.numel() == N
    a, lda, pa = _operand(a)
    b, ldb, pb = _operand(b)
    out = _lib.empty(a, M, N)
    flags = (EPI_BIAS if bias is not None else 0) | (EPI_RESID if residual is not None else 0) | (0, EPI_RELU, EPI_RELU_LAST)[relu]
    rc = lib.tnnb_gemm_bf16_norm(pa, pb, out, M, N, K, lda, ldb, N, bias, gamma, beta, mean, var, eps, residual,
                                 N if residual is not None else 0, flags, split_k, _lib.status_addr(a.device), _lib.raw_stream())
    _lib.check_rc(rc, "tnnb_gemm_bf16_norm")
    LAUNCHES["count"] += 1
    return out


def gemm_batched(a: torch.Tensor, b: torch.Tensor, *, a_t: bool = False, b_t: bool = False,
                 out_dtype: Optional[torch.dtype] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``out[i] = op(a[i]) @ op(b[i]).T`` for every ``i`` of the leading dimension, in one launch of the batched
    tcgen05 kernel. a: ``[G, M, K]`` (``[G, K, M]`` with ``a_t``), b: ``[G, N, K]`` (``[G, K, N]`` with ``b_t``); the
    last dimension must be contiguous, the row pitch a multiple of 8 elements. ``out``: ``[G, M, N]`` bf16 or fp32,
    possibly a view with a padded row pitch."""
    G = a.shape[0]
    M = a.shape[2] if a_t else a.shape[1]
    K = a.shape[1] if a_t else a.shape[2]
    N = b.shape[2] if b_t else b.shape[1]
    assert b.shape[0] == G and (b.shape[1] if b_t else b.shape[2]) == K
    if out is None:
        out = torch.empty(G, M, N, dtype=out_dtype or a.dtype, device=a.device)
    if not a.is_cuda:
        A = (a.transpose(1, 2) if a_t else a).float()
        B = (b.transpose(1, 2) if b_t else b).float()
        out.copy_((A @ B.transpose(1, 2)).to(out.dtype))
        return out
    assert a.stride(2) == 1 and b.stride(2) == 1 and out.stride(2) == 1
    items = [Heads(t, 0, t.stride(1), G, 1, 0, t.stride(0), t.stride(0)) for t in (a, b, out)]
    gemm_heads(*items, M, N, K, G, a_t=a_t, b_t=b_t)
    return out


_HEADS_DECLARED = False


class Heads:
    """``count`` matrices ``[rows, cols]`` inside a 2-D tensor ``t``: item ``i`` is head ``(i + first) % heads`` of sequence
    ``(i + first) // heads``. ``stride_h`` / ``stride_b`` / ``ld``: elements between heads, sequences and rows."""
    __slots__ = ("t", "ptr", "ld", "heads", "seqs", "first", "stride_h", "stride_b")

    def __init__(self, t, offset, ld, heads, seqs, first, stride_h, stride_b):
        self.t, self.ptr = t, t.data_ptr() + offset * t.element_size()
        self.ld, self.heads, self.seqs, self.first, self.stride_h, self.stride_b = ld, heads, seqs, first, stride_h, stride_b


def gemm_heads(a: Heads, b: Heads, out: Heads, M: int, N: int, K: int, count: int, *, a_t: bool = False, b_t: bool = False) -> None:
    """``out[i] = op(a[i]) @ op(b[i]).T`` for ``count`` items in one launch (CUDA; operands bf16, ``out`` bf16 or fp32)."""
    global _HEADS_DECLARED
    import ctypes
    lib = _lib.load()
    if not _HEADS_DECLARED:
        vp, ll, i = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
        _lib.declare(lib, "tnnb_gemm_bf16_heads", [vp, vp, vp, i, i, i, i, i, ll, ll, ll, i, vp, vp, i, vp, vp])
        _HEADS_DECLARED = True
    assert a.t.dtype == torch.bfloat16 and b.t.dtype == torch.bfloat16 and out.t.dtype in (torch.bfloat16, torch.float32)
    layout = (ctypes.c_int * 9)(a.heads, a.seqs, a.first, b.heads, b.seqs, b.first, out.heads, out.seqs, out.first)
    strides = (ctypes.c_longlong * 6)(a.stride_h, a.stride_b, b.stride_h, b.stride_b, out.stride_h, out.stride_b)
    # (addresses only: both arrays live until the call returns)
    rc = lib.tnnb_gemm_bf16_heads(a.ptr, b.ptr, out.ptr, M, N, K, int(a_t), int(b_t), a.ld, b.ld, out.ld, count,
                                  ctypes.addressof(layout), ctypes.addressof(strides),
                                  64 if out.t.dtype == torch.float32 else 0, _lib.status_addr(a.t.device), _lib.raw_stream())
    _lib.check_rc(rc, "tnnb_gemm_bf16_heads")
    LAUNCHES["count"] += 1
