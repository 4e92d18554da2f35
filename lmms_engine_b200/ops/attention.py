"""Packed variable-length attention.

``varlen_attn`` keeps the signature of the reference dispatcher
(src/lmms_engine/kernels/attention.py:20-51): flat ``q [Tq, Hq, D]``, ``k/v [Tk, Hkv, D]``
plus ``cu_seqlens`` boundaries, causal or full, optional left sliding window, GQA.
CUDA bf16 inputs run the tcgen05 kernels of ``csrc/attention_sm100.cu``; anything else
runs a per-document fp32 reference (also the oracle of the GPU tests).
"""
from __future__ import annotations

import math
import os
from typing import Optional, Tuple

import torch

from . import _cuda

_cuda.register("b200_attn_fwd", "attention_sm100", "ppppppp" + "iiiiii" + "llll" + "fii" + "ps")
_cuda.register("b200_attn_bwd", "attention_sm100", "ppppppppppppp" + "iiiiii" + "llllllll" + "fii" + "ps")
_cuda.register("b200_qk_norm_rope_parts", "elementwise", "")
_cuda.register("b200_qk_norm_rope_fwd", "elementwise", "ppppppp" + "liii" + "ll" + "f" + "s")
_cuda.register("b200_qk_norm_rope_bwd", "elementwise", "pppppppp" + "liii" + "ll" + "s")
_cuda.register("b200_attn_small_fwd", "attention_small", "ppppppp" + "iiiiii" + "llll" + "fii" + "ps")
_cuda.register("b200_attn_small_bwd", "attention_small", "ppppppppppp" + "iiiiii" + "llllllll" + "fii" + "ps")
_cuda.register("b200_attn_bwd_v2", "attention_bwd_sm100", "pppppppppppp" + "iiiiii" + "llllllll" + "fii" + "ps")

# "split": dK/dV and dQ in two reduction-free kernels (default); "fused": the single-kernel
# variant that reduces dQ across key blocks with fp32 red.global
BACKWARD_IMPL = os.environ.get("LMMS_B200_ATTN_BWD", "split")


def varlen_attn_ref(q, k, v, cu_q, cu_k, causal=True, softmax_scale=None, window_left: int = -1):
    """fp32 per-document attention; bottom-right aligned causal mask like flash-attn."""
    Hq, Hkv, D = q.shape[1], k.shape[1], q.shape[2]
    scale = softmax_scale if softmax_scale is not None else 1.0 / math.sqrt(D)
    out = torch.empty_like(q)
    cq, ck = cu_q.tolist(), cu_k.tolist()
    for d in range(len(cq) - 1):
        qd = q[cq[d] : cq[d + 1]].float().transpose(0, 1)  # [Hq, Lq, D]
        kd = k[ck[d] : ck[d + 1]].float().transpose(0, 1)
        vd = v[ck[d] : ck[d + 1]].float().transpose(0, 1)
        if Hq != Hkv:
            kd = kd.repeat_interleave(Hq // Hkv, 0)
            vd = vd.repeat_interleave(Hq // Hkv, 0)
        lq, lk = qd.shape[1], kd.shape[1]
        s = torch.matmul(qd, kd.transpose(1, 2)) * scale
        qi = torch.arange(lq, device=q.device).unsqueeze(1) + (lk - lq)
        kj = torch.arange(lk, device=q.device).unsqueeze(0)
        mask = torch.ones(lq, lk, dtype=torch.bool, device=q.device)
        if causal:
            mask &= kj <= qi
        if window_left >= 0:
            mask &= kj >= qi - window_left
        s = s.masked_fill(~mask, float("-inf"))
        p = torch.softmax(s, dim=-1)
        p = torch.nan_to_num(p, nan=0.0)
        out[cq[d] : cq[d + 1]] = torch.matmul(p, vd).transpose(0, 1).to(q.dtype)
    return out


def _token_stride_ok(t: torch.Tensor) -> bool:
    return t.stride(2) == 1 and t.stride(1) == t.shape[2] and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0


# Longest document of the one-CTA-per-document kernels (csrc/attention_small.cu).  They need the caller's word that no
# document is longer, so only callers that build the boundaries on the host from the lengths themselves pass ``max_len``.
# The line lies at the tile: a longer document would need a loop over keys, which the tcgen05 kernels do better.
SMALL_DOC = 64


def _fwd(q, k, v, cu_q, cu_k, causal, scale, window_left, small=False):
    Tq, Hq, D = q.shape
    Tk, Hkv, _ = k.shape
    o = torch.empty((Tq, Hq, D), dtype=q.dtype, device=q.device)
    lse = torch.empty((Hq, Tq), dtype=torch.float32, device=q.device)
    st = _cuda.status_word(q.device)
    _cuda.call(
        "b200_attn_small_fwd" if small else "b200_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
        lse.data_ptr(), cu_q.data_ptr(), cu_k.data_ptr(), cu_q.numel() - 1, Tq, Tk, Hq, Hkv, D, q.stride(0), k.stride(0),
        v.stride(0), o.stride(0), float(scale), int(causal), int(window_left), st.data_ptr(), _cuda.stream(),
    )
    return o, lse


def _bwd(q, k, v, o, lse, do, cu_q, cu_k, causal, scale, window_left, dq, dk, dv, small=False):
    """Writes the gradients into ``dq, dk, dv`` (rows of contiguous heads at any 16-byte row stride)."""
    do = do if _token_stride_ok(do) else do.clone(memory_format=torch.contiguous_format)
    Tq, Hq, D = q.shape
    Tk, Hkv, _ = k.shape
    st = _cuda.status_word(q.device)
    # the single-kernel variant converts its fp32 accumulator into a dense dq
    out_q = dq if BACKWARD_IMPL == "split" or small or dq.is_contiguous() else torch.empty((Tq, Hq, D), dtype=q.dtype, device=q.device)
    strides = (q.stride(0), k.stride(0), v.stride(0), o.stride(0), do.stride(0), out_q.stride(0), dk.stride(0), dv.stride(0))
    tail = (cu_q.data_ptr(), cu_k.data_ptr(), cu_q.numel() - 1, Tq, Tk, Hq, Hkv, D, *strides, float(scale), int(causal),
            int(window_left), st.data_ptr(), _cuda.stream())
    if small:
        _cuda.call("b200_attn_small_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
                   dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), *tail)
        return
    delta = torch.empty((Hq, Tq), dtype=torch.float32, device=q.device)
    if BACKWARD_IMPL == "split":
        # two reduction-free kernels (dK/dV per key block, dQ per query block)
        _cuda.call("b200_attn_bwd_v2", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
                   delta.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), *tail)
        return
    dq_acc = torch.empty((Tq, Hq, D), dtype=torch.float32, device=q.device)
    _cuda.call("b200_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
               delta.data_ptr(), dq_acc.data_ptr(), out_q.data_ptr(), dk.data_ptr(), dv.data_ptr(), *tail)
    if out_q is not dq:
        dq.copy_(out_q)


class _VarlenAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, cu_q, cu_k, causal, scale, window_left):
        q = q if _token_stride_ok(q) else q.contiguous()
        k = k if _token_stride_ok(k) else k.contiguous()
        v = v if _token_stride_ok(v) else v.contiguous()
        o, lse = _fwd(q, k, v, cu_q, cu_k, causal, scale, window_left)
        ctx.save_for_backward(q, k, v, o, lse, cu_q, cu_k)
        ctx.cfg = (causal, scale, window_left)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse, cu_q, cu_k = ctx.saved_tensors
        dq, dk, dv = (torch.empty(t.shape, dtype=q.dtype, device=q.device) for t in (q, k, v))
        _bwd(q, k, v, o, lse, do, cu_q, cu_k, *ctx.cfg, dq, dk, dv)
        return dq, dk, dv, None, None, None, None, None


def _rotate(x, ldx, y, cos, sin, heads, D, conj):
    _cuda.call("b200_rope_apply", x.data_ptr(), y.data_ptr(), cos.data_ptr(), sin.data_ptr(), y.shape[0], heads, D, D, ldx, y.stride(0),
               int(conj), _cuda.stream())


def _rotated(qkv, cos, sin, n_q, n_kv, D, wq, wk, eps):
    """q and k heads of the projection rows, normalised per head where weights are given, rotated: ``([T, n_q + n_kv, D], rstd)``."""
    T = qkv.shape[0]
    rot = torch.empty((T, n_q + n_kv, D), dtype=qkv.dtype, device=qkv.device)
    if wq is None:
        _rotate(qkv, qkv.stride(0), rot, cos, sin, n_q + n_kv, D, False)
        return rot, None
    rstd = torch.empty((T, n_q + n_kv), dtype=torch.float32, device=qkv.device)
    _cuda.call("b200_qk_norm_rope_fwd", qkv.data_ptr(), rot.data_ptr(), wq.data_ptr(), wk.data_ptr(), cos.data_ptr(), sin.data_ptr(),
               rstd.data_ptr(), T, n_q, n_kv, D, qkv.stride(0), rot.stride(0), float(eps), _cuda.stream())
    return rot, rstd


class _RopeAttnFn(torch.autograd.Function):
    """(Per-head RMSNorm of q and k +) rotary embedding + attention on the rows of ONE projection
    ``[T, (n_q + 2 n_kv) * D]`` (heads of q, then k, then v).

    As separate operations on slices of the projection, the backward pass builds three zero-filled gradients of its whole
    size and adds them (five passes over it, twice that for a 3-way view); here the attention backward writes its three
    gradients into the rows of one buffer and the rotation (and norm) runs in place on the q and k part.  Query and key heads
    are neighbours in a row, so both are handled by one launch."""

    @staticmethod
    def forward(ctx, qkv, wq, wk, cos, sin, cu, n_q, n_kv, D, eps, causal, scale, window_left, small):
        rot, rstd = _rotated(qkv, cos, sin, n_q, n_kv, D, wq, wk, eps)
        v = qkv[:, (n_q + n_kv) * D:].view(qkv.shape[0], n_kv, D)
        o, lse = _fwd(rot[:, :n_q], rot[:, n_q:], v, cu, cu, causal, scale, window_left, small)
        ctx.save_for_backward(rot, qkv, o, lse, cu, cos, sin, wq, wk, rstd)
        ctx.cfg = (causal, scale, window_left)
        ctx.dims = (n_q, n_kv, D, small)
        return o

    @staticmethod
    def backward(ctx, do):
        rot, qkv, o, lse, cu, cos, sin, wq, wk, rstd = ctx.saved_tensors
        n_q, n_kv, D, small = ctx.dims
        T = rot.shape[0]
        v = qkv[:, (n_q + n_kv) * D:].view(T, n_kv, D)
        d = torch.empty((T, n_q + 2 * n_kv, D), dtype=rot.dtype, device=rot.device)
        _bwd(rot[:, :n_q], rot[:, n_q:], v, o, lse, do, cu, cu, *ctx.cfg, d[:, :n_q], d[:, n_q:n_q + n_kv], d[:, n_q + n_kv:], small)
        dwq = dwk = None
        if wq is None:
            _rotate(d, d.stride(0), d, cos, sin, n_q + n_kv, D, True)
        else:
            part = torch.empty((_cuda.fn("b200_qk_norm_rope_parts")(), 2, D), dtype=torch.float32, device=rot.device)
            _cuda.call("b200_qk_norm_rope_bwd", d.data_ptr(), qkv.data_ptr(), wq.data_ptr(), wk.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                       rstd.data_ptr(), part.data_ptr(), T, n_q, n_kv, D, qkv.stride(0), d.stride(0), _cuda.stream())
            dwq, dwk = part.sum(0).to(wq.dtype).unbind(0)
        return (d.view(T, -1), dwq, dwk) + (None,) * 11


def _fused_rows_ok(qkv, cos, sin, n_q, n_kv, D, wq, wk) -> bool:
    """Rows, tables and norm weights that the fused kernels read: bf16 rows on 16-byte boundaries, whole-head rotation, fp32
    tables of exactly these rows; with norms, heads of 64 or 128 (a lane group owns a head)."""
    def plain(w):
        return (type(w) in (torch.Tensor, torch.nn.Parameter) and w.is_cuda and w.dtype == torch.bfloat16 and w.shape == (D,)
                and w.is_contiguous() and w.data_ptr() % 16 == 0)
    return (qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.dim() == 2 and qkv.shape[0] > 0 and qkv.shape[1] == (n_q + 2 * n_kv) * D
            and qkv.stride(1) == 1 and qkv.stride(0) % 8 == 0 and qkv.data_ptr() % 16 == 0 and D % 8 == 0 and D <= 128
            and n_q % n_kv == 0 and cos.dtype == sin.dtype == torch.float32 and cos.is_cuda and sin.is_cuda
            and cos.shape == sin.shape == (qkv.shape[0], D) and not (cos.requires_grad or sin.requires_grad)
            and cos.data_ptr() % 16 == 0 and sin.data_ptr() % 16 == 0
            and (wq is None) == (wk is None) and (wq is None or (D in (64, 128) and plain(wq) and plain(wk))))


def rope_attention(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, cu_seqlens: torch.Tensor, n_q: int, n_kv: int, D: int,
                   causal: bool, softmax_scale: float, window_left: int = -1, max_len: Optional[int] = None,
                   norms: Optional[Tuple[torch.Tensor, torch.Tensor, float]] = None) -> Optional[torch.Tensor]:
    """Rotary embedding over whole heads (behind a per-head RMSNorm with ``norms`` = weights of q and k, eps), then attention,
    from one projection's rows; ``None`` where the fused form does not apply (other dtypes, partial rotation, rows off 16-byte
    boundaries) and the caller runs the operations one by one.
    ``max_len``: no document is longer, from a caller that made the boundaries; ``None`` where it is not known."""
    wq, wk, eps = norms if norms is not None else (None, None, 0.0)
    if not _fused_rows_ok(qkv, cos, sin, n_q, n_kv, D, wq, wk):
        return None
    cu = cu_seqlens.to(torch.int32).contiguous()
    small = max_len is not None and max_len <= SMALL_DOC and cu.numel() <= 65536
    return _RopeAttnFn.apply(qkv, wq, wk, cos.contiguous(), sin.contiguous(), cu, n_q, n_kv, D, float(eps), bool(causal),
                             float(softmax_scale), int(window_left), small)


def rope_heads(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, n_q: int, n_kv: int, D: int,
               norms: Optional[Tuple[torch.Tensor, torch.Tensor, float]] = None) -> Optional[Tuple[torch.Tensor, torch.Tensor]]:
    """The first half of ``rope_attention`` without gradients: ``q [T, n_q, D]`` and ``k [T, n_kv, D]`` as they enter attention (and
    a key / value cache), or ``None``."""
    wq, wk, eps = norms if norms is not None else (None, None, 0.0)
    if torch.is_grad_enabled() or not _fused_rows_ok(qkv, cos, sin, n_q, n_kv, D, wq, wk):
        return None
    rot, _ = _rotated(qkv, cos.contiguous(), sin.contiguous(), n_q, n_kv, D, wq, wk, eps)
    return rot[:, :n_q], rot[:, n_q:]


def varlen_attn(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    cu_seqlens_q: torch.Tensor,
    cu_seqlens_k: Optional[torch.Tensor] = None,
    max_seqlen_q: Optional[int] = None,
    max_seqlen_k: Optional[int] = None,
    causal: bool = True,
    softmax_scale: Optional[float] = None,
    window_size: Tuple[int, int] = (-1, -1),
    dropout_p: float = 0.0,
    backend: Optional[str] = None,
) -> torch.Tensor:
    """Attention over packed documents.  ``max_seqlen_*`` are accepted for signature
    compatibility; the kernel derives its schedule from ``cu_seqlens`` on the device, so
    no host synchronisation is needed to obtain them."""
    if dropout_p != 0.0:
        raise NotImplementedError("attention dropout is not supported")
    if cu_seqlens_k is None:
        cu_seqlens_k = cu_seqlens_q
    D = q.shape[-1]
    scale = softmax_scale if softmax_scale is not None else 1.0 / math.sqrt(D)
    window_left = int(window_size[0]) if window_size is not None else -1
    window_right = int(window_size[1]) if window_size is not None and len(window_size) > 1 else -1
    if window_right >= 0 and not causal:
        # a causal mask already limits the right side to 0; a finite right window without it is a
        # different mask, which neither the kernel nor the reference formulation below implements
        raise NotImplementedError(f"window_size[1] = {window_right} (right window) is only supported together with causal=True")
    native = q.is_cuda and q.dtype == torch.bfloat16 and D % 8 == 0 and D <= 128 and backend != "reference"
    if native:
        cu_q = cu_seqlens_q.to(torch.int32).contiguous()
        cu_k = cu_seqlens_k.to(torch.int32).contiguous()
        return _VarlenAttnFn.apply(q, k, v, cu_q, cu_k, bool(causal), float(scale), window_left)
    return varlen_attn_ref(q, k, v, cu_seqlens_q, cu_seqlens_k, causal, scale, window_left)
