"""SwiGLU: ``silu(gate) * up`` and the fused MLP built on it.

``swiglu_mlp`` runs gate and up projections in ONE tcgen05 GEMM whose epilogue applies
SiLU*mul while the accumulators are still in TMEM; gate/up pre-activations are kept
(bf16) for backward so no GEMM is recomputed.  The reference gets the elementwise part
from Liger's ``LigerSwiGLUMLP`` and the GEMMs from cuBLAS
(src/lmms_engine/models/qwen2/monkey_patch.py:76-77, 114-115).
"""
from __future__ import annotations

import torch

from . import _cuda
from . import gemm as _gemm


def swiglu_ref(g: torch.Tensor, u: torch.Tensor) -> torch.Tensor:
    return (torch.nn.functional.silu(g.float()) * u.float()).to(g.dtype)


class _SwiGLUFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, g, u):
        g = g.contiguous()
        u = u.contiguous()
        h = torch.empty_like(g)
        _cuda.call("b200_swiglu_fwd", g.data_ptr(), u.data_ptr(), h.data_ptr(), g.numel(), _cuda.stream())
        ctx.save_for_backward(g, u)
        return h

    @staticmethod
    def backward(ctx, dh):
        g, u = ctx.saved_tensors
        dh = dh.contiguous()
        dg = torch.empty_like(g)
        du = torch.empty_like(u)
        _cuda.call(
            "b200_swiglu_bwd", dh.data_ptr(), g.data_ptr(), u.data_ptr(), dg.data_ptr(), du.data_ptr(), g.numel(),
            _cuda.stream(),
        )
        return dg, du


def swiglu(g: torch.Tensor, u: torch.Tensor) -> torch.Tensor:
    if g.is_cuda and g.dtype == torch.bfloat16 and g.numel() % 8 == 0:
        return _SwiGLUFn.apply(g, u)
    return swiglu_ref(g, u)


class _SwiGLUMLPFn(torch.autograd.Function):
    """down( silu(x Wg^T) * (x Wu^T) ) with the first two GEMMs and the activation fused."""

    @staticmethod
    def forward(ctx, x, wg, wu, wd):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        h, g, u = _gemm.gemm_swiglu(x2, wg, wu, store_gu=True)
        y = _gemm.matmul_nt(h, wd)
        ctx.save_for_backward(x2, wg, wu, wd, g, u)
        ctx.shp = shp
        return y.view(*shp[:-1], wd.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, wg, wu, wd, g, u = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        # recompute h (elementwise) instead of keeping a third [T, I] tensor alive
        h = torch.empty_like(g)
        _cuda.call("b200_swiglu_fwd", g.data_ptr(), u.data_ptr(), h.data_ptr(), g.numel(), _cuda.stream())
        dwd = _gemm.matmul_tn(dy2, h) if ctx.needs_input_grad[3] else None
        dh = _gemm.matmul_nn(dy2, wd, out=h)  # reuse h's storage
        # dg, du overwrite g, u in place
        _cuda.call(
            "b200_swiglu_bwd", dh.data_ptr(), g.data_ptr(), u.data_ptr(), g.data_ptr(), u.data_ptr(), g.numel(),
            _cuda.stream(),
        )
        dwg = _gemm.matmul_tn(g, x2) if ctx.needs_input_grad[1] else None
        dwu = _gemm.matmul_tn(u, x2) if ctx.needs_input_grad[2] else None
        dx = None
        if ctx.needs_input_grad[0]:
            dx = _gemm.matmul_nn(g, wg)
            dx = _gemm.gemm(u, wu, b_mn_major=True, cin=dx, beta=1.0, out=dx)
            dx = dx.view(ctx.shp)
        return dx, dwg, dwu, dwd


def swiglu_mlp(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, wd: torch.Tensor) -> torch.Tensor:
    native = (
        x.is_cuda
        and x.dtype == torch.bfloat16
        and wg.dtype == torch.bfloat16
        and x.shape[-1] % 8 == 0
        and wg.shape[0] % 8 == 0
        and wg.is_contiguous()
        and wu.is_contiguous()
        and wd.is_contiguous()
    )
    if native and _gemm.LINEAR_BACKEND == "tcgen05":
        return _SwiGLUMLPFn.apply(x, wg, wu, wd)
    lin = torch.nn.functional.linear
    return lin(swiglu(lin(x, wg), lin(x, wu)), wd)


class _GatedMLPFn(torch.autograd.Function):
    """``swiglu_mlp`` with biases and an inner width that may be any number (3420 in the windowed vision tower): rows of the
    inner activations are padded to 16 bytes, which is all that TMA needs, and the products stop at the true width."""

    @staticmethod
    def forward(ctx, x, wg, bg, wu, bu, wd, bd):
        shp = x.shape
        x2 = _rows16(x.reshape(-1, shp[-1]))
        # whole padded rows are saved: a hook on saved tensors (offloading) copies a view without its padding, which the
        # elementwise pass of the backward would read past
        h, g, u = _gemm.gemm_swiglu(x2, wg, wu, True, bg, bu, whole_rows=True)
        y = _gemm.gemm(h[:, :wg.shape[0]], _padded(wd), bias=bd)
        # h too, as three linears keep it: computing it again is a pass over all three
        ctx.save_for_backward(x2, wg, wu, wd, g, u, h)
        ctx.shp, ctx.biases = shp, (bg is not None, bu is not None, bd is not None)
        return y.view(*shp[:-1], wd.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, wg, wu, wd, g, u, h = ctx.saved_tensors
        need = ctx.needs_input_grad
        dy2 = _rows16(dy.reshape(-1, dy.shape[-1]))
        M, inter = x2.shape[0], wg.shape[0]
        ld = (inter + 7) // 8 * 8
        # the elementwise pass runs over whole padded rows: the padding holds anything and is not read again
        dh, dg, du = (torch.empty((M, ld), dtype=g.dtype, device=g.device) for _ in range(3))
        dwd = None
        if need[5]:
            dwd = torch.empty((wd.shape[0], ld), dtype=wd.dtype, device=wd.device)[:, :inter]
            _gemm.matmul_tn(dy2, h[:, :inter], out=dwd)
        _gemm.matmul_nn(dy2, _padded(wd), out=dh[:, :inter])
        _cuda.call("b200_swiglu_bwd", dh.data_ptr(), g.data_ptr(), u.data_ptr(), dg.data_ptr(), du.data_ptr(), M * ld, _cuda.stream())
        dg, du = dg[:, :inter], du[:, :inter]
        dx = None
        if need[0]:
            dx = _gemm.matmul_nn(dg, wg)
            dx = _gemm.gemm(du, wu, b_mn_major=True, cin=dx, beta=1.0, out=dx).view(ctx.shp)
        dwg = _gemm.matmul_tn(dg, x2) if need[1] else None
        dwu = _gemm.matmul_tn(du, x2) if need[3] else None
        has_g, has_u, has_d = ctx.biases
        return (dx, dwg, _gemm.column_sum(dg) if has_g and need[2] else None, dwu, _gemm.column_sum(du) if has_u and need[4] else None, dwd,
                _gemm.column_sum(dy2) if has_d and need[6] else None)


def _rows16(t):
    return t if t.is_contiguous() and t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def _padded(wd):
    """The down projection with rows on 16-byte boundaries (one copy of the weight where its width is not a multiple of 8);
    the padding lies outside every tensor map."""
    n, i = wd.shape
    if i % 8 == 0:
        return wd
    return torch.empty((n, (i + 7) // 8 * 8), dtype=wd.dtype, device=wd.device)[:, :i].copy_(wd)


# Rows x width x inner width from which an inner width that is no multiple of 8 takes the fused function: below, host time decides,
# and the library's three linears launch less.  Forward + backward, us, linears / fused: 100 x 1280 x 3420 360 / 515, 2000 x 256 x
# 516 375 / 503, 22000 x 256 x 516 (2.9e9) 700 / 683, 2000 x 1280 x 3420 (8.8e9) 854 / 508, 22000 x 1280 x 3420 6540 / 1640.
UNALIGNED_MIN = 1 << 31


def gated_mlp(x, wg, bg, wu, bu, wd, bd) -> torch.Tensor:
    """``(silu(x wg^T + bg) * (x wu^T + bu)) wd^T + bd``; any of the biases may be ``None``.

    One fused function: as three linears, an inner width that is no multiple of 8 went to the library's unaligned kernels (49 of
    the 94 device ms of an eight-block tower with 3420 over 21.9k patches, forward + backward).  Such a width takes the linears
    where the products are small (``UNALIGNED_MIN``)."""
    plain = (torch.Tensor, torch.nn.Parameter)
    native = (
        _gemm.LINEAR_BACKEND == "tcgen05" and x.is_cuda and x.dtype == torch.bfloat16 and x.numel() > 0 and wg.shape == wu.shape
        and (wg.shape[0] % 8 == 0 or x.numel() * wg.shape[0] >= UNALIGNED_MIN)
        and x.shape[-1] % 8 == 0 and wg.shape[1] == x.shape[-1] and wd.shape[0] % 8 == 0 and wd.shape[1] == wg.shape[0]
        and all(type(w) in plain and w.is_cuda and w.dtype == torch.bfloat16 and w.is_contiguous() and w.data_ptr() % 16 == 0
                for w in (wg, wu, wd))
        and all(b is None or (type(b) in plain and b.is_cuda and b.dtype == torch.bfloat16 and b.is_contiguous() and b.shape == (w.shape[0],))
                for b, w in ((bg, wg), (bu, wu), (bd, wd)))
    )
    if native:
        return _GatedMLPFn.apply(x, wg, bg, wu, bu, wd, bd)
    g, u = _gemm.linear(x, wg, bg), _gemm.linear(x, wu, bu)
    return _gemm.linear(swiglu(g, u), wd, bd)
