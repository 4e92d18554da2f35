"""One new token per sequence through all layers of a decoder in one native call (``csrc/decode.cu``).

``decode_layers`` takes the place of the layer loop when a forward pass against a ``PackedKVCache`` feeds at most one token
to each of at most 64 sequences, without gradients, on plain bf16 CUDA weights of the dense decoder layers
(``decoder_lm.DecoderLayer``) or the hybrid ones (``qwen3_5.Qwen35Layer``).  Everything else - prompts, sparse MLPs, sharded
weights, subclassed, patched, parametrised or hooked modules, norms of different eps, other head dims - returns ``None`` and
runs layer by layer.  The numbers are those of the layer loop up to the order of fp32 sums: every intermediate is rounded to
bf16 at the same place.
"""
from __future__ import annotations

from array import array
from functools import lru_cache
from typing import Optional

import torch

from ..ops import _cuda
from ..ops import gemm as gemm_ops
from .plain_call import global_hooks, own_forward

_cuda.register("b200_decode_layers", "decode", "ppi" + "pppp" + "fff" + "ppppp" + "p" + "l" + "pp" + "s")

MAX_SEQS = 64  # kDecSeqs of the kernels: per-sequence tables travel as kernel arguments
_BF16 = torch.bfloat16
_PARAM = torch.nn.Parameter


class _Unfit(Exception):
    pass


@lru_cache(maxsize=None)
def _sms(dev) -> int:
    return torch.cuda.get_device_properties(dev).multi_processor_count


def _plain(module, cls) -> dict:
    """Parameters of a module whose call is only the arithmetic of its class (``plain_call.own_call`` with the part that is the
    same for all modules of a class done once per pass, and without backward hooks: there is no backward pass)."""
    d = module.__dict__
    if type(module) is not cls or d["_forward_hooks"] or d["_forward_pre_hooks"] or "forward" in d:
        raise _Unfit
    return d["_parameters"]


def _fill(rec, items) -> None:
    """``rec[slot]`` = address of every plain bf16 weight ``(slot, weight, shape)``."""
    for slot, w, shape in items:
        if type(w) is not _PARAM or w.dtype is not _BF16 or w.shape != shape or not (w.is_cuda and w.is_contiguous()):
            raise _Unfit
        p = w.data_ptr()
        if p & 15:
            raise _Unfit
        rec[slot] = p


def _own(module, cls=torch.nn.Linear) -> dict:
    """Parameters of a projection.  Its layer reads the weight and never calls the module, so hooks on it do not matter, but a
    subclass (a parametrisation makes one) may compute its weight on access."""
    if type(module) is not cls:
        raise _Unfit
    return module.__dict__["_parameters"]


def _norm(module, cls, eps):
    own = _plain(module, cls)
    if module.__dict__.get("eps") != eps:  # one eps for all norms of the call
        raise _Unfit
    return own.get("weight")


def _attention(items, att, cls, norm_cls, eps, window, shapes, gated):
    _plain(att, cls)
    m = att.__dict__["_modules"]
    if getattr(att, "nsa", None) is not None or getattr(att, "window", (-1, -1))[0] != window:
        raise _Unfit
    q_shape, kv_shape, q_bias, kv_bias, head, o_shape, o_bias = shapes
    q, k, v, o = _own(m["q_proj"]), _own(m["k_proj"]), _own(m["v_proj"]), _own(m["o_proj"])
    items += ((1, q.get("weight"), q_shape), (2, k.get("weight"), kv_shape), (3, v.get("weight"), kv_shape), (11, o.get("weight"), o_shape))
    for slot, own, shape in ((5, q, q_bias), (6, k, kv_bias), (7, v, kv_bias)):
        if own.get("bias") is not None:
            items.append((slot, own["bias"], shape))
    if gated and o.get("bias") is not None:  # the ungated layer adds none
        items.append((19, o["bias"], o_bias))
    if gated or att.cfg.qk_norm:
        items += ((9, _norm(m["q_norm"], norm_cls, eps), head), (10, _norm(m["k_norm"], norm_cls, eps), head))


def _delta(items, net, cls, eps, H):
    own = _plain(net, cls)
    m = net.__dict__["_modules"]
    # the gated output norm is a weight without a call of its own; its eps stands at the layer
    if net.eps != eps or type(m["norm"]) is not torch.nn.Module:
        raise _Unfit
    key, val, hv = net.key_dim, net.value_dim, net.hv
    heads, conv = (hv, H), 2 * key + val
    items += ((1, _own(m["in_proj_qkv"]).get("weight"), (conv, H)), (2, _own(m["in_proj_z"]).get("weight"), (val, H)),
              (3, _own(m["in_proj_b"]).get("weight"), heads), (4, _own(m["in_proj_a"]).get("weight"), heads),
              (9, _own(m["conv1d"], torch.nn.Conv1d).get("weight"), (conv, 1, net.kernel)), (10, own.get("A_log"), (hv,)),
              (16, own.get("dt_bias"), (hv,)), (17, m["norm"].__dict__["_parameters"].get("weight"), (net.dv,)),
              (11, _own(m["out_proj"]).get("weight"), (H, val)))


def _delta_state(store, net, seqs, where):
    """Tail and state buffers of every live sequence: ``(pointers, new store entries)``; the old ones are read and new ones
    written, as in the layer loop: value heads that share key channels read the same old rows, and a caller may hold the state
    of an earlier token."""
    ptrs, new = [], []
    at, tail_shape, state_shape = where.get_device(), (net.kernel - 1, 2 * net.key_dim + net.value_dim), (net.hv, net.dk, net.dv)
    for i in seqs:
        tail, S = store.get(i, (None, None))
        if tail is None:
            tail = torch.zeros(tail_shape, dtype=_BF16, device=where.device)
        if S is None:
            S = torch.zeros(state_shape, dtype=torch.float32, device=where.device)
        if tail.shape != tail_shape or S.shape != state_shape or tail.get_device() != at or S.get_device() != at:
            raise _Unfit
        if not (tail.is_contiguous() and S.is_contiguous() and tail.dtype is _BF16 and S.dtype is torch.float32 and S.data_ptr() % 16 == 0):
            tail, S = tail.to(_BF16).contiguous(), S.float().clone(memory_format=torch.contiguous_format)
        tail_out, S_out = torch.empty_like(tail), torch.empty_like(S)
        ptrs += (tail.data_ptr(), tail_out.data_ptr(), S.data_ptr(), S_out.data_ptr())
        new.append((i, (tail_out, S_out), tail, S))  # the old ones until the kernels are queued
    return ptrs, new


def decode_layers(backbone, embeds: torch.Tensor, ctx) -> Optional[torch.Tensor]:
    cache = ctx.kv_cache
    M = embeds.shape[0]
    if (M > MAX_SEQS or not embeds.is_cuda or embeds.dtype is not _BF16 or torch.is_grad_enabled() or not ctx.causal
            or ctx.sp_size > 1 or ctx.tp_size > 1 or ctx.deepstack is not None or gemm_ops.LINEAR_BACKEND != "tcgen05" or global_hooks()):
        return None
    seqs = [i for i, n in enumerate(cache.new_lens) if n]
    if len(seqs) != M or any(cache.new_lens[i] != 1 for i in seqs):
        return None
    try:
        return _run(backbone, embeds, ctx, cache, seqs)
    except _Unfit:
        return None


def _run(backbone, embeds, ctx, cache, seqs):
    from .decoder_lm import Attention, DecoderLayer, RMSNorm, SwiGLUMLP

    cfg, dev, M = backbone.cfg, embeds.device, embeds.shape[0]
    H, I, D, nq, nkv = cfg.hidden_size, cfg.intermediate_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    if H % 8 or I % 8 or D not in (64, 128) or nq // nkv > 16 or (nq * D) % 8:
        raise _Unfit
    rot = ctx.cos.shape[-1]
    if rot % 2 or rot > D or ctx.cos.dtype is not torch.float32 or ctx.cos.shape[0] != M:
        raise _Unfit
    cache.decode_window = -1
    layers = backbone.layers._modules
    first = next(iter(layers.values()), None)
    if type(first) is DecoderLayer:
        cache.decode_window = getattr(first.self_attn, "window", (-1, -1))[0]
        hybrid, layer_cls, att_cls, norm_cls, norm_off = None, DecoderLayer, Attention, RMSNorm, 0.0
    else:
        from . import qwen3_5 as hybrid

        if type(first) is not hybrid.Qwen35Layer:
            raise _Unfit
        layer_cls, att_cls, norm_cls, norm_off = hybrid.Qwen35Layer, hybrid.GatedAttention, hybrid.ZRMSNorm, 1.0
    if not all(map(own_forward, (layer_cls, att_cls, norm_cls, SwiGLUMLP))) or (hybrid is not None and not own_forward(hybrid.GatedDeltaNet)):
        raise _Unfit
    table, types, nets = array("Q"), array("i"), []
    rec0 = [0] * 24
    hk = hv = taps = 0
    gated, eps, window = hybrid is not None, cfg.rms_norm_eps, cache.decode_window
    q_rows = nq * D * (2 if gated else 1)
    shapes = ((q_rows, H), (nkv * D, H), (q_rows,), (nkv * D,), (D,), (H, nq * D), (H,))
    row, wide, narrow = (H,), (I, H), (H, I)
    for layer in layers.values():
        _plain(layer, layer_cls)
        m = layer.__dict__["_modules"]
        rec, items, mlp = rec0[:], [], m["mlp"]
        _plain(mlp, SwiGLUMLP)
        if mlp.tp_group is not None:
            raise _Unfit
        if gated and "linear_attn" in m:
            net = m["linear_attn"]
            _delta(items, net, hybrid.GatedDeltaNet, eps, H)
            if net.dk != 128 or net.dv != 128 or net.hv % 8 or net.hv % net.hk or not 2 <= net.kernel <= 8:
                raise _Unfit
            hk, hv, taps = net.hk, net.hv, net.kernel
            nets.append(net)
            types.append(2)
        else:
            att = m["self_attn"]
            _attention(items, att, att_cls, norm_cls, eps, window, shapes, gated)
            k, v = cache.slabs(att.layer_idx, nkv, D, _BF16, dev)
            if k.dtype is not _BF16 or k.device != dev or k.shape[1:] != (nkv, D):
                raise _Unfit
            rec[16], rec[17] = k.data_ptr(), v.data_ptr()
            types.append(1 if gated else 0)
        mm = mlp.__dict__["_modules"]
        items += ((0, _norm(m["input_layernorm"], norm_cls, eps), row), (12, _norm(m["post_attention_layernorm"], norm_cls, eps), row),
                  (13, _own(mm["gate_proj"]).get("weight"), wide), (14, _own(mm["up_proj"]).get("weight"), wide),
                  (15, _own(mm["down_proj"]).get("weight"), narrow))
        _fill(rec, items)
        table.extend(rec)
    last = [0]
    _fill(last, ((0, _norm(backbone._modules["norm"], norm_cls, eps), row),))
    final = last[0]

    # the states are replaced after the call: what declines here leaves them as they were
    gdn, news = array("Q"), []
    for net in nets:
        store = cache.state.setdefault(net.layer_idx, {})
        ptrs, new = _delta_state(store, net, seqs, embeds)
        gdn.extend(ptrs)
        news.append((store, new))
    have = array("i", [cache.had[i] for i in seqs])
    base = array("i", [cache.base[i] for i in seqs])
    longest = max(have) + 1
    if cache.decode_window >= 0:
        longest = min(longest, cache.decode_window + 1)
    # shares of a key head: enough to fill the chip about twice or 512 keys each (a batch waits for its longest sequence),
    # whichever are more, and at least 64 keys each
    splits = max(1, min(max(-(-2 * _sms(dev) // (nkv * M)), -(-longest // 512)), -(-longest // 64), 64))
    np_ = max(nq * D * 2 + 2 * nkv * D if len(nets) < len(types) else 0, (2 * hk + 2 * hv) * 128 + 2 * hv)
    work = torch.empty(2 * M * (np_ + max(nq * D, hv * 128) + I + H) + 4096, dtype=torch.uint8, device=dev)
    n_ws = M * nkv * splits * (nq // nkv) * (D + 2)
    shares = torch.empty(n_ws if splits > 1 else 1, dtype=torch.float32, device=dev)
    count = cache.decode_counters(M * nkv, dev)
    res = embeds.clone(memory_format=torch.contiguous_format)
    hidden = torch.empty_like(res)
    cos, sin = ctx.cos.contiguous(), ctx.sin.contiguous()
    dims = array("i", [M, H, nq, nkv, D, rot, I, cache.decode_window, splits, hk, hv, taps])
    a = lambda x: x.buffer_info()[0]  # noqa: E731
    _cuda.call("b200_decode_layers", a(table), a(types), len(types), a(dims), a(base), a(have), a(gdn) if nets else None,
               float(cfg.rms_norm_eps), norm_off, D ** -0.5, cos.data_ptr(), sin.data_ptr(), res.data_ptr(), hidden.data_ptr(), final,
               work.data_ptr(), work.numel(), shares.data_ptr(), count.data_ptr(), _cuda.stream())
    for store, new in news:
        for i, entry, _, _ in new:
            store[i] = entry
    return hidden
