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
from .plain_call import global_hooks, own_call

_cuda.register("b200_decode_layers", "decode", "ppi" + "pppp" + "fff" + "ppppp" + "p" + "l" + "pp" + "s")

MAX_SEQS = 64  # kDecSeqs of the kernels: per-sequence tables travel as kernel arguments
_BF16 = torch.bfloat16


class _Unfit(Exception):
    pass


@lru_cache(maxsize=None)
def _sms(dev) -> int:
    return torch.cuda.get_device_properties(dev).multi_processor_count


def _plain(module, cls) -> dict:
    """Parameters of a module whose call is only the arithmetic of its class."""
    if not own_call(module, cls):
        raise _Unfit
    return module._parameters


def _at(w, shape) -> int:
    if w is None or w.dtype is not _BF16 or type(w) is not torch.nn.Parameter or not w.is_cuda or w.shape != shape or not w.is_contiguous():
        raise _Unfit
    p = w.data_ptr()
    if p & 15:
        raise _Unfit
    return p


def _opt(w, shape) -> int:
    return 0 if w is None else _at(w, shape)


def _norm(module, cls, cfg, width) -> int:
    own = _plain(module, cls)
    if module.eps != cfg.rms_norm_eps:  # one eps for all norms of the call
        raise _Unfit
    return _at(own.get("weight"), (width,))


def _weight(module, shape, cls=torch.nn.Linear) -> int:
    """Weight of a projection.  Its layer reads the weight and never calls the module, so hooks on it do not matter, but a
    subclass may compute its weight on access."""
    if type(module) is not cls:
        raise _Unfit
    return _at(module._parameters.get("weight"), shape)


def _mlp(rec, mlp, cls, H, I):
    _plain(mlp, cls)
    if mlp.tp_group is not None:
        raise _Unfit
    m = mlp._modules
    rec[13] = _weight(m["gate_proj"], (I, H))
    rec[14] = _weight(m["up_proj"], (I, H))
    rec[15] = _weight(m["down_proj"], (H, I))


def _attention(rec, att, cls, norm_cls, cfg, cache, dev, H, nq, nkv, D, gated):
    _plain(att, cls)
    m = att._modules
    if getattr(att, "nsa", None) is not None or getattr(att, "window", (-1, -1))[0] != cache.decode_window:
        raise _Unfit
    rows = nq * D * (2 if gated else 1)
    for i, (name, n) in enumerate((("q_proj", rows), ("k_proj", nkv * D), ("v_proj", nkv * D))):
        rec[1 + i] = _weight(m[name], (n, H))
        rec[5 + i] = _opt(m[name]._parameters.get("bias"), (n,))
    if gated or att.cfg.qk_norm:
        rec[9] = _norm(m["q_norm"], norm_cls, cfg, D)
        rec[10] = _norm(m["k_norm"], norm_cls, cfg, D)
    rec[11] = _weight(m["o_proj"], (H, nq * D))
    rec[19] = _opt(m["o_proj"]._parameters.get("bias"), (H,)) if gated else 0  # the ungated layer adds none
    k, v = cache.slabs(att.layer_idx, nkv, D, _BF16, dev)
    if k.dtype is not _BF16 or k.device != dev or k.shape[1:] != (nkv, D):
        raise _Unfit
    rec[16], rec[17] = k.data_ptr(), v.data_ptr()


def _delta(rec, net, cls, cfg, H):
    own = _plain(net, cls)
    m = net._modules
    # the gated output norm is a weight without a call of its own; its eps stands at the layer
    if net.eps != cfg.rms_norm_eps or type(m["norm"]) is not torch.nn.Module:
        raise _Unfit
    key, val, hv = net.key_dim, net.value_dim, net.hv
    for i, (name, n) in enumerate((("in_proj_qkv", 2 * key + val), ("in_proj_z", val), ("in_proj_b", hv), ("in_proj_a", hv))):
        rec[1 + i] = _weight(m[name], (n, H))
    rec[9] = _weight(m["conv1d"], (2 * key + val, 1, net.kernel), torch.nn.Conv1d)
    rec[10], rec[16] = _at(own.get("A_log"), (hv,)), _at(own.get("dt_bias"), (hv,))
    rec[17] = _at(m["norm"]._parameters.get("weight"), (net.dv,))
    rec[11] = _weight(m["out_proj"], (H, val))


def _delta_state(store, net, seqs, device):
    """Tail and state buffers of every live sequence: ``(pointers, new store entries)``; the old ones are read and new ones
    written, as in the layer loop: value heads that share key channels read the same old rows, and a caller may hold the state
    of an earlier token."""
    ptrs, new = [], []
    for i in seqs:
        tail, S = store.get(i, (None, None))
        if tail is None:
            tail = torch.zeros((net.kernel - 1, 2 * net.key_dim + net.value_dim), dtype=_BF16, device=device)
        if S is None:
            S = torch.zeros((net.hv, net.dk, net.dv), dtype=torch.float32, device=device)
        if tail.shape != (net.kernel - 1, 2 * net.key_dim + net.value_dim) or S.shape != (net.hv, net.dk, net.dv) \
                or tail.device != device or S.device != device:
            raise _Unfit
        if not (tail.is_contiguous() and S.is_contiguous() and tail.dtype is _BF16 and S.dtype is torch.float32 and S.data_ptr() % 16 == 0):
            tail, S = tail.to(_BF16).contiguous(), S.float().clone(memory_format=torch.contiguous_format)
        tail_out, S_out = torch.empty_like(tail), torch.empty_like(S)
        ptrs += (tail.data_ptr(), tail_out.data_ptr(), S.data_ptr(), S_out.data_ptr())
        new.append((i, tail, S, (tail_out, S_out)))
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
    table, types, nets = array("Q"), array("i"), []
    rec0 = [0] * 24
    hk = hv = taps = 0
    for layer in layers.values():
        rec = rec0[:]
        _plain(layer, layer_cls)
        m = layer._modules
        if hybrid is not None and "linear_attn" in m:
            net = m["linear_attn"]
            _delta(rec, net, hybrid.GatedDeltaNet, cfg, H)
            if net.dk != 128 or net.dv != 128 or net.hv % 8 or net.hv % net.hk or not 2 <= net.kernel <= 8:
                raise _Unfit
            hk, hv, taps = net.hk, net.hv, net.kernel
            nets.append(net)
            types.append(2)
        else:
            _attention(rec, m["self_attn"], att_cls, norm_cls, cfg, cache, dev, H, nq, nkv, D, hybrid is not None)
            types.append(0 if hybrid is None else 1)
        for at, name in ((0, "input_layernorm"), (12, "post_attention_layernorm")):
            rec[at] = _norm(m[name], norm_cls, cfg, H)
        _mlp(rec, m["mlp"], SwiGLUMLP, H, I)
        table.extend(rec)
    final = _norm(backbone._modules["norm"], norm_cls, cfg, H)

    # the states are replaced after the call: what declines here leaves them as they were
    gdn, news = array("Q"), []
    for net in nets:
        store = cache.state.setdefault(net.layer_idx, {})
        ptrs, new = _delta_state(store, net, seqs, dev)
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
    has_attn = any(t != 2 for t in types)
    np_ = max(nq * D * 2 + 2 * nkv * D if has_attn else 0, (2 * hk + 2 * hv) * 128 + 2 * hv)
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
        for i, _, _, entry in new:
            store[i] = entry
    return hidden
