"""One new token per sequence through all layers of a decoder in one native call (``csrc/decode.cu``).

``decode_layers`` takes the place of the layer loop when a forward pass against a ``PackedKVCache`` feeds at most one token
to each of at most 64 sequences, without gradients, on plain bf16 CUDA weights of the dense decoder layers
(``decoder_lm.DecoderLayer``) or the hybrid ones (``qwen3_5.Qwen35Layer``).  Everything else - prompts, sparse MLPs, sharded
weights, modules with forward hooks, other head dims - returns ``None`` and runs layer by layer.  The numbers are those of
the layer loop up to the order of fp32 sums: every intermediate is rounded to bf16 at the same place.
"""
from __future__ import annotations

from array import array
from typing import Optional

import torch

from ..ops import _cuda
from ..ops import gemm as gemm_ops

_cuda.register("b200_decode_layers", "decode", "ppi" + "pppp" + "fff" + "ppppp" + "p" + "l" + "pp" + "s")

MAX_SEQS = 64  # kDecSeqs of the kernels: per-sequence tables travel as kernel arguments
_BF16 = torch.bfloat16


class _Unfit(Exception):
    pass


def _plain(module) -> dict:
    """Parameters of a module whose call is only its arithmetic."""
    if module._forward_hooks or module._forward_pre_hooks:
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


def _norm(module, cfg, H) -> int:
    if module.eps != cfg.rms_norm_eps:
        raise _Unfit
    return _at(_plain(module)["weight"], (H,))


def _mlp(rec, mlp, H, I):
    if mlp.tp_group is not None:
        raise _Unfit
    _plain(mlp)
    m = mlp._modules
    rec[13] = _at(_plain(m["gate_proj"])["weight"], (I, H))
    rec[14] = _at(_plain(m["up_proj"])["weight"], (I, H))
    rec[15] = _at(_plain(m["down_proj"])["weight"], (H, I))


def _attention(rec, att, cache, dev, H, nq, nkv, D, gated):
    m = att._modules
    _plain(att)
    if getattr(att, "nsa", None) is not None or getattr(att, "window", (-1, -1))[0] != cache.decode_window:
        raise _Unfit
    rows = nq * D * (2 if gated else 1)
    for i, (name, n) in enumerate((("q_proj", rows), ("k_proj", nkv * D), ("v_proj", nkv * D))):
        p = _plain(m[name])
        rec[1 + i] = _at(p["weight"], (n, H))
        rec[5 + i] = _opt(p["bias"], (n,))
    if "q_norm" in m:
        rec[9] = _at(_plain(m["q_norm"])["weight"], (D,))
        rec[10] = _at(_plain(m["k_norm"])["weight"], (D,))
    p = _plain(m["o_proj"])
    rec[11] = _at(p["weight"], (H, nq * D))
    rec[19] = _opt(p["bias"], (H,))
    k, v = cache.slabs(att.layer_idx, nkv, D, _BF16, dev)
    if k.dtype is not _BF16 or k.device != dev or k.shape[1:] != (nkv, D):
        raise _Unfit
    rec[16], rec[17] = k.data_ptr(), v.data_ptr()


def _delta(rec, net, H):
    m = net._modules
    own = _plain(net)
    key, val, hv = net.key_dim, net.value_dim, net.hv
    for i, (name, n) in enumerate((("in_proj_qkv", 2 * key + val), ("in_proj_z", val), ("in_proj_b", hv), ("in_proj_a", hv))):
        rec[1 + i] = _at(_plain(m[name])["weight"], (n, H))
    rec[9] = _at(_plain(m["conv1d"])["weight"], (2 * key + val, 1, net.kernel))
    rec[10], rec[16] = _at(own["A_log"], (hv,)), _at(own["dt_bias"], (hv,))
    rec[17] = _at(m["norm"]._parameters["weight"], (net.dv,))
    rec[11] = _at(_plain(m["out_proj"])["weight"], (H, val))


def _delta_state(store, net, seqs, device):
    """Tail and state buffers of every live sequence: ``(pointers, new store entries)``; the old tail is read and a new one
    written, because value heads that share key channels read the same old rows."""
    ptrs, new = [], []
    for i in seqs:
        tail, S = store.get(i, (None, None))
        if tail is None:
            tail = torch.zeros((net.kernel - 1, 2 * net.key_dim + net.value_dim), dtype=_BF16, device=device)
        if S is None:
            S = torch.zeros((net.hv, net.dk, net.dv), dtype=torch.float32, device=device)
        if not (tail.is_contiguous() and S.is_contiguous() and tail.dtype is _BF16 and S.dtype is torch.float32 and S.data_ptr() % 16 == 0):
            tail, S = tail.to(_BF16).contiguous(), S.float().clone()
        out = torch.empty_like(tail)
        ptrs += (tail.data_ptr(), out.data_ptr(), S.data_ptr())
        new.append((i, tail, out, S))
    return ptrs, new


def decode_layers(backbone, embeds: torch.Tensor, ctx) -> Optional[torch.Tensor]:
    cache = ctx.kv_cache
    M = embeds.shape[0]
    if (M > MAX_SEQS or not embeds.is_cuda or embeds.dtype is not _BF16 or torch.is_grad_enabled() or not ctx.causal
            or ctx.sp_size > 1 or ctx.tp_size > 1 or ctx.deepstack is not None or gemm_ops.LINEAR_BACKEND != "tcgen05"):
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
    norm_off = 0.0
    cache.decode_window = -1
    layers = backbone.layers._modules
    first = next(iter(layers.values()))
    if type(first) is DecoderLayer:
        cache.decode_window = first.self_attn.window[0]
        hybrid = None
    else:
        from . import qwen3_5 as hybrid

        if type(first) is not hybrid.Qwen35Layer:
            raise _Unfit
        norm_off = 1.0
    table, types, nets = array("Q"), array("i"), []
    rec0 = [0] * 24
    hk = hv = taps = 0
    for layer in layers.values():
        rec = rec0[:]
        _plain(layer)
        m = layer._modules
        mlp = m["mlp"]
        if type(mlp) is not SwiGLUMLP:
            raise _Unfit
        if hybrid is None:
            att = m["self_attn"]
            if type(layer) is not DecoderLayer or type(att) is not Attention or type(m["input_layernorm"]) is not RMSNorm:
                raise _Unfit
            _attention(rec, att, cache, dev, H, nq, nkv, D, False)
            types.append(0)
        else:
            if type(layer) is not hybrid.Qwen35Layer:
                raise _Unfit
            if "linear_attn" in m:
                net = m["linear_attn"]
                if type(net) is not hybrid.GatedDeltaNet or net.dk != 128 or net.dv != 128 or net.hv % 8 or net.hv % net.hk or not 2 <= net.kernel <= 8:
                    raise _Unfit
                _delta(rec, net, H)
                hk, hv, taps = net.hk, net.hv, net.kernel
                nets.append(net)
                types.append(2)
            else:
                if type(m["self_attn"]) is not hybrid.GatedAttention:
                    raise _Unfit
                _attention(rec, m["self_attn"], cache, dev, H, nq, nkv, D, True)
                types.append(1)
        for at, name in ((0, "input_layernorm"), (12, "post_attention_layernorm")):
            rec[at] = _norm(m[name], cfg, H)
        _mlp(rec, mlp, H, I)
        table.extend(rec)
    final = _norm(backbone._modules["norm"], cfg, H)

    # nothing below declines: the states are replaced only here
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
    splits = max(1, min(max(-(-296 // (nkv * M)), -(-longest // 512)), -(-longest // 64), 64))
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
        for i, _, tail, S in new:
            store[i] = (tail, S)
    return hidden
