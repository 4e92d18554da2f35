"""Performance cases: the work that users of this engine run, through its public entry points.

A case is a plain dict; ``prepare`` builds what a program has in hand before the call (weights, optimizer state, inputs),
``run`` is one pass.  The kinds and what they stand for:

``step``      one optimizer step of a packed dense decoder on one GPU: forward, backward, clipping, update (the training
              loop of the native runtime): AdamW, or at the headline width Muon on the matrices and AdamW on the rest.
``hybrid``    one accumulation micro-step (forward + backward into the flat gradient) of the Gated-DeltaNet / gated
              attention hybrid decoder on a packed batch.
``moe``       one sparse block, forward + backward: router, permutation, grouped expert MLP, weighted combine.
``vision``    a vision tower on packed patches, forward + backward: windowed + full attention over images, or per-frame
              attention over video frames with the deepstack outputs.
``attention`` packed variable-length attention by itself, forward + backward.
``decode``    one sequence: the prompt once, then one token per call against the key / value cache.
``rollout``   a batch of ragged sequences advanced together against the packed cache, one token each per call.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

DEV = "cuda"

# Widths as they stand in this repository's benchmark, examples and tests.
DENSE = {
    # the kernel smoke run
    "small": dict(vocab_size=4096, hidden_size=512, intermediate_size=1408, num_attention_heads=4, num_key_value_heads=2, head_dim=128),
    # the example configurations with 1024 hidden units (QK-norm, tied head)
    "h1024": dict(vocab_size=151936, hidden_size=1024, intermediate_size=3072, num_attention_heads=16, num_key_value_heads=8,
                  head_dim=128, attention_bias=False, qk_norm=True, tie_word_embeddings=True),
    # the headline training configuration
    "h3584": dict(vocab_size=152064, hidden_size=3584, intermediate_size=18944, num_attention_heads=28, num_key_value_heads=4,
                  head_dim=128, attention_bias=True, tie_word_embeddings=False),
}
HYBRID = dict(vocab_size=32000, hidden_size=2048, intermediate_size=6144, num_attention_heads=16, num_key_value_heads=4, head_dim=128,
              linear_conv_kernel_dim=4, linear_key_head_dim=128, linear_value_head_dim=128, linear_num_key_heads=16,
              linear_num_value_heads=32, partial_rotary_factor=0.25)
MOE = dict(hidden_size=2048, num_experts=128, num_experts_per_tok=8, moe_intermediate_size=768)
VIT_IMAGE = dict(hidden_size=1280, intermediate_size=3420, num_heads=16, patch_size=14, temporal_patch_size=2, spatial_merge_size=2,
                 in_channels=3, window_size=112, out_hidden_size=3584)
VIT_VIDEO = dict(hidden_size=1152, intermediate_size=4304, num_heads=16, patch_size=16, temporal_patch_size=2, spatial_merge_size=2,
                 in_channels=3, out_hidden_size=4096, num_position_embeddings=2304, hidden_act="gelu_pytorch_tanh")


def listed():
    return [
        # the smallest training step: launches and host work count
        dict(name="step_small", kind="step", width="small", layers=2, tokens=1024, max_len=600, muon=False),
        # many narrow layers on a short packed row, as when a small model is tuned
        dict(name="step_h1024", kind="step", width="h1024", layers=28, tokens=4096, max_len=2048, muon=False),
        # the headline row of 16384 tokens at its width; two layers, so that the state fits several times
        dict(name="step_h3584", kind="step", width="h3584", layers=2, tokens=16384, max_len=8192, muon=True),
        # one period of the hybrid stack on a long packed row
        dict(name="hybrid_16k", kind="hybrid", layers=4, tokens=16384, max_len=8192),
        # one sparse block of the mixture-of-experts configuration on its row of 8192 tokens
        dict(name="moe_8k", kind="moe", tokens=8192),
        # eight images of a multi-image sample through the windowed tower (seven windowed blocks and a full one)
        dict(name="vision_images", kind="vision", tower="image", depth=8, items=8, side_h=896, side_w=672, frames=1),
        # one video clip through the per-frame tower
        dict(name="vision_video", kind="vision", tower="video", depth=9, items=1, side_h=448, side_w=640, frames=40),
        # long causal documents, grouped heads
        dict(name="attention_16k", kind="attention", tokens=16384, max_len=8192, heads=28, kv_heads=4, dim=128, causal=True),
        # an interactive continuation on a small model
        dict(name="decode_h1024", kind="decode", family="dense", width="h1024", layers=28, prompt=300, new=24),
        # a long prompt at the headline width; layers of that width differ only in number, and eight keep the rounding of
        # bf16 activations, which every further layer amplifies, small against the outputs
        dict(name="decode_h3584", kind="decode", family="dense", width="h3584", layers=8, prompt=6000, new=32),
        # one period of the hybrid stack generating
        dict(name="decode_hybrid", kind="decode", family="hybrid", width="hybrid", layers=4, prompt=1000, new=24),
        # a policy-gradient rollout: 48 ragged prompts advanced together
        dict(name="rollout_48", kind="rollout", width="h1024", layers=28, seqs=48, max_prompt=1024, new=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "hybrid", "moe", "vision", "vision", "attention", "decode", "decode", "rollout"])
    if kind == "step":
        width = rng.choice(["small", "h1024", "h3584"])
        if width == "small":
            return dict(kind=kind, width=width, layers=rng.randint(1, 4), tokens=_log_int(rng, 200, 16384), max_len=_log_int(rng, 150, 4096), muon=False)
        if width == "h1024":
            return dict(kind=kind, width=width, layers=rng.randint(4, 28), tokens=_log_int(rng, 600, 8192), max_len=_log_int(rng, 300, 4096), muon=False)
        return dict(kind=kind, width=width, layers=rng.randint(1, 2), tokens=_log_int(rng, 1000, 16384), max_len=_log_int(rng, 300, 8192), muon=True)
    if kind == "hybrid":
        return dict(kind=kind, layers=rng.choice([1, 2, 3, 4]), tokens=_log_int(rng, 500, 16384), max_len=_log_int(rng, 200, 8192))
    if kind == "moe":
        return dict(kind=kind, tokens=_log_int(rng, 300, 16384))
    if kind == "vision":
        if rng.random() < 0.5:
            return dict(kind=kind, tower="image", depth=rng.randint(2, 8), items=rng.randint(1, 10), side_h=28 * rng.randint(8, 40),
                        side_w=28 * rng.randint(8, 28), frames=1)
        return dict(kind=kind, tower="video", depth=rng.randint(3, 9), items=rng.randint(1, 2), side_h=32 * rng.randint(7, 18),
                    side_w=32 * rng.randint(7, 18), frames=2 * rng.randint(2, 20))
    if kind == "attention":
        heads, kv = rng.choice([(28, 4), (32, 8), (16, 16), (16, 4)])
        return dict(kind=kind, tokens=_log_int(rng, 500, 16384), max_len=_log_int(rng, 200, 8192), heads=heads, kv_heads=kv,
                    dim=rng.choice([128, 128, 80, 64]), causal=rng.random() < 0.75)
    if kind == "decode":
        family = rng.choice(["dense", "dense", "hybrid"])
        if family == "hybrid":
            return dict(kind=kind, family=family, width="hybrid", layers=rng.randint(1, 4), prompt=_log_int(rng, 30, 3000), new=rng.randint(4, 24))
        width = rng.choice(["h1024", "h3584"])
        layers = rng.randint(8, 28) if width == "h1024" else rng.randint(2, 8)
        return dict(kind=kind, family=family, width=width, layers=layers, prompt=_log_int(rng, 30, 6000), new=rng.randint(4, 24))
    return dict(kind=kind, width="h1024", layers=rng.randint(8, 28), seqs=rng.randint(2, 48), max_prompt=_log_int(rng, 60, 1024), new=rng.randint(3, 12))


# ---------------------------------------------------------------------------------------------------- shapes of a case
def _lengths(total, max_len):
    """Ragged document lengths up to ``max_len`` that fill ``total`` exactly, fixed by the case."""
    rng = random.Random(7919 * total + max_len)
    out, left = [], total
    while left > 0:
        n = min(left, rng.randint(max(1, min(128, max_len // 4)), max_len))
        out.append(n)
        left -= n
    return out


def _prompt_lengths(case):
    rng = random.Random(31 * case["seqs"] + case["max_prompt"])
    return [rng.randint(max(1, case["max_prompt"] // 16), case["max_prompt"]) for _ in range(case["seqs"])]


def _grid(case):
    p = 14 if case["tower"] == "image" else 16
    t = 1 if case["tower"] == "image" else case["frames"] // 2
    m = 2 * p
    out = []
    for i in range(case["items"]):  # every item a little smaller than the one before it
        h, w = max(m, case["side_h"] - i * m), case["side_w"]
        out.append((t, h // m * 2, w // m * 2))
    return out


def _cu(lengths):
    at, out = 0, [0]
    for n in lengths:
        at += n
        out.append(at)
    return torch.tensor(out, dtype=torch.int32, device=DEV)


def _dense_model(case):
    from lmms_engine_b200.mapping_func import create_model_from_config

    return create_model_from_config("qwen2", dict(DENSE[case["width"]], num_hidden_layers=case["layers"]), device=DEV, dtype=torch.bfloat16)


def _hybrid_model(case):
    from lmms_engine_b200.mapping_func import create_model_from_config

    # built in the default type and cast, as the trainers do: the decay parameters are drawn in fp32
    return create_model_from_config("qwen3_5_text", dict(HYBRID, num_hidden_layers=case["layers"]), device=DEV).to(torch.bfloat16)


# ---------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed + 1)
    return {"case": case, **_PREPARE[case["kind"]](case, gen)}


def _ids(n, vocab, gen):
    return torch.randint(0, vocab, (n,), device=DEV, generator=gen)


def _prepare_step(case, gen):
    from lmms_engine_b200.parallel.owner_sharded import OwnerShardedRuntime

    model = _dense_model(case)
    rt = OwnerShardedRuntime(model, None, lr=2e-4, weight_decay=0.01, use_muon=case["muon"], max_grad_norm=1.0)
    return dict(model=model, rt=rt, ids=_ids(case["tokens"], DENSE[case["width"]]["vocab_size"], gen),
                cu=_cu(_lengths(case["tokens"], case["max_len"])))


def _prepare_hybrid(case, gen):
    from lmms_engine_b200.parallel.owner_sharded import OwnerShardedRuntime

    model = _hybrid_model(case)
    rt = OwnerShardedRuntime(model, None, lr=1e-5)
    return dict(model=model, rt=rt, ids=_ids(case["tokens"], HYBRID["vocab_size"], gen), cu=_cu(_lengths(case["tokens"], case["max_len"])))


def _randn(shape, gen, scale=1.0):
    return (torch.randn(shape, device=DEV, generator=gen, dtype=torch.float32) * scale).to(torch.bfloat16)


def _prepare_moe(case, gen):
    from lmms_engine_b200.models.moe_lm import MoEConfig, SparseMoeBlock

    with torch.device(DEV):
        block = SparseMoeBlock(MoEConfig(num_hidden_layers=1, **MOE)).to(torch.bfloat16)
    with torch.no_grad():
        for p in block.parameters():
            p.normal_(0.0, 0.02)
    h = MOE["hidden_size"]
    return dict(block=block, x=_randn((case["tokens"], h), gen).requires_grad_(True), dy=_randn((case["tokens"], h), gen, 1e-3))


def _prepare_vision(case, gen):
    from lmms_engine_b200.models.vision import Qwen3VisionTower, Qwen25VisionTower, VisionConfig
    from lmms_engine_b200.parallel.owner_sharded import OwnerShardedRuntime

    depth = case["depth"]
    if case["tower"] == "image":
        cfg, cls = VisionConfig.from_dict(dict(VIT_IMAGE, depth=depth, fullatt_block_indexes=[depth - 1])), Qwen25VisionTower
    else:
        taps = sorted({depth // 3 - 1, 2 * depth // 3 - 1, depth - 1})
        cfg, cls = VisionConfig.from_dict(dict(VIT_VIDEO, depth=depth, deepstack_visual_indexes=taps)), Qwen3VisionTower
    with torch.device(DEV):
        tower = cls(cfg).to(torch.bfloat16)
    rt = OwnerShardedRuntime(tower, None, lr=1e-5)
    grid = _grid(case)
    n = sum(t * h * w for t, h, w in grid)
    merged = n // 4
    dys = [_randn((merged, cfg.out_hidden_size), gen, 1e-3) for _ in range(1 if case["tower"] == "image" else 1 + len(cfg.deepstack_visual_indexes))]
    return dict(tower=tower, rt=rt, patches=_randn((n, 3 * 2 * cfg.patch_size ** 2), gen), grid=torch.tensor(grid), dys=dys)


def _prepare_attention(case, gen):
    t, d = case["tokens"], case["dim"]
    q = _randn((t, case["heads"], d), gen).requires_grad_(True)
    k = _randn((t, case["kv_heads"], d), gen).requires_grad_(True)
    v = _randn((t, case["kv_heads"], d), gen).requires_grad_(True)
    return dict(q=q, k=k, v=v, do=_randn((t, case["heads"], d), gen), cu=_cu(_lengths(t, case["max_len"])))


def _prepare_decode(case, gen):
    model = _hybrid_model(case) if case["family"] == "hybrid" else _dense_model(case)
    vocab = HYBRID["vocab_size"] if case["family"] == "hybrid" else DENSE[case["width"]]["vocab_size"]
    return dict(model=model.eval(), prompt=_ids(case["prompt"], vocab, gen), new=_ids(case["new"], vocab, gen))


def _prepare_rollout(case, gen):
    vocab = DENSE[case["width"]]["vocab_size"]
    lens = _prompt_lengths(case)
    return dict(model=_dense_model(case).eval(), prompt=_ids(sum(lens), vocab, gen), lens=lens, prompt_cu=_cu(lens),
                new=_ids(case["new"] * case["seqs"], vocab, gen).view(case["new"], case["seqs"]))


_PREPARE = dict(step=_prepare_step, hybrid=_prepare_hybrid, moe=_prepare_moe, vision=_prepare_vision, attention=_prepare_attention,
                decode=_prepare_decode, rollout=_prepare_rollout)


# ---------------------------------------------------------------------------------------------------- run
def run(state):
    return _RUN[state["case"]["kind"]](state)


def _run_step(s):
    rt = s["rt"]
    loss = s["model"](input_ids=s["ids"], labels=s["ids"], cu_seqlens=s["cu"])["loss"]
    loss.backward()
    norm = rt.step()
    return dict(loss=loss.detach(), norm=norm, weights=rt.P, muon_masters=rt.mu_master, adam_masters=rt.ad_master)


def _run_hybrid(s):
    rt = s["rt"]
    rt.zero_grad()
    loss = s["model"](input_ids=s["ids"], labels=s["ids"], cu_seqlens=s["cu"])["loss"]
    loss.backward()
    return dict(loss=loss.detach(), grads=rt.G)


def _run_moe(s):
    block, x = s["block"], s["x"]
    x.grad = None
    block.zero_grad(set_to_none=True)
    y, aux = block(x)
    (y, aux_w) = (y, 1e-3 * aux)
    torch.autograd.backward([y, aux_w], [s["dy"], None])
    e = block.experts
    return dict(y=y.detach(), aux=aux.detach(), dx=x.grad, d_gate=block.gate.weight.grad, d_gate_up=e.gate_up_proj.grad, d_down=e.down_proj.grad)


def _run_vision(s):
    s["rt"].zero_grad()
    out = s["tower"](s["patches"], s["grid"])
    outs = [out] if torch.is_tensor(out) else [out[0], *out[1]]
    torch.autograd.backward(outs, s["dys"])
    return dict(features=[o.detach() for o in outs], grads=s["rt"].G)


def _run_attention(s):
    from lmms_engine_b200.ops.attention import varlen_attn

    q, k, v = s["q"], s["k"], s["v"]
    q.grad = k.grad = v.grad = None
    o = varlen_attn(q, k, v, s["cu"], causal=s["case"]["causal"])
    o.backward(s["do"])
    return dict(o=o.detach(), dq=q.grad, dk=k.grad, dv=v.grad)


@torch.no_grad()
def _run_decode(s):
    from lmms_engine_b200.models.generation import GenerationState

    model, new = s["model"], s["new"]
    n = new.numel()
    st = GenerationState(model, s["prompt"].numel() + n, s["prompt"].device)
    hidden = st.prefill(s["prompt"])
    logits = [model.lm_head(hidden)]
    for i in range(n):
        hidden = st.step(new[i:i + 1])
        logits.append(model.lm_head(hidden))
    return torch.cat(logits)


@torch.no_grad()
def _run_rollout(s):
    from lmms_engine_b200.models.kv_cache import PackedKVCache

    model, lens, new = s["model"], s["lens"], s["new"]
    steps, seqs = new.shape
    cache = PackedKVCache(s["case"]["layers"], [n + steps for n in lens], device=s["prompt"].device)
    pos = cache.advance(lens)
    hidden = model(input_ids=s["prompt"], cu_seqlens=s["prompt_cu"], position_ids=pos, kv_cache=cache)["hidden_states"]
    logits = [model.lm_head(hidden.index_select(0, (s["prompt_cu"][1:] - 1).long()))]
    cu = torch.arange(seqs + 1, dtype=torch.int32, device=s["prompt"].device)
    for i in range(steps):
        pos = cache.advance([1] * seqs)
        hidden = model(input_ids=new[i], cu_seqlens=cu, position_ids=pos, kv_cache=cache)["hidden_states"]
        logits.append(model.lm_head(hidden))
    return torch.stack(logits)


_RUN = dict(step=_run_step, hybrid=_run_hybrid, moe=_run_moe, vision=_run_vision, attention=_run_attention, decode=_run_decode, rollout=_run_rollout)


# ---------------------------------------------------------------------------------------------------- work
def _dense_params(w, layers):
    h, i = w["hidden_size"], w["intermediate_size"]
    q, kv = w["num_attention_heads"] * w["head_dim"], w["num_key_value_heads"] * w["head_dim"]
    mats = [(q, h), (kv, h), (kv, h), (h, q), (i, h), (i, h), (h, i)]
    return layers * sum(a * b for a, b in mats), mats


def _causal_pairs(lengths):
    return sum(n * (n + 1) / 2 for n in lengths)


def _work_step(case):
    w = DENSE[case["width"]]
    body, mats = _dense_params(w, case["layers"])
    head = w["vocab_size"] * w["hidden_size"]
    heads = head * (1 if w.get("tie_word_embeddings") else 2)
    t = case["tokens"]
    attn = 4 * w["num_attention_heads"] * w["head_dim"] * _causal_pairs(_lengths(t, case["max_len"])) * case["layers"]
    ns = sum(5 * (4.0 * min(m) ** 2 * max(m) + 2.0 * min(m) ** 3) for m in mats) * case["layers"] if case["muon"] else 0.0
    # weights read forward and backward, gradients written and read, masters and moments read and written
    return {"bytes": (body + heads) * 2.0 * 5 + body * (16.0 if case["muon"] else 24.0) + heads * 24.0, "flops": 6.0 * (body + head) * t + 3.5 * attn + ns}


def _hybrid_layer_params():
    h, i = HYBRID["hidden_size"], HYBRID["intermediate_size"]
    key, val = 16 * 128, 32 * 128
    linear = h * (2 * key + 2 * val + 2 * 32) + val * h
    full = h * (2 * 16 * 128 + 2 * 4 * 128) + 16 * 128 * h
    return linear + 3 * h * i, full + 3 * h * i


def _hybrid_sizes(layers):
    n_full = sum(1 for i in range(layers) if (i + 1) % 4 == 0)
    lin, full = _hybrid_layer_params()
    return n_full, (layers - n_full) * lin + n_full * full


def _delta_flops_per_token():
    # per head and token of a 64-token chunk: three products with the chunk's keys / values, three with the state
    return 32 * (2 * 64 * 128 * 3 + 2 * 128 * 128 * 3 + 64 * 64 / 2)


def _work_hybrid(case):
    n_full, body = _hybrid_sizes(case["layers"])
    head = HYBRID["vocab_size"] * HYBRID["hidden_size"]
    t = case["tokens"]
    attn = 4 * 16 * 128 * _causal_pairs(_lengths(t, case["max_len"])) * n_full
    flops = 6.0 * (body + head) * t + 3.5 * attn + 3.0 * (case["layers"] - n_full) * _delta_flops_per_token() * t
    return {"bytes": (body + 2 * head) * 2.0 * 4 + case["layers"] * t * HYBRID["hidden_size"] * 2.0 * 8, "flops": flops}


def _work_moe(case):
    t, h, i, e, k = case["tokens"], MOE["hidden_size"], MOE["moe_intermediate_size"], MOE["num_experts"], MOE["num_experts_per_tok"]
    return {"bytes": 3.0 * h * i * e * 2 * 2 + 4.0 * t * h * 2, "flops": 6.0 * t * k * 3 * h * i + 6.0 * t * h * e}


def _work_vision(case):
    grid = _grid(case)
    n = sum(t * h * w for t, h, w in grid)
    c = VIT_IMAGE if case["tower"] == "image" else VIT_VIDEO
    h, i, p = c["hidden_size"], c["intermediate_size"], c["patch_size"]
    mlp = (3 if case["tower"] == "image" else 2) * h * i
    block = 4 * h * h + mlp
    hidden = 4 * h
    merger = hidden * hidden + hidden * c["out_hidden_size"]
    mergers = 1 if case["tower"] == "image" else 4
    full = sum(t * (hh * ww) ** 2 for t, hh, ww in grid)
    if case["tower"] == "image":
        pairs = (case["depth"] - 1) * n * 64 + full
    else:
        pairs = case["depth"] * full
    params = case["depth"] * block + mergers * merger + 6 * p * p * h
    flops = 6.0 * n * (case["depth"] * block + 6 * p * p * h) + 6.0 * (n / 4) * mergers * merger + 3.5 * 4 * h * pairs
    return {"bytes": params * 2.0 * 3 + n * 6 * p * p * 2.0 * 2 + n / 4 * c["out_hidden_size"] * 2.0 * 2 * mergers, "flops": flops}


def _work_attention(case):
    t, d = case["tokens"], case["dim"]
    lengths = _lengths(t, case["max_len"])
    pairs = _causal_pairs(lengths) if case["causal"] else sum(n * n for n in lengths)
    rows = t * d * 2.0
    return {"bytes": rows * (case["heads"] * 4 + case["kv_heads"] * 4), "flops": 3.5 * 4 * case["heads"] * d * pairs}


def _work_decode(case):
    t, n = case["prompt"], case["new"]
    if case["family"] == "hybrid":
        n_full, body = _hybrid_sizes(case["layers"])
        head = HYBRID["vocab_size"] * HYBRID["hidden_size"]
        kv = n_full * 2 * 4 * 128 * 2.0
        attn = 4 * 16 * 128 * n_full * t * t / 2
        state = (case["layers"] - n_full) * 32 * 128 * 128 * 4.0 * 2
    else:
        w = DENSE[case["width"]]
        body, _ = _dense_params(w, case["layers"])
        head = w["vocab_size"] * w["hidden_size"]
        kv = case["layers"] * 2 * w["num_key_value_heads"] * w["head_dim"] * 2.0
        attn = 4 * w["num_attention_heads"] * w["head_dim"] * case["layers"] * t * t / 2
        state = 0.0
    return {"bytes": (n + 1) * (body + head) * 2.0 + n * (t + n / 2) * kv + n * state, "flops": 2.0 * body * (t + n) + 2.0 * head * (n + 1) + attn}


def _work_rollout(case):
    w = DENSE[case["width"]]
    body, _ = _dense_params(w, case["layers"])
    head = w["vocab_size"] * w["hidden_size"]
    lens, n = _prompt_lengths(case), case["new"]
    kv = case["layers"] * 2 * w["num_key_value_heads"] * w["head_dim"] * 2.0
    attn = 4 * w["num_attention_heads"] * w["head_dim"] * case["layers"] * _causal_pairs(lens)
    return {"bytes": (n + 1) * (body + head) * 2.0 + n * (sum(lens) + case["seqs"] * n / 2) * kv,
            "flops": 2.0 * body * (sum(lens) + case["seqs"] * n) + 2.0 * head * case["seqs"] * (n + 1) + attn}


_WORK = dict(step=_work_step, hybrid=_work_hybrid, moe=_work_moe, vision=_work_vision, attention=_work_attention, decode=_work_decode, rollout=_work_rollout)


def work(case):
    return _WORK[case["kind"]](case)


# Largest relative 2-norm / element difference of another correct implementation at the same precision.  Measured as the
# difference of the same pass on library products and the other attention backward, and against the same model in fp32:
#   step       weights 6e-4 / 0.022 (Adam's first updates are signs: elements whose gradient is rounding noise flip)
#   hybrid     gradients 0.010 / 0.26 between the two, 0.041 against fp32
#   moe        the same router decisions, so only the products' and the combine's bf16 rounding remains (2^-9 a rounding)
#   vision     gradients 0.007 / 0.23 between the two, features 0.011 and gradients 0.017 / 0.54 against fp32
#   attention  bf16 probabilities and score gradients: 2^-9 each, four roundings on the way to dQ and dK
#   decode     logits 0.027 / 0.14 (headline width, eight layers), 0.013 / 0.07 (1024 units), 0.025 / 0.12 (hybrid) against fp32
_TOLERANCE = dict(
    step={"rel": 0.0025, "max": 0.09}, hybrid={"rel": 0.03, "max": 0.99}, moe={"rel": 0.01, "max": 0.4}, vision={"rel": 0.03, "max": 0.95},
    attention={"rel": 0.015, "max": 0.5}, decode={"rel": 0.03, "max": 0.5}, rollout={"rel": 0.03, "max": 0.3})


def tolerance(case):
    return dict(_TOLERANCE[case["kind"]])
