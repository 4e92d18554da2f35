"""One-token passes through the native layer loop against the layer-by-layer path on the same cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DENSE = dict(vocab_size=512, hidden_size=256, intermediate_size=520, num_hidden_layers=2, rms_norm_eps=1e-6)


def _model(kind, **sizes):
    from lmms_engine_b200.mapping_func import create_model_from_config

    torch.manual_seed(3)
    if kind == "hybrid":
        cfg = dict(DENSE, num_attention_heads=4, num_key_value_heads=2, head_dim=128, linear_conv_kernel_dim=4, linear_key_head_dim=128,
                   linear_value_head_dim=128, linear_num_key_heads=4, linear_num_value_heads=8, partial_rotary_factor=0.25,
                   full_attention_interval=2)
        m = create_model_from_config("qwen3_5_text", dict(cfg, **sizes))
    else:
        heads, kv, dim, extra = {"grouped": (14, 2, 128, {}), "normed": (4, 2, 128, dict(attention_bias=False, qk_norm=True)),
                                 "narrow": (4, 4, 64, {}), "wide_group": (12, 1, 128, {}),
                                 "window": (4, 2, 128, dict(sliding_window=70, use_sliding_window=True))}[kind]
        m = create_model_from_config("qwen2", dict(DENSE, num_attention_heads=heads, num_key_value_heads=kv, head_dim=dim, **{**extra, **sizes}))
    m = m.to("cuda", torch.bfloat16).eval()
    with torch.no_grad():
        for n, p in m.named_parameters():
            if "norm" in n:
                p.add_(torch.randn_like(p) * 0.1)
            elif n.endswith("bias") and "dt_bias" not in n:
                p.copy_(torch.randn_like(p) * 0.1)
    return m


def _run_tokens(model, prompts, steps):
    from lmms_engine_b200.models.kv_cache import PackedKVCache

    gen = torch.Generator(device="cuda").manual_seed(5)
    n, out = len(prompts), []
    cache = PackedKVCache(len(model.model.layers), [p + steps for p in prompts], device=torch.device("cuda", 0))
    ids = torch.randint(0, 512, (sum(prompts),), device="cuda", generator=gen)
    with torch.no_grad():
        pos = cache.advance(prompts)
        cu = torch.tensor([0] + torch.tensor(prompts).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        model(input_ids=ids, cu_seqlens=cu, position_ids=pos, kv_cache=cache)
        for s in range(steps):
            live = [1 if (i + s) % 3 or n == 1 else 0 for i in range(n)]  # sequences pause and resume
            pos = cache.advance(live)
            m = sum(live)
            tok = torch.randint(0, 512, (m,), device="cuda", generator=gen)
            cu = torch.arange(m + 1, dtype=torch.int32, device="cuda")
            out.append(model(input_ids=tok, cu_seqlens=cu, position_ids=pos, kv_cache=cache)["hidden_states"])
    return torch.cat(out).float()


def _go(model, prompts, steps, native):
    from lmms_engine_b200.models import decode_path
    from lmms_engine_b200.ops import _cuda

    keep = decode_path.MAX_SEQS
    decode_path.MAX_SEQS = keep if native else 0
    try:
        out = _run_tokens(model, prompts, steps)
        _cuda.check_status()
    finally:
        decode_path.MAX_SEQS = keep
    return out


@pytest.mark.parametrize("kind,prompts", [("grouped", [1]), ("grouped", [63, 64, 65, 700]), ("normed", [2100]), ("normed", [5] * 7 + [130] * 11),
                                          ("narrow", [17, 300]), ("wide_group", [129, 40]), ("window", [50, 200]), ("hybrid", [100]),
                                          ("hybrid", [64, 1, 130]), ("normed", list(range(1, 41))), ("normed", list(range(1, 65)))])
def test_one_call_matches_layer_loop(kind, prompts, monkeypatch):
    """Both paths round every intermediate to bf16 at the same place, so only elements whose fp32 sums land on either side of
    a rounding boundary differ, by one bf16 step (2^-8); two layers carry a few of those into an output of rms 1."""
    from lmms_engine_b200.ops import _cuda

    model = _model(kind)
    seen, real = [], _cuda.call
    monkeypatch.setattr(_cuda, "call", lambda name, *a: (seen.append(name), real(name, *a))[1])
    want = _go(model, prompts, 5, False)
    assert "b200_decode_layers" not in seen
    got = _go(model, prompts, 5, True)
    assert seen.count("b200_decode_layers") == 5 + all(n == 1 for n in prompts)  # prompts of one token are such a pass too
    assert torch.isfinite(got).all()
    rel = ((got - want).norm() / want.norm()).item()
    assert rel < 2.0 ** -7, rel


def test_native_path_is_taken_and_hooks_keep_the_layer_loop():
    from lmms_engine_b200.ops import _cuda

    model = _model("grouped")
    _go(model, [10], 1, True)
    seen, real = [], _cuda.call
    try:
        _cuda.call = lambda name, *a: (seen.append(name), real(name, *a))[1]
        _go(model, [10], 2, True)
        assert seen.count("b200_decode_layers") == 2
        del seen[:]
        hook = model.model.layers[1].mlp.register_forward_hook(lambda *a: None)
        _go(model, [10], 2, True)
        hook.remove()
        assert "b200_decode_layers" not in seen
    finally:
        _cuda.call = real


class _ScaledLinear(torch.nn.Linear):
    """Computes its weight on access, as a quantised or adapted projection does."""

    @property
    def weight(self):
        return self._parameters["weight"] * 1.5


class _Twice(torch.nn.Module):
    def forward(self, w):
        return 2 * w


def _negated(cls):
    return type("Negated" + cls.__name__, (cls,), {"forward": lambda self, *a: cls.forward(self, *(-x for x in a))})


def _change(model, what, monkeypatch):
    from torch.nn.utils import parametrize

    from lmms_engine_b200.models import decoder_lm

    layer = model.model.layers[1]
    if what == "parametrized":
        parametrize.register_parametrization(layer.self_attn.o_proj, "weight", _Twice())
    elif what == "computed weight":
        layer.mlp.up_proj.__class__ = _ScaledLinear
    elif what in ("q_norm eps", "k_norm eps"):
        getattr(layer.self_attn, what[:6]).eps = 0.5
    elif what == "post norm eps":
        layer.post_attention_layernorm.eps = 0.5
    elif what == "q_norm subclass":
        layer.self_attn.q_norm.__class__ = _negated(type(layer.self_attn.q_norm))
    elif what == "post norm subclass":
        layer.post_attention_layernorm.__class__ = _negated(type(layer.post_attention_layernorm))
    elif what == "final norm subclass":
        model.model.norm.__class__ = _negated(type(model.model.norm))
    elif what == "instance forward":
        layer.mlp.forward = lambda x: 0.5 * x
    elif what == "class forward":
        monkeypatch.setattr(decoder_lm.SwiGLUMLP, "forward", lambda self, x: 0.5 * x)
    elif what == "global hook":
        return torch.nn.modules.module.register_module_forward_hook(lambda m, a, out: 0.5 * out if m is layer.mlp else None).remove
    elif what == "delta eps":
        model.model.layers[0].linear_attn.eps = 0.5
    elif what == "delta projection":
        model.model.layers[0].linear_attn.in_proj_z.__class__ = _ScaledLinear
    return lambda: None


@pytest.mark.parametrize("kind,what", [("normed", w) for w in (
    "parametrized", "computed weight", "q_norm eps", "k_norm eps", "post norm eps", "q_norm subclass", "post norm subclass",
    "final norm subclass", "instance forward", "class forward", "global hook")] + [("hybrid", "delta eps"), ("hybrid", "delta projection")])
def test_modules_that_are_more_than_their_weights_keep_the_layer_loop(kind, what, monkeypatch):
    """Whatever a call of the module would do beyond its class's arithmetic on plain parameters has to happen: the pass runs
    layer by layer, which is what it is compared with (bit by bit: it is the same code)."""
    from lmms_engine_b200.ops import _cuda

    model = _model(kind)
    before = _go(model, [10], 2, False)
    undo = _change(model, what, monkeypatch)
    try:
        want = _go(model, [10], 2, False)
        seen, real = [], _cuda.call
        monkeypatch.setattr(_cuda, "call", lambda name, *a: (seen.append(name), real(name, *a))[1])
        got = _go(model, [10], 2, True)
    finally:
        undo()
    assert not torch.equal(want, before), "the change has no effect on the output"
    assert torch.equal(got, want)
    assert "b200_decode_layers" not in seen


def test_cache_advances_under_a_default_device():
    """``torch.set_default_device("cuda")`` and ``with torch.device("cuda")`` make factory calls return device tensors."""
    from lmms_engine_b200.models.kv_cache import PackedKVCache

    with torch.device("cuda"):
        cache = PackedKVCache(1, [8, 8, 8], device=torch.device("cuda", 0))
        assert cache.advance([3, 0, 2]).tolist() == [0, 1, 2, 0, 1]
        assert cache.advance([1, 1, 1]).tolist() == [3, 0, 2]
        assert cache.advance([0, 2, 0]).tolist() == [1, 2]


def test_rotary_frequencies_are_kept_per_stream_and_not_from_a_capture():
    """The first pass may be a capture, a trace or on another stream: none of them leaves values behind that a later pass
    reads before they exist."""
    import copy

    from torch._subclasses.fake_tensor import FakeTensorMode

    from lmms_engine_b200.ops import rope

    backbone = _model("grouped").model
    pos = torch.arange(5, device="cuda")
    want = rope.rope_table(pos, rope.inv_freq(128, backbone.cfg.rope_theta, device=pos.device))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        backbone.rope_tables(pos)
    with FakeTensorMode():
        backbone._frequencies(128, pos.device)
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(backbone.rope_tables(pos), want))
    here = backbone._frequencies(128, pos.device)
    with torch.cuda.stream(torch.cuda.Stream()):
        there = backbone._frequencies(128, pos.device)
    assert there is not here and backbone._frequencies(128, pos.device) is here
    assert not hasattr(copy.deepcopy(backbone), "_fp32_frequencies")


@pytest.mark.parametrize("seqs,hidden", [(6, 6136), (4, 8184), (6, 6144), (6, 12280), (6, 12288)])
def test_rows_of_the_fused_norm_at_the_edges_of_shared_memory(seqs, hidden):
    """Of six sequences four have a token in a pass, of four up to three.  Rows that fill shared memory up to the limit without
    an opt-in (which covers a kernel's static part too), one step past it, up to the largest that the fused norm takes, and one
    past that.  Against the same weights in fp32: no further off than the layer loop, whose roundings are as many (a few per
    cent apart over some ten thousand values)."""
    model = _model("grouped", hidden_size=hidden)
    prompts = [5, 9, 1, 7, 3, 2][:seqs]
    loop, got = _go(model, prompts, 2, False), _go(model, prompts, 2, True)
    want = _go(model.float(), prompts, 2, False)
    assert (got - want).norm() < 1.15 * (loop - want).norm()


def test_threads_with_different_row_sizes():
    """Host threads that generate with models of different widths: neither lowers the other's shared-memory limit."""
    import threading

    models = [_model("grouped", hidden_size=h) for h in (6400, 12000)]
    prompts, errors = [3, 4, 5, 6, 1, 2], []

    def work(m):
        try:
            for _ in range(8):
                with torch.cuda.stream(torch.cuda.Stream()):
                    assert torch.isfinite(_run_tokens(m, prompts, 3)).all()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(m,)) for m in models]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]


def test_an_earlier_recurrent_state_stays_as_it_was():
    """A caller that keeps the entries of ``PackedKVCache.state`` can go back to them: a token replaces them and writes into
    none."""
    from lmms_engine_b200.models.kv_cache import PackedKVCache

    model = _model("hybrid")
    cache = PackedKVCache(len(model.model.layers), [40], device=torch.device("cuda", 0))
    one = torch.tensor([0, 1], dtype=torch.int32, device="cuda")

    def token(t):
        return model(input_ids=torch.tensor([t], device="cuda"), cu_seqlens=one, position_ids=cache.advance([1]), kv_cache=cache)["hidden_states"]

    with torch.no_grad():
        cu = torch.tensor([0, 30], dtype=torch.int32, device="cuda")
        model(input_ids=torch.arange(30, device="cuda"), cu_seqlens=cu, position_ids=cache.advance([30]), kv_cache=cache)
        token(3)
        held = {layer: dict(entries) for layer, entries in cache.state.items()}
        copies = {layer: {i: tuple(t.clone() for t in e) for i, e in entries.items()} for layer, entries in held.items()}
        first = token(7)
        token(9)
        assert held and all(torch.equal(a, b) for layer in held for i in held[layer] for a, b in zip(held[layer][i], copies[layer][i]))
        cache.state, cache.lens = {layer: dict(e) for layer, e in held.items()}, [31]
        assert torch.equal(token(7), first)


def _one_token(model, cache, embeds):
    """A pass of one token with given embeddings (the layer loop where the one-call path declines)."""
    from lmms_engine_b200.models.decoder_lm import PackedContext

    pos = cache.advance([1])
    ctx = PackedContext(torch.tensor([0, 1], dtype=torch.int32, device="cuda"), 1, *model.model.rope_tables(pos), True)
    ctx.kv_cache = cache
    with torch.no_grad():
        return model.model(embeds, ctx)


def test_decay_of_a_token_is_as_precise_as_in_the_layer_loop(monkeypatch):
    """A token of zeros leaves only the decay of the state: exp(-exp(A) softplus(dt)) against 64 bits, decays down to e^-13."""
    from lmms_engine_b200.models import decode_path
    from lmms_engine_b200.models.kv_cache import PackedKVCache

    model = _model("hybrid", linear_num_value_heads=256, linear_num_key_heads=8, num_hidden_layers=1)
    net = model.model.layers[0].linear_attn
    with torch.no_grad():
        net.A_log.copy_(torch.linspace(-4.0, 1.5, 256))
        net.dt_bias.copy_(torch.randn(256) * 1.5)
    want = (-net.A_log.double().exp() * torch.nn.functional.softplus(net.dt_bias.double())).exp()
    err = {}
    for native in (True, False):
        monkeypatch.setattr(decode_path, "MAX_SEQS", 64 if native else 0)
        cache = PackedKVCache(1, [4], device=torch.device("cuda", 0))
        cache.state[0] = {0: (torch.zeros(3, 2 * net.key_dim + net.value_dim, device="cuda", dtype=torch.bfloat16),
                              torch.ones(256, 128, 128, device="cuda"))}
        _one_token(model, cache, torch.zeros(1, 256, device="cuda", dtype=torch.bfloat16))
        got = cache.state[0][0][1]
        assert torch.equal(got, got[:, :1, :1].expand_as(got))
        err[native] = ((got[:, 0, 0].double() / want) - 1).abs()
    assert err[True].norm() < 1.1 * err[False].norm() + 1e-7, (err[True].norm().item(), err[False].norm().item())
