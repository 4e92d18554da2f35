"""tcgen05 varlen attention (forward and backward) against the fp32 per-document reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(lens, Hq, Hkv, D, causal, window=-1, seed=0):
    from lmms_engine_b200.ops import attention, _cuda

    torch.manual_seed(seed)
    T = sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    q = torch.randn(T, Hq, D, device="cuda").to(torch.bfloat16).requires_grad_()
    k = torch.randn(T, Hkv, D, device="cuda").to(torch.bfloat16).requires_grad_()
    v = torch.randn(T, Hkv, D, device="cuda").to(torch.bfloat16).requires_grad_()
    o = attention.varlen_attn(q, k, v, cu, cu, causal=causal, window_size=(window, -1))
    do = torch.randn_like(o)
    o.backward(do)
    _cuda.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf = attention.varlen_attn_ref(qr, kr, vr, cu, cu, causal=causal, window_left=window)
    orf.backward(do.float())
    assert (o.float() - orf).abs().max().item() < 3e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item() / (b.abs().max().item() + 1e-6)
        assert err < 3e-2, (name, err)


@pytest.mark.parametrize("lens", [[128], [256, 128], [1, 37, 130, 257, 64], [700, 3, 1025]])
@pytest.mark.parametrize("causal", [True, False])
def test_attn_d128_gqa(lens, causal):
    _case(lens, 4, 2, 128, causal)


def test_attn_d64_mha():
    _case([300, 17, 129], 2, 2, 64, True)


def test_attn_d80_vision_noncausal():
    _case([64, 1024, 400], 4, 4, 80, False)


def test_attn_d72_vision_noncausal():
    _case([256, 100], 2, 2, 72, False)


def test_attn_sliding_window():
    _case([600, 300], 4, 1, 128, True, window=200)


def test_attn_qwen7b_heads():
    _case([2048, 1000], 28, 4, 128, True)


def test_attn_strided_qkv_views():
    from lmms_engine_b200.ops import attention

    T, Hq, Hkv, D = 500, 4, 2, 128
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device="cuda").to(torch.bfloat16)
    q = qkv[:, : Hq * D].view(T, Hq, D)
    k = qkv[:, Hq * D : (Hq + Hkv) * D].view(T, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D :].view(T, Hkv, D)
    cu = torch.tensor([0, 200, 500], dtype=torch.int32, device="cuda")
    o = attention.varlen_attn(q, k, v, cu, cu, causal=True)
    ref = attention.varlen_attn_ref(q.float(), k.float(), v.float(), cu, cu, causal=True)
    assert (o.float() - ref).abs().max().item() < 3e-2


def test_cu_seqlens_past_the_tensor_raise_status_not_a_fault():
    """A cu_seqlens table that reaches past the packed tensor makes the kernel raise its status word and skip
    the document; nothing is written out of bounds and the context stays usable."""
    from lmms_engine_b200.ops import _cuda, attention

    T, H, D = 256, 2, 64
    q = torch.randn(T, H, D, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(T, H, D, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(T, H, D, device="cuda", dtype=torch.bfloat16)
    bad = torch.tensor([0, 128, 384], dtype=torch.int32, device="cuda")  # the second document ends 128 rows past T
    attention.varlen_attn(q, k, v, bad, bad, causal=True)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="bad shape"):
        _cuda.check_status()
    good = torch.tensor([0, 128, 256], dtype=torch.int32, device="cuda")
    out = attention.varlen_attn(q, k, v, good, good, causal=True)
    ref = attention.varlen_attn_ref(q, k, v, good, good, True, 1.0 / D ** 0.5, -1)
    assert (out.float() - ref.float()).abs().max() < 3e-2
    _cuda.check_status()
    with pytest.raises(NotImplementedError):
        attention.varlen_attn(q, k, v, good, good, causal=False, window_size=(-1, 16))


@pytest.mark.parametrize("causal", [True, False])
def test_queries_shorter_than_keys_bottom_right_aligned(causal):
    """Documents whose keys are a visible prefix followed by the queries' own tokens (the attention splits of the
    unified model): the causal mask is aligned to the END of the keys."""
    from lmms_engine_b200.ops import attention, _cuda

    torch.manual_seed(0)
    lq, lk = [5, 130, 64, 1], [40, 130, 300, 129]
    cu_q = torch.tensor([0] + list(torch.tensor(lq).cumsum(0)), dtype=torch.int32, device="cuda")
    cu_k = torch.tensor([0] + list(torch.tensor(lk).cumsum(0)), dtype=torch.int32, device="cuda")
    q = torch.randn(sum(lq), 4, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    k = torch.randn(sum(lk), 2, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    v = torch.randn(sum(lk), 2, 64, device="cuda").to(torch.bfloat16).requires_grad_()
    o = attention.varlen_attn(q, k, v, cu_q, cu_k, causal=causal)
    do = torch.randn_like(o)
    o.backward(do)
    _cuda.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    orf = attention.varlen_attn_ref(qr, kr, vr, cu_q, cu_k, causal=causal)
    orf.backward(do.float())
    assert (o.float() - orf).abs().max().item() < 3e-2
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item() / (b.abs().max().item() + 1e-6)
        assert err < 3e-2, (name, err)


@pytest.mark.parametrize("lens,n_q,n_kv,D,causal,window,max_len", [
    ((64, 1, 17, 63, 48, 16), 3, 3, 80, False, -1, 64),      # windows of a vision tower, ragged edges
    ((33, 64, 5), 4, 2, 72, True, -1, 64),                   # grouped heads, a head of 72 (rotation in fours), causal
    ((64, 64, 31), 4, 1, 128, True, 9, 64),
    ((2, 64), 2, 2, 64, False, -1, 64),
    ((130, 1, 127, 257), 4, 2, 80, False, -1, None),         # the long-document kernels behind the same entry
    ((40,) * 70 + (200,), 2, 1, 128, True, -1, None),        # more documents than one step of the block search
])
def test_rope_attention_matches_separate_operations(lens, n_q, n_kv, D, causal, window, max_len):
    """Against the fp32 formulation of both operations.  Outputs and gradients carry four bf16 roundings of 2^-9 each on
    the way (rotated rows, probabilities, score gradients, the result), so 2^-6 of the 2-norm bounds them."""
    from lmms_engine_b200.ops import _cuda, attention, rope

    torch.manual_seed(3)
    T = sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * D).bfloat16()
    ang = torch.randn(T, D // 2).repeat(1, 2)
    cos, sin, do = ang.cos(), ang.sin(), torch.randn(T, n_q, D).bfloat16()
    ref = qkv.float().requires_grad_()
    q, k, v = ref.view(T, -1, D).split([n_q, n_kv, n_kv], 1)
    want = attention.varlen_attn_ref(rope.rope_apply_ref(q, cos, sin), rope.rope_apply_ref(k, cos, sin), v, cu, cu, causal, D ** -0.5, window)
    want.backward(do.float())
    x = qkv.cuda().requires_grad_()
    got = attention.rope_attention(x, cos.cuda(), sin.cuda(), cu.cuda(), n_q, n_kv, D, causal, D ** -0.5, window, max_len)
    got.backward(do.cuda())
    _cuda.check_status()
    for a, b in ((got.detach(), want.detach()), (x.grad, ref.grad)):
        assert torch.isfinite(a).all()
        assert (a.float().cpu() - b).norm() < 2 ** -6 * b.norm()


def test_small_document_kernel_refuses_a_longer_document():
    """The promise of ``max_len`` is checked: the document is skipped and the status word raised, nothing is read past a tile."""
    from lmms_engine_b200.ops import _cuda, attention

    x = torch.randn(70, 3 * 64, device="cuda", dtype=torch.bfloat16)
    cs = torch.ones(70, 64, device="cuda")
    attention.rope_attention(x, cs, cs, torch.tensor([0, 70], dtype=torch.int32, device="cuda"), 1, 1, 64, False, 0.125, max_len=64)
    with pytest.raises(RuntimeError):
        _cuda.check_status()


@pytest.mark.parametrize("lens,n_q,n_kv,D", [((1,), 1, 1, 128), ((70, 3), 5, 1, 64), ((64, 129, 30), 4, 2, 128)])
def test_head_norm_rotation_attention(lens, n_q, n_kv, D):
    """Per-head norm + rotation + attention from the projection's rows against the fp32 formulation (six bf16 roundings of
    2^-9 on the way: 2^-6 of the 2-norm bounds them), one head group past the end of the work included (odd head counts)."""
    from lmms_engine_b200.ops import _cuda, attention, norm, rope

    torch.manual_seed(4)
    T = sum(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    qkv = (2.0 * torch.randn(T, (n_q + 2 * n_kv) * D)).bfloat16()
    wq, wk = (1 + 0.3 * torch.randn(D)).bfloat16(), (1 + 0.3 * torch.randn(D)).bfloat16()
    ang = torch.randn(T, D // 2).repeat(1, 2)
    cos, sin, do = ang.cos(), ang.sin(), torch.randn(T, n_q, D).bfloat16()
    ref = [t.float().requires_grad_() for t in (qkv, wq, wk)]
    q, k, v = ref[0].view(T, -1, D).split([n_q, n_kv, n_kv], 1)
    q, k = norm.rmsnorm_ref(q, ref[1], 1e-6), norm.rmsnorm_ref(k, ref[2], 1e-6)
    want = attention.varlen_attn_ref(rope.rope_apply_ref(q, cos, sin), rope.rope_apply_ref(k, cos, sin), v, cu, cu, True, D ** -0.5)
    want.backward(do.float())
    dev = [t.cuda().requires_grad_() for t in (qkv, wq, wk)]
    got = attention.rope_attention(dev[0], cos.cuda(), sin.cuda(), cu.cuda(), n_q, n_kv, D, True, D ** -0.5, norms=(dev[1], dev[2], 1e-6))
    got.backward(do.cuda())
    _cuda.check_status()
    for a, b in [(got.detach(), want.detach())] + [(x.grad, r.grad) for x, r in zip(dev, ref)]:
        assert torch.isfinite(a).all()
        assert (a.float().cpu() - b).norm() < 2 ** -6 * b.norm() + 1e-5
    with torch.no_grad():
        q2, k2 = attention.rope_heads(dev[0], cos.cuda(), sin.cuda(), n_q, n_kv, D, (dev[1], dev[2], 1e-6))
        q1 = rope.rope_apply(norm.rmsnorm(dev[0][:, :n_q * D].reshape(-1, D), dev[1], 1e-6).view(T, n_q, D), cos.cuda(), sin.cuda())
    assert torch.equal(q2, q1) and k2.shape == (T, n_kv, D)  # the sums run in the order of the separate kernels


@pytest.mark.parametrize("D,heads,kv", [(64, 6, 2), (128, 5, 1), (128, 4, 4)])
@pytest.mark.parametrize("lens", [(1,), (130, 7, 64)])
def test_fused_head_norm_gives_the_bits_of_the_separate_passes(D, heads, kv, lens):
    """An attention layer with the per-head norms read by the fused kernels and with the norms called (a hook asks for that):
    outputs and all gradients but the two norm weights' are equal bit by bit; those are fp32 sums over the rows in another
    order, rounded once."""
    from lmms_engine_b200.models.decoder_lm import Attention, DecoderConfig, PackedContext
    from lmms_engine_b200.ops import _cuda

    torch.manual_seed(5)
    T, H = sum(lens), 256
    cfg = DecoderConfig(hidden_size=H, num_attention_heads=heads, num_key_value_heads=kv, head_dim=D, qk_norm=True, attention_bias=True)
    with torch.device("cuda"):
        layer = Attention(cfg, 0).to(torch.bfloat16)
        with torch.no_grad():
            layer.q_norm.weight.add_(0.3 * torch.randn(D))
            layer.k_norm.weight.add_(0.3 * torch.randn(D))
        ang = torch.randn(T, D // 2).repeat(1, 2)
        cu = torch.tensor([0] + torch.tensor(lens, device="cpu").cumsum(0).tolist(), dtype=torch.int32)
        x, dy = torch.randn(T, H).bfloat16(), torch.randn(T, H).bfloat16()
    ctx = PackedContext(cu, max(lens), ang.cos(), ang.sin(), True)

    def run():
        layer.zero_grad(set_to_none=True)
        xs, n0 = x.clone().requires_grad_(), _cuda.launch_count
        y = layer(xs, ctx)
        y.backward(dy)
        return _cuda.launch_count - n0, {"y": y.detach(), "x": xs.grad, **{n: p.grad.clone() for n, p in layer.named_parameters()}}

    fused_launches, fused = run()
    hooks = [m.register_forward_hook(lambda *a: None) for m in (layer.q_norm, layer.k_norm)]
    separate_launches, separate = run()
    for h in hooks:
        h.remove()
    assert fused_launches < separate_launches
    for name, a in fused.items():
        b = separate[name]
        if "norm" in name:
            assert ((a.float() - b.float()).abs() <= 2 ** -8 * b.float().abs() + 1e-6 * T ** 0.5).all(), name
        else:
            assert torch.equal(a, b), name
