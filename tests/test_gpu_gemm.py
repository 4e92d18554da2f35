"""tcgen05 GEMM against an fp32 PyTorch reference (all operand layouts and epilogues)."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", dtype=torch.float32) * scale).to(torch.bfloat16)


def _check(out, ref, tol=2e-2):
    err = (out.float() - ref).abs().max().item()
    den = ref.abs().max().item() + 1e-6
    assert err / den < tol, f"rel err {err / den:.4f}"


SHAPES = [(128, 256, 64), (256, 512, 128), (384, 768, 320), (200, 264, 72), (1024, 3584, 3584), (4096, 2304, 512),
          (77, 40, 24)]


@pytest.fixture(autouse=True, params=["pair", "single"])
def tile_mode(request):
    """Every test runs with 256 x 256 tiles on CTA pairs (the default) and with one-CTA tiles only."""
    from lmms_engine_b200.ops import _cuda

    set_mode = _cuda.fn("b200_gemm_set_pair_mode")
    set_mode(1 if request.param == "pair" else 0)
    yield request.param
    set_mode(1)


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nt(M, N, K):
    from lmms_engine_b200.ops import gemm, _cuda

    a, b = _rand(M, K), _rand(N, K)
    out = gemm.gemm(a, b)
    _check(out, a.float() @ b.float().t())
    _cuda.check_status()


@pytest.mark.parametrize("M,N,K", SHAPES[:-1] + [(80, 40, 24)])
def test_gemm_nn_b_mn_major(M, N, K):
    from lmms_engine_b200.ops import gemm, _cuda

    a, b = _rand(M, K), _rand(K, N)
    out = gemm.gemm(a, b, b_mn_major=True)
    _check(out, a.float() @ b.float())
    _cuda.check_status()


@pytest.mark.parametrize("M,N,K", SHAPES[:-1] + [(80, 40, 24)])
def test_gemm_tn_both_mn_major(M, N, K):
    from lmms_engine_b200.ops import gemm, _cuda

    a, b = _rand(K, M), _rand(K, N)
    out = gemm.gemm(a, b, a_mn_major=True, b_mn_major=True)
    _check(out, a.float().t() @ b.float())
    _cuda.check_status()


def test_gemm_bias_beta():
    from lmms_engine_b200.ops import gemm

    M, N, K = 300, 520, 192
    a, b, c, bias = _rand(M, K), _rand(N, K), _rand(M, N), _rand(N)
    out = gemm.gemm(a, b, alpha=0.5, beta=2.0, bias=bias, cin=c)
    _check(out, 0.5 * (a.float() @ b.float().t()) + bias.float() + 2.0 * c.float())


@pytest.mark.parametrize("M,K", [(512, 256), (3584, 1024), (640, 200)])
def test_gemm_symmetric(M, K):
    from lmms_engine_b200.ops import gemm

    x = _rand(M, K, scale=0.1)
    out = gemm.gemm(x, x, symmetric=True)
    ref = x.float() @ x.float().t()
    _check(out, ref)
    assert torch.equal(out, out.t()), "mirrored store must make the result exactly symmetric"
    a = out
    out2 = gemm.gemm(a, a, alpha=2.0, beta=-3.0, cin=a, symmetric=True)
    _check(out2, 2.0 * (a.float() @ a.float().t()) - 3.0 * a.float())


@pytest.mark.parametrize("M,I,K", [(256, 384, 128), (1000, 688, 256), (4096, 18944, 3584)])
def test_gemm_swiglu(M, I, K):
    from lmms_engine_b200.ops import gemm

    x, wg, wu = _rand(M, K), _rand(I, K, scale=0.05), _rand(I, K, scale=0.05)
    h, g, u = gemm.gemm_swiglu(x, wg, wu, store_gu=True)
    gr, ur = x.float() @ wg.float().t(), x.float() @ wu.float().t()
    _check(g, gr)
    _check(u, ur)
    _check(h, torch.nn.functional.silu(g.float()) * u.float(), tol=1e-2)
    h2, _, _ = gemm.gemm_swiglu(x, wg, wu, store_gu=False)
    assert torch.equal(h, h2)


@pytest.mark.parametrize("M,N,K", [(256, 1024, 128), (333, 4104, 256)])
def test_gemm_stats(M, N, K):
    from lmms_engine_b200.ops import gemm

    x, w = _rand(M, K), _rand(N, K, scale=0.2)
    logits, stats = gemm.gemm_stats(x, w)
    ref = x.float() @ w.float().t()
    _check(logits[:, :N], ref)
    lf = logits[:, :N].float()
    mx = stats[..., 0].max(dim=1).values
    lse = mx + torch.log((stats[..., 1] * torch.exp(stats[..., 0] - mx[:, None])).sum(1))
    assert torch.allclose(lse, torch.logsumexp(lf, dim=1), atol=2e-3, rtol=1e-4)


def test_linear_autograd_matches_torch():
    from lmms_engine_b200.ops import gemm

    x = _rand(2, 192, 320).requires_grad_()
    w = _rand(456 // 8 * 8, 320, scale=0.05).requires_grad_()
    b = _rand(456 // 8 * 8).requires_grad_()
    y = gemm.linear(x, w, b)
    dy = _rand(*y.shape)
    y.backward(dy)
    xr, wr, br = (t.detach().float().requires_grad_() for t in (x, w, b))
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(dy.float())
    _check(y, yr.detach())
    _check(x.grad, xr.grad)
    _check(w.grad, wr.grad)
    _check(b.grad, br.grad)


@pytest.mark.parametrize("M", [1, 4, 8, 9, 16, 17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("N,K", [(8, 8), (1000, 520), (4608, 3584)])
def test_few_rows(M, N, K):
    """Weight-streaming product of at most 64 rows: tile edges of the row groups, ragged K and N, bias, strided input."""
    from lmms_engine_b200.ops import gemm, _cuda

    torch.manual_seed(M * N + K)
    x = torch.randn(M, K + 8, device="cuda").to(torch.bfloat16)[:, :K]
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    b = torch.randn(N, device="cuda").to(torch.bfloat16)
    want = x.float() @ w.float().t()
    # one rounding to bf16 (2^-9 of the value) on top of fp32 sums
    for bias, ref in ((None, want), (b, want + b.float())):
        y = gemm.matmul_nt(x, w, bias)
        _cuda.check_status()
        assert ((y.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4 * K ** 0.5).all()


@pytest.mark.parametrize("M,N,K,few", [(1, 16384, 64, True), (1, 16392, 64, False), (1, 16392, 2048, True), (4, 16392, 8192, False),
                                       (5, 12288, 64, True), (16, 12296, 64, False), (17, 8192, 64, True), (32, 8200, 64, False),
                                       (33, 4096, 64, True), (48, 4104, 64, False), (49, 3584, 64, True), (64, 3592, 64, False),
                                       (65, 64, 64, False)])
def test_few_rows_take_the_kernel_that_is_faster(M, N, K, few, monkeypatch):
    """Both sides of every line of the rule; either kernel gives fp32 sums rounded once."""
    from lmms_engine_b200.ops import gemm, _cuda

    seen, real = [], _cuda.call
    monkeypatch.setattr(_cuda, "call", lambda name, *a: (seen.append(name), real(name, *a))[1])
    x, w, b = _rand(M, K), _rand(N, K, scale=0.05), _rand(N)
    y = gemm.matmul_nt(x, w, b)
    assert ("b200_skinny_linear" in seen) == few
    want = x.float() @ w.float().t() + b.float()
    assert ((y.float() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4 * K ** 0.5).all()


@pytest.mark.parametrize("P,K,inter,N,biases", [(1, 64, 36, 64, True), (65, 72, 100, 136, True), (300, 128, 130, 64, False),
                                               (257, 1280, 3420, 1280, True), (129, 64, 3, 8, True)])
def test_gated_mlp_any_width(P, K, inter, N, biases):
    """Inner widths that are no multiple of 8 (rows padded to 16 bytes, products stop at the true width): against fp32
    linears.  Two bf16 roundings between the products and one of the result: 2^-6 of the 2-norm bounds them."""
    from lmms_engine_b200.ops import swiglu

    torch.manual_seed(0)
    shapes = [(P, K), (inter, K), (inter,), (inter, K), (inter,), (N, inter), (N,)]
    raw = [torch.randn(s) * (1.0 if i == 0 else K ** -0.5 if i < 5 else inter ** -0.5) for i, s in enumerate(shapes)]
    raw = [t.bfloat16() for t in raw]
    if not biases:
        raw[2] = raw[4] = raw[6] = None
    ref = [None if t is None else t.float().requires_grad_() for t in raw]
    F = torch.nn.functional
    want = F.linear(F.silu(F.linear(ref[0], ref[1], ref[2])) * F.linear(ref[0], ref[3], ref[4]), ref[5], ref[6])
    dy = torch.randn(P, N).bfloat16()
    want.backward(dy.float())
    dev = [None if t is None else t.cuda().requires_grad_() for t in raw]
    got = swiglu.gated_mlp(*dev)
    got.backward(dy.cuda(), retain_graph=True)
    first = [None if t is None else t.grad.clone() for t in dev]
    for a, b in [(got.detach(), want.detach())] + [(f, r.grad) for f, r in zip(first, ref) if r is not None]:
        assert torch.isfinite(a).all()
        assert (a.float().cpu() - b).norm() < 2 ** -6 * b.norm() + 1e-6
    got.backward(dy.cuda())  # the saved activations are not overwritten: a second pass adds the same gradients
    for t, f in zip(dev, first):
        if t is not None:
            assert torch.equal(t.grad, f + f)


@pytest.mark.parametrize("P,K,inter,N,biases", [(1, 64, 36, 64, True), (65, 72, 100, 136, True), (300, 128, 130, 64, False),
                                               (257, 1280, 3420, 1280, True), (129, 64, 3, 8, True)])
def test_gated_mlp_fused_at_small_sizes(P, K, inter, N, biases, monkeypatch):
    """Unaligned widths below the line run as linears; the fused function has to hold there too."""
    from lmms_engine_b200.ops import swiglu, _cuda

    seen, real = [], _cuda.call
    monkeypatch.setattr(_cuda, "call", lambda name, *a: (seen.append(name), real(name, *a))[1])
    test_gated_mlp_any_width(P, K, inter, N, biases)
    assert "b200_gemm_swiglu_bf16" not in seen
    monkeypatch.setattr(swiglu, "UNALIGNED_MIN", 0)
    test_gated_mlp_any_width(P, K, inter, N, biases)
    assert "b200_gemm_swiglu_bf16" in seen


@pytest.mark.parametrize("inter", [36, 40])
def test_gated_mlp_under_saved_tensor_hooks(inter):
    """Activations that are moved to the host and back between the passes come back without the strides of a view."""
    from lmms_engine_b200.ops import swiglu

    torch.manual_seed(0)
    raw = [_rand(130, 64), _rand(inter, 64, scale=0.1), _rand(inter), _rand(inter, 64, scale=0.1), _rand(inter), _rand(72, inter, scale=0.1), _rand(72)]
    dy, grads = _rand(130, 72), []
    for hooked in (False, True):
        leaves = [t.clone().requires_grad_() for t in raw]
        with torch.autograd.graph.save_on_cpu(pin_memory=True) if hooked else contextlib.nullcontext():
            y = swiglu._GatedMLPFn.apply(*leaves)
        y.backward(dy)
        grads.append([t.grad for t in leaves])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("inter", [36, 40])
@pytest.mark.parametrize("wrong", ["gate", "up", "both", "bias", "down"])
def test_gated_mlp_refuses_shapes_that_do_not_match(inter, wrong):
    """Weights narrower or wider than the rows and short biases are refused on the host, as three linears refuse them: the
    kernel takes one width for all and would read past the end."""
    from lmms_engine_b200.ops import swiglu

    K, N = 64, 64
    for d in (-8, 8):
        wg, bg, wu, bu, wd, bd = _rand(inter, K), _rand(inter), _rand(inter, K), _rand(inter), _rand(N, inter), _rand(N)
        if wrong == "gate":
            wg = _rand(inter, K + d)
        elif wrong == "up":
            wu = _rand(inter, K + d)
        elif wrong == "both":
            wg, wu = _rand(inter, K + d), _rand(inter, K + d)
        elif wrong == "bias":
            bu = _rand(inter + d)
        else:
            wd = _rand(N, inter + d)
        with pytest.raises((ValueError, RuntimeError)):
            swiglu.gated_mlp(_rand(130, K), wg, bg, wu, bu, wd, bd)


@pytest.mark.parametrize("rows,N,ld", [(1, 8, 8), (31, 256, 256), (33, 260, 264), (1000, 1152, 1152), (4097, 3420, 3424), (7, 1, 8)])
def test_column_sum(rows, N, ld):
    """Remainders of the row and column tiles; rows wider than N hold NaN that may not reach a sum.  fp32 sums, one rounding."""
    from lmms_engine_b200.ops import gemm

    torch.manual_seed(0)
    x = torch.full((rows, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
    x[:, :N] = torch.randn(rows, N, device="cuda").bfloat16()
    want = x[:, :N].double().sum(0)
    got = gemm.column_sum(x[:, :N])
    assert got.shape == (N,) and got.dtype == torch.bfloat16
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6 * rows).all()
