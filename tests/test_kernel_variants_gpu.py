"""Branches of the dispatch rules at the sizes where they change hands, against 64-bit references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm()).item()


def _rand(*s, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(dtype)


@pytest.mark.parametrize("M", [1, 7, 9, 3000])
@pytest.mark.parametrize("D", [8, 264, 512, 1024, 1032, 1020])
@pytest.mark.parametrize("layer", [False, True])
def test_norm_backward_column_sums(M, D, layer):
    from megalodon_b200 import ops
    torch.manual_seed(D)
    x, w, b, g = _rand(M, D), _rand(D, scale=0.2), _rand(D), _rand(M, D)
    xs = [x.clone().requires_grad_(True), w.clone().requires_grad_(True), b.clone().requires_grad_(True)]
    rs = [t.double().requires_grad_(True) for t in (x, w, b)]
    if layer:
        ops.layer_norm(xs[0], xs[1], xs[2], 1e-5, weight_offset=1.0).backward(g)
        torch.nn.functional.layer_norm(rs[0], (D,), rs[1] + 1.0, rs[2], 1e-5).backward(g.double())
    else:
        ops.rms_norm(xs[0], xs[1], 1e-5, weight_offset=1.0).backward(g)
        (rs[0] * torch.rsqrt(rs[0].pow(2).mean(-1, keepdim=True) + 1e-5) * (rs[1] + 1.0)).backward(g.double())
    for a, r in list(zip(xs, rs))[:3 if layer else 2]:
        assert _rel(a.grad, r.grad) < 2.0 ** -8         # fp32 sums, one rounding


@pytest.mark.parametrize("V", [8, 4096, 4104, 1000, 1003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_cross_entropy_rows(V, dtype):
    """Vectorised and scalar rows; masked-out logits (minus infinity), a whole leading stretch of them included."""
    from megalodon_b200 import ops
    torch.manual_seed(V)
    x = _rand(6, V, dtype=dtype, scale=3.0)
    x[1, : V // 2] = float("-inf")
    x[2, 1:] = torch.finfo(dtype).min
    t = torch.tensor([0, V - 1, 0, -100, V // 2, V - 2], device="cuda")
    a, r = x.clone().requires_grad_(True), x.double().requires_grad_(True)
    loss = ops.cross_entropy(a, t)
    want = torch.nn.functional.cross_entropy(r, t, reduction="none")
    torch.testing.assert_close(loss.double(), want, rtol=2e-6, atol=2e-6)
    g = torch.rand(6, device="cuda")
    loss.backward(g)
    want.backward(g.double())
    assert _rel(a.grad, r.grad) < (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5)
    assert a.grad[3].abs().max() == 0


@pytest.mark.parametrize("n", [1, 7, 4096, 100003])
def test_gradient_norm_and_scale(n):
    from megalodon_b200.ops import cuda_ops
    g = _rand(n + 1)[1:] if n % 2 else _rand(n)             # (an offset of one element: the scalar path)
    acc = torch.zeros((), dtype=torch.float64, device="cuda")
    cuda_ops.sum_squares(g, acc)
    assert abs(acc.item() / g.double().pow(2).sum().item() - 1) < 1e-5
    want = (g.float() * 0.3).bfloat16()
    cuda_ops.scale_by_ptr(g, torch.tensor([0.3], device="cuda"))
    assert torch.equal(g, want)


# lengths around the 8-column pieces, the 128-row tile (one CTA / CTA pair) and the 256-column tile; several
# sequences and heads in one launch
@pytest.mark.parametrize("B,L,H,dk,dv", [(1, 5, 2, 16, 24), (3, 37, 1, 64, 64), (2, 128, 2, 32, 40), (2, 129, 3, 64, 72),
                                         (2, 257, 2, 128, 256), (3, 777, 1, 64, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_any_length(B, L, H, dk, dv, causal):
    from megalodon_b200 import ops
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(L)
    q, k, v = _rand(B, L, H, dk, scale=dk ** -0.25), _rand(B, L, H, dk, scale=dk ** -0.25), _rand(B, L, H, dv)
    g = _rand(B, L, H, dv)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = ops.attention(*leaves, 0.7, 0.0, causal, True)
    out.backward(g)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = torch.einsum("blhd,bmhd->bhlm", ref[0], ref[1]) * 0.7
    if causal:
        s = s.masked_fill(torch.ones(L, L, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.einsum("bhlm,bmhd->blhd", torch.softmax(s, -1), ref[2])
    want.backward(g.double())
    # probabilities, scores' gradients and results are rounded to 8 bits once each
    assert _rel(out, want) < 2.0 ** -7
    for a, b in zip(leaves, ref):
        assert _rel(a.grad, b.grad) < 2.0 ** -6
    cuda_ops.check_kernel_errors()


@pytest.mark.parametrize("slen,past", [(37, 0), (96, 0), (33, 20), (192, 0)])
def test_causal_marker_equals_the_explicit_mask(slen, past):
    """The unfused model without dropout: `CAUSAL` against the additive mask it stands for."""
    from megalodon_b200.modules.moving_average_gated_attention import CAUSAL, _InnerAttention
    torch.manual_seed(slen)
    H, dk, dv, c, B = 2, 32, 64, 96, 2
    inner = _InnerAttention(dk, dv, H, c, 0.1, None).eval()
    q, k, v = _rand(B, slen, H * dk, scale=0.5), _rand(B, slen, H * dk, scale=0.5), _rand(B, slen, H * dv)
    kv = (_rand(B, past, H, dk, scale=0.5), _rand(B, past, H, dv), past)
    rows = min(slen, c)
    assert inner.causal_mask(q, rows, past) is CAUSAL
    mask = torch.full((1, 1, rows, rows + past), float("-inf"), device="cuda").triu(past + 1).bfloat16()
    got, kv1 = inner(q, k, v, CAUSAL, None, kv)
    want, kv2 = inner(q, k, v, mask, None, kv)
    assert _rel(got, want) < 2.0 ** -6 and torch.equal(kv1[0], kv2[0]) and kv1[2] == kv2[2]
    assert torch.is_tensor(inner.train().causal_mask(q, rows, past))       # dropout acts on the probabilities
