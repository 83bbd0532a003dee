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
