"""Causal attention of fewer (or more) queries than keys, wider than one 256-column tile: every product of that
route contracts whole rows, so a masked column that is not zero is a key from the future."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm()).item()


def _rand(*s, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(dtype)


def _hidden(L1, L2):
    """True where query r may not see key c."""
    return torch.arange(L2, device="cuda") > torch.arange(L1, device="cuda").unsqueeze(-1) + (L2 - L1)


def _probs(s):
    """Causal softmax in the dtype of s; a row without keys gives zeros."""
    hide = _hidden(*s.shape[-2:])
    return torch.softmax(s.masked_fill(hide, -1e30), -1) * ~hide


# 600 new tokens behind 500 cached ones; an odd key count (scalar rows); a single short query block; more queries
# than keys (the first rows see nothing)
@pytest.mark.parametrize("B,L1,L2,H", [(2, 600, 1100, 2), (1, 333, 905, 1), (1, 2, 777, 2), (1, 24, 2048, 1), (1, 300, 264, 2)])
def test_rectangular_causal_attention(B, L1, L2, H):
    from megalodon_b200 import ops
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(L2)
    dk, dv = 32, 72
    q, k = _rand(B, L1, H, dk, scale=dk ** -0.25), _rand(B, L2, H, dk, scale=dk ** -0.25)
    v, g = _rand(B, L2, H, dv), _rand(B, L1, H, dv)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    torch.cuda.empty_cache()        # the score buffers are uninitialised memory: make that NaN
    poison = [torch.full((B * H * L1 * (-(-L2 // 128) * 128),), float("nan"), dtype=q.dtype, device="cuda") for _ in range(3)]
    del poison
    out = ops.attention(*leaves, 0.7, 0.0, True, True)
    out.backward(g)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    p = _probs(torch.einsum("blhd,bmhd->bhlm", ref[0], ref[1]) * 0.7)
    want = torch.einsum("bhlm,bmhd->blhd", p, ref[2])
    want.backward(g.double())
    # scores, probabilities, their gradients and the results are rounded to 8 bits once each
    assert _rel(out, want) < 2.0 ** -6
    for a, b in zip(leaves, ref):
        assert _rel(a.grad, b.grad) < 2.0 ** -5
    cuda_ops.check_kernel_errors()


@pytest.mark.parametrize("slen,past", [(600, 500), (401, 300)])
def test_unfused_model_against_a_cached_prefix(slen, past):
    """Several tokens behind a cached prefix: the marker that stands for the additive mask, and the mask itself."""
    from megalodon_b200.modules.moving_average_gated_attention import CAUSAL, _InnerAttention
    torch.manual_seed(slen)
    H, dk, dv, c, B = 2, 32, 64, 1200, 2
    inner = _InnerAttention(dk, dv, H, c, 0.1, None).eval()
    q, k, v = _rand(B, slen, H * dk, scale=0.5), _rand(B, slen, H * dk, scale=0.5), _rand(B, slen, H * dv)
    kv = (_rand(B, past, H, dk, scale=0.5), _rand(B, past, H, dv), past)
    assert inner.causal_mask(q, slen, past) is CAUSAL
    mask = torch.full((1, 1, slen, slen + past), float("-inf"), device="cuda").triu(past + 1).bfloat16()
    got, _ = inner(q, k, v, CAUSAL, None, kv)
    want, _ = inner(q, k, v, mask, None, kv)
    assert _rel(got, want) < 2.0 ** -6


# the operator by itself: rows wider than a tile, vectorised and scalar, square and not
@pytest.mark.parametrize("L1,L2", [(600, 600), (40, 700), (40, 701), (300, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_softmax_operator_clears_masked_columns(L1, L2, dtype):
    from megalodon_b200 import ops
    torch.manual_seed(L2)
    x, g = _rand(2, L1, L2, dtype=dtype), _rand(2, L1, L2, dtype=dtype)
    a, r = x.clone().requires_grad_(True), x.double().requires_grad_(True)
    y, want = ops.attention_softmax(a, 0.0, True, True), _probs(r)
    y.backward(g)
    want.backward(g.double())
    tol = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    assert _rel(y, want) < tol and _rel(a.grad, r.grad) < 4 * tol      # (the gradient starts from the rounded y)
    assert (y[:, _hidden(L1, L2)] == 0).all() and (a.grad[:, _hidden(L1, L2)] == 0).all()


@pytest.mark.parametrize("L2", [2048, 2040])
def test_backward_memory_without_the_fused_softmax(L2):
    """The gradients of the probabilities are held for a bounded number of sequences, whatever the batch."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(0)
    B, L1, H, d = 5, 2048, 8, 16
    q, k, v, g = _rand(B, L1, H, d), _rand(B, L2, H, d), _rand(B, L2, H, d), _rand(B, L1, H, d)

    def grads(s):
        leaves = [t[s].clone().requires_grad_(True) for t in (q, k, v)]
        out = cuda_ops.attention(*leaves, 0.25, 0.0, True, True)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        res = torch.autograd.grad(out, leaves, g[s])
        torch.cuda.synchronize()
        return res, torch.cuda.max_memory_allocated() - before
    cuda_ops.set_fused_attention_softmax(False)
    try:
        whole, peak = grads(slice(0, B))
        assert peak < (128 << 20) + (32 << 20), peak        # 64 MB a sequence, and the results
        for b in range(B):
            one, _ = grads(slice(b, b + 1))
            for a, r in zip(one, whole):
                assert torch.equal(a[0], r[b])
    finally:
        cuda_ops.set_fused_attention_softmax(True)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dropout", [0.0, 0.5])
def test_attention_of_no_sequences(causal, dropout):
    from megalodon_b200 import ops
    leaves = [torch.empty(0, 16, 2, 16, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3)]
    out = ops.attention(*leaves, 1.0, dropout, causal, True)
    out.sum().backward()
    assert out.shape == (0, 16, 2, 16) and all(t.grad.shape == t.shape for t in leaves)


@pytest.mark.parametrize("shape,stride,offset", [((1, 16, 2, 16), (1001, 32, 16, 1), 0), ((2, 1, 2, 16), (32, 7, 16, 1), 0),
                                                 ((2, 16, 1, 16), (256, 16, 13, 1), 0), ((2, 16, 2, 16), (512, 32, 16, 1), 3)])
def test_attention_of_odd_strides(shape, stride, offset):
    """Dimensions of size one may carry any stride and a view may start anywhere; both count as contiguous."""
    from megalodon_b200 import ops
    torch.manual_seed(0)
    ts = [torch.as_strided(_rand(4096), shape, stride, offset) for _ in range(4)]
    assert all(t.is_contiguous() for t in ts)
    res = []
    for norm in (lambda t: t, lambda t: t.clone(memory_format=torch.contiguous_format)):
        leaves = [norm(t).detach().requires_grad_(True) for t in ts[:3]]
        out = ops.attention(*leaves, 1.0, 0.0, True, True)
        res.append([out, *torch.autograd.grad(out, leaves, norm(ts[3]))])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("pieces", [(512, 511), (300, 700), (5, 900, 100)])
def test_model_in_pieces_against_the_whole(fused, pieces):
    """Several tokens at a time against a growing cache give the logits of one call over all of them."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.utils import init_cache, set_random_seed
    cfg = ModelConf(num_layers=2, model_dim=256, num_heads=2, z_dim=128, value_dim=512, ffn_hidden_dim=384, chunk_size=1024,
                    vocab_size=520, swiglu=True, norm_num_groups=16, efficient_attn="fused" if fused else None)
    set_random_seed(3)
    model = build_model(cfg, "fp16", False, True).eval()
    tok = torch.randint(0, 520, (2, sum(pieces)), device="cuda")
    with torch.no_grad():
        want, _ = model(tok, cache=init_cache(2, model, torch.float16))
        cache, at = init_cache(2, model, torch.float16), 0
        for n in pieces:
            got, cache = model(tok[:, at:at + n], cache=cache)
            # some ten roundings to 2^-11 a layer on either side, adding up like a random walk
            assert _rel(got, want[:, at:at + n]) < (2 * 10 * cfg.num_layers) ** 0.5 * 2.0 ** -11, n
            at += n
