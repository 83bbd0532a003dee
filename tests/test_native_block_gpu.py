"""The block as one native call against the same block through its modules."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-30)).item()


def _block(dtype=torch.bfloat16, chunk=256, swiglu=True, fused="fused", affine=True, **kw):
    from megalodon_b200.config import ModelConf
    from megalodon_b200.models.mega import MegaBlock
    torch.manual_seed(0)
    cfg = ModelConf(num_layers=1, model_dim=256, num_heads=2, z_dim=128, value_dim=512, ffn_hidden_dim=384, chunk_size=chunk,
                    vocab_size=64, swiglu=swiglu, norm_num_groups=16, efficient_attn=fused, norm_affine=affine, **kw)
    block = MegaBlock(cfg, 0).cuda()
    with torch.no_grad():
        for p in block.parameters():
            p.add_(torch.randn_like(p) * 0.05)
    return block.to(dtype)


def _freqs(block, L):
    a = block.mega
    ang = torch.outer(torch.arange(min(L, a.chunk_size), device="cuda").float(), torch.rand(a.z_head_dim // 2, device="cuda"))
    return torch.polar(torch.ones_like(ang), ang)


def _calls(monkeypatch):
    from megalodon_b200.modules import native_block
    calls = []
    inner = native_block._MegaBlock.forward
    monkeypatch.setattr(native_block._MegaBlock, "forward",
                        staticmethod(lambda ctx, *a: (calls.append(1), inner(ctx, *a))[1]))
    return calls


def _through_modules(monkeypatch, f):
    from megalodon_b200.modules import native_block
    with monkeypatch.context() as m:
        m.setattr(native_block, "forward", lambda *a, **k: None)
        return f()


def _flat(o):
    if isinstance(o, torch.Tensor):
        return [torch.view_as_real(o) if o.is_complex() else o]
    return [t for x in o for t in _flat(x)] if isinstance(o, (tuple, list)) else [] if o is None else [torch.tensor(o)]


@pytest.mark.parametrize("B,L", [(1, 2), (1, 37), (3, 37), (2, 255), (2, 256), (1, 768)])
@pytest.mark.parametrize("dtype,swiglu,fused,affine", [(torch.bfloat16, True, "fused", True), (torch.float16, False, None, True),
                                                       (torch.bfloat16, False, "fused", False)])
def test_without_gradients(monkeypatch, B, L, dtype, swiglu, fused, affine):
    """Same kernels in the same order, so the same bits: outputs, running statistics, EMA state and cached keys.  (A row
    sum is one contribution, or two added in either order, up to 512 keys.)"""
    from megalodon_b200.modules.moving_average_gated_attention import CAUSAL
    block = _block(dtype, swiglu=swiglu, fused=fused, affine=affine).eval()
    calls = _calls(monkeypatch)
    x, freqs = torch.randn(B, L, 256, device="cuda").to(dtype), _freqs(block, L)
    mask = None if fused else CAUSAL
    prev = (torch.full((B,), 5, device="cuda"), torch.randn(B, 16, device="cuda").to(dtype) * 0.1,
            torch.rand(B, 16, device="cuda").to(dtype) + 0.5)
    hx = torch.view_as_complex(torch.randn(B, 256, 16, 2, device="cuda"))
    states = [dict(), dict(carry=(*prev, hx), piece=(1, 2, 2 * L)), dict(carry=(*prev, hx), piece=(1, 3, 3 * L)),
              dict(carry=(*prev, hx), piece=(1, 2, 2 * L, True)), dict(cache=((None, None, 0), (None, None, None), None)),
              dict(cache=((None, None, 0), prev, hx))]
    with torch.no_grad():
        for kw in states:
            calls.clear()
            got = _flat(block(x, freqs, mask, **kw))
            assert calls
            want = _flat(_through_modules(monkeypatch, lambda: block(x, freqs, mask, **kw)))
            assert len(got) == len(want)
            for a, b in zip(got, want):
                assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)


@pytest.mark.parametrize("B,L", [(3, 2), (2, 512), (2, 16640)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_prior_statistics(monkeypatch, B, L, dtype):
    """The prior that the kernel spreads over the batch, in both forms of the scan (one launch up to 16384 steps), against
    the expanded one: the same bits, and another prior gives others."""
    block = _block(dtype).eval()
    calls = _calls(monkeypatch)
    x, freqs = torch.randn(B, L, 256, device="cuda").to(dtype), _freqs(block, L)
    with torch.no_grad():
        block.mega.timenorm.prior_count.fill_(3)
        block.mega.timenorm.prior_logv.uniform_(-2.0, 2.0)
        got = _flat(block(x, freqs, piece=(0, 2, 2 * L)))
        assert calls
        want = _flat(_through_modules(monkeypatch, lambda: block(x, freqs, piece=(0, 2, 2 * L))))
        for a, b in zip(got, want):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
        block.mega.timenorm.prior_logv.add_(1.0)
        assert not torch.equal(_flat(block(x, freqs, piece=(0, 2, 2 * L)))[0], got[0])


@pytest.mark.parametrize("B,L,swiglu,fused,affine,dtype", [(2, 40, True, "fused", True, torch.bfloat16),
                                                           (1, 37, False, None, True, torch.bfloat16),
                                                           (2, 256, True, None, False, torch.float16),
                                                           (1, 512, False, "fused", True, torch.bfloat16)])
def test_gradients(monkeypatch, B, L, swiglu, fused, affine, dtype):
    """Of the input, the carried state and every parameter.  The native block rounds some sums of gradients once where
    autograd rounds every addition."""
    from megalodon_b200.modules.moving_average_gated_attention import CAUSAL
    block = _block(dtype, swiglu=swiglu, fused=fused, affine=affine)
    calls = _calls(monkeypatch)
    freqs, mask = _freqs(block, L), None if fused else CAUSAL
    x = torch.randn(B, 2 * L, 256, device="cuda").to(dtype)
    g = torch.randn_like(x)

    def run():
        leaf = x.clone().requires_grad_(True)
        parts, carry = [], None
        for i, piece in enumerate(leaf.split(L, dim=1)):           # (two pieces: the second one's x has gaps between rows)
            y, carry = block(piece, freqs, mask, None, carry, (i, 2, 2 * L))
            parts.append(y)
        out = torch.cat(parts, 1)
        return [out, *torch.autograd.grad(out, [leaf, *block.parameters()], g)]
    got = run()
    assert len(calls) == 2
    want = _through_modules(monkeypatch, run)
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert _rel(a, b) < 2.0 ** -6, (a.shape, _rel(a, b))


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("L", [64, 512])
def test_a_kept_graph_is_walked_again(monkeypatch, native, L):
    """Two backward passes over one graph, the block's own and its attention's: the same gradients."""
    from megalodon_b200.modules import native_block
    if not native:
        monkeypatch.setattr(native_block, "forward", lambda *a, **k: None)
    block = _block()
    x = torch.randn(2, L, 256, device="cuda").bfloat16().requires_grad_(True)
    y, _ = block(x, _freqs(block, L))
    g = torch.randn_like(y)
    first = torch.autograd.grad(y, [x, *block.parameters()], g, retain_graph=True)
    for a, b in zip(first, torch.autograd.grad(y, [x, *block.parameters()], g)):
        assert _rel(b, a) < 1e-5             # (column sums are added in any order)


def test_what_stays_with_the_modules(monkeypatch):
    """Hooks, replaced modules, dropout, frozen parameters, one token, cached keys, doubles and other options."""
    from megalodon_b200.ops import cuda_ops
    calls = _calls(monkeypatch)
    x = torch.randn(2, 64, 256, device="cuda").bfloat16()

    def native(block, x=x, grad=False, **kw):
        calls.clear()
        with torch.set_grad_enabled(grad):
            block(x.clone().requires_grad_(grad), _freqs(block, x.shape[1]), None, **kw)
        return bool(calls)

    assert native(_block()) and native(_block(), grad=True)
    b = _block()
    seen = []
    b.mega.wz.register_forward_hook(lambda *a: seen.append(1))
    b.nffn.register_forward_hook(lambda *a: seen.append(1))
    assert not native(b) and len(seen) >= 1
    b = _block()

    class Adapter(type(b.mega.wv)):
        pass
    b.mega.wv.__class__ = Adapter
    assert not native(b)
    b = _block()
    b.nffn.fc2.weight.requires_grad_(False)
    assert native(b) and not native(b, grad=True)
    assert not native(_block(), x=x[:, :1])
    assert not native(_block(hidden_dropout=0.1), grad=True) and native(_block(hidden_dropout=0.1).eval())
    assert not native(_block().float(), x=x.float())
    assert not native(_block(rescale_nffn=True))
    k = torch.randn(2, 8, 2, 64, device="cuda").bfloat16()
    v = torch.randn(2, 8, 2, 256, device="cuda").bfloat16()
    b = _block().eval()
    calls.clear()
    with torch.no_grad():
        b(x, _freqs(b, 64), None, ((k, v, 8), (None, None, None), None))
    assert not calls
    cuda_ops.set_attention_recompute_scores(True)
    try:
        assert not native(_block(), grad=True)
    finally:
        cuda_ops.set_attention_recompute_scores(False)


def test_a_model_with_the_native_block_through_checkpoints_and_units(monkeypatch):
    """Sharded units (weight gradients in the flat buffer), a recomputed block, two pieces a sequence, two backward passes."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.utils import set_random_seed
    calls = _calls(monkeypatch)
    cfg = ModelConf(num_layers=2, model_dim=256, num_heads=2, z_dim=128, value_dim=512, ffn_hidden_dim=384, chunk_size=128,
                    vocab_size=96, swiglu=True, norm_num_groups=16, efficient_attn="fused", layerwise_ckpt=True, ckpt_layers=1)
    toks = torch.randint(0, 96, (2, 257), device="cuda")

    def run():
        junk = torch.full((64 << 20,), 1e30, device="cuda")     # what a range that nothing writes would show
        del junk
        set_random_seed(0)
        model = build_model(cfg, "bf16", False, True)
        model._wrapped.seq_microbatch_chunks = 1
        out = []
        for _ in range(2):
            losses, _ = model(toks[:, :-1], targets=toks[:, 1:])
            losses.mean().backward()
            out.append(losses.detach())
        model.grad_all_reduce()
        return out + [p._grad_shard.float() for p in model.params_with_grad]
    got = run()
    assert len(calls) == 2 * (2 * 3)            # two passes: pieces times (checkpointed: twice, the other once)
    want = _through_modules(monkeypatch, run)
    assert torch.equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert _rel(a, b) < 2.0 ** -6


@pytest.mark.parametrize("L,swiglu,kernels", [(256, True, 21), (256, False, 19), (37, True, 17)])
def test_launches_are_counted_where_they_are_made(L, swiglu, kernels):
    """TimestepNorm three, EMA one, six norms and element-wise ones (without the gate, which is torch's, for few rows, and
    without SwiGLU), three of attention, eight products (seven; few rows: the four projections in one)."""
    from megalodon_b200.ops import cuda_ops
    block = _block(swiglu=swiglu).eval()
    x, freqs = torch.randn(1, L, 256, device="cuda").bfloat16(), _freqs(block, L)
    with torch.no_grad():
        block(x, freqs)                          # (in eval mode the EMA's coefficients are computed once)
        before = cuda_ops.count_launches()
        block(x, freqs)
    assert cuda_ops.count_launches() - before == kernels
