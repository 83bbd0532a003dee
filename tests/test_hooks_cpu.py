"""Hooks and replaced sub-modules: a faster route around a module's call must not pass them by."""
import contextlib

import pytest
import torch


def _model(**kw):
    from megalodon_b200.config import ModelConf
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.utils import set_random_seed
    cfg = dict(num_layers=2, model_dim=64, num_heads=2, z_dim=32, value_dim=128, ffn_hidden_dim=128, cema_ndim=4,
               chunk_size=16, vocab_size=96, swiglu=True, norm_num_groups=8, efficient_attn="fused")
    cfg.update(kw)
    set_random_seed(0)
    return build_model(ModelConf(**cfg), "fp32", False, True)


def _block(model, i=0):
    layer = model._wrapped.layers[i]
    while hasattr(layer, "_wrapped"):
        layer = layer._wrapped
    return layer


def _modules(model):
    a, out = _block(model).mega, model._wrapped.output
    return {"wz": a.wz, "wr": a.wr, "wv": a.wv, "final_norm": out.final_norm, "output": out, "output.output": out.output}


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("kind", ["forward", "pre", "global"])
def test_hooks_fire(grad, kind):
    model = _model()
    toks = torch.randint(0, 96, (2, 16))
    with torch.no_grad():
        want, _ = model(toks)
    seen, handles = set(), []
    names = {id(m): n for n, m in _modules(model).items()}
    if kind == "global":
        handles.append(torch.nn.modules.module.register_module_forward_hook(
            lambda m, a, o: seen.add(names.get(id(m)))))
    for n, m in _modules(model).items():
        if kind == "forward":
            handles.append(m.register_forward_hook(lambda m, a, o, n=n: (seen.add(n), None)[1]))
        elif kind == "pre":
            handles.append(m.register_forward_pre_hook(lambda m, a, n=n: (seen.add(n), None)[1]))
    try:
        with contextlib.nullcontext() if grad else torch.no_grad():
            got, _ = model(toks)
    finally:
        for h in handles:
            h.remove()
    assert set(_modules(model)) <= seen
    torch.testing.assert_close(got.detach(), want, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("name", ["wz", "wr"])
def test_a_replaced_projection_is_called(name):
    from megalodon_b200.parallel.model_parallel import ColumnParallelLinear

    class Adapter(ColumnParallelLinear):
        def forward(self, x):
            return super().forward(x).roll(1, -1)

    model = _model()
    toks = torch.randint(0, 96, (2, 16))
    layer = getattr(_block(model).mega, name)
    outs = []
    for cls in (ColumnParallelLinear, Adapter):
        layer.__class__ = cls
        with torch.no_grad():
            outs.append(model(toks)[0])
    layer.__class__ = ColumnParallelLinear
    h = layer.register_forward_hook(lambda m, a, o: o.roll(1, -1))
    with torch.no_grad():
        outs.append(model(toks)[0])
    h.remove()
    assert (outs[1] - outs[0]).abs().max() > 1e-4
    torch.testing.assert_close(outs[1], outs[2], rtol=1e-6, atol=1e-6)


def test_a_replaced_output_projection_is_called():
    model = _model()
    toks = torch.randint(0, 96, (2, 16))
    out = model._wrapped.output
    with torch.no_grad():
        want, _ = model(toks)
        h = out.output.register_forward_hook(lambda m, a, o: o + 1.0)
        got, _ = model(toks)
        h.remove()
        h = out.register_forward_hook(lambda m, a, o: (o[0] + 2.0, o[1]))
        more, _ = model(toks)
        h.remove()
    torch.testing.assert_close(got, want + 1.0)
    torch.testing.assert_close(more, want + 2.0)


def _attentions(model):
    return [_block(model, i).mega for i in range(2)]


def test_marker_for_the_causal_mask_stays_among_its_own(monkeypatch):
    """`CAUSAL` is handed only to layers that know it: a replaced or observed attention gets the mask itself, and dropout
    in any layer asks for it too."""
    from megalodon_b200 import ops
    from megalodon_b200.modules.moving_average_gated_attention import CAUSAL, _InnerAttention
    model = _model(efficient_attn=None, attention_dropout=0.1)
    model.eval()
    toks = torch.randint(0, 96, (2, 12))
    with torch.no_grad():
        want, _ = model(toks)
    monkeypatch.setattr(ops, "attention_native", lambda *a: True)
    masks = []

    class Recorder(_InnerAttention):
        def forward(self, xq, xk, xv, mask, *rest):
            masks.append(mask)
            return super().forward(xq, xk, xv, mask, *rest)

    class Foreign(torch.nn.Module):                          # knows nothing of the marker
        def __init__(self, inner):
            super().__init__()
            self.call = [inner]

        def forward(self, *args):
            masks.append(args[3])
            return self.call[0](*args)

    def run():
        masks.clear()
        with torch.no_grad():
            got, _ = model(toks)
        torch.testing.assert_close(got, want, rtol=1e-4, atol=1e-4)
    x = torch.zeros(1, 1, 64)
    assert model._wrapped._causal_mask(x, 12, 0) is CAUSAL
    run()
    last = _attentions(model)[1]
    last.inner_attention.__class__ = Recorder
    run()
    assert torch.is_tensor(masks[0])
    last.inner_attention.__class__ = _InnerAttention
    plain = last.inner_attention
    last.inner_attention = Foreign(plain)
    run()
    assert torch.is_tensor(masks[0])
    last.inner_attention = plain
    h = plain.register_forward_pre_hook(lambda m, a: masks.append(a[3]))
    run()
    h.remove()
    assert torch.is_tensor(masks[0])
    plain.train()                                            # dropout acts in this layer alone
    assert torch.is_tensor(model._wrapped._causal_mask(x, 12, 0))


def test_mask_of_layers_that_are_not_the_models_own(monkeypatch):
    from megalodon_b200 import ops
    model = _model(efficient_attn=None)._wrapped
    monkeypatch.setattr(ops, "attention_native", lambda *a: True)
    x = torch.zeros(1, 1, 64)
    model.layers = torch.nn.ModuleList([model.layers[0], torch.nn.Identity()])
    assert torch.is_tensor(model._causal_mask(x, 12, 0))
    model.layers = torch.nn.ModuleList()
    assert torch.is_tensor(model._causal_mask(x, 12, 3))
