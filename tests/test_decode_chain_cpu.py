"""Host side of the native decode step, on the CPU: what is launched in which order, with the launches recorded
instead of made."""
import pytest
import torch


class _Recorder:
    """Stands for the extension: every call is noted, nothing runs."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return {"skinny_gemm": 0, "decode_attend_splits": 2}.get(name)
        return call


def _session(monkeypatch, **kw):
    from megalodon_b200.config import ModelConf
    from megalodon_b200.decoding import DecodeSession
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.ops import _ext
    from megalodon_b200.utils import set_random_seed
    cfg = dict(num_layers=3, model_dim=64, num_heads=2, z_dim=32, value_dim=128, ffn_hidden_dim=128, cema_ndim=4,
               chunk_size=16, vocab_size=96, swiglu=True, norm_num_groups=8, efficient_attn="fused")
    cfg.update(kw)
    set_random_seed(0)
    model = build_model(ModelConf(**cfg), "fp32", False, True)
    rec = _Recorder()
    sess = DecodeSession(model, 2, torch.float32, use_graph=False)
    assert not sess._native                             # (no GPU)
    monkeypatch.setattr(_ext, "require", lambda: rec)
    sess._native = True
    sess._native_buffers()
    rec.calls.clear()
    return sess, rec


@pytest.mark.parametrize("training", [False, True])
def test_ema_coefficients_precede_the_chain(monkeypatch, training):
    """The links read p, q and gamma ahead of their wait, which is right only if nothing between two links writes
    them: whatever computes them has to be launched before the first."""
    sess, rec = _session(monkeypatch)
    for layer in sess.mega.layers:
        while hasattr(layer, "_wrapped"):
            layer = layer._wrapped
        cema = layer.mega.cema
        inner = cema._calc_coeffs
        monkeypatch.setattr(cema, "_calc_coeffs",
                            lambda inner=inner: (rec.calls.append(("coeffs", ())), inner())[1])
    sess.model.train(training)
    for _ in range(2):
        rec.calls.clear()
        sess.step(torch.tensor([1, 2]))
        names = [n for n, _ in rec.calls]
        assert names.count("decode_norm_ema") == 4
        assert "coeffs" not in names[names.index("decode_norm_ema"):]
        # the first link waits for everything before it; only the later ones may run ahead
        links = [a[-1] for n, a in rec.calls if n == "decode_norm_ema"]
        assert links == [False, True, True, True]
