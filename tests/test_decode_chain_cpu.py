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


def _block(sess, i=1):
    layer = sess.mega.layers[i]
    while hasattr(layer, "_wrapped"):
        layer = layer._wrapped
    return layer


def _spots(sess):
    b, out = _block(sess), sess.mega.output
    return {"embed": sess.mega.embed, "wrapper": sess.mega.layers[1], "block": b, "mega": b.mega, "wz": b.mega.wz,
            "wr": b.mega.wr, "wv": b.mega.wv, "rmsnorm": b.mega.rmsnorm, "nffn": b.nffn, "fc1": b.nffn.fc1,
            "fc3": b.nffn.fc3, "norm": b.nffn.norm, "output": out, "output.output": out.output}


def test_hooks_and_adapters_take_the_step_through_the_modules(monkeypatch):
    """Also when they come after the session was made; without them the chain runs again."""
    sess, rec = _session(monkeypatch)
    reached = []
    monkeypatch.setattr(sess, "_native_step", lambda: (reached.append("chain"), torch.zeros(2, 96))[1])
    tok = torch.tensor([1, 2])
    for name, mod in _spots(sess).items():
        h = mod.register_forward_hook(lambda m, a, o, name=name: (reached.append(name), None)[1])
        assert not sess._as_built(), name
        h.remove()
        cls = type(mod)
        mod.__class__ = type("Adapter", (cls,), {})
        assert not sess._as_built() or name == "wrapper", name
        mod.__class__ = cls
    b = _block(sess)
    b.nffn.fc1.bias = torch.nn.Parameter(torch.zeros(128))       # a bias that the chain has no place for
    assert not sess._as_built()
    b.nffn.fc1.bias = None
    sess.step(tok)
    assert reached == ["chain"]


def test_updated_weights_are_gathered_before_the_chain(monkeypatch):
    """An optimiser step or a load since the last token: the compute-dtype weights are brought up to date first."""
    sess, rec = _session(monkeypatch)
    events = []
    inner = sess.model.materialize_views
    monkeypatch.setattr(sess.model, "materialize_views", lambda: (events.append("gather"), inner())[1])
    monkeypatch.setattr(sess, "_native_step", lambda: (events.append("chain"), torch.zeros(2, 96))[1])
    tok = torch.tensor([1, 2])
    sess.step(tok)
    unit = sess.model._units()[1]
    with torch.no_grad():
        unit.flat_param.mul_(1.5)
    sess.step(tok)
    assert events == ["chain", "gather", "chain"] and all(u._full_is_valid() for u in sess.model._units())


def test_step_through_the_modules_takes_fp32_statistics(monkeypatch):
    """A native session's running statistics are fp32 whatever its dtype; the modules want them in the dtype."""
    sess, _ = _session(monkeypatch)
    sess.dtype = torch.bfloat16
    count, mean, var = sess._stats(sess.layers[0]["norm"])
    assert mean.dtype == var.dtype == torch.bfloat16 and count.dtype == torch.int64


def test_logits_of_a_step_outlive_the_next(monkeypatch):
    """Eager steps hand out memory of their own, the one after a capture that did not work among them."""
    import contextlib
    sess, _ = _session(monkeypatch)
    sess.use_graph = True
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: None)

    @contextlib.contextmanager
    def no_capture(*a, **k):
        raise RuntimeError("not capturable")
        yield
    monkeypatch.setattr(torch.cuda, "graph", no_capture)
    outs = [sess.step(torch.tensor([1, 2])) for _ in range(5)]
    held = {o.data_ptr() for o in outs}
    assert not sess.use_graph and len(held) == 5 and sess._buf["logits"].data_ptr() not in held


def test_launches_are_counted(monkeypatch):
    from megalodon_b200.ops import cuda_ops
    sess, rec = _session(monkeypatch)
    before = cuda_ops.count_launches()
    sess.step(torch.tensor([1, 2]))
    # (attention is two launches: the splits and their combination)
    made = sum(2 if name == "decode_attend" else 1 for name, _ in rec.calls if name != "decode_attend_splits")
    assert made == 8 * sess.mega.num_layers + 2 and cuda_ops.count_launches() - before == made


def test_a_session_on_the_model_inside_its_root_unit(monkeypatch):
    """Its units cannot all be brought up to date from here: after an update the step goes through their own calls."""
    from megalodon_b200.decoding import DecodeSession
    sess, _ = _session(monkeypatch)
    inner = DecodeSession(sess.mega, 2, torch.float32, use_graph=False)
    reached = []
    inner._native = True
    monkeypatch.setattr(inner, "_native_step", lambda: (reached.append("chain"), torch.zeros(2, 96))[1])
    assert inner._weights_current()
    inner.step(torch.tensor([1, 2]))
    assert reached == ["chain"]
    with torch.no_grad():
        inner._units()[0].flat_param.mul_(1.5)
    assert not inner._weights_current()
