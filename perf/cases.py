"""The work whose speed counts: training steps, perplexity scoring, prefill, short prompts and decoding.

Every case goes through the public entry points a user's program calls (`build_model`, `model(...)`,
`grad_all_reduce`, `clip_grad_norm_`, `build_optimizer`, `inference`, `init_cache`, `DecodeSession`) with a
model of `ModelStore` (or the small two-layer shape of the smoke test) cut to a few layers: a layer costs
the same at any depth, and one optimiser step, one vocabulary projection and one call's fixed cost stay in.
Weights are drawn from the seed with the scales of the model's own initialisation (plus non-zero norm
scales, biases and attention gains, as in a trained model), rounded to 16 bits so that a 64-bit statement
of the model sees the same numbers, and loaded as a checkpoint is.

`exact` is that statement: the whole model in 64-bit torch, the EMA as a long convolution.
"""
from __future__ import annotations

import dataclasses
import math
import weakref

import torch
import torch.nn.functional as F

from megalodon_b200.config import ModelConf, OptimConf
from megalodon_b200.decoding import DecodeSession
from megalodon_b200.inference import inference
from megalodon_b200.models.mega import ModelStore, build_model
from megalodon_b200.optim import build_optimizer
from megalodon_b200.utils import clip_grad_norm_, init_cache

_SMALL = ModelConf(num_layers=2, model_dim=512, num_heads=2, z_dim=256, value_dim=1024, ffn_hidden_dim=1024,
                   chunk_size=256, vocab_size=1024, swiglu=True, norm_num_groups=32)
_VOCAB = 32000
_EPS = 1e-5


def _case(name, kind, model, layers, batch, length, *, fused, ckpt=0, steps=0, dtype="bf16"):
    return {"name": name, "kind": kind, "model": model, "layers": layers, "batch": batch, "length": length,
            "fused": fused, "ckpt": ckpt, "steps": steps, "dtype": dtype}


def listed():
    return [
        # a debugging-size model: an optimiser step is launches and host work
        _case("train_small", "train", "small", 2, 2, 512, fused=True),
        # mega200M as it ships (unfused attention, SiLU feed-forward), documents shorter than a chunk
        _case("train_200m_ragged", "train", "mega200M", 4, 4, 1000, fused=False),
        # the 1.3B of the PG19 runs: SwiGLU, shared embedding, two chunks a sequence
        _case("train_1b", "train", "mega1.3B_pg19", 3, 2, 4096, fused=True),
        # the headline shape: 4096-wide, 4096-token chunks fed one by one, part of the layers checkpointed
        _case("train_7b", "train", "mega7B_32k", 2, 1, 8192, fused=True, ckpt=1),
        # perplexity of one long odd-sized text, streamed chunk by chunk through the cache
        _case("score_1b_ragged", "score", "mega1.3B", 6, 1, 5003, fused=True),
        # perplexity of a batch of short odd-sized texts on the model as it ships
        _case("score_200m_batch", "score", "mega200M", 12, 8, 777, fused=False),
        # long-context prefill of the 7B shape
        _case("prefill_7b", "prefill", "mega7B_32k", 3, 1, 16384, fused=True),
        # time to the first token of a short chat turn: the smallest forward call
        _case("prompt_200m", "prompt", "mega200M", 12, 1, 37, fused=False),
        # token-by-token decoding, one user, small model: launches
        _case("decode_200m", "decode", "mega200M", 12, 1, 300, fused=True, steps=16),
        # one user, 7B width: streams the weights
        _case("decode_7b", "decode", "mega7B_32k", 4, 1, 1111, fused=True, steps=16),
        # sixteen users at once on the 1.3B
        _case("decode_1b_batch", "decode", "mega1.3B_pg19", 6, 16, 700, fused=True, steps=16),
    ]


_MODELS = {"small": 2, "mega200M": 12, "mega1.3B": 8, "mega1.3B_pg19": 8, "mega7.1B": 4, "mega7.3B": 4,
           "mega7B_32k": 4}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _memory(case):
    """About how much of the card one state and its pass take: three states at once have to fit."""
    cfg = _conf(case)
    B, L, c, train = case["batch"], case["length"], cfg.chunk_size, case["kind"] == "train"
    params = cfg.num_layers * _numel(_block_shapes(cfg)) + _numel(_root_shapes(cfg))
    tokens, live = B * L, cfg.num_layers - case["ckpt"] + 1 if train else 1
    scores = B * cfg.num_heads * L * min(L, c) * (2 if case["fused"] else 16)
    acts = tokens * 2 * (12 * cfg.model_dim + 5 * cfg.value_dim + 4 * cfg.ffn_hidden_dim)
    logits = tokens * cfg.vocab_size * (8 if train else 6 if case["kind"] != "prefill" else 0)
    kv = 4 * cfg.num_layers * B * c * (cfg.z_dim + cfg.value_dim) if case["kind"] == "decode" else 0
    return params * (20 if train else 6) + live * (scores + acts) + logits + kv


def draw(rng):
    """A training step, a scoring call, a prefill, a prompt or a decoding run of any model of the store, from
    a few tokens to several chunks, no dearer than the largest listed case of its kind."""
    dearest = {}
    for c in listed():
        dearest[c["kind"]] = max(dearest.get(c["kind"], 0.0), work(c)["flops"])
    while True:
        kind = rng.choice(["train", "train", "score", "prefill", "prompt", "decode", "decode"])
        model = rng.choice(sorted(_MODELS))
        chunk = _conf({"model": model, "layers": 1, "fused": True, "ckpt": 0}).chunk_size
        layers = rng.randint(1, min(4, _MODELS[model]) if kind == "train" else _MODELS[model])
        batch, steps, ckpt = _log_int(rng, 1, 8), 0, 0
        if kind == "train":
            length = chunk * rng.randint(1, 4) if rng.random() < 0.5 else _log_int(rng, 33, chunk - 1)
            ckpt = rng.randint(0, layers)
        elif kind == "score":
            length = _log_int(rng, 65, 4 * chunk)
        elif kind == "prefill":
            length = chunk * rng.randint(1, 8)
        elif kind == "prompt":
            length = _log_int(rng, 5, chunk - 1)
        else:
            batch, length, steps = _log_int(rng, 1, 32), _log_int(rng, 9, chunk - 40), rng.randint(4, 24)
        c = _case("", kind, model, layers, batch, length, fused=rng.random() < 0.7, ckpt=ckpt, steps=steps,
                  dtype="fp16" if kind != "train" and rng.random() < 0.15 else "bf16")
        if kind == "decode":
            c["fused"] = True
        del c["name"]
        if _memory(c) < 14e9 and work(c)["flops"] <= (dearest["prefill"] / 8 if kind == "prompt" else dearest[kind]):
            return c


# ------------------------------------------------------------------------------------------ model and weights
def _conf(case) -> ModelConf:
    base = _SMALL if case["model"] == "small" else ModelStore[case["model"]]
    return dataclasses.replace(base, num_layers=case["layers"], efficient_attn="fused" if case["fused"] else None,
                               vocab_size=_VOCAB if base.vocab_size == -1 else base.vocab_size,
                               layerwise_ckpt=case["ckpt"] > 0, ckpt_layers=case["ckpt"])


def _block_shapes(cfg):
    """Parameters of one block in the order of the model's modules (the order of a unit's flat buffer)."""
    D, Z, V, N, H = cfg.model_dim, cfg.z_dim, cfg.value_dim, cfg.cema_ndim, cfg.ffn_hidden_dim
    out = [("mega.gamma", (2, Z)), ("mega.beta", (2, Z)),
           ("mega.timenorm.weight", (D,)), ("mega.timenorm.bias", (D,)),
           ("mega.cema.alpha", (D, N, 1)), ("mega.cema.delta", (D, N, 1)), ("mega.cema.theta", (D, 1, 1)),
           ("mega.cema.gamma", (D, N, 2)), ("mega.cema.omega", (D, 1)),
           ("mega.rmsnorm.weight", (D,)),
           ("mega.wv.weight", (V, D)), ("mega.wv.bias", (V,)), ("mega.wz.weight", (Z, D)), ("mega.wz.bias", (Z,)),
           ("mega.wr.weight", (V, D)), ("mega.wr.bias", (V,)), ("mega.wh1.weight", (D, D)), ("mega.wh1.bias", (D,)),
           ("mega.wh2.weight", (D, V)),
           ("nffn.norm.weight", (D,)), ("nffn.norm.bias", (D,)), ("nffn.fc1.weight", (H, D)),
           ("nffn.fc2.weight", (D, H))]
    return out + [("nffn.fc3.weight", (H, D))] if cfg.swiglu else out


def _root_shapes(cfg):
    out = [("embed.weight", (cfg.vocab_size, cfg.model_dim)), ("output.final_norm.weight", (cfg.model_dim,)),
           ("output.final_norm.bias", (cfg.model_dim,))]
    return out if cfg.share_emb else out + [("output.output.weight", (cfg.vocab_size, cfg.model_dim))]


def _units(cfg):
    """[[(name, shape), ...] per unit of the sharded model], the root first."""
    return [_root_shapes(cfg)] + [[(f"layers.{i}.{n}", s) for n, s in _block_shapes(cfg)]
                                  for i in range(cfg.num_layers)]


def _weights(cfg, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    low = torch.float16 if dtype == "fp16" else torch.bfloat16
    D = cfg.model_dim
    out = {}
    for unit in _units(cfg):
        for name, shape in unit:
            w = torch.randn(shape, generator=gen, device="cuda")
            last = name.rsplit(".", 1)[-1]
            if name.endswith("cema.theta"):
                at = torch.randperm(D, generator=gen, device="cuda") + 1
                f = torch.exp(at.double() * (-math.log(D) / D)).float()
                w = torch.log(f / (1.0 - f)).view(shape)
            elif name.endswith(("cema.alpha", "cema.delta")):
                w.mul_(0.2)
            elif name.endswith("cema.omega"):
                w.mul_(0.25)
            elif name.endswith("cema.gamma"):
                pass
            elif name in ("embed.weight", "output.output.weight"):
                w.mul_(D ** -0.5)
            elif len(shape) == 2 and last == "weight":
                w.mul_((3.0 * shape[1]) ** -0.5)
            elif name.endswith("mega.gamma"):
                w.mul_(0.3)
            elif name.endswith("mega.beta"):
                w.mul_(0.05)
            else:
                w.mul_(0.1)
            out[name] = w.to(low).float()
    if cfg.share_emb:
        out["output.output.weight"] = out["embed.weight"]
    return out


def _tokens(case, cfg, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    n = case["length"] + 1 + case["steps"]
    return torch.randint(0, cfg.vocab_size, (case["batch"], n), generator=gen, device="cuda")


# ------------------------------------------------------------------------------------------------ the passes
class _Owner:
    """Lives as long as a training state.  The parameter views of the last step hold the model through their
    autograd node, which the garbage collector cannot see into: when the state goes they are replaced."""

    def __init__(self, model):
        weakref.finalize(self, model.materialize_views).atexit = False


def prepare(case, seed):
    cfg, kind = _conf(case), case["kind"]
    model = build_model(cfg, case["dtype"])
    model.load_state_dict(_weights(cfg, case["dtype"], seed))
    tok = _tokens(case, cfg, seed)
    L = case["length"]
    state = {"kind": kind, "model": model, "dtype": case["dtype"]}
    low = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
    if kind == "train":
        state["x"], state["y"] = tok[:, :-1].contiguous(), tok[:, 1:].contiguous()
        if L > cfg.chunk_size:
            model._wrapped.seq_microbatch_chunks = 1
        state["owner"] = _Owner(model)
        state["opt"], state["sched"] = build_optimizer(model, OptimConf(), 10000, case["dtype"])
        return state
    model.eval()
    state["x"] = tok[:, :L].contiguous()
    state["low"] = low
    if kind == "score":
        state["y"] = tok[:, 1:L + 1].contiguous()
    elif kind == "decode":
        with torch.inference_mode():
            cache = init_cache(case["batch"], model, low)
            _, state["cache"] = model(state["x"], cache=cache)
            state["next"] = tok[:, L:L + case["steps"]].t().contiguous()
            session = DecodeSession(model, case["batch"], low)
            for _ in range(3):                     # a serving program's session is past its first requests
                session.load_cache(state["cache"])
                session.step(state["next"][0])
        state["session"] = session
    return state


def run(state):
    kind, model = state["kind"], state["model"]
    if kind == "train":
        opt = state["opt"]
        opt.zero_grad()
        losses, _ = model(state["x"], targets=state["y"])
        losses.mean().backward()
        model.grad_all_reduce()
        norm = clip_grad_norm_(model, 1.0)
        grads = [p._grad_shard for p in model.params_with_grad]
        opt.step()
        state["sched"].step()
        return {"losses": losses, "norm": norm, "grads": grads, "weights": [p.data for p in model.parameters()]}
    if kind == "score":
        return inference(model, state["x"], state["y"], state["dtype"])
    with torch.inference_mode():
        if kind == "prefill":
            logits, (layers, _) = model(state["x"], prefill=True)
            return {"logits": logits, "ema": [layer[2] for layer in layers]}
        if kind == "prompt":
            cache = init_cache(state["x"].shape[0], model, state["low"])
            logits, (layers, _) = model(state["x"], cache=cache)
            return {"logits": logits, "k": [layer[0][0] for layer in layers], "v": [layer[0][1] for layer in layers],
                    "ema": [layer[2] for layer in layers]}
        session, out = state["session"], []
        session.load_cache(state["cache"])
        for tok in state["next"]:                  # the given token wins, as inside a prompt
            out.append(session.step(tok).clone())
        return torch.stack(out)


# ---------------------------------------------------------------------------------------------- what it costs
def _numel(shapes):
    return sum(math.prod(s) for _, s in shapes)


def work(case):
    cfg = _conf(case)
    D, Z, V, N, c = cfg.model_dim, cfg.z_dim, cfg.value_dim, cfg.cema_ndim, cfg.chunk_size
    block = _numel(_block_shapes(cfg)) * cfg.num_layers
    vocab = cfg.vocab_size * D
    params = block + _numel(_root_shapes(cfg))
    B, L, T = case["batch"], case["length"], case["steps"]

    def attention(n):                              # causal products of n tokens in chunks
        full, rest = divmod(n, c)
        return 2.0 * (Z + V) * (full * c * (c + 1) / 2 + rest * (rest + 1) / 2)

    ema = 8.0 * N * D                              # complex state update and read-out a token
    if case["kind"] == "decode":
        first, kv = L % c, 2 * (Z + V) * cfg.num_layers
        keys = sum((first + t) % c + 1 for t in range(T))
        flops = T * B * (2.0 * (block + vocab) + ema * cfg.num_layers) + 2.0 * B * keys * (Z + V) * cfg.num_layers
        state = B * cfg.num_layers * D * N * 8
        return {"bytes": T * (2.0 * (block + vocab) + 2.0 * state + 4.0 * B * cfg.vocab_size) + 1.0 * B * keys * kv,
                "flops": flops}
    tokens = B * L
    out_tokens = B if case["kind"] == "prefill" else tokens
    flops = 2.0 * tokens * block + 2.0 * out_tokens * vocab + cfg.num_layers * (B * attention(L) + tokens * ema)
    if case["kind"] == "train":
        # three passes of products; masters and moments read and written, 16-bit weights written and read
        return {"bytes": params * (24.0 + 2.0 + 2.0 + 2.0), "flops": 3.0 * flops}
    logits = 0.0 if case["kind"] == "score" else 4.0 * out_tokens * cfg.vocab_size
    return {"bytes": 2.0 * (block + vocab) + logits, "flops": flops}


def tolerance(case):
    # 16-bit activations through a few layers.  Seen against the 64-bit statement: losses 0.0007, logits
    # 0.012 after decoding, gradients 0.011; single gradients 0.2 of their root mean square between two runs
    # of the same inputs (sums of scores are added in any order).  About four times that, as far as allowed.
    if case["kind"] == "score":
        return {"rel": 0.003, "max": 0.05}
    return {"rel": 0.03, "max": 0.99 if case["kind"] == "train" else 0.5}


# ------------------------------------------------------------------------------------- the model in 64 bits
def _timestep_norm(x, groups, weight, bias):
    B, L, D = x.shape
    xg = x.view(B, L, groups, D // groups)
    n = torch.arange(1, L + 1, device=x.device, dtype=x.dtype).view(1, L, 1)
    mean = xg.mean(-1).cumsum(1) / n
    var = (xg * xg).mean(-1).cumsum(1) / n - mean * mean
    y = (xg - mean.unsqueeze(-1)) * torch.rsqrt(var.clamp_min(0.0) + _EPS).unsqueeze(-1)
    return y.reshape(B, L, D) * (weight + 1.0) + bias


def _rms_norm(x, weight=None):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + _EPS)
    return y if weight is None else y * (weight + 1.0)


def _ema(x, W, pre, N, want_state):
    """y and the last state of the complex EMA, through its kernel k_l = Re sum_n gamma_n p_n q_n^l."""
    B, L, D = x.shape
    alpha, delta = torch.sigmoid(W[pre + "alpha"]).view(D, N), torch.sigmoid(W[pre + "delta"]).view(D, N)
    theta = torch.sigmoid(W[pre + "theta"]).view(D, 1) * (2.0 * math.pi / N)
    logq = torch.complex(torch.log1p(-alpha * delta), theta * torch.arange(1, N + 1, device=x.device))
    gamma = torch.view_as_complex(W[pre + "gamma"].contiguous()) * math.sqrt(1.0 / N)
    blk = 64
    A = -(-L // blk)
    steps = torch.arange(blk, device=x.device, dtype=x.dtype)
    inner = torch.exp(steps.view(blk, 1, 1) * logq)                                   # [blk, D, N]
    outer = torch.exp((blk * torch.arange(A, device=x.device, dtype=x.dtype)).view(A, 1, 1) * logq)
    k = torch.einsum("adn,bdn->dab", outer * (gamma * alpha), inner).real.reshape(D, A * blk)[:, :L]
    n = 2 * L
    y = torch.stack([torch.fft.irfft(torch.fft.rfft(xb.t(), n=n) * torch.fft.rfft(k, n=n), n=n)[:, :L].t()
                     for xb in x])
    y = y + x * W[pre + "omega"].view(D)
    h = None
    if want_state:
        xp = F.pad(x, (0, 0, A * blk - L, 0)).view(B, A, blk, D).to(inner.dtype)
        part = torch.einsum("bajd,jdn->badn", xp, inner.flip(0))
        h = torch.zeros(B, D, N, dtype=inner.dtype, device=x.device)
        for a in range(A):
            h = h * torch.exp(blk * logq) + part[:, a]
        h = h * alpha
    return y, h


def _attend(q, k, v):
    """Causal attention of [B, L, H, d] within one chunk, a few heads at a time."""
    L = q.shape[1]
    hidden = torch.ones(L, L, dtype=torch.bool, device=q.device).triu(1)
    out = []
    for b in range(q.shape[0]):
        s = torch.einsum("lhd,mhd->hlm", q[b], k[b]).masked_fill(hidden, float("-inf"))
        out.append(torch.einsum("hlm,mhd->lhd", torch.softmax(s, -1), v[b]))
    return torch.stack(out)


def _block(x, W, pre, cfg, freqs, want_state):
    B, L, D = x.shape
    c, H = cfg.chunk_size, cfg.num_heads
    m = pre + "mega."
    t = _timestep_norm(x, cfg.norm_num_groups, W[m + "timenorm.weight"], W[m + "timenorm.bias"])
    e, h = _ema(t, W, m + "cema.", cfg.cema_ndim, want_state)
    mx = _rms_norm(e, W[m + "rmsnorm.weight"])
    z = _rms_norm(F.linear(mx, W[m + "wz.weight"], W[m + "wz.bias"]).view(B, L, H, -1)).reshape(B, L, -1)
    d = z.shape[-1] // H
    rot = torch.polar(torch.ones_like(freqs), freqs)[torch.arange(L, device=x.device) % c].view(1, L, 1, d // 2)
    qk = []
    for i in range(2):
        u = (z * (W[m + "gamma"][i] + 1.0) / math.sqrt(d) + W[m + "beta"][i]).view(B, L, H, d // 2, 2)
        qk.append(torch.view_as_real(torch.view_as_complex(u.contiguous()) * rot).reshape(B, L, H, d))
    v = F.silu(F.linear(t, W[m + "wv.weight"], W[m + "wv.bias"])).view(B, L, H, -1)
    r = F.silu(F.linear(mx, W[m + "wr.weight"], W[m + "wr.bias"]))
    a = torch.cat([_attend(qk[0][:, s:s + c], qk[1][:, s:s + c], v[:, s:s + c]) for s in range(0, L, c)], dim=1)
    y = (F.linear(mx, W[m + "wh1.weight"], W[m + "wh1.bias"]) + F.linear(a.reshape(B, L, -1) * r, W[m + "wh2.weight"])
         + x)
    f = F.layer_norm(y, (D,), W[pre + "nffn.norm.weight"] + 1.0, W[pre + "nffn.norm.bias"], _EPS)
    u = F.silu(F.linear(f, W[pre + "nffn.fc1.weight"]))
    if cfg.swiglu:
        u = u * F.linear(f, W[pre + "nffn.fc3.weight"])
    return F.linear(u, W[pre + "nffn.fc2.weight"]) + x, (qk[1], v, h)


def _hidden(tokens, W, cfg, low, want_state=False):
    x = F.embedding(tokens, W["embed.weight"])
    if cfg.scale_emb:
        x = x * math.sqrt(cfg.model_dim)
    d = cfg.z_dim // cfg.num_heads
    base = torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d
    # the table of rotary frequencies is a buffer of the model and has the model's 16-bit type
    f = (1.0 / torch.pow(torch.tensor(10000.0, dtype=torch.float64, device=x.device), base)).float().to(low).double()
    freqs = torch.outer(torch.arange(cfg.chunk_size, dtype=torch.float64, device=x.device), f)
    states = []
    for i in range(cfg.num_layers):
        x, st = _block(x, W, f"layers.{i}.", cfg, freqs, want_state)
        states.append(st)
    x = _timestep_norm(x, cfg.norm_num_groups, W["output.final_norm.weight"], W["output.final_norm.bias"])
    return x, states


def _nll(x, W, targets):
    """Losses of hidden states, a few thousand rows of logits at a time."""
    out = []
    for xs, ts in zip(x.flatten(0, 1).split(4096), targets.flatten().split(4096)):
        out.append(F.cross_entropy(F.linear(xs, W["output.output.weight"]), ts, reduction="none"))
    return torch.cat(out).view(targets.shape)


def _flat(tensors):
    """A unit's flat buffer: every parameter padded to a multiple of 64 values."""
    return torch.cat([F.pad(t.reshape(-1), (0, -t.numel() % 64)) for t in tensors])


def exact(case, seed):
    cfg, kind = _conf(case), case["kind"]
    W = {k: v.double() for k, v in _weights(cfg, case["dtype"], seed).items()}
    tok = _tokens(case, cfg, seed)
    low = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
    L = case["length"]
    if kind == "train":
        names = [[n for n, _ in unit] for unit in _units(cfg)]
        for unit in names:
            for n in unit:
                W[n].requires_grad_(True)
        if cfg.share_emb:
            W["output.output.weight"] = W["embed.weight"]
        losses = _nll(_hidden(tok[:, :-1], W, cfg, low)[0], W, tok[:, 1:]).flatten()
        losses.mean().backward()
        grads = [_flat([W[n].grad for n in unit]) for unit in names]
        norm = torch.stack([g.square().sum() for g in grads]).sum().sqrt()
        grads = [g * torch.clamp(1.0 / (norm + 1e-6), max=1.0) for g in grads]
        o = OptimConf()
        lr = o.lr * o.lr_init_ratio
        weights = []
        for unit, g in zip(names, grads):
            w = _flat([W[n].detach() for n in unit])
            weights.append(w * (1.0 - lr * o.weight_decay) - lr * g / (g.abs() + o.epsilon))
        return {"losses": losses.detach(), "norm": norm, "grads": grads, "weights": weights}
    with torch.no_grad():
        if kind == "score":
            return _nll(_hidden(tok[:, :L], W, cfg, low)[0], W, tok[:, 1:L + 1])
        if kind == "decode":
            x, _ = _hidden(tok[:, :L + case["steps"]], W, cfg, low)
            return F.linear(x[:, L:], W["output.output.weight"]).transpose(0, 1).contiguous()
        x, states = _hidden(tok[:, :L], W, cfg, low, want_state=True)
        ema = [h for _, _, h in states]
        if kind == "prefill":
            return {"logits": F.linear(x[:, -1], W["output.output.weight"]), "ema": ema}
        return {"logits": F.linear(x, W["output.output.weight"]), "k": [k for k, _, _ in states],
                "v": [v for _, v, _ in states], "ema": ema}
