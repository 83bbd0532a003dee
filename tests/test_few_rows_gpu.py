"""Products with few rows and the kernels of the native decode step, against 64-bit / module references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm()).item()


# rows around the padding to 16 and the largest accepted; features around the 128-row tile; K with a ragged
# 64-block, fewer blocks than a split would need, and a long one
@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 8), (100, 72), (136, 4104), (2056, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_skinny_products(M, N, K, dtype):
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(M + N + K)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def rand(*s):
        return torch.randn(*s, device="cuda")
    x = rand(M, K).to(dtype)
    w, w2 = (rand(N, K) / K ** 0.5).to(dtype), (rand(N, K) / K ** 0.5).to(dtype)
    b, add = rand(N).to(dtype), rand(M, N + 8).to(dtype)[:, :N]
    lin, lin2 = x.double() @ w.double().t(), x.double() @ w2.double().t()
    outs = [torch.full((M, N), float("nan"), device="cuda") for _ in range(3)]
    # three jobs of one launch: bias + addend, SiLU, SwiGLU
    rc = cuda_ops._C().skinny_gemm([x, x, x], [w, w, w], [None, None, w2], [b, b, None], [add, None, None], [0, 1, 2],
                                   outs, False, err)
    assert rc == 0 and err.item() == 0
    silu = torch.nn.functional.silu
    # fp32 accumulation: the tensor core adds 16 products at a time and truncates, which a sum of K terms of
    # either sign shows as up to K / 16 steps of 2^-24 each, far below sqrt(K) * 2^-20 of the result's norm
    tol = max(4e-6, K ** 0.5 * 2.0 ** -20)
    for got, want in zip(outs, (lin + b.double() + add.double(), silu(lin + b.double()), silu(lin) * lin2)):
        assert _rel(got, want) < tol, (_rel(got, want), tol)
    low = torch.empty(M, N, dtype=dtype, device="cuda")
    assert cuda_ops._C().skinny_gemm([x], [w], [None], [None], [None], [0], [low], False, err) == 0
    assert _rel(low, lin) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)


def test_few_row_rule_agrees_with_the_tiles():
    """`gemm` sends 1 row, few rows and many rows to three kernels; strided rows and an addend included."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(3)
    w = (torch.randn(264, 520, device="cuda") / 520 ** 0.5).bfloat16()
    big = torch.randn(200, 3, 520, device="cuda").bfloat16()
    add = torch.randn(200, 264, device="cuda").bfloat16()
    for M in (1, 2, 63, 64, 65, 200):
        x = big[:M, 1]                                  # row stride 1560
        ref = x.double() @ w.double().t()
        y, _ = cuda_ops.gemm(x, w)
        assert _rel(y, ref) < 2.0 ** -8
        z = cuda_ops.linear_add(x, w, None, add[:M])
        assert _rel(z, ref + add[:M].double()) < 2.0 ** -7
    cuda_ops.check_kernel_errors()


@pytest.mark.parametrize("D,G,N,B", [(512, 32, 16, 1), (1024, 32, 16, 3), (96, 3, 4, 2), (4096, 64, 16, 2), (64, 1, 32, 1),
                                     (2048, 32, 16, 9), (8192, 8, 32, 1)])
def test_decode_norm_ema(D, G, N, B):
    from megalodon_b200.ops import cuda_ops, reference
    torch.manual_seed(D)
    dev = "cuda"
    x = torch.randn(B, D, device=dev).bfloat16()
    w, b, rw, omega = (torch.randn(D, device=dev).mul_(0.1).bfloat16() for _ in range(4))
    count = torch.tensor(([0, 5, 1000] * 3)[:B], device=dev)
    mean, var = torch.randn(B, G, device=dev) * 0.1, torch.rand(B, G, device=dev) + 0.5
    p = torch.rand(D, N, device=dev)
    q = torch.polar(torch.rand(D, N, device=dev), torch.randn(D, N, device=dev))
    ga = torch.view_as_complex(torch.randn(D, N, 2, device=dev))
    hx = torch.view_as_complex(torch.randn(B, D, N, 2, device=dev))
    ty, c1, m1, v1 = reference.timestep_norm(x.double()[:, None], count, mean.double(), var.double(), w.double(),
                                             b.double(), None, G, 1e-5, 1.0)
    t_ref = ty[:, 0].to(torch.bfloat16)
    h_ref = q.to(torch.complex128) * hx.to(torch.complex128) + p.double() * t_ref.double()[:, :, None]
    y_ref = ((ga.to(torch.complex128) * h_ref).sum(-1).real + omega.double() * t_ref.double())
    mx_ref = y_ref * torch.rsqrt(y_ref.pow(2).mean(-1, keepdim=True) + 1e-5) * (rw.double() + 1.0)
    t, mx = torch.empty_like(x), torch.empty_like(x)
    cuda_ops._C().decode_norm_ema(x, w, b, count, mean, var, t, p, torch.view_as_real(q), torch.view_as_real(ga), omega,
                                  torch.view_as_real(hx), rw, mx, None, 0, 1e-5, 1e-5, False)
    assert torch.equal(count, c1) and _rel(mean, m1) < 1e-6 and _rel(var, v1) < 1e-6
    # one rounding to 8 bits each way (t), and of y and mx
    assert _rel(t, ty[:, 0]) < 2.0 ** -8 and _rel(torch.view_as_real(hx), torch.view_as_real(h_ref)) < 2.0 ** -8
    assert _rel(mx, mx_ref) < 2.0 ** -7
    pos = torch.tensor([6], device=dev)
    cuda_ops._C().decode_norm_ema(x, w, b, count, mean, var, t, None, None, None, None, None, None, None, pos, 7, 1e-5,
                                  0.0, False)
    assert pos.item() == 0 and torch.equal(count, c1 + 1)


@pytest.mark.parametrize("B,H,C,dk,dv,pos", [(1, 1, 40, 8, 8, 0), (2, 3, 100, 72, 200, 99), (1, 4, 4096, 256, 2048, 700),
                                             (33, 2, 64, 16, 4096, 31)])
def test_decode_attend(B, H, C, dk, dv, pos):
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(pos)
    dev = "cuda"

    def rand(*s):
        return torch.randn(*s, device=dev)
    z, v, gate = rand(B, H * dk).bfloat16(), rand(B, H * dv).bfloat16(), rand(B, H * dv).bfloat16()
    gamma, beta = (rand(2, H * dk) * 0.3).bfloat16(), (rand(2, H * dk) * 0.3).bfloat16()
    kb, vb = rand(B, H, C, dk).bfloat16(), rand(B, H, C, dv).bfloat16()
    kb[:, :, pos:] = float("nan")                      # neither the stale slots nor slot `pos` may be read
    vb[:, :, pos:] = float("nan")
    ang = torch.outer(torch.arange(C, device=dev).float(), torch.rand(dk // 2, device=dev))
    freqs = torch.polar(torch.ones_like(ang), ang)
    zn = z.double().view(B, H, dk)
    zn = zn * torch.rsqrt(zn.pow(2).mean(-1, keepdim=True) + 1e-5)
    qk = []
    for i in range(2):
        u = zn * (gamma[i].double().view(H, dk) + 1.0) / dk ** 0.5 + beta[i].double().view(H, dk)
        u = torch.view_as_complex(u.view(B, H, dk // 2, 2).contiguous()) * freqs[pos].to(torch.complex128)
        qk.append(torch.view_as_real(u).reshape(B, H, dk))
    keys = torch.cat([kb[:, :, :pos].double(), qk[1].bfloat16().double()[:, :, None]], 2)
    vals = torch.cat([vb[:, :, :pos].double(), v.double().view(B, H, 1, dv)], 2)
    pr = torch.softmax(torch.einsum("bhd,bhcd->bhc", qk[0], keys), -1)
    ref = torch.einsum("bhc,bhcd->bhd", pr, vals).reshape(B, -1) * gate.double()
    out = torch.empty(B, H * dv, device=dev, dtype=torch.bfloat16)
    splits = cuda_ops._C().decode_attend_splits(B * H, C)
    part = torch.empty(B * H * splits * (dv + 2), device=dev)
    cuda_ops._C().decode_attend(z, gamma, beta, torch.view_as_real(freqs), v, kb, vb, torch.tensor([pos], device=dev),
                                gate, out, part, 1e-5, False)
    # fp32 scores; one rounding of the result (and a key that may round the other way)
    assert _rel(out, ref) < 2.0 ** -7
    assert _rel(kb[:, :, pos], qk[1]) < 2.0 ** -8 and torch.equal(vb[:, :, pos].reshape(B, -1), v)


@pytest.mark.parametrize("B,H,C,dk,dv,dtype", [(1, 1, 96, 256, 2048, torch.bfloat16), (2, 1, 96, 64, 512, torch.float16),
                                               (1, 1, 300, 72, 264, torch.bfloat16), (20, 1, 96, 256, 136, torch.bfloat16),
                                               (50, 2, 40, 32, 4096, torch.float16), (300, 1, 12, 8, 24, torch.bfloat16)])
def test_decode_attention_in_one_launch(B, H, C, dk, dv, dtype):
    """Clusters over the keys: fewer keys than splits, the edges of a ring stage and of a box, several column blocks,
    widths that do and do not suit the tensor cores, more heads than fill the GPU."""
    from megalodon_b200 import ops
    torch.manual_seed(dv)
    q = torch.randn(B, H, dk, device="cuda").to(dtype)
    k, v = torch.randn(B, H, C, dk, device="cuda").to(dtype), torch.randn(B, H, C, dv, device="cuda").to(dtype)
    for pos in sorted({0, 1, 14, 15, 16, 31, 32, 33, C // 2, C - 1} & set(range(C))):
        kn, vn = k.clone(), v.clone()
        kn[:, :, pos + 1:] = float("nan")
        vn[:, :, pos + 1:] = float("nan")
        out = ops.decode_attention(q, kn, vn, torch.tensor([pos], device="cuda"), 0.4)
        s = torch.einsum("bhd,bhcd->bhc", q.double(), k[:, :, :pos + 1].double()) * 0.4
        ref = torch.einsum("bhc,bhcd->bhd", torch.softmax(s, -1), v[:, :, :pos + 1].double())
        # fp32 throughout, one rounding
        assert _rel(out, ref) < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11), pos


@pytest.mark.parametrize("B,dk", [(1, 256), (2, 64), (28, 32), (64, 128), (1, 72), (12, 64)])
def test_decode_attention_with_infinite_keys(B, dk):
    """A key with an infinity against the query has no weight (its score is minus infinity) and spoils nothing."""
    from megalodon_b200 import ops
    torch.manual_seed(dk)
    q = torch.rand(B, 1, dk, device="cuda").bfloat16() + 0.5
    k, v = torch.randn(B, 1, 40, dk, device="cuda").bfloat16(), torch.randn(B, 1, 40, 256, device="cuda").bfloat16()
    k[:, :, 3, 1] = float("-inf")
    k[:, :, 17, dk - 1] = float("-inf")
    s = torch.einsum("bhd,bhcd->bhc", q.double(), k.double()) * 0.1
    ref = torch.einsum("bhc,bhcd->bhd", torch.softmax(s, -1), v.double())
    out = ops.decode_attention(q, k, v, torch.tensor([39], device="cuda"), 0.1)
    assert _rel(out, ref) < 2.0 ** -8                # fp32 throughout, one rounding


@pytest.mark.parametrize("B,H", [(1, 1), (1, 2), (32, 1), (64, 2), (200, 1)])
def test_decode_attend_with_a_small_query_in_fp16(B, H):
    """Query entries of 4e-6 (the query is held in fp32) against keys of 2e4: scores of about one, which 16-bit parts of
    the query would get wrong by a hundredth."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(B)
    dk, dv, C, pos, dev, dt = 64, 256, 96, 80, "cuda", torch.float16

    def rand(*s):
        return torch.randn(*s, device=dev)
    z, v, gate = rand(B, H * dk).to(dt), rand(B, H * dv).to(dt), rand(B, H * dv).to(dt)
    gamma, beta = torch.full((2, H * dk), -1.0, device=dev, dtype=dt), (rand(2, H * dk) * 4e-6).to(dt)      # q, k = beta, rotated
    kb, vb = (rand(B, H, C, dk) * 2e4).clamp(-6e4, 6e4).to(dt), rand(B, H, C, dv).to(dt)
    ang = torch.outer(torch.arange(C, device=dev).float(), torch.rand(dk // 2, device=dev))
    freqs = torch.polar(torch.ones_like(ang), ang)
    q, k = (torch.view_as_real(torch.view_as_complex(b.double().view(H, dk // 2, 2)) * freqs[pos].to(torch.complex128))
            .reshape(1, H, dk).expand(B, H, dk) for b in beta)
    keys = torch.cat([kb[:, :, :pos].double(), k.half().double()[:, :, None]], 2)
    vals = torch.cat([vb[:, :, :pos].double(), v.double().view(B, H, 1, dv)], 2)
    pr = torch.softmax(torch.einsum("bhd,bhcd->bhc", q, keys), -1)
    ref = torch.einsum("bhc,bhcd->bhd", pr, vals).reshape(B, -1) * gate.double()
    out = torch.empty(B, H * dv, device=dev, dtype=dt)
    part = torch.empty(B * H * cuda_ops._C().decode_attend_splits(B * H, C) * (dv + 2), device=dev)
    cuda_ops._C().decode_attend(z, gamma, beta, torch.view_as_real(freqs), v, kb, vb, torch.tensor([pos], device=dev), gate,
                                out, part, 1e-5, False)
    assert _rel(out, ref) < 2.0 ** -11               # fp32 throughout, one rounding


@pytest.mark.parametrize("D,G,N,B", [(512, 32, 16, 1), (96, 3, 4, 2), (4096, 64, 16, 3), (64, 1, 32, 1), (2048, 64, 16, 40),
                                     (80, 10, 2, 2), (8192, 8, 32, 1)])
def test_decode_norm_ema_in_parts(D, G, N, B):
    """The norm + EMA link whose RMSNorm factor is left to the products against the one that applies it, twice in a row
    (the count, which also tells who came last), and the products that apply it."""
    from megalodon_b200.ops import cuda_ops
    C = cuda_ops._C()
    torch.manual_seed(D)

    def rand(*s):
        return torch.randn(*s, device="cuda")
    w, b, rw, omega = (rand(D).mul_(0.1).bfloat16() for _ in range(4))
    p, q, ga = torch.rand(D, N, device="cuda"), rand(D, N, 2) * 0.4, rand(D, N, 2)
    state = [torch.arange(B, device="cuda"), rand(B, G) * 0.1, torch.rand(B, G, device="cuda") + 0.5, rand(B, D, N, 2)]
    other = [t.clone() for t in state]
    weight, bias = (rand(96, D) * D ** -0.5).bfloat16(), rand(96).bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for step in range(2):
        x = rand(B, D).bfloat16()
        outs = []
        for (count, mean, var, hx), sq in ((state, None), (other, torch.empty(B, G, device="cuda"))):
            t, mx = torch.empty_like(x), torch.empty_like(x)
            args = (x, w, b, count, mean, var, t, p, q, ga, omega, hx, rw, mx, None, 0, 1e-5, 1e-5)
            C.decode_norm_ema(*args, *([] if sq is None else [sq]), False)
            y = torch.empty(B, 96, device="cuda")
            assert C.skinny_gemm([mx], [weight], [None], [bias], [None], [0], [y], False, err,
                                 [] if sq is None else [sq], 1e-5) == 0
            outs.append((t, y))
        assert torch.equal(state[0], other[0]) and (state[0] == torch.arange(B, device="cuda") + step + 1).all()
        assert _rel(other[1], state[1]) < 1e-6 and _rel(other[2], state[2]) < 1e-6
        # (a rounding of t may fall the other way, and so may one of mx)
        assert _rel(outs[1][0], outs[0][0]) < 2.0 ** -12 and _rel(other[3], state[3]) < 2.0 ** -12
        assert _rel(outs[1][1], outs[0][1]) < 2.0 ** -7
    assert err.item() == 0


@pytest.mark.parametrize("D,G,N,B", [(2056, 257, 16, 2), (4112, 514, 4, 3)])
def test_decode_norm_ema_in_parts_with_more_groups_than_threads(D, G, N, B):
    """Groups that only a prime over 256 of them bundles into 32 features: every part of the sum of squares is written.
    Against the step in 64 bits."""
    _norm_ema_in_parts(D, G, N, B, 3)


@pytest.mark.parametrize("D,G,N,B,steps", [(512, 32, 16, 2, 2 ** 32 - 1), (1024, 8, 2, 3, 2 ** 40 + 5), (16384, 512, 2, 1, 2 ** 32 + 1)])
def test_decode_norm_ema_in_parts_after_many_steps(D, G, N, B, steps):
    """Counts beyond 32 bits, with as many CTAs to a row as there can be."""
    _norm_ema_in_parts(D, G, N, B, steps)
    _norm_ema_in_parts(D, G, N, B, steps + 1)


def _norm_ema_in_parts(D, G, N, B, steps_before):
    """The link and a product behind it, once, against the step in 64 bits from a count of `steps_before` on."""
    from megalodon_b200.ops import cuda_ops, reference
    C = cuda_ops._C()
    torch.manual_seed(D)

    def rand(*s):
        return torch.randn(*s, device="cuda")
    w, b, rw, omega = (rand(D).mul_(0.1).bfloat16() for _ in range(4))
    p, q, ga, hx = torch.rand(D, N, device="cuda"), rand(D, N, 2) * 0.4, rand(D, N, 2), rand(B, D, N, 2)
    count, mean, var = torch.full((B,), steps_before, device="cuda"), rand(B, G) * 0.1, torch.rand(B, G, device="cuda") + 0.5
    x, weight = rand(B, D).bfloat16(), (rand(96, D) * D ** -0.5).bfloat16()
    ty, _, m1, v1 = reference.timestep_norm(x.double()[:, None], count, mean.double(), var.double(), w.double(), b.double(),
                                            None, G, 1e-5, 1.0)
    t64 = ty[:, 0].bfloat16().double()
    ga64, q64, h64 = (torch.view_as_complex(z.double()) for z in (ga, q, hx))
    y = (ga64 * (q64 * h64 + p.double() * t64[:, :, None])).sum(-1).real + omega.double() * t64
    want = (y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * (rw.double() + 1.0)) @ weight.double().t()
    t, mx, sq = torch.empty_like(x), torch.empty_like(x), torch.full((B, G), float("nan"), device="cuda")
    C.decode_norm_ema(x, w, b, count, mean, var, t, p, q, ga, omega, hx, rw, mx, None, 0, 1e-5, 1e-5, sq, False)
    out, err = torch.empty(B, 96, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    assert C.skinny_gemm([mx], [weight], [None], [None], [None], [0], [out], False, err, [sq], 1e-5) == 0 and err.item() == 0
    assert (count == steps_before + 1).all() and _rel(mean, m1) < 1e-6 and _rel(var, v1) < 1e-6
    assert _rel(out, want) < 2.0 ** -7               # roundings of t, of y and of y (1 + w) to 8 bits


@pytest.mark.parametrize("swiglu,B,D,H,share", [(True, 1, 256, 2, False), (False, 5, 512, 1, True)])
def test_native_session_matches_cache_path(swiglu, B, D, H, share):
    """The native chain, eager and replayed, against the growing cache; one step across the chunk boundary."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.decoding import DecodeSession
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.ops import cuda_ops
    from megalodon_b200.utils import init_cache, set_random_seed
    cfg = ModelConf(num_layers=2, model_dim=D, num_heads=H, z_dim=128, value_dim=512, ffn_hidden_dim=384,
                    chunk_size=64, vocab_size=520, swiglu=swiglu, norm_num_groups=16, efficient_attn="fused",
                    share_emb=share, scale_emb=share)
    set_random_seed(1)
    model = build_model(cfg, "bf16", False, False).eval()
    tok = torch.randint(0, 520, (B, 76), device="cuda")
    with torch.no_grad():
        fresh = DecodeSession(model, B, use_graph=False)
        assert fresh._native
        cache = init_cache(B, model, torch.bfloat16)
        for i in range(3):                              # from no past at all
            ref, cache = model(tok[:, i:i + 1], cache=cache)
            assert _rel(fresh.step(tok[:, i]), ref[:, -1]) < 3e-2
        _, cache = model(tok[:, 3:60], cache=cache)
        sess = DecodeSession(model, B)
        sess.load_cache(cache)
        for i in range(60, 72):
            ref, cache = model(tok[:, i:i + 1], cache=cache)
            assert _rel(sess.step(tok[:, i]), ref[:, -1]) < 3e-2, i
        assert sess._graph is not None
    cuda_ops.check_kernel_errors()


@pytest.mark.parametrize("dtype", ["bf16", "fp16"])
@pytest.mark.parametrize("training,use_graph", [(False, False), (True, False), (True, True)])
def test_native_session_without_cached_coefficients(dtype, training, use_graph):
    """A session on a model whose EMA coefficients nobody has computed yet - just put in eval mode, or left in training
    mode, where every eager step and the captured graph compute them anew - against the growing cache."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.decoding import DecodeSession
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.ops import cuda_ops
    from megalodon_b200.utils import init_cache, set_random_seed
    cfg = ModelConf(num_layers=4, model_dim=1024, num_heads=1, z_dim=128, value_dim=1024, ffn_hidden_dim=1024,
                    chunk_size=64, vocab_size=520, swiglu=True, norm_num_groups=32, efficient_attn="fused")
    set_random_seed(2)
    model = build_model(cfg, dtype, False, False)
    t = torch.bfloat16 if dtype == "bf16" else torch.float16
    tok = torch.randint(0, 520, (2, 40), device="cuda")
    model.train(training)
    sess = DecodeSession(model, 2, t, use_graph=use_graph)
    assert sess._native
    got = [sess.step(tok[:, i]).clone() for i in range(8)]
    assert model.training == training and (sess._graph is not None) == use_graph
    model.eval()
    cache = init_cache(2, model, t)
    eps = 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
    with torch.no_grad():
        for i in range(8):
            ref, cache = model(tok[:, i:i + 1], cache=cache)
            # some ten roundings a layer on either side, each of about 0.4 eps, adding up like a random walk (0.0143 seen
            # in bf16, 0.0017 in fp16); half as much again
            assert _rel(got[i], ref[:, -1]) < 0.6 * (2 * 10 * cfg.num_layers) ** 0.5 * eps, i
    cuda_ops.check_kernel_errors()


def test_native_session_in_fp16_with_large_ema_outputs():
    """EMA outputs that are over 65504 when multiplied by 1 + w but not normalised, against the modules."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.decoding import DecodeSession
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.utils import init_cache, set_random_seed
    cfg = ModelConf(num_layers=1, model_dim=256, num_heads=1, z_dim=64, value_dim=256, ffn_hidden_dim=256, chunk_size=64,
                    vocab_size=264, swiglu=True, norm_num_groups=8, efficient_attn="fused")
    set_random_seed(5)
    model = build_model(cfg, "fp16", False, False).eval()
    block = model._wrapped.layers[0]
    while hasattr(block, "_wrapped"):
        block = block._wrapped
    tok = torch.randint(0, 264, (2, 6), device="cuda")
    with torch.no_grad():
        model.materialize_views()
        block.mega.cema.omega.fill_(6000.0)
        block.mega.rmsnorm.weight.fill_(9.0)
        sess = DecodeSession(model, 2, torch.float16, use_graph=False)
        assert sess._native
        cache = init_cache(2, model, torch.float16)
        for i in range(4):
            ref, cache = model(tok[:, i:i + 1], cache=cache)
            # some ten roundings on either side, each of about 0.4 x 2^-11, adding up like a random walk; half as much again
            assert _rel(sess.step(tok[:, i]), ref[:, -1]) < 0.6 * 20 ** 0.5 * 2.0 ** -11


@pytest.mark.parametrize("D,G,B", [(2048, 32, 64), (4096, 64, 40), (1024, 2, 64)])
def test_decode_norm_ema_with_more_clusters_than_fit(D, G, B):
    """Clusters that wait for room start late and one by one; every row still gets the whole row's sum of squares."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(D)
    N = 16
    x = torch.randn(B, D, device="cuda").bfloat16()
    w, b, rw, omega = (torch.randn(D, device="cuda").mul_(0.1).bfloat16() for _ in range(4))
    p, q = torch.rand(D, N, device="cuda"), torch.randn(D, N, 2, device="cuda") * 0.5
    ga = torch.randn(D, N, 2, device="cuda")
    t, mx = torch.empty_like(x), torch.empty_like(x)
    for _ in range(20):
        count = torch.zeros(B, dtype=torch.int64, device="cuda")
        mean, var = torch.zeros(B, G, device="cuda"), torch.ones(B, G, device="cuda")
        hx = torch.zeros(B, D, N, 2, device="cuda")
        cuda_ops._C().decode_norm_ema(x, w, b, count, mean, var, t, p, q, ga, omega, hx, rw, mx, None, 0, 1e-5, 1e-5, False)
        y = ((ga[..., 0].double() * p.double()).sum(-1) + omega.double()) * t.double()      # no past: h = p t
        ref = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * (rw.double() + 1.0)
        rows = (mx.double() - ref).norm(dim=1) / ref.norm(dim=1)
        assert rows.max() < 2.0 ** -7, rows
        assert (count == 1).all()


def test_native_session_with_hooks_adapters_and_new_weights():
    """What the chain does not know about is left to the modules: hooks from the start or added later, an adapter in the
    place of a projection; and weights changed between two eager steps are the ones used."""
    from megalodon_b200.config import ModelConf
    from megalodon_b200.decoding import DecodeSession
    from megalodon_b200.models.mega import build_model
    from megalodon_b200.parallel.model_parallel import ColumnParallelLinear
    from megalodon_b200.utils import init_cache, set_random_seed
    cfg = ModelConf(num_layers=2, model_dim=256, num_heads=1, z_dim=64, value_dim=256, ffn_hidden_dim=256,
                    chunk_size=64, vocab_size=264, swiglu=True, norm_num_groups=8, efficient_attn="fused")
    set_random_seed(4)
    model = build_model(cfg, "fp16", False, False).eval()
    tok = torch.randint(0, 264, (2, 12), device="cuda")

    class Adapter(ColumnParallelLinear):
        def forward(self, x):
            return super().forward(x).roll(1, -1)

    def run(steps, between=lambda i: None):
        """the same steps through a session and through the growing cache, `between(i)` before step i of either"""
        sess = DecodeSession(model, 2, torch.float16, use_graph=False)
        outs = []
        for session in (True, False):
            cache = init_cache(2, model, torch.float16)
            rows = []
            with torch.no_grad():
                for i in range(steps):
                    undo = between(i)
                    if session:
                        rows.append(sess.step(tok[:, i]).clone())
                    else:
                        y, cache = model(tok[:, i:i + 1], cache=cache)
                        rows.append(y[:, -1])
                    if undo is not None:
                        undo()
            outs.append(torch.stack(rows))
        # some ten roundings a layer on either side, each of about 0.4 x 2^-11, adding up like a random walk (0.0012 seen);
        # half as much again
        assert _rel(*outs) < 0.6 * (2 * 10 * cfg.num_layers) ** 0.5 * 2.0 ** -11
        return sess._native, outs[0]

    block = model._wrapped.layers[1]
    while hasattr(block, "_wrapped"):
        block = block._wrapped
    native, plain = run(4)
    assert native
    wr = block.mega.wr
    wr.__class__ = Adapter                                   # from the start
    native, adapted = run(4)
    assert not native and _rel(adapted, plain) > 1e-2
    wr.__class__ = ColumnParallelLinear

    def hook(i):                                             # for some of the steps
        if i % 2:
            return block.nffn.fc1.register_forward_hook(lambda m, a, o: o * 0.5).remove
    native, hooked = run(6, hook)
    assert native and _rel(hooked[:4], plain) > 1e-2 and torch.equal(hooked[0], plain[0])

    unit = model._units()[2]

    def update(i):
        if i == 2:
            keep = unit.flat_param.detach().clone()
            unit.flat_param.mul_(1.25)
            return lambda: unit.flat_param.copy_(keep)       # (the steps run under no_grad)
    native, moved = run(4, update)
    assert native and torch.equal(moved[:2], plain[:2]) and _rel(moved[2:], plain[2:]) > 1e-3


@pytest.mark.parametrize("B,H,C,dk,dv,pos,offset", [(2, 3, 40, 16, 12, 20, 0), (1, 2, 700, 64, 2061, 699, 0), (3, 1, 64, 8, 1, 5, 0),
                                                    (2, 2, 300, 32, 64, 130, 1), (1, 1, 16, 8, 4100, 0, 3)])
def test_decode_attention_of_any_value_width(B, H, C, dk, dv, pos, offset):
    """Value rows that are no whole 16-byte pieces, or start between two."""
    from megalodon_b200 import ops
    torch.manual_seed(dv)
    q, k = torch.randn(B, H, dk, device="cuda").bfloat16(), torch.randn(B, H, C, dk, device="cuda").bfloat16()
    v = torch.randn(B * H * C * dv + offset, device="cuda").bfloat16()[offset:].view(B, H, C, dv)
    k[:, :, pos + 1:] = float("nan")
    v[:, :, pos + 1:] = float("nan")
    assert ops.decode_attention_native(q, k)
    out = ops.decode_attention(q, k, v, torch.tensor([pos], device="cuda"), 0.4)
    s = torch.einsum("bhd,bhcd->bhc", q.double(), k[:, :, :pos + 1].double()) * 0.4
    ref = torch.einsum("bhc,bhcd->bhd", torch.softmax(s, -1), v[:, :, :pos + 1].double())
    assert out.shape == ref.shape and _rel(out, ref) < 2.0 ** -8       # fp32 throughout, one rounding
