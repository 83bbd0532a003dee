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
                                         (2, 257, 2, 128, 256), (3, 777, 1, 64, 128),
                                         (1, 907, 2, 256, 2048)])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_any_length(B, L, H, dk, dv, causal):
    from megalodon_b200 import ops
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(L)
    q, k, v = _rand(B, L, H, dk, scale=dk ** -0.25), _rand(B, L, H, dk, scale=dk ** -0.25), _rand(B, L, H, dv)
    g = _rand(B, L, H, dv)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    # the score buffer is uninitialised memory: whatever a product reads without another having written it is NaN
    torch.cuda.empty_cache()
    poison = [torch.full((B * H * L * (-(-L // 128) * 128),), float("nan"), dtype=q.dtype, device="cuda") for _ in range(3)]
    del poison
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


@pytest.mark.parametrize("D,N", [(1, 1), (37, 16), (512, 32), (100, 5)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cema_coefficients(D, N, dtype):
    from megalodon_b200 import ops
    from megalodon_b200.ops import reference
    torch.manual_seed(D)
    ps = [_rand(D, N, 1, dtype=dtype), _rand(D, N, 1, dtype=dtype), _rand(D, 1, 1, dtype=dtype, scale=3.0),
          _rand(D, N, 2, dtype=dtype)]
    a = [t.clone().requires_grad_(True) for t in ps]
    b = [t.double().requires_grad_(True) for t in ps]
    sc = N ** -0.5
    p, q, g = ops.cema_coeffs(*a, sc)
    pd = torch.sigmoid(b[0])
    qd = torch.polar(1.0 - pd * torch.sigmoid(b[1]),
                     torch.sigmoid(b[2]) * (2 * torch.pi / N) * torch.arange(1, N + 1, device="cuda").view(1, N, 1))
    gd = torch.view_as_complex(b[3]) * sc
    rp, rq, rg = reference.cema_coeffs(*ps, sc)
    for got, ref, want in ((p, rp, pd), (q, rq, qd), (g, rg, gd)):
        assert got.shape == ref.shape and got.dtype == ref.dtype
        assert ((got - want).abs().norm() / want.abs().norm()).item() < 4e-7
    cp, cq, cg = torch.randn_like(pd), torch.randn_like(qd), torch.randn_like(gd)
    for outs in ((p, q, g), (pd, qd, gd)):
        loss = (outs[0] * cp).sum() + (outs[1] * cq.conj()).real.sum() + (outs[2] * cg.conj()).real.sum()
        loss.backward()
    for x, y in zip(a, b):
        assert _rel(x.grad, y.grad) < (2e-5 if dtype == torch.float32 else 2.0 ** -8)
    p, q, g = ops.cema_coeffs(*a, sc)                       # one output alone
    assert torch.autograd.grad(p.sum(), a[0])[0].shape == a[0].shape


@pytest.mark.parametrize("rows", [1, 2, 64, 65, 300])
def test_linear_group_matches_separate_layers(rows):
    from megalodon_b200 import ops
    torch.manual_seed(rows)
    K, sizes = 264, (64, 136, 264)
    x, add = _rand(rows, K), _rand(rows, sizes[2])
    ws, bs = [_rand(n, K, scale=K ** -0.5) for n in sizes], [_rand(n) for n in sizes]
    gs = [_rand(rows, n) for n in sizes]
    leaves = [t.clone().requires_grad_(True) for t in (x, add, *ws, *bs)]
    lw, lb = leaves[2:5], leaves[5:]
    outs = ops.linear_group(leaves[0], [(lw[0], lb[0], None), (lw[1], None, None), (lw[2], lb[2], leaves[1])])
    torch.autograd.backward(outs, gs)
    ref = [t.double().requires_grad_(True) for t in (x, add, *ws, *bs)]
    rw, rb = ref[2:5], ref[5:]
    want = [ref[0] @ rw[0].t() + rb[0], ref[0] @ rw[1].t(), ref[0] @ rw[2].t() + rb[2] + ref[1]]
    torch.autograd.backward(want, [g.double() for g in gs])
    for o, w in zip(outs, want):
        assert _rel(o, w) < 2.0 ** -7
    for i, (a, r) in enumerate(zip(leaves, ref)):
        if i != 6:
            assert _rel(a.grad, r.grad) < 2.0 ** -7, i      # dx: rounded after each of the three products
    # an output that nobody used
    out = ops.linear_group(leaves[0], [(lw[0], lb[0], None), (lw[1], None, None)])
    leaves[0].grad = None
    out[1].backward(gs[1])
    assert _rel(leaves[0].grad, gs[1].double() @ ws[1].double()) < 2.0 ** -7


# lengths at which the scans change the steps of a segment (4, 8, 16, 32 of at most 512 segments) and leave the
# one-kernel form; a padded stretch and a carried past
@pytest.mark.parametrize("L", [1, 3, 5, 37, 2048, 2049, 4097, 8193, 16385])
@pytest.mark.parametrize("masked", [False, True])
def test_timestep_norm_segments(L, masked):
    from megalodon_b200 import ops
    from megalodon_b200.ops import reference
    torch.manual_seed(L)
    B, G, D = 2, 3, 24
    x, g = _rand(B, L, D, dtype=torch.float32), _rand(B, L, D, dtype=torch.float32)
    w, b = _rand(D, dtype=torch.float32, scale=0.2), _rand(D, dtype=torch.float32)
    count = torch.tensor([0, 11], device="cuda")
    mean, var = _rand(B, G, dtype=torch.float32, scale=0.3), torch.rand(B, G, device="cuda") + 0.5
    mask = None
    if masked:
        mask = torch.zeros(B, L, dtype=torch.bool, device="cuda")
        mask[0, : L // 3] = True
        mask[1, L // 2: L // 2 + 5] = True
    gm, gv = _rand(B, G, dtype=torch.float32), _rand(B, G, dtype=torch.float32)

    def grads(f, dt):
        leaves = [t.to(dt).requires_grad_(True) for t in (x, mean, var, w, b)]
        y, c, m, v = f(leaves[0], count, leaves[1], leaves[2], leaves[3], leaves[4], mask, G, 1e-5, 1.0)
        return (y, m, v), torch.autograd.grad((y * g.to(dt)).sum() + (m * gm.to(dt)).sum() + (v * gv.to(dt)).sum(),
                                              leaves), c
    got, dgot, c1 = grads(ops.timestep_norm, torch.float32)
    want, dwant, c2 = grads(reference.timestep_norm, torch.float64)
    assert torch.equal(c1, c2)
    for a, r in zip(got, want):
        assert _rel(a, r) < 2e-6
    for a, r in zip(dgot, dwant):
        assert _rel(a, r) < 2e-5, (a.shape, _rel(a, r))


@pytest.mark.parametrize("tile", [64, 128, 256, 512])
@pytest.mark.parametrize("M,N,K", [(100, 72, 136), (128, 64, 64), (300, 200, 264), (777, 264, 1032), (513, 768, 264)])
def test_tiles(tile, M, N, K):
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(M)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b, bias = _rand(M, K), _rand(N, K, scale=K ** -0.5), _rand(N)
    ref = a.double() @ b.double().t() + bias.double()
    for a_mn, b_mn in ((False, False), (False, True), (True, True)):
        if a_mn and M % 8:
            continue
        A = a.t().contiguous() if a_mn else a
        B = b.t().contiguous() if b_mn else b
        for dtype, tol in ((0, 2e-6), (1, 2.0 ** -8)):      # fp32 leaves through the staging buffers too
            out, _, rc = cuda_ops._C().gemm(A, B, None, bias, 0, a_mn, b_mn, False, dtype, 0, 1.0, err, tile=tile)
            assert rc == 0 and err.item() == 0
            assert _rel(out, ref) < tol


@pytest.mark.parametrize("tile", [64, 128, 256, 512])
@pytest.mark.parametrize("M,batch", [(4096, 1), (4097, 2), (8448, 1), (12301, 1)])
def test_tiles_in_bands(tile, M, batch):
    """The tile walk in bands of rows: one band, a last band of one row, equal bands, a ragged last tile."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(M)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b = _rand(batch, M, 72), _rand(batch, 520, 72, scale=72 ** -0.5)
    out, _, rc = cuda_ops._C().gemm(a, b, None, None, 0, False, False, False, 1, 0, 1.0, err, tile=tile)
    assert rc == 0 and err.item() == 0
    ref = a.double() @ b.double().transpose(1, 2)
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()   # every tile: fp32 sums, one rounding


@pytest.mark.parametrize("tile", [64, 128, 256, 512])
@pytest.mark.parametrize("M,N", [(300, 200), (513, 264), (100, 77)])
def test_epilogues(tile, M, N):
    """Bias (vector and scalar reads), SiLU with its pre-activation, addend and accumulation through the staging buffers,
    last columns that are no whole piece included; nothing beyond them is written."""
    from megalodon_b200.ops import cuda_ops
    C = cuda_ops._C()
    torch.manual_seed(M)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, b = _rand(M, 136), _rand(N, 136, scale=136 ** -0.5)
    prod = a.double() @ b.double().t()
    ld = -(-N // 8) * 8 + 8

    def close(got, want):
        return ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()     # fp32 sums, one rounding

    for dt, off in ((torch.bfloat16, 0), (torch.float32, 0), (torch.float16, 1)):
        bias = _rand(N + off, dtype=dt)[off:]
        for add in (None, "aux", "accumulate"):
            buf = torch.full((M, ld), 7.0, device="cuda", dtype=torch.bfloat16)
            aux = _rand(M, ld)[:, :N]
            if add == "accumulate":
                buf[:, :N] = aux
            out, _, rc = C.gemm(a, b, buf[:, :N], bias, 0, False, False, False, 1, 0, 0.5, err, tile=tile,
                                accumulate=add == "accumulate", aux=aux if add == "aux" else None)
            assert rc == 0 and (buf[:, N:] == 7.0).all()
            assert close(buf[:, :N], 0.5 * prod + bias.double() + (aux.double() if add else 0.0))
        if N % 8 == 0:
            for code, odt in ((1, torch.bfloat16), (0, torch.float32)):
                out, pre, rc = C.gemm(a, b, None, bias, 1, False, False, True, code, 0, 1.0, err, tile=tile)
                assert rc == 0 and out.dtype == odt and close(pre, prod + bias.double())
                assert close(out, torch.nn.functional.silu(prod + bias.double()))
    assert err.item() == 0


@pytest.mark.parametrize("B,L,D", [(1, 1, 8), (2, 15, 24), (1, 16, 16), (3, 17, 40), (1, 255, 264), (2, 256, 16), (1, 257, 8),
                                   (1, 700, 32), (2, 1024, 48), (3, 17, 1024), (5, 300, 648)])
@pytest.mark.parametrize("carried", [False, True])
def test_ema_on_tensor_cores(B, L, D, carried):
    """Chunks, tiles and features that are no whole ones, several sequences to a CTA, against the recurrence in 64 bits:
    outputs rounded once, the last state to 32-bit sums."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(L)
    N, dev = 16, "cuda"
    x = _rand(B, L, D)
    p = torch.rand(D, N, device=dev) * 0.8 + 0.1
    q = torch.polar(1.0 - torch.rand(D, N, device=dev).pow(3) * 0.9, torch.rand(D, N, device=dev) * 3.0)
    gamma = torch.view_as_complex(torch.randn(D, N, 2, device=dev) * 0.25)
    omega = torch.randn(D, device=dev)
    hx = torch.view_as_complex(torch.randn(B, D, N, 2, device=dev)) if carried else None
    y, last = cuda_ops._C().cema_fwd(x, p, torch.view_as_real(q), torch.view_as_real(gamma), omega,
                                     None if hx is None else torch.view_as_real(hx), True)
    h = torch.zeros(B, D, N, dtype=torch.complex128, device=dev) if hx is None else hx.to(torch.complex128)
    want, size = (torch.empty(B, L, D, dtype=torch.float64, device=dev) for _ in range(2))
    for t in range(L):
        h = q.to(torch.complex128) * h + p.double() * x[:, t].double().unsqueeze(-1)
        want[:, t] = (gamma.to(torch.complex128) * h).sum(-1).real + omega.double() * x[:, t].double()
        size[:, t] = (gamma.abs().double() * h.abs()).sum(-1) + omega.abs().double() * x[:, t].abs().double()
    assert _rel(last, torch.view_as_real(h)) < 2e-6
    # one rounding of the result, and of 32 + 16 terms summed in fp32 what they cancel (2^-24 each, and of their powers)
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -24 * 64 * size).all()


@pytest.mark.parametrize("B,L,D", [(1, 3, 8), (2, 16, 48), (4, 128, 1024), (2, 129, 24), (3, 257, 1024)])
def test_ema_on_tensor_cores_for_short_sequences(B, L, D):
    """Around the length up to which the scan needs one pass, where the choice between the two follows another line, and
    several short sequences to a CTA."""
    from megalodon_b200.ops import cuda_ops
    per = cuda_ops._C().cema_tensor_plan(B, L, D, torch.cuda.get_device_properties(0).multi_processor_count)
    assert per == (2 if D == 1024 else 1)
    test_ema_on_tensor_cores(B, L, D, True)


@pytest.mark.parametrize("bad", [float("inf"), float("nan"), -float("inf")])
def test_ema_with_infinities_stays_causal(bad):
    """What comes before an infinity or NaN in a feature, and the other features, do not see it."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(3)
    B, L, D, N = 2, 600, 32, 16
    x = _rand(B, L, D)
    p, q = torch.rand(D, N, device="cuda"), torch.rand(D, N, 2, device="cuda") * 0.6
    gamma, omega = torch.randn(D, N, 2, device="cuda") * 0.25, torch.randn(D, device="cuda")
    clean, _ = cuda_ops._C().cema_fwd(x, p, q, gamma, omega, None, True)
    x2 = x.clone()
    x2[1, 300, 5] = bad
    y, last = cuda_ops._C().cema_fwd(x2, p, q, gamma, omega, None, True)
    keep = torch.ones(B, L, D, dtype=torch.bool, device="cuda")
    keep[1, 300:, 5] = False
    assert torch.isfinite(y[keep]).all() and _rel(y[keep], clean[keep]) < 2.0 ** -9
    assert not torch.isfinite(y[1, 300:, 5]).any() and not torch.isfinite(last[1, 5]).all()


def test_ema_with_growing_states():
    """Powers that overflow within a tile, where the recurrence itself does not: only the last steps have inputs."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(4)
    B, L, D, N = 1, 500, 16, 16
    x = torch.zeros(B, L, D, device="cuda", dtype=torch.bfloat16)
    x[:, 480:] = _rand(B, 20, D)
    p, q = torch.rand(D, N, device="cuda"), torch.randn(D, N, 2, device="cuda") * 2
    gamma, omega = torch.randn(D, N, 2, device="cuda") * 0.25, torch.randn(D, device="cuda")
    y, last = cuda_ops._C().cema_fwd(x, p, q, gamma, omega, None, True)
    tail, tail_last = cuda_ops._C().cema_fwd(x[:, 480:].float().contiguous(), p, q, gamma, omega, None, True)
    assert (y[:, :480] == 0).all() and _rel(y[:, 480:], tail) < 2.0 ** -8 and _rel(last, tail_last) < 1e-5


def test_operators_without_gradients_match_the_recorded_ones():
    """The short route under no_grad against the autograd function, and what the latter refuses stays refused."""
    from megalodon_b200 import ops
    torch.manual_seed(0)
    x, w, b = _rand(70, 64), _rand(128, 64, scale=0.1), _rand(128)
    rec = ops.linear(x.clone().requires_grad_(True), w, b, "silu")
    with torch.no_grad():
        got = ops.linear(x, w.clone().requires_grad_(True), b, "silu")
    assert rec.requires_grad and not got.requires_grad and torch.equal(rec, got)
    with torch.no_grad(), torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        with pytest.raises(Exception):
            ops.linear(dual, w, b, "silu")
    with torch.no_grad(), pytest.raises(Exception):
        torch.func.vmap(lambda r: ops.rms_norm(r, None, 1e-5))(x)


def test_gate_is_rounded_after_its_activation(monkeypatch):
    """The gate SiLU(r) leaves the product's epilogue rounded once; rounding r first shows as up to |r| times that."""
    from megalodon_b200.modules.moving_average_gated_attention import MovingAverageGatedAttention, ops
    torch.manual_seed(5)
    m = MovingAverageGatedAttention(mdim=64, zdim=16, hdim=128, num_heads=1, ndim=4, chunk_size=32,
                                    efficient_attn="fused", norm_num_groups=4).cuda().bfloat16()
    with torch.no_grad():
        m.wr.weight.normal_(std=0.3)                       # r with a deviation of 2.4
    x = _rand(3, 32, 64)
    monkeypatch.setattr(m.inner_attention, "forward", lambda q, k, v, *a: (torch.ones_like(v), None))
    seen = []
    monkeypatch.setattr(ops, "memory_efficient_dropout", lambda t, p, training: (seen.append(t.detach()), t)[1])
    freqs = torch.polar(torch.ones(32, 8, device="cuda"), torch.rand(32, 8, device="cuda"))
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            m(x, freqs)
        mx, gate = seen
        seen.clear()
        want = torch.nn.functional.silu(mx.double() @ m.wr.weight.double().t() + m.wr.bias.double())
        # one rounding to 8 significant bits is at most 2^-8 of the value; the sum behind it is fp32
        assert ((gate.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 4e-6).all()


@pytest.mark.parametrize("rows", [1, 2, 64, 65, 300])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_linear_group_with_a_gate(rows, dtype):
    from megalodon_b200 import ops
    torch.manual_seed(rows)
    K, sizes = 264, (64, 136, 264)
    x, add, v = _rand(rows, K, dtype=dtype), _rand(rows, sizes[2], dtype=dtype), _rand(rows, sizes[1], dtype=dtype)
    ws, bs = [_rand(n, K, scale=K ** -0.5, dtype=dtype) for n in sizes], [_rand(n, dtype=dtype) for n in sizes]
    gs = [_rand(rows, n, dtype=dtype) for n in sizes]
    leaves = [t.clone().requires_grad_(True) for t in (x, add, *ws, *bs, v)]

    def outs(t):
        return [t[0] @ t[2].t() + t[5], torch.nn.functional.silu(t[0] @ t[3].t() + t[6]) * t[8], t[0] @ t[4].t() + t[7] + t[1]]

    def group(t):
        a, r, c = ops.linear_group(t[0], [(t[2], t[5], None), (t[3], t[6], None, True), (t[4], t[7], t[1], False)])
        return [a, ops.gate(r, t[8]), c]
    got = group(leaves)
    torch.autograd.backward(got, gs)
    ref = [t.double().requires_grad_(True) for t in (x, add, *ws, *bs, v)]
    want = outs(ref)
    torch.autograd.backward(want, [g.double() for g in gs])
    with torch.no_grad():
        again = group(leaves)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for i, (o, n, w) in enumerate(zip(got, again, want)):
        # one rounding; two where the gate is rounded before it is applied (few rows)
        assert _rel(o, w) < eps * (1 + (i == 1)) and _rel(n, w) < eps * (1 + (i == 1))
    for i, (a, r) in enumerate(zip(leaves, ref)):
        # dx and what comes through the gate: rounded once more on the way
        assert _rel(a.grad, r.grad) < (2 if i in (0, 3, 6, 8) else 1) * eps, i
    # the gate alone, and the group without it
    a, r, c = ops.linear_group(leaves[0], [(leaves[2], leaves[5], None), (leaves[3], None, None, True)])[:2] + [None]
    da, = torch.autograd.grad(ops.gate(r, v), leaves[0], gs[1], retain_graph=True)
    z = x.double() @ ws[1].double().t()
    s = torch.sigmoid(z)
    assert _rel(da, (gs[1].double() * v.double() * s * (1 + z * (1 - s))) @ ws[1].double()) < 2 * eps
    assert _rel(torch.autograd.grad(a, leaves[0], gs[0])[0], gs[0].double() @ ws[0].double()) < 2 * eps


@pytest.mark.parametrize("n", [7, 4096, 100003])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_swiglu_of_a_wider_input(n, dtype):
    """a in fp32 against b in 16 bits, whole pieces and a tail, aligned and not."""
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(n)
    for off in (0, 1):
        a = _rand(n + off, dtype=torch.float32, scale=3.0)[off:]
        b, g = _rand(n + off, dtype=dtype)[off:], _rand(n + off, dtype=dtype)[off:]
        ad, bd = a.double(), b.double()
        s = torch.sigmoid(ad)
        eps = 1.01 * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
        out = cuda_ops._C().swiglu_fwd(a, b)
        da, db = cuda_ops._C().swiglu_bwd(g, a, b)
        for got, want in ((out, ad * s * bd), (da, g.double() * bd * (s + ad * s * (1 - s))), (db, g.double() * ad * s)):
            assert got.dtype == dtype and ((got.double() - want).abs() <= eps * want.abs() + 1e-6).all()
    with pytest.raises(Exception):
        cuda_ops._C().swiglu_fwd(a, b[:-1])


def _coefficient_args(dtype=torch.float32, D=12, N=4):
    torch.manual_seed(D)
    return [_rand(D, N, 1, dtype=dtype), _rand(D, N, 1, dtype=dtype), _rand(D, 1, 1, dtype=dtype),
            _rand(D, N, 2, dtype=dtype)]


def test_cema_coefficients_differentiate_twice():
    """A penalty on the gradient of a function of p, q and gamma, against the element-wise operations in 64 bits."""
    from megalodon_b200 import ops

    def coeffs64(alpha, delta, theta, gamma, scale):
        p = torch.sigmoid(alpha)
        n = torch.arange(1, 5, device="cuda", dtype=torch.float64).view(1, 4, 1)
        q = torch.polar(1.0 - p * torch.sigmoid(delta), torch.sigmoid(theta) * (2 * torch.pi / 4) * n)
        return p, q, torch.view_as_complex(gamma) * scale

    def second(f, args):
        p, q, g = f(*args, 0.5)
        loss = (p ** 2).sum() + (q.real ** 3).sum() + q.imag.abs().sum() + (g.abs() ** 4).sum()
        first = torch.autograd.grad(loss, args, create_graph=True)
        return [*first, *torch.autograd.grad(sum((x ** 2).sum() for x in first), args)]
    base = _coefficient_args()
    got = second(ops.cema_coeffs, [t.clone().requires_grad_(True) for t in base])
    want = second(coeffs64, [t.double().requires_grad_(True) for t in base])
    for a, b in zip(got, want):
        assert _rel(a.detach(), b.detach()) < 2e-5
    # some of the parameters, some of the outputs
    alpha = base[0].clone().requires_grad_(True)
    q = ops.cema_coeffs(alpha, *base[1:], 0.5)[1]
    first, = torch.autograd.grad(q.real.sum(), alpha, create_graph=True)
    assert torch.autograd.grad(first.sum(), alpha)[0].abs().sum() > 0
    theta = base[2].clone().requires_grad_(True)             # p and gamma do not depend on it
    p, q, g = ops.cema_coeffs(*base[:2], theta, base[3], 0.5)
    first, = torch.autograd.grad(p.sum() + q.real.sum() + g.abs().sum(), theta, create_graph=True)
    assert torch.autograd.grad(first.sum(), theta)[0].abs().sum() > 0


def test_cema_coefficients_under_transforms_and_other_types():
    from megalodon_b200 import ops
    from megalodon_b200.ops import reference
    args = _coefficient_args()
    want = reference.cema_coeffs(*args, 0.5)
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            got = ops.cema_coeffs(*[t.double() for t in args], 0.5)
            assert all(_rel(torch.view_as_real(a) if a.is_complex() else a, torch.view_as_real(b) if b.is_complex() else b)
                       < 1e-6 for a, b in zip(got, want))
            _, tangents = torch.func.jvp(lambda a: ops.cema_coeffs(a, *args[1:], 0.5)[0], (args[0],),
                                         (torch.ones_like(args[0]),))
            s = torch.sigmoid(args[0])
            assert _rel(tangents, s * (1 - s)) < 1e-6
            batch = torch.stack([args[0], args[0] + 1.0])
            ps = torch.func.vmap(lambda a: ops.cema_coeffs(a, *args[1:], 0.5)[0])(batch)
            assert _rel(ps, torch.sigmoid(batch)) < 1e-6


@pytest.mark.parametrize("rows", [1, 5, 300])
def test_empty_sums(rows):
    """No rows: every weight gradient is a sum of nothing, zero.  No features: bias and addend alone."""
    from megalodon_b200 import ops
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(0)
    poison = [torch.full((1 << 14,), float("nan"), device="cuda") for _ in range(8)]
    del poison
    x, w, b = _rand(0, 64).requires_grad_(True), _rand(32, 64).requires_grad_(True), _rand(32).requires_grad_(True)
    add = _rand(0, 32).requires_grad_(True)
    for out in (ops.linear(x, w, b), ops.linear(x, w, b, "silu"), ops.linear_add(x, w, b, add),
                ops.linear_group(x, [(w, b, None), (w, b, add)])[1]):
        dx, dw, db = torch.autograd.grad(out.sum(), (x, w, b))
        assert dx.shape == x.shape and (dw == 0).all() and (db == 0).all()
    x, w, add = _rand(rows, 0), _rand(32, 0), _rand(rows, 32)
    b = b.detach()
    assert torch.equal(cuda_ops.gemm(x, w, b)[0], b.expand(rows, 32))
    assert torch.equal(cuda_ops.gemm(x, w, b, softmax=dict(aux=add))[0], b + add)
    target = _rand(32, 64)
    for accumulate, want in ((True, target.clone()), (False, torch.zeros_like(target))):
        cuda_ops.gemm(_rand(0, 32), _rand(0, 64), a_mn=True, b_mn=True, out=target, accumulate=accumulate)
        assert torch.equal(target, want)


class _Pending:
    """What a sharded weight carries while its all-gather is left to the first product (one GPU: the row blocks of two
    ranks as two tensors)."""

    def __init__(self, w, blocks):
        self.w, self.blocks, self.pending, self.how = w, blocks, True, None

    def sources(self):
        return [b.data_ptr() for b in self.blocks], 1

    def done(self):
        self.pending, self.how = False, "product"

    def pull_now(self):
        self.w.copy_(torch.cat(self.blocks))
        self.pending, self.how = False, "pull"


@pytest.mark.parametrize("rows", [1, 5, 64, 300])
@pytest.mark.parametrize("grad", [False, True])
def test_linear_group_gathers_sharded_weights(rows, grad):
    """No kernel may read a weight that has not been gathered; where the shape allows it the product gathers it."""
    from megalodon_b200 import ops
    from megalodon_b200.ops import cuda_ops
    torch.manual_seed(rows)
    K, sizes = 128, (256, 512, 256)
    x, add, v = _rand(rows, K), _rand(rows, sizes[2]), _rand(rows, sizes[1])
    true = [_rand(n, K, scale=K ** -0.5) for n in sizes]
    bs = [_rand(n) for n in sizes]
    ws, specs = [], []
    for t in true:
        w = torch.full_like(t, float("nan"))
        blocks = [t[: t.shape[0] // 2].clone(), t[t.shape[0] // 2:].clone()]
        w[t.shape[0] // 2:] = blocks[1]                     # this rank's own rows are in place
        w._gather_spec = _Pending(w, blocks)
        specs.append(w._gather_spec)
        ws.append(w)
    xl = x.clone().requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        a, r, c = ops.linear_group(xl, [(ws[0], bs[0], None), (ws[1], bs[1], None, True), (ws[2], bs[2], add)])
        b = ops.gate(r, v)
    torch.cuda.synchronize()
    assert [s.how for s in specs] == ["product" if rows > 128 else "pull"] * 3
    lin = [x.double() @ t.double().t() + bias.double() for t, bias in zip(true, bs)]
    want = [lin[0], torch.nn.functional.silu(lin[1]) * v.double(), lin[2] + add.double()]
    for got, ref in zip((a, b, c), want):
        assert _rel(got, ref) < 2.0 ** -7
    assert all(torch.equal(w, t) for w, t in zip(ws, true))
    if grad:
        dx, = torch.autograd.grad([a, c], xl, [a.detach(), c.detach()])
        ref = a.double() @ true[0].double() + c.double() @ true[2].double()
        assert _rel(dx, ref) < 2.0 ** -7
    cuda_ops.check_kernel_errors()


def test_fp32_products_without_gradients_refuse_what_linear_refuses():
    from megalodon_b200 import ops
    x, w = _rand(70, 64), _rand(128, 64, scale=0.1)
    with torch.no_grad():
        assert ops.linear_fp32_out(x, w).dtype == torch.float32
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
            with pytest.raises(Exception):
                ops.linear_fp32_out(dual, w)
        with pytest.raises(Exception):
            torch.func.vmap(lambda r: ops.linear_fp32_out(r[None], w))(x)


@pytest.mark.parametrize("tile", [64, 128, 256, 512])
def test_silu_of_large_negative_values(tile):
    """SiLU(x) down to where exp(-x) leaves fp32: results that bf16 holds are not flushed to zero."""
    from megalodon_b200.ops import cuda_ops
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a, w = torch.zeros(130, 64, device="cuda").bfloat16(), torch.zeros(72, 64, device="cuda").bfloat16()
    a[:, 0] = 1.0
    w[:, 0] = -torch.linspace(80.0, 88.5, 72, device="cuda").bfloat16()
    out, _, rc = cuda_ops._C().gemm(a, w, None, None, 1, False, False, False, 1, 0, 1.0, err, tile=tile)
    x = w[:, 0].double()
    # one rounding to 8 bits; exp in fp32 is off by some 88 steps of 2^-23
    assert rc == 0 and ((out.double() / (x * torch.sigmoid(x)) - 1.0).abs() < 2.0 ** -8).all()


def test_silu_of_the_epilogue_in_fp32():
    """Against 64 bits over all of fp32's useful range, and at its ends."""
    from megalodon_b200.ops import cuda_ops
    err = torch.zeros(1, dtype=torch.int32, device="cuda")

    def silu(x):
        a, w = torch.zeros(8, 64, device="cuda").bfloat16(), torch.zeros(x.numel(), 64, device="cuda").bfloat16()
        out, _, rc = cuda_ops._C().gemm(a, w, None, x, 1, False, False, False, 0, 0, 1.0, err)
        assert rc == 0
        return out[0]
    torch.manual_seed(0)
    x = torch.rand(1 << 16, device="cuda") * 176.0 - 88.0
    want = x.double() * torch.sigmoid(x.double())
    # exp in fp32 is a power of two whose exponent x log2(e) has two roundings, of the constant and of the product, half a
    # step each: |x| steps of 2^-23 of the result; the power is off by two, and three roundings more
    assert ((silu(x).double() / want - 1.0).abs() <= (x.double().abs() + 5) * 2.0 ** -23).all()
    inf = float("inf")
    got = silu(torch.tensor([0.0, inf, 3e38, -100.0, -3e38, 1e-38, -1e-38, 1e-40], device="cuda")).tolist()
    assert got[:5] == [0.0, inf, 3.0000000054977558e38, 0.0, 0.0]
    assert all(abs(g - w) <= 2.0 ** -149 for g, w in zip(got[5:], (5e-39, -5e-39, 5e-41)))
    assert silu(torch.tensor([-inf, float("nan")] * 4, device="cuda")).isnan().all()
