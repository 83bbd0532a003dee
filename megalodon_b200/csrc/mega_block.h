// A MEGA block forward and backward as one call each, over the operator functions of bindings.cpp (which includes this
// file in its unnamed namespace): the same kernels in the same order as the modules launch them, without an interpreter,
// a module call and an autograd node between two of them.
//
// A launch through the modules costs the host 20 to 27 us, more than most kernels of a small model take; from here some
// 9 without gradients (21 launches of a block in 178 us, Python's checks among them; 15 a launch both ways with autograd).  Modules / native, ms: a training step of two 512-wide layers 9.8 / 5.9, of four 1024-wide ones 8.6 / 6.7; scoring
// 8 x 777 tokens in twelve 1024-wide layers 8.4 / 6.2; a prompt of 37 tokens there 6.7 / 3.2.
#pragma once

enum BlockParam {
  kTsnW, kTsnB, kOmega, kRmsW, kWv, kBv, kWz, kBz, kWr, kBr, kWh1, kBh1, kGamma, kBeta, kWh2, kLnW, kLnB, kFc1, kFc3, kFc2,
  kBlockParams
};
using Params = std::vector<OptTensor>;

struct BlockDims {
  int64_t groups, heads, dk, dv, chunk;
  double tsn_eps, rms_eps, z_eps, ln_eps;
};
BlockDims block_dims(const std::vector<int64_t>& d, const std::vector<double>& eps) {
  TORCH_CHECK(d.size() == 5 && eps.size() == 4, "mega_block: sizes");
  return {d[0], d[1], d[2], d[3], d[4], eps[0], eps[1], eps[2], eps[3]};
}

struct GemmArgs {
  OptTensor out, bias, aux, row_in, row_in2, row_out;
  int64_t act = 0, mode = 0, epi = 0;
  bool a_mn = false, b_mn = false, want_pre = false, accumulate = false;
  double alpha = 1.0;
  at::ScalarType out_type = at::ScalarType::Undefined;
};
class Launcher {
 public:
  explicit Launcher(const Tensor& err) : err_(err), before_(mb::thread_launches()) {}
  // kernels launched since
  int64_t count() const { return mb::thread_launches() - before_; }

  std::tuple<Tensor, OptTensor> gemm(const Tensor& a, const Tensor& b, const GemmArgs& g) {
    const at::ScalarType t = g.out.has_value() ? g.out->scalar_type()
                                               : (g.out_type == at::ScalarType::Undefined ? a.scalar_type() : g.out_type);
    const int64_t code = t == at::kFloat ? 0 : (t == at::kBFloat16 ? 1 : 2);
    auto [c, pre, rc] = ::gemm(a, b, g.out, g.bias, g.act, g.a_mn, g.b_mn, g.want_pre, code, g.mode, g.alpha, err_, {}, 0,
                               {}, g.accumulate, {}, 0, g.epi, g.row_in, g.row_in2, g.row_out, g.aux, 0, 0);
    TORCH_CHECK(rc == 0, "tcgen05 GEMM launch failed with code ", rc);
    return {c, pre};
  }
  // act(x w^T + bias) + aux with the route of a linear layer's forward: few rows on the streaming kernel
  std::tuple<Tensor, OptTensor> linear(const Tensor& x, const Tensor& w, GemmArgs g) {
    if (x.size(0) <= mb::kSkinnyMaxRows && !g.want_pre && !(g.aux.has_value() && g.act != 0)) {
      const at::ScalarType t = g.out_type == at::ScalarType::Undefined ? x.scalar_type() : g.out_type;
      if (!g.out.has_value()) g.out = torch::empty({x.size(0), w.size(0)}, x.options().dtype(t));
      const int64_t rc = skinny_gemm({x}, {w}, {OptTensor()}, {g.bias}, {g.aux}, {g.act}, {*g.out}, false, err_, {}, 0.0);
      TORCH_CHECK(rc == 0 || rc == -1, "few-row product: launch failed with code ", rc);
      if (rc == 0) return {*g.out, OptTensor()};
    }
    return gemm(x, w, g);
  }
  Tensor err() const { return err_; }

 private:
  Tensor err_;
  long long before_;
};

// Every size that the kernels take on trust.
void check_block(const Tensor& x, const Tensor& count, const Tensor& mean, const Tensor& var, const OptTensor& hx,
                 const Tensor& p, const Params& w, const BlockDims& d, bool prior) {
  const int64_t B = x.size(0), D = x.size(2), N = p.size(1), V = d.heads * d.dv, S = d.heads * d.dk;
  auto is = [&](int i, std::vector<int64_t> shape) {
    TORCH_CHECK(w[i].has_value() && w[i]->sizes() == at::IntArrayRef(shape) && w[i]->is_contiguous(),
                "mega_block: parameter ", i, " has another shape");
  };
  auto of = [&](int i, int64_t n) {
    TORCH_CHECK(!w[i].has_value() || (w[i]->numel() == n && w[i]->is_contiguous()), "mega_block: parameter ", i, " has another size");
  };
  is(kTsnW, {D}); is(kTsnB, {D}); is(kWv, {V, D}); is(kWz, {S, D}); is(kWr, {V, D}); is(kWh1, {D, D}); is(kWh2, {D, V});
  is(kGamma, {2, S}); is(kBeta, {2, S});
  TORCH_CHECK(w[kFc1].has_value() && w[kFc1]->dim() == 2 && w[kOmega].has_value());
  const int64_t F = w[kFc1]->size(0);
  is(kFc1, {F, D}); is(kFc2, {D, F});
  if (w[kFc3].has_value()) is(kFc3, {F, D});
  of(kOmega, D); of(kRmsW, D); of(kBv, V); of(kBz, S); of(kBr, V); of(kBh1, D); of(kLnW, D); of(kLnB, D);
  const int64_t n = prior ? 1 : B;
  TORCH_CHECK(count.numel() == n && mean.numel() == n * d.groups && var.numel() == n * d.groups && p.numel() == D * N &&
              (!hx.has_value() || hx->numel() == 2 * B * D * N), "mega_block: state of another size");
  TORCH_CHECK(x.size(1) <= d.chunk || x.size(1) % d.chunk == 0, "mega_block: not a whole number of chunks");
}

Tensor heads_view(const Tensor& t) { return t.permute({0, 2, 1, 3}); }

// x [B, L, D] etc. -> {out, count, mean, var, k, v[, h]}, what the backward pass needs (empty without `keep`), launches.
// count, mean, var: the running statistics before x, or with `prior` one count, mean and log variance; hx [B, D, N, 2]; p, q, gamma: EMA coefficients (fp32, real pairs)
std::tuple<std::vector<Tensor>, Params, int64_t> mega_block_fwd(
    const Tensor& x, const Tensor& count, const Tensor& mean, const Tensor& var, const OptTensor& hx, const Tensor& p,
    const Tensor& q, const Tensor& gamma, const Tensor& freqs, const Params& w, const std::vector<int64_t>& dims,
    const std::vector<double>& eps, bool want_last, bool keep, bool prior, const Tensor& err) {
  TORCH_CHECK(w.size() == kBlockParams && x.dim() == 3 && x.numel() > 0 && !(keep && prior), "mega_block: arguments");
  c10::cuda::CUDAGuard guard(x.device());
  const BlockDims d = block_dims(dims, eps);
  check_block(x, count, mean, var, hx, p, w, d, prior);
  Launcher run(err);
  const auto T = x.scalar_type();
  const auto f32 = x.options().dtype(at::kFloat);
  const Tensor xc = x.contiguous();
  const int64_t B = xc.size(0), L = xc.size(1), D = xc.size(2), rows = B * L;
  const Tensor pm = mean.to(T).contiguous(), pv = var.to(T).contiguous();
  const std::vector<Tensor> tsn = timestep_norm_fwd_from(xc, count.contiguous(), pm, pv, *w[kTsnW], 1.0, *w[kTsnB],
                                                         OptTensor(), d.groups, d.tsn_eps, prior);
  const Tensor& t = tsn[0];
  const Tensor omega = w[kOmega]->view({D});
  const auto [ema, h] = cema_fwd_any(t, p, q, gamma, omega, hx, want_last);
  const auto [mx, mx_rstd] = rms_norm_fwd(ema, w[kRmsW], 1.0, d.rms_eps);
  const Tensor x2 = xc.view({rows, D}), t2 = t.view({rows, D}), m2 = mx.view({rows, D});

  // the projections of mx; the gate leaves as fp32 pre-activation, for few rows without gradients as its 16-bit SiLU
  const int64_t S = d.heads * d.dk, V = d.heads * d.dv;
  Tensor z = torch::empty({rows, S}, x.options()), r, hres = torch::empty({rows, D}, x.options()), v;
  OptTensor v_pre;
  bool few = rows <= mb::kSkinnyMaxRows && !keep;
  if (few) {
    r = torch::empty({rows, V}, x.options());
    v = torch::empty({rows, V}, x.options());
    const OptTensor none;
    const int64_t rc = skinny_gemm({m2, m2, m2, t2}, {*w[kWz], *w[kWr], *w[kWh1], *w[kWv]}, {none, none, none, none},
                                   {w[kBz], w[kBr], w[kBh1], w[kBv]}, {none, none, x2, none}, {0, 1, 0, 1}, {z, r, hres, v},
                                   false, err, {}, 0.0);
    TORCH_CHECK(rc == 0 || rc == -1, "few-row products: launch failed with code ", rc);
    few = rc == 0;
  }
  if (!few) {
    r = torch::empty({rows, V}, f32);
    GemmArgs gz, gr, gh;
    gz.out = z; gz.bias = w[kBz];
    gr.out = r; gr.bias = w[kBr];
    gh.out = hres; gh.bias = w[kBh1]; gh.aux = x2;
    run.linear(m2, *w[kWz], gz);
    run.linear(m2, *w[kWr], gr);
    run.linear(m2, *w[kWh1], gh);
  }
  const auto [zn, z_rstd] = rms_norm_fwd(z.view({rows * d.heads, d.dk}), OptTensor(), 1.0, d.z_eps);
  const Tensor zn3 = zn.view({B, L, S});
  const int64_t c = std::min(L, d.chunk), n = rows / c, ld = (c + 127) / 128 * 128;
  const Tensor rmax = torch::empty({n, d.heads, c}, f32), rsum = torch::empty({n, d.heads, c}, f32);
  const auto [qr, kr] = qk_rotary_fwd_rows(zn3, *w[kGamma], *w[kBeta], freqs, d.dk, rmax, rsum);
  if (!few) {
    GemmArgs gv;
    gv.bias = w[kBv]; gv.act = 1; gv.want_pre = keep;
    std::tie(v, v_pre) = run.linear(t2, *w[kWv], gv);
  }

  // chunk-local causal attention: scores twice (row maxima, then exponentials and row sums), P V over the row sums
  const Tensor qh = heads_view(qr.view({n, c, d.heads, d.dk})), kh = heads_view(kr.view({n, c, d.heads, d.dk}));
  const Tensor vh = heads_view(v.view({n, c, d.heads, d.dv}));
  const Tensor P = torch::empty({n, d.heads, c, ld}, x.options()), attn = torch::empty({n, c, d.heads, d.dv}, x.options());
  const Tensor Pv = P.narrow(-1, 0, c);
  GemmArgs gs;
  gs.out = Pv; gs.mode = 1; gs.epi = 1; gs.row_out = rmax;
  run.gemm(qh, kh, gs);
  gs.epi = 2; gs.row_in = rmax; gs.row_out = rsum;
  run.gemm(qh, kh, gs);
  GemmArgs go;
  go.out = heads_view(attn); go.mode = 2; go.b_mn = true; go.epi = 3; go.row_in = rsum;
  run.gemm(Pv, vh, go);

  const Tensor a2 = attn.view({rows, V});
  const Tensor gated = few ? a2 * r : swiglu_fwd(r, a2);
  GemmArgs gy;
  gy.aux = hres; gy.out = torch::empty_like(hres);
  const Tensor y = std::get<0>(run.linear(gated, *w[kWh2], gy));

  // feed-forward branch; the block's input is its residual
  const auto [f, ln_mean, ln_rstd] = layer_norm_fwd(y, w[kLnW], w[kLnB], 1.0, d.ln_eps);
  Tensor a, b, u;
  if (w[kFc3].has_value()) {
    a = std::get<0>(run.linear(f, *w[kFc1], {}));
    b = std::get<0>(run.linear(f, *w[kFc3], {}));
    u = swiglu_fwd(a, b);
  } else {
    GemmArgs g1;
    g1.act = 1; g1.want_pre = keep;
    OptTensor pre;
    std::tie(u, pre) = run.linear(f, *w[kFc1], g1);
    if (pre.has_value()) a = *pre;
  }
  GemmArgs g2;
  g2.aux = x2; g2.out = torch::empty_like(x2);
  const Tensor out = std::get<0>(run.linear(u, *w[kFc2], g2)).view({B, L, D});

  std::vector<Tensor> outs{out, tsn[1], tsn[2], tsn[3], kr, v.view({B, L, V})};
  if (h.has_value()) outs.push_back(*h);
  Params saved;
  if (keep)
    saved = {xc, pm, tsn[1], tsn[4], tsn[5], t, omega, ema, mx_rstd, mx, z, z_rstd, zn, qr, kr, v, v_pre, P, rsum, attn, r,
             gated, y, ln_mean, ln_rstd, f, a, b.defined() ? OptTensor(b) : OptTensor(), u};
  return {outs, saved, run.count()};
}

// Gradients of x, mean, var, hx, p, q, gamma (hx's also where it was absent) and of the parameters, and the launches.
// sinks: for a weight matrix the place of its gradient, written or (adds) added to, which leaves none to return.
std::tuple<Params, int64_t> mega_block_bwd(const Tensor& dout, const OptTensor& dmean, const OptTensor& dvar,
                                           const OptTensor& dh, const Params& saved, const OptTensor& hx, const Tensor& p,
                                           const Tensor& q, const Tensor& gamma, const Tensor& freqs, const Params& w,
                                           const Params& sinks, const std::vector<bool>& adds,
                                           const std::vector<int64_t>& dims, const std::vector<double>& eps,
                                           const Tensor& err) {
  TORCH_CHECK(w.size() == kBlockParams && sinks.size() == kBlockParams && adds.size() == kBlockParams && saved.size() == 29,
              "mega_block: arguments");
  c10::cuda::CUDAGuard guard(dout.device());
  const BlockDims d = block_dims(dims, eps);
  Launcher run(err);
  int at = 0;
  auto next = [&]() -> const Tensor& { return *saved[at++]; };
  const Tensor &x = next(), &pm = next(), &count = next(), &cummean = next(), &cumrstd = next(), &t = next();
  const Tensor &omega = next(), &ema = next(), &mx_rstd = next(), &mx = next(), &z = next(), &z_rstd = next();
  const Tensor &zn = next(), &qr = next(), &kr = next(), &v = next(), &v_pre = next(), &P = next(), &rsum = next();
  const Tensor &attn = next(), &r = next(), &gated = next(), &y = next(), &ln_mean = next(), &ln_rstd = next();
  const Tensor &f = next(), &a = next();
  const OptTensor& b = saved[at++];
  const Tensor& u = next();
  const auto T = x.scalar_type();
  const int64_t B = x.size(0), L = x.size(1), D = x.size(2), rows = B * L, S = d.heads * d.dk, V = d.heads * d.dv;
  const Tensor t2 = t.view({rows, D}), m2 = mx.view({rows, D});
  Params dw(kBlockParams);

  auto weight_grad = [&](int i, const Tensor& g, const Tensor& in) {     // g^T in
    GemmArgs a;
    a.a_mn = a.b_mn = true;
    a.out = sinks[i]; a.accumulate = sinks[i].has_value() && adds[i];
    const Tensor res = std::get<0>(run.gemm(g, in, a));
    if (!sinks[i].has_value()) dw[i] = res;
  };
  auto input_grad = [&](const Tensor& g, int i, const OptTensor& onto) {  // g w, added to `onto`
    GemmArgs a;
    a.b_mn = true;
    a.out = onto; a.accumulate = onto.has_value();
    return std::get<0>(run.gemm(g, *w[i], a));
  };
  auto bias_grad = [&](int i, const Tensor& g) {
    if (!w[i].has_value()) return;
    dw[i] = colsum(g, dtype_code(*w[i]));
  };

  // feed-forward branch
  const Tensor g = dout.reshape({rows, D}).contiguous();
  const Tensor du = input_grad(g, kFc2, {});
  weight_grad(kFc2, g, u);
  Tensor df;
  if (b.has_value()) {
    const auto [da, db] = swiglu_bwd(du, a, *b);
    df = input_grad(da, kFc1, {});
    input_grad(db, kFc3, df);
    weight_grad(kFc1, da, f);
    weight_grad(kFc3, db, f);
  } else {
    const Tensor da = silu_bwd(du, a);
    df = input_grad(da, kFc1, {});
    weight_grad(kFc1, da, f);
  }
  const auto [dy, dlnw, dlnb] = layer_norm_bwd(df, y, w[kLnW], 1.0, ln_mean, ln_rstd);
  dw[kLnW] = dlnw;
  if (w[kLnB].has_value()) dw[kLnB] = dlnb;

  // gate and attention
  const Tensor dgated = input_grad(dy, kWh2, {});
  weight_grad(kWh2, dy, gated);
  const auto [dr, dattn] = swiglu_bwd(dgated, r, attn.view({rows, V}));
  const int64_t n = attn.size(0), c = attn.size(1);
  const Tensor q4 = qr.view({n, c, d.heads, d.dk}), k4 = kr.view({n, c, d.heads, d.dk}), v4 = v.view({n, c, d.heads, d.dv});
  const Tensor do4 = dattn.view({n, c, d.heads, d.dv});
  const Tensor dq = torch::empty_like(q4), dk = torch::empty_like(k4), dv = torch::empty_like(v4);
  const auto [dos, delta] = attn_bwd_prep(do4, attn, rsum);
  const Tensor Pv = P.narrow(-1, 0, c);
  {
    GemmArgs a;
    a.out = heads_view(dv); a.mode = 3; a.a_mn = a.b_mn = true;
    run.gemm(Pv, heads_view(dos), a);
    // dS in memory of its own: a graph that is kept is walked again, and then wants the probabilities
    const Tensor dS = torch::empty_like(P).narrow(-1, 0, c);
    GemmArgs s;
    s.out = dS; s.mode = 1; s.epi = 4; s.row_in = rsum; s.row_in2 = delta; s.aux = Pv;
    run.gemm(heads_view(do4), heads_view(v4), s);
    GemmArgs qg;
    qg.out = heads_view(dq); qg.mode = 2; qg.b_mn = true;
    run.gemm(dS, heads_view(k4), qg);
    GemmArgs kg;
    kg.out = heads_view(dk); kg.mode = 3; kg.a_mn = kg.b_mn = true;
    run.gemm(dS, heads_view(q4), kg);
  }
  const Tensor gv = silu_bwd(dv.view({rows, V}), v_pre);
  weight_grad(kWv, gv, t2);
  bias_grad(kBv, gv);
  const auto [dzn, dgamma, dbeta] = qk_rotary_bwd(dq.view({B, L, S}), dk.view({B, L, S}), zn.view({B, L, S}), *w[kGamma],
                                                  freqs, d.dk);
  dw[kGamma] = dgamma.to(w[kGamma]->scalar_type());
  dw[kBeta] = dbeta.to(w[kBeta]->scalar_type());
  const Tensor dz = std::get<0>(rms_norm_bwd(dzn.view({rows * d.heads, d.dk}), z.view({rows * d.heads, d.dk}), OptTensor(),
                                             1.0, z_rstd)).view({rows, S});

  // projections of mx
  const Tensor dmx = input_grad(dz, kWz, {});
  input_grad(dr, kWr, dmx);
  input_grad(dy, kWh1, dmx);
  weight_grad(kWz, dz, m2);
  weight_grad(kWr, dr, m2);
  weight_grad(kWh1, dy, m2);
  bias_grad(kBz, dz);
  bias_grad(kBr, dr);
  bias_grad(kBh1, dy);

  // norms and EMA
  const auto [dema, drms] = rms_norm_bwd(dmx.view({B, L, D}), ema, w[kRmsW], 1.0, mx_rstd);
  dw[kRmsW] = drms;
  const std::vector<Tensor> ce = cema_bwd_any(dema, t, p, q, gamma, omega, hx, dh);
  dw[kOmega] = ce[4].view(w[kOmega]->sizes()).to(w[kOmega]->scalar_type());
  const Tensor dt = ce[0];
  input_grad(gv, kWv, dt.view({rows, D}));
  const auto stat = [&](const OptTensor& s) { return s.has_value() ? OptTensor(s->to(T).contiguous()) : s; };
  const std::vector<Tensor> ts = timestep_norm_bwd(dt, stat(dmean), stat(dvar), x, pm, count, cummean, cumrstd, *w[kTsnW],
                                                   1.0, OptTensor(), d.groups);
  dw[kTsnW] = ts[3];
  dw[kTsnB] = ts[4];
  // both residual additions hand their gradient on
  const Tensor dx = ts[0];
  mb::add_two(dx.data_ptr(), dy.data_ptr(), g.data_ptr(), dx.numel(), dtype_code(dx), stream());

  Params out{dx, ts[1], ts[2], ce[5], ce[1], ce[2], ce[3]};
  out.insert(out.end(), dw.begin(), dw.end());
  return {out, run.count()};
}
