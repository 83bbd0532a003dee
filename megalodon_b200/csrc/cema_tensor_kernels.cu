// Forward complex EMA on the tensor cores (bf16 activations, 16 states), one pass over the sequence.
//
// The scan of cema_kernels.cu spends ten FMAs per state and step, and its FMA pipes bound it.  Over chunks of 16 steps
// the same recurrence is three small products per feature, with x exact in 16 bits:
//
//   S = X E      [16 chunks x 16 steps] x [16 x 32]   what a chunk adds to the state: E = p q^(15 - step), re and im
//   H            state before each chunk: H <- q^16 H + S, a scan over 16 chunks in registers, fp32 (a thread has two
//                adjacent chunks of four states, so three exchanges across the warp do)
//   Y = X K + H F                                     K: the causal kernel Re sum gamma p q^(j - i) (omega on its
//                                                     diagonal), F: gamma q^(step + 1)
//
// A warp has one feature, whose E, K and F stay in its registers; a CTA has 16 features and walks the sequence in tiles
// of 256 steps, so there are no segments, no second pass and no combination between them.  Nothing is held or multiplied
// in fewer than 24 bits: an fp32 factor is the sum of three bf16 parts (x needs one; of H F the six products above
// 2^-24 are taken), products and sums are fp32.  Against the recurrence in 64 bits, 16-bit results rounded the other way
// and the last state's relative error: 1.5e-4 and 5.7e-8 (scan), 1.1e-4 and 4.8e-8 (this) after 1000 steps, 9.7e-5 and
// 5.9e-8, 7.1e-5 and 5.0e-8 after 8192.
//
// Tiles lie in shared memory feature by feature, which makes a lane's share of a fragment 8 contiguous bytes: the places
// of a fragment along the contraction, and the columns of the result, are dealt out as steps 4 t .. 4 t + 3 of thread t.
//
// A tile of a feature with infinities or NaN, and all of one whose powers overflow, takes the recurrence step by step: in
// the products a zero of K times an infinity would reach back in time.
//
// us, scan / this (B x L x D): 1 x 300 x 1024 35 / 12, 8 x 777 x 1024 88 / 52, 1 x 907 x 2048 39 / 18, 2 x 2048 x 2048
// 97 / 53, 1 x 4096 x 4096 169 / 104, 1 x 16384 x 4096 586 / 376.  What bounds it is latency: sixteen warps fill an SM's
// registers (128 a thread), a scheduler issues in 48 % of the cycles, the tensor pipe is busy in 24 %, the wavefronts of
// shared memory in 39 %.  Setting a warp up takes some 5 us, a tile 2.9.
#include "common.cuh"
#include "kernels.h"

namespace mb {
namespace {

constexpr int kFeat = 16;                 // features, and warps, of a CTA
constexpr int kSteps = 256;               // steps of a tile: 16 chunks of 16
constexpr int kPitch = kSteps + 4;        // elements between features: a half-warp's two octets fall into different banks
constexpr int kStates = 16;

// An fp32 value and what its rounding left: some 48 bits.  (Doubles would do, but not their conversions: 16 lanes a cycle.)
struct ff {
  float h, l;
};
struct cff {
  ff re, im;
};
struct WarpTables {
  cff pow[17][kStates + 1];               // q^l (rows apart by a bank group)
  cff tile[kStates];                      // q^256
  float2 hop[4][kStates];                 // q^16, q^32, q^64, q^128
  float2 pair[8][kStates];                // q^(32 g)
  float2 state[kStates], q[kStates], gamma[kStates];
  float p[kStates];
  ff kern[16];
};
struct __align__(16) Smem {
  __nv_bfloat16 x[2][kFeat][kPitch];      // inputs, replaced by the outputs
  WarpTables t[kFeat];
};

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// a, b as sums of three bf16 parts
__device__ __forceinline__ void split3(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = pack_bf16(a, b);
  a -= __uint_as_float(p0 << 16);
  b -= __uint_as_float(p0 & 0xffff0000u);
  p1 = pack_bf16(a, b);
  p2 = pack_bf16(a - __uint_as_float(p1 << 16), b - __uint_as_float(p1 & 0xffff0000u));
}
__device__ __forceinline__ void split3(ff a, ff b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {     // (the third with .l)
  split3(a.h, b.h, p0, p1, p2);
  p2 = pack_bf16(a.h - __uint_as_float(p0 << 16) - __uint_as_float(p1 << 16) + a.l,
                 b.h - __uint_as_float(p0 & 0xffff0000u) - __uint_as_float(p1 & 0xffff0000u) + b.l);
}
// Sums and products without loss (Knuth's and Dekker's, the latter with a fused multiply-add); the intrinsics keep the
// compiler from contracting
__device__ __forceinline__ ff two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), v = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v))};
}
__device__ __forceinline__ ff join(ff a, float e) {
  const float h = __fadd_rn(a.h, __fadd_rn(a.l, e));
  return {h, __fadd_rn(__fadd_rn(a.l, e), __fsub_rn(a.h, h))};
}
__device__ __forceinline__ ff mul(ff a, ff b) {
  const float p = __fmul_rn(a.h, b.h);
  return {p, fmaf(a.h, b.l, fmaf(a.l, b.h, fmaf(a.h, b.h, -p)))};
}
__device__ __forceinline__ ff add(ff a, ff b) { return join(two_sum(a.h, b.h), __fadd_rn(a.l, b.l)); }
__device__ __forceinline__ cff cmul(cff a, cff b) {
  const ff t = mul(a.im, b.im);
  return {add(mul(a.re, b.re), {-t.h, -t.l}), add(mul(a.re, b.im), mul(a.im, b.re))};
}
// Re and Im of a z, rounded once
__device__ __forceinline__ float2 cmul_rounded(float2 a, cff z) {
  const float u = a.y * z.im.h, v = a.y * z.re.h;
  const float ul = fmaf(a.x, z.re.l, fmaf(-a.y, z.im.l, -fmaf(a.y, z.im.h, -u)));
  const float vl = fmaf(a.x, z.im.l, fmaf(a.y, z.re.l, fmaf(a.y, z.re.h, -v)));
  const float p = a.x * z.re.h, r = a.x * z.im.h;
  const ff re = two_sum(p, -u), im = two_sum(r, v);
  return make_float2(re.h + (re.l + (ul + fmaf(a.x, z.re.h, -p))), im.h + (im.l + (vl + fmaf(a.x, z.im.h, -r))));
}
__device__ __forceinline__ cff widen(float2 z) { return {{z.x, 0.f}, {z.y, 0.f}}; }
__device__ __forceinline__ float2 rounded(cff z) { return make_float2(z.re.h, z.im.h); }
__device__ __forceinline__ float2 cmul2(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// z += q s
__device__ __forceinline__ void cfma(float& re, float& im, float2 q, float sr, float si) {
  re = fmaf(q.x, sr, fmaf(-q.y, si, re));
  im = fmaf(q.x, si, fmaf(q.y, sr, im));
}
__device__ __forceinline__ bool odd_bf16(uint32_t w) {       // an infinity or NaN in either half
  return (w & 0x7f80u) == 0x7f80u || (w & 0x7f800000u) == 0x7f800000u;
}

__global__ void __launch_bounds__(kFeat * 32, 1)
cema_fwd_tensor_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ p, const float2* __restrict__ q,
                       const float2* __restrict__ gamma, const OmegaRef omega, const float2* __restrict__ hx,
                       __nv_bfloat16* __restrict__ y, float2* __restrict__ h_last, int B, int L, int D, int per) {
  begin_dependent();
  extern __shared__ uint8_t raw[];
  Smem& sm = *reinterpret_cast<Smem*>(raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int f0 = blockIdx.x * kFeat, b0 = blockIdx.y * per, tiles = (L + kSteps - 1) / kSteps;
  const int all = tiles * min(per, B - b0);               // tiles of this CTA: sequences b0, b0 + 1, ... one after another
  const bool live = f0 + warp < D;
  const int d = live ? f0 + warp : D - 1;
  const float om = load_any(omega.p, omega.dtype, d);
  WarpTables& tb = sm.t[warp];
  const float2 *qd = tb.q, *gd = tb.gamma;
  const float* pd = tb.p;

  // this thread's piece of a tile: eight features of one step
  const int oct = lane & 1, step = warp * 16 + (lane >> 1);
  const bool has = f0 + 8 * oct < D;
  struct Place {                     // of that piece, from tile to tile
    int s;
    long long i;
  };
  const long long first = ((long long)b0 * L + step) * D + f0 + 8 * oct, skip = (long long)(L - tiles * kSteps) * D;
  Place from{step, first}, to = from;
  auto advance = [&](Place& p) {
    p.s += kSteps;
    p.i += (long long)kSteps * D;
    if (p.s >= tiles * kSteps) {
      p.s = step;
      p.i += skip;
    }
  };
  auto load = [&]() {
    const uint4 v = has && from.s < L ? *reinterpret_cast<const uint4*>(x + from.i) : make_uint4(0u, 0u, 0u, 0u);
    advance(from);
    return v;
  };
  auto put = [&](int k, const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
      reinterpret_cast<unsigned short&>(sm.x[k & 1][8 * oct + i][step]) = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
  };
  auto store = [&](int k) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = (uint32_t) reinterpret_cast<const unsigned short&>(sm.x[k & 1][8 * oct + 2 * i][step]) |
             (uint32_t) reinterpret_cast<const unsigned short&>(sm.x[k & 1][8 * oct + 2 * i + 1][step]) << 16;
    if (has && to.s < L) *reinterpret_cast<uint4*>(y + to.i) = make_uint4(w[0], w[1], w[2], w[3]);
    advance(to);
  };
  uint4 next = load();
  float H0[4][2];                 // state before the tile, states 4 j + t
  auto start = [&](int b) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 z = hx != nullptr ? hx[((long long)b * D + d) * kStates + 4 * j + t] : make_float2(0.f, 0.f);
      H0[j][0] = z.x;
      H0[j][1] = z.y;
    }
  };
  start(b0);

  // ---------------------------------------------------------------- fragments of E, K and F
  // Powers and what is made of them carry some 48 bits: a factor that is off is off by the same amount in every chunk,
  // which adds up over a long memory where the scan's roundings average out.  Half of the warp makes q^0 .. q^8, the
  // other q^8 .. q^16.
  const int n16 = lane & 15, upper = lane >> 4;
  bool overflow;
  {
    const float2 q0 = q[d * kStates + n16], g0 = gamma[d * kStates + n16];
    tb.p[n16] = p[d * kStates + n16];
    tb.q[n16] = q0;
    tb.gamma[n16] = g0;
    const cff qq = widen(q0);
    cff z = {{1.f, 0.f}, {0.f, 0.f}};
    if (upper) {
      z = cmul(qq, qq);
      z = cmul(z, z);
      z = cmul(z, z);
    }
#pragma unroll 1
    for (int l = 0; l < 8; ++l) {
      tb.pow[8 * upper + l][n16] = z;
      z = cmul(z, qq);
    }
    if (upper) tb.pow[16][n16] = z;
  }
  __syncwarp();
  {
    const cff q16 = tb.pow[16][n16], q32 = cmul(q16, q16), q64 = cmul(q32, q32), q128 = cmul(q64, q64);
    // pair[2 i], pair[2 i + 1] for i = 0, 1 of one half, 2, 3 of the other
    const cff one = {{1.f, 0.f}, {0.f, 0.f}}, four = upper ? q128 : one, six = cmul(four, q64);
    tb.pair[4 * upper][n16] = rounded(four);
    tb.pair[4 * upper + 1][n16] = rounded(cmul(four, q32));
    tb.pair[4 * upper + 2][n16] = rounded(six);
    tb.pair[4 * upper + 3][n16] = rounded(cmul(six, q32));
    tb.hop[2 * upper][n16] = rounded(upper ? q64 : q16);
    tb.hop[2 * upper + 1][n16] = rounded(upper ? q128 : q32);
    const cff q256 = cmul(q128, q128);
    if (upper) tb.tile[n16] = q256;
    overflow = __any_sync(0xffffffffu, !isfinite(q256.re.h) || !isfinite(q256.im.h));
    // k_l for l = n16, half of the states each
    ff k = {upper == 0 && n16 == 0 ? om : 0.f, 0.f};
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      const int n = 8 * upper + i;
      k = add(k, mul({pd[n], 0.f}, {cmul_rounded(gd[n], tb.pow[n16][n]).x, 0.f}));
    }
    const ff other = {__shfl_xor_sync(0xffffffffu, k.h, 16), __shfl_xor_sync(0xffffffffu, k.l, 16)};
    if (!upper) tb.kern[n16] = add(k, other);
  }
  __syncwarp();
  uint32_t E[4][3][2], K[2][3][2], F[2][2][3][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = 4 * j + (g >> 1);
    const ff pn = {pd[n], 0.f};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const cff &z0 = tb.pow[15 - 4 * t - 2 * i][n], &z1 = tb.pow[14 - 4 * t - 2 * i][n];
      split3(mul(pn, (g & 1) ? z0.im : z0.re), mul(pn, (g & 1) ? z1.im : z1.re), E[j][0][i], E[j][1][i], E[j][2][i]);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int at = 4 * (g >> 1) + (g & 1) + 2 * u;          // step of column g of result tile u
    auto lag = [&](int i) { return at >= 4 * t + i ? tb.kern[max(at - 4 * t - i, 0)] : ff{0.f, 0.f}; };
#pragma unroll
    for (int i = 0; i < 2; ++i) split3(lag(2 * i), lag(2 * i + 1), K[u][0][i], K[u][1][i], K[u][2][i]);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int n = 8 * s + 4 * i + t;
        const float2 z = cmul_rounded(gd[n], tb.pow[at + 1][n]);
        split3(z.x, -z.y, F[s][u][0][i], F[s][u][1][i], F[s][u][2][i]);
      }
    }
  }

  // One barrier a tile: a thread takes the outputs of tile k - 1 from where it then puts the inputs of tile k + 1.
  put(0, next);
  if (all > 1) next = load();
  int b = b0, seq_k = 0;          // the tile's sequence, its number there
  for (int k = 0; k < all; ++k) {
    __syncthreads();
    if (k > 0) store(k - 1);
    if (k + 1 < all) put(k + 1, next);
    if (k + 2 < all) next = load();
    const int valid = min(kSteps, L - seq_k * kSteps);
    __nv_bfloat16* row = sm.x[k & 1][warp];
    uint2* plo = reinterpret_cast<uint2*>(row + 32 * g + 4 * t);            // chunk 2 g
    uint2* phi = reinterpret_cast<uint2*>(row + 32 * g + 16 + 4 * t);       // chunk 2 g + 1
    const uint2 lo = *plo, hi = *phi;
    bool odd = overflow || odd_bf16(lo.x) || odd_bf16(lo.y) || odd_bf16(hi.x) || odd_bf16(hi.y);
#pragma unroll
    for (int j = 0; j < 4; ++j) odd = odd || !isfinite(H0[j][0]) || !isfinite(H0[j][1]);
    if (!__any_sync(0xffffffffu, odd)) {
      const uint32_t a[4] = {lo.x, hi.x, lo.y, hi.y};
      float S[4][4], Y[2][4], Z[2][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) S[j][i] = 0.f;
#pragma unroll
        for (int r = 2; r >= 0; --r) mma(S[j], a, E[j][r]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int i = 0; i < 4; ++i) Y[u][i] = Z[u][i] = 0.f;
#pragma unroll
        for (int r = 2; r >= 0; --r) mma(Y[u], a, K[u][r]);
      }
      // S[j][0..1], S[j][2..3]: what chunks 2 g and 2 g + 1 add to state 4 j + t
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = 4 * j + t;
        const float2 q16 = tb.hop[0][n];
        float wr = S[j][2], wi = S[j][3];                        // both chunks together, then all up to them
        cfma(wr, wi, q16, S[j][0], S[j][1]);
#pragma unroll
        for (int lev = 0; lev < 3; ++lev) {
          const float sr = __shfl_up_sync(0xffffffffu, wr, 4 << lev), si = __shfl_up_sync(0xffffffffu, wi, 4 << lev);
          if (g >= 1 << lev) cfma(wr, wi, tb.hop[lev + 1][n], sr, si);
        }
        float br = __shfl_up_sync(0xffffffffu, wr, 4), bi = __shfl_up_sync(0xffffffffu, wi, 4);
        float er = __shfl_sync(0xffffffffu, wr, 28 + t), ei = __shfl_sync(0xffffffffu, wi, 28 + t);
        if (g == 0) br = bi = 0.f;
        cfma(br, bi, tb.pair[g][n], H0[j][0], H0[j][1]);         // before chunk 2 g
        S[j][2] = S[j][0];
        S[j][3] = S[j][1];
        cfma(S[j][2], S[j][3], q16, br, bi);                     // before chunk 2 g + 1
        S[j][0] = br;
        S[j][1] = bi;
        const cff q256 = tb.tile[n];
        cfma(er, ei, make_float2(q256.re.l, q256.im.l), H0[j][0], H0[j][1]);
        cfma(er, ei, make_float2(q256.re.h, q256.im.h), H0[j][0], H0[j][1]);
        H0[j][0] = er;
        H0[j][1] = ei;
      }
      if (h_last != nullptr && seq_k == tiles - 1) {
        // the state after the last step: that before its chunk, and the chunk's steps one by one
        const int c = (valid - 1) / 16, rest = valid - 16 * c;
        if (g == c / 2) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tb.state[4 * j + t] = c % 2 == 0 ? make_float2(S[j][0], S[j][1]) : make_float2(S[j][2], S[j][3]);
        }
        __syncwarp();
        if (lane < kStates && live) {
          float2 z = tb.state[lane];
          const float2 qq = qd[lane];
          const float pn = pd[lane];
          for (int i = 0; i < rest; ++i) {
            const float xv = __bfloat162float(row[16 * c + i]);
            z = cmul2(qq, z);
            z.x = fmaf(pn, xv, z.x);
          }
          h_last[((long long)b * D + d) * kStates + lane] = z;
        }
        __syncwarp();
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        uint32_t h[3][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          split3(S[2 * s + i][0], S[2 * s + i][1], h[0][2 * i], h[1][2 * i], h[2][2 * i]);
          split3(S[2 * s + i][2], S[2 * s + i][3], h[0][2 * i + 1], h[1][2 * i + 1], h[2][2 * i + 1]);
        }
        // (two chains of sums: the small products and the large ones)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          mma(Z[u], h[2], F[s][u][0]);
          mma(Y[u], h[1], F[s][u][0]);
          mma(Z[u], h[0], F[s][u][2]);
          mma(Y[u], h[0], F[s][u][1]);
          mma(Z[u], h[1], F[s][u][1]);
          mma(Y[u], h[0], F[s][u][0]);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int i = 0; i < 4; ++i) Y[u][i] += Z[u][i];
      }
      *plo = make_uint2(pack_bf16(Y[0][0], Y[0][1]), pack_bf16(Y[1][0], Y[1][1]));
      *phi = make_uint2(pack_bf16(Y[0][2], Y[0][3]), pack_bf16(Y[1][2], Y[1][3]));
    } else {
      // step by step, a state a lane (both halves of the warp alike)
      if (g == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) tb.state[4 * j + t] = make_float2(H0[j][0], H0[j][1]);
      }
      __syncwarp();
      const int n = lane & 15;
      float2 z = tb.state[n];
      const float2 qq = qd[n], c = gd[n];
      const float pn = pd[n];
#pragma unroll 1
      for (int i = 0; i < valid; ++i) {
        const float xv = __bfloat162float(row[i]);
        z = cmul2(qq, z);
        z.x = fmaf(pn, xv, z.x);
        const float out = subwarp_sum<16>(fmaf(c.x, z.x, -c.y * z.y)) + om * xv;
        __syncwarp();
        if (lane == 0) row[i] = __float2bfloat16_rn(out);
      }
      __syncwarp();
      if (lane < 16) tb.state[n] = z;
      if (h_last != nullptr && seq_k == tiles - 1 && lane < 16 && live)
        h_last[((long long)b * D + d) * kStates + n] = z;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 s = tb.state[4 * j + t];
        H0[j][0] = s.x;
        H0[j][1] = s.y;
      }
    }
    if (++seq_k == tiles && k + 1 < all) {
      seq_k = 0;
      start(++b);
    }
  }
  __syncthreads();
  store(all - 1);
}

}  // namespace

// Sequences of a CTA; 0 where the scan is the faster one.  That is where few features have a long sequence, which only the
// scan divides: 16384 x 1024 167 us there, 185 here; 16384 x 512 109 and 184; 4096 x 1024 64 and 51; 2048 x 512 41 and 28.
// The lines in between: the scan takes 32 us and 8 for a million elements, or in one pass (up to 128 steps) 7.5 and 0.13 a
// step, this 5 and 2.85 a tile of 256 steps for every wave of CTAs.  One pass, scan / this: 1 x 2 x 1024 7.6 / 9.0 us,
// 1 x 37 x 1024 12.3 / 9.0, 4 x 128 x 1024 23.9 / 12.3, 16 x 128 x 1024 24.4 / 30.6, 128 x 100 x 128 20.9 / 28.6.  A CTA has 16 features of as many sequences as make that least: it is set up once for all of them, and
// waves are filled better (8 x 777 x 1024 67 -> 52 us, 2 x 2048 x 2048 57 -> 53, 32 x 1000 x 1024 240 -> 196; of one sequence
// each, 1 % the slower for the bookkeeping).
int cema_tensor_plan(int B, int L, int D, int sms) {
  const int groups = div_up(D, kFeat), tiles = div_up(L, kSteps);
  int per = 1;
  double us = 1e30;
  for (int n = 1; n <= B;) {                      // n sequences a CTA, the fewest that make so many CTAs
    const int ctas = div_up(B, n);
    const double t = div_up((long long)groups * ctas, sms) * (5.0 + 2.85 * tiles * n);
    if (t < us) us = t, per = n;
    n = ctas == 1 ? B + 1 : (B - 1) / (ctas - 1) + 1;
  }
  return us > (L <= kCemaSegLen ? 7.5 + 0.13 * L : 32.0 + 8e-6 * B * L * D) ? 0 : per;
}

// y (and h_last, if given) of the EMA; false where the scan is to run
bool cema_fwd_tensor(const void* x, const float* p, const float* q, const float* gamma, OmegaRef omega, const float* hx,
                     void* y, float* h_last, int B, int L, int D, int N, int x_dtype, cudaStream_t st) {
  if (N != kStates || x_dtype != kBF16 || D % 8 != 0 || L < 1 || B < 1 || B > 65535 || !aligned16(x) || !aligned16(y))
    return false;
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  const int groups = div_up(D, kFeat), per = cema_tensor_plan(B, L, D, sms);
  if (per == 0) return false;
  static std::atomic<unsigned long long> configured{0};
  if (!allow_dynamic_smem(cema_fwd_tensor_kernel, sizeof(Smem), configured)) return false;
  launch_dependent(cema_fwd_tensor_kernel, dim3(groups, div_up(B, per)), dim3(kFeat * 32), sizeof(Smem), st,
                   (const __nv_bfloat16*)x, p, (const float2*)q, (const float2*)gamma, omega, (const float2*)hx,
                   (__nv_bfloat16*)y, (float2*)h_last, B, L, D, per);
  return true;
}

}  // namespace mb
