// One token through a MEGA block with a fixed-shape state: everything between the matrix products.
//
//   decode_norm_ema   TimestepNorm step -> complex-EMA step -> RMSNorm, state updated in place
//   decode_attend     per-head RMSNorm of z, query / key affine and rotary, key / value appended to the
//                     buffers, attention of one query over the filled slots split over the keys
//   decode_combine    the partial results of the splits put together, times the gate
//   decode_layer_norm LayerNorm of the feed-forward branch
//
// A step is bound by its chain of launches, not by bytes: per layer these four and four products
// (skinny_gemm.cu) replace some thirty-five launches.  All of them are written as links of a programmatic
// dependent launch chain: `pdl_wait` before the first access to anything another kernel writes.
#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace mb {
namespace {

using namespace ptx;

constexpr int kDecThreads = 256;

// ---------------------------------------------------------------- TimestepNorm + EMA + RMSNorm
// A cluster of `cl` CTAs shares one row: every CTA owns G / cl whole groups and their D / cl features, so only
// the sum of squares of the RMSNorm crosses CTAs (through distributed shared memory).  The EMA state is the
// bulk of the traffic (8 N bytes a feature read and written, 20 N bytes of coefficients): a thread owns two
// states (16 bytes of h, q and gamma each), the N / 2 threads of a feature add up with shuffles.
template <typename T, int THREADS>
__global__ void __launch_bounds__(THREADS)
decode_norm_ema_kernel(const __grid_constant__ DecodeNormEma p, int cl) {
  extern __shared__ float sm[];
  __shared__ float scratch[32];
  __shared__ float csum[8];
  if (cl > 1) cluster_arrive();    // awaited before the first store into another CTA: by then all have started
  const int rank = blockIdx.x % cl, b = blockIdx.x / cl;
  const int dl = p.D / cl, gl = p.G / cl, gs = p.D / p.G;
  float* xs = sm;                 // dl: input, later the EMA output
  float* ts = xs + dl;            // dl: normalised input as the products see it
  float* gm = ts + dl;            // gl means, gl reciprocal deviations
  float* gr = gm + gl;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row0 = (long long)b * p.D + rank * dl;
  // State and statistics were last written, and the coefficients computed, before the first link of the chain, which
  // waits for everything ahead of it (the caller launches nothing that writes them between two links): the first items'
  // are loaded and the rest requested in L2 while the predecessor finishes.
  const int per = p.N / 2;         // threads of a feature
  const int total = p.hx != nullptr ? dl * per : 0;
  constexpr int kBatch = 4;        // items of a thread whose loads are in flight together
  const long long c0 = (long long)rank * dl * per;           // first item of this CTA
  float4* hx = reinterpret_cast<float4*>(p.hx) + (long long)b * p.D * per + c0;
  float4 h[kBatch], q[kBatch], ga[kBatch];
  float2 pp[kBatch];
  auto load_items = [&](int base) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = base + u * THREADS + threadIdx.x;
      if (i < total) {
        h[u] = hx[i];
        q[u] = __ldg(reinterpret_cast<const float4*>(p.q) + c0 + i);
        ga[u] = __ldg(reinterpret_cast<const float4*>(p.gamma) + c0 + i);
        pp[u] = __ldg(reinterpret_cast<const float2*>(p.p) + c0 + i);
      }
    }
  };
  load_items(0);
  for (int i = kBatch * THREADS + threadIdx.x * 8; i < total; i += THREADS * 8) {     // 8 items: 128 bytes
    asm volatile("prefetch.global.L2 [%0];" ::"l"(hx + i));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float4*>(p.q) + c0 + i));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float4*>(p.gamma) + c0 + i));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float2*>(p.p) + c0 + i));
  }
  const double n0 = (double)p.count[b];
  float u_old = 0.f, v_old = 0.f;                             // of this warp's first group
  if (warp < gl) {
    u_old = p.mean[(long long)b * p.G + rank * gl + warp];
    v_old = p.var[(long long)b * p.G + rank * gl + warp];
  }
  pdl_wait();
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < dl; i += THREADS) xs[i] = to_f(reinterpret_cast<const T*>(p.x)[row0 + i]);
  __syncthreads();
  for (int g = warp; g < gl; g += THREADS / 32) {
    float s = 0.f;
    for (int i = lane; i < gs; i += 32) s += xs[g * gs + i];
    const float u = warp_sum(s) / gs;
    float v = 0.f;
    for (int i = lane; i < gs; i += 32) {
      const float d = xs[g * gs + i] - u;
      v = fmaf(d, d, v);
    }
    v = warp_sum(v) / gs;
    if (lane == 0) {
      // the group's features are one sample of weight one, merged into the running population
      const long long gi = (long long)b * p.G + rank * gl + g;
      const double u0 = g == warp ? u_old : p.mean[gi], v0 = g == warp ? v_old : p.var[gi], ud = u;
      const double mean = (n0 * u0 + ud) / (n0 + 1.0);
      const double var = fmax((n0 * (v0 + u0 * u0) + ((double)v + ud * ud)) / (n0 + 1.0) - mean * mean, 0.0);
      p.mean[gi] = (float)mean;
      p.var[gi] = (float)var;
      gm[g] = (float)mean;
      gr[g] = rsqrtf((float)var + p.eps);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < dl; i += THREADS) {
    const int f = rank * dl + i, g = i / gs;
    const T t = from_f<T>((xs[i] - gm[g]) * gr[g] * (to_f(reinterpret_cast<const T*>(p.w)[f]) + 1.f) +
                          to_f(reinterpret_cast<const T*>(p.b)[f]));
    reinterpret_cast<T*>(p.t_out)[row0 + i] = t;
    ts[i] = to_f(t);
  }
  if (p.hx == nullptr) {           // the norm alone (before the vocabulary projection)
    if (cl > 1) {
      cluster_wait();
      cluster_sync_all();          // every CTA of the row has read the count
    } else {
      __syncthreads();
    }
    if (rank == 0 && threadIdx.x == 0) {
      p.count[b] += 1;
      if (b == 0 && p.pos != nullptr) p.pos[0] = (p.pos[0] + 1) % p.chunk;
    }
    return;
  }
  __syncthreads();
  float sq = 0.f;
  for (int base = 0; base < total; base += kBatch * THREADS) {
    if (base > 0) load_items(base);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = base + u * THREADS + threadIdx.x;
      const bool on = i < total;
      const int fl = on ? i / per : 0;
      float acc = 0.f;
      const float t = ts[fl];
      if (on) {
        float4 n;
        n.x = fmaf(q[u].x, h[u].x, fmaf(-q[u].y, h[u].y, pp[u].x * t));
        n.y = fmaf(q[u].x, h[u].y, q[u].y * h[u].x);
        n.z = fmaf(q[u].z, h[u].z, fmaf(-q[u].w, h[u].w, pp[u].y * t));
        n.w = fmaf(q[u].z, h[u].w, q[u].w * h[u].z);
        hx[i] = n;
        acc = ga[u].x * n.x - ga[u].y * n.y + ga[u].z * n.z - ga[u].w * n.w;
      }
      for (int o = per / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (on && i % per == 0) {
        const float y = to_f(from_f<T>(fmaf(to_f(reinterpret_cast<const T*>(p.omega)[rank * dl + fl]), t, acc)));
        xs[fl] = y;
        sq = fmaf(y, y, sq);
      }
    }
  }
  sq = block_sum(sq, scratch);     // (its barriers also publish xs)
  if (cl > 1) {
    cluster_wait();
    if (threadIdx.x < cl) st_cluster_f32(map_to_cta(smem_u32(csum + rank), threadIdx.x), sq);
    cluster_sync_all();
    sq = 0.f;
    for (int r = 0; r < cl; ++r) sq += csum[r];
  }
  const float rstd = rsqrtf(sq / p.D + p.rms_eps);
  for (int i = threadIdx.x; i < dl; i += THREADS) {
    const int f = rank * dl + i;
    float v = xs[i] * rstd;
    if (p.rms_w != nullptr) v *= to_f(reinterpret_cast<const T*>(p.rms_w)[f]) + 1.f;
    reinterpret_cast<T*>(p.mx_out)[row0 + i] = from_f<T>(v);
  }
  if (rank == 0 && threadIdx.x == 0) p.count[b] += 1;     // every CTA of the row read it before the barrier above
}

// ---------------------------------------------------------------- attention of one query
// Keys of one (sequence, head) handled by a CTA; the same rule in both kernels.
__device__ __forceinline__ int keys_per_split(int n, int splits) { return max(8, (n + splits - 1) / splits); }

// CTA = (split, sequence x head).  A split reads its keys once (a warp per key) and its value rows once
// (16-byte pieces; eight rows in flight per thread while the eight before them are added up), and leaves max, sum and the un-normalised fp32 row.  The
// number of splits is fixed by the buffers' shape (about two CTAs per SM), the keys per split by the
// position, so the launch can sit in a CUDA graph; splits beyond the filled slots leave at once.
// Before: one CTA per 256 value columns walked all keys with 2-byte loads - 177 us at 4 heads, 1100 keys,
// d_v 2048 (18 MB of values), now 14.6 with the combination; 16 sequences of 2 heads, 700 keys (103 MB): 31.5 us
// (54.5 with eight rows in flight and nothing behind them).
// VEC: value rows of whole 16-byte pieces.  Otherwise (a width that is no multiple of 8, or a buffer that starts
// anywhere) their pieces are put together element by element; the partial rows are padded to `padded_width`.
__host__ __device__ __forceinline__ int padded_width(int dv) { return (dv + 7) & ~7; }

template <typename T, bool VEC>
__global__ void __launch_bounds__(kDecThreads, 2)
decode_attend_kernel(const __grid_constant__ DecodeAttend p) {
  extern __shared__ float sm[];
  __shared__ float scratch[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.y, b = bh / p.H, h = bh - b * p.H;
  float* qs = sm;                       // dk
  float* kn = qs + p.dk;                // dk: this token's key
  float* red = kn + p.dk;               // kDecThreads * 8: partial rows of the thread groups
  float* sc = red + kDecThreads * 8;    // scores of this split
  // In the chain `pos` and the older slots were written by launches long before the predecessor, which itself
  // waited for them: they may be read, and the split's keys and values fetched into L2, ahead of the wait - as
  // long as all of them leave room for the products' weights there (16 tokens at 1.4 MB a layer 9.0 -> 8.6 ms, at
  // 103 MB 13.9 -> 14.3 ms, hence the line between).
  if (p.z == nullptr) pdl_wait();
  const int at = (int)min(p.pos[0], (long long)p.C - 1);
  const int n = at + 1;
  const int per = keys_per_split(n, gridDim.x);
  const int lo = blockIdx.x * per, hi = min(n, lo + per);
  if (VEC && lo < hi && warp == 0 && (long long)n * gridDim.y * (p.dk + p.dv) * (long long)sizeof(T) <= (32 << 20)) {
    const T* k0 = reinterpret_cast<const T*>(p.k_buf) + ((long long)bh * p.C + lo) * p.dk;
    const T* v0 = reinterpret_cast<const T*>(p.v_buf) + ((long long)bh * p.C + lo) * p.dv;
    for (int j = lane; j < hi - lo; j += 32) {
      bulk_prefetch_l2(v0 + (long long)j * p.dv, p.dv * sizeof(T));
      bulk_prefetch_l2(k0 + (long long)j * p.dk, p.dk * sizeof(T));
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  if (lo >= hi) return;
  T* krow = reinterpret_cast<T*>(p.k_buf) + (long long)bh * p.C * p.dk;
  T* vrow = reinterpret_cast<T*>(p.v_buf) + (long long)bh * p.C * p.dv;
  const bool fused = p.z != nullptr;
  const bool mine = fused && at >= lo && at < hi;
  if (fused) {
    const T* zr = reinterpret_cast<const T*>(p.z) + (long long)bh * p.dk;
    float s = 0.f;
    for (int i = tid; i < p.dk; i += kDecThreads) {
      const float v = to_f(zr[i]);
      qs[i] = v;
      s = fmaf(v, v, s);
    }
    const float rstd = rsqrtf(block_sum(s, scratch) / p.dk + p.eps);
    const float inv = rsqrtf((float)p.dk);
    const T *ga = reinterpret_cast<const T*>(p.gamma) + h * p.dk, *be = reinterpret_cast<const T*>(p.beta) + h * p.dk;
    const int S = p.H * p.dk;
    for (int i = tid; i < p.dk / 2; i += kDecThreads) {
      const float2 f = reinterpret_cast<const float2*>(p.freqs)[(long long)at * (p.dk / 2) + i];
      const float z0 = qs[2 * i] * rstd, z1 = qs[2 * i + 1] * rstd;
      const float a0 = z0 * (to_f(ga[2 * i]) + 1.f) * inv + to_f(be[2 * i]);
      const float a1 = z1 * (to_f(ga[2 * i + 1]) + 1.f) * inv + to_f(be[2 * i + 1]);
      const float c0 = z0 * (to_f(ga[S + 2 * i]) + 1.f) * inv + to_f(be[S + 2 * i]);
      const float c1 = z1 * (to_f(ga[S + 2 * i + 1]) + 1.f) * inv + to_f(be[S + 2 * i + 1]);
      qs[2 * i] = a0 * f.x - a1 * f.y;
      qs[2 * i + 1] = a0 * f.y + a1 * f.x;
      const T k0 = from_f<T>(c0 * f.x - c1 * f.y), k1 = from_f<T>(c0 * f.y + c1 * f.x);
      kn[2 * i] = to_f(k0);
      kn[2 * i + 1] = to_f(k1);
      if (mine) {
        krow[(long long)at * p.dk + 2 * i] = k0;
        krow[(long long)at * p.dk + 2 * i + 1] = k1;
      }
    }
  } else {
    const T* qr = reinterpret_cast<const T*>(p.q) + (long long)bh * p.dk;
    for (int i = tid; i < p.dk; i += kDecThreads) qs[i] = to_f(qr[i]);
  }
  // The first value rows of the first column block are under way while the scores are computed.
  const T* vnew = fused ? reinterpret_cast<const T*>(p.v_new) + (long long)bh * p.dv : nullptr;
  const int dvp = padded_width(p.dv);
  const int ct0 = min(kDecThreads, dvp / 8), ng0 = kDecThreads / ct0, grp0 = tid / ct0;
  const int c0 = (tid - grp0 * ct0) * 8;
  auto load_rows = [&](uint4 (&raw)[8], int j0, int step, int c, bool on) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u * step;
      raw[u] = make_uint4(0u, 0u, 0u, 0u);
      if (!on || j >= hi) continue;
      const T* src = mine && j == at ? vnew + c : vrow + (long long)j * p.dv + c;
      if constexpr (VEC) {
        raw[u] = *reinterpret_cast<const uint4*>(src);
      } else {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (c + i < p.dv) w[i / 2] |= (uint32_t)reinterpret_cast<const unsigned short*>(src)[i] << (16 * (i & 1));
        raw[u] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  };
  uint4 next[8];
  load_rows(next, lo + grp0, ng0, c0, grp0 < ng0);
  __syncthreads();
  for (int j0 = lo + warp * 4; j0 < hi; j0 += kDecThreads / 32 * 4) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = lane * 8; c < p.dk; c += 256) {
      float kv[4][8];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + u;
        if (j < hi && !(mine && j == at)) load8(krow + (long long)j * p.dk + c, kv[u]);
        else {
#pragma unroll
          for (int i = 0; i < 8; ++i) kv[u][i] = mine && j == at ? kn[c + i] : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float qv = qs[c + i];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fmaf(qv, kv[u][i], acc[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float s = warp_sum(acc[u]);
      if (lane == 0 && j0 + u < hi) sc[j0 + u - lo] = s * p.scale;
    }
  }
  __syncthreads();
  float m = -INFINITY;
  for (int j = tid; j < hi - lo; j += kDecThreads) m = fmaxf(m, sc[j]);
  m = block_max(m, scratch);
  const float ref = m == -INFINITY ? 0.f : m;      // a split whose keys all have weight zero
  float sum = 0.f;
  for (int j = tid; j < hi - lo; j += kDecThreads) {
    const float e = __expf(sc[j] - ref);
    sc[j] = e;
    sum += e;
  }
  sum = block_sum(sum, scratch);
  __syncthreads();
  const long long part = (long long)bh * gridDim.x + blockIdx.x;
  if (tid == 0) reinterpret_cast<float2*>(p.part_ml)[part] = make_float2(m, sum);
  float* dst = p.part_acc + part * dvp;
  for (int col0 = 0; col0 < dvp; col0 += kDecThreads * 8) {
    const int ct = min(kDecThreads, (dvp - col0) / 8);     // threads across the columns
    const int ng = kDecThreads / ct;                        // groups of them, each every ng-th key
    const int grp = tid / ct, c = col0 + (tid - grp * ct) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (grp < ng) {
      if (col0 > 0) load_rows(next, lo + grp, ng, c, true);
      for (int j0 = lo + grp; j0 < hi; j0 += ng * 8) {
        uint4 raw[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) raw[u] = next[u];
        load_rows(next, j0 + ng * 8, ng, c, true);       // (nothing beyond the split's last key)
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = j0 + u * ng;
          if (j < hi) {
            if (VEC && mine && j == at) *reinterpret_cast<uint4*>(vrow + (long long)j * p.dv + c) = raw[u];
            float v[8];
            load8(reinterpret_cast<const T*>(&raw[u]), v);
            const float e = sc[j - lo];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = fmaf(e, v[i], acc[i]);
          }
        }
      }
    }
    if (ng == 1) {
      if (grp == 0) store8(dst + c, acc);
    } else {
      __syncthreads();
      if (grp < ng) store8(red + tid * 8, acc);
      __syncthreads();
      for (int i = tid; i < ct * 8; i += kDecThreads) {
        float s = 0.f;
        for (int g = 0; g < ng; ++g) s += red[g * ct * 8 + i];
        dst[col0 + i] = s;
      }
    }
  }
}

// out = gate * sum_s exp(m_s - m) acc_s / sum_s exp(m_s - m) l_s; CTA = 128 columns of one (sequence, head),
// 32 threads of four columns times 8 strands of splits.
template <typename T>
__global__ void __launch_bounds__(kDecThreads)
decode_combine_kernel(const __grid_constant__ DecodeAttend p, int splits) {
  __shared__ float wgt[kDecodeMaxSplits];
  __shared__ float4 red[8][32];
  const int tid = threadIdx.x, strand = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.y, c = blockIdx.x * 128 + lane * 4;
  pdl_wait();
  pdl_launch_dependents();
  // (the position of the step is still in place: it moves on after the last layer)
  const int n = (int)min(p.pos[0], (long long)p.C - 1) + 1;
  const int per = keys_per_split(n, splits);
  const int active = (n + per - 1) / per;
  if (strand == 0) {
    const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + (long long)bh * splits;
    float m = -INFINITY, l = 0.f;
    for (int s = lane; s < active; s += 32) m = fmaxf(m, ml[s].x);
    m = warp_max(m);
    for (int s = lane; s < active; s += 32) l += __expf(ml[s].x - m) * ml[s].y;
    l = warp_sum(l);
    for (int s = lane; s < active; s += 32) wgt[s] = __expf(ml[s].x - m) / l;
  }
  __syncthreads();
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  const int dvp = padded_width(p.dv);
  if (c < dvp) {
    const float* src = p.part_acc + (long long)bh * splits * dvp + c;
#pragma unroll 4
    for (int s = strand; s < active; s += 8) {
      const float4 v = *reinterpret_cast<const float4*>(src + (long long)s * dvp);
      const float w = wgt[s];
      a.x = fmaf(w, v.x, a.x); a.y = fmaf(w, v.y, a.y); a.z = fmaf(w, v.z, a.z); a.w = fmaf(w, v.w, a.w);
    }
  }
  red[strand][lane] = a;
  __syncthreads();
  if (tid < 128 && blockIdx.x * 128 + tid < p.dv) {
    float v = 0.f;
#pragma unroll
    for (int s = 0; s < 8; ++s) v += reinterpret_cast<const float*>(&red[s][0])[tid];
    const long long o = (long long)bh * p.dv + blockIdx.x * 128 + tid;
    if (p.gate != nullptr) v *= to_f(reinterpret_cast<const T*>(p.gate)[o]);
    reinterpret_cast<T*>(p.out)[o] = from_f<T>(v);
  }
}

// ---------------------------------------------------------------- LayerNorm of a few rows
template <typename T>
__global__ void __launch_bounds__(kDecThreads)
decode_layer_norm_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b, T* __restrict__ y,
                         int D, float eps) {
  extern __shared__ float sm[];
  __shared__ float scratch[32];
  const long long row = (long long)blockIdx.x * D;
  pdl_wait();
  pdl_launch_dependents();
  float s = 0.f;
  for (int i = threadIdx.x * 8; i < D; i += kDecThreads * 8) {
    float v[8];
    load8(x + row + i, v);
    store8(sm + i, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[j];
  }
  const float mean = block_sum(s, scratch) / D;
  float q = 0.f;
  for (int i = threadIdx.x; i < D; i += kDecThreads) {
    const float d = sm[i] - mean;
    q = fmaf(d, d, q);
  }
  const float rstd = rsqrtf(block_sum(q, scratch) / D + eps);
  for (int i = threadIdx.x * 8; i < D; i += kDecThreads * 8) {
    float o[8], wv[8], bv[8];
    if (w != nullptr) load8(w + i, wv);
    if (b != nullptr) load8(b + i, bv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v = (sm[i + j] - mean) * rstd;
      if (w != nullptr) v *= wv[j] + 1.f;
      if (b != nullptr) v += bv[j];
      o[j] = v;
    }
    store8(y + row + i, o);
  }
}

template <int THREADS = kDecThreads, typename... KArgs, typename... Args>
cudaError_t launch_link(void (*kern)(KArgs...), dim3 grid, size_t smem, int cluster, bool pdl, cudaStream_t st,
                        Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (cluster > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = cluster;
    attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

}  // namespace

bool decode_norm_ema_ok(int D, int G, int N) {
  return G >= 1 && D % G == 0 && D <= 16384 && (N == 2 || N == 4 || N == 8 || N == 16 || N == 32);
}

int decode_norm_ema(const DecodeNormEma& p, int B, int dtype, bool pdl, cudaStream_t st) {
  if (B == 0) return 0;
  // as many CTAs per row as share its groups evenly (a cluster of 8 at the most)
  int cl = 8;
  while (cl > 1 && p.G % cl != 0) cl /= 2;
  const size_t smem = sizeof(float) * (2 * (p.D / cl) + 2 * (p.G / cl));
  cudaError_t e = cudaSuccess;
  // Few rows: 512 threads, one CTA per SM.  A cluster of eight such CTAs takes half of a GPC, so from nine rows on
  // some would wait for a second wave and 256 threads, two CTAs per SM, are the better ones (4096 features, one row:
  // 9.4 against 14.2 us; 2048 features, 16 rows: 12.9 against 10.0 us).
  MB_DISPATCH_16BIT(dtype, {
    auto wide = decode_norm_ema_kernel<scalar_t, 512>;
    auto narrow = decode_norm_ema_kernel<scalar_t, 256>;
    if (smem > 40 * 1024) {
      e = cudaFuncSetAttribute(wide, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(narrow, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    }
    if (e == cudaSuccess)
      e = B <= 8 ? launch_link<512>(wide, dim3(B * cl), smem, cl, pdl, st, p, cl)
                 : launch_link<256>(narrow, dim3(B * cl), smem, cl, pdl, st, p, cl);
  });
  return e == cudaSuccess ? 0 : -3;
}

int decode_attend_splits(int BH, int C, int num_sms) {
  int s = 2 * num_sms / (BH > 0 ? BH : 1);         // one wave of two CTAs per SM
  const int least = div_up(C, 16384);              // the scores of a split sit in shared memory
  if (s < least) s = least;
  return s < 1 ? 1 : (s > kDecodeMaxSplits ? kDecodeMaxSplits : s);
}

int decode_attend(const DecodeAttend& p, int B, int splits, int dtype, bool pdl, cudaStream_t st) {
  if (B == 0) return 0;
  if (p.z != nullptr && (p.dv % 8 != 0 || !aligned16(p.v_buf))) return -1;      // (the new value row leaves in pieces)
  const int BH = B * p.H;
  const int keys = div_up(p.C, splits) < 8 ? 8 : div_up(p.C, splits);
  const size_t smem = sizeof(float) * (2 * p.dk + kDecThreads * 8 + keys);
  cudaError_t e = cudaSuccess;
  MB_DISPATCH_16BIT(dtype, {
    const bool vec = p.dv % 8 == 0 && aligned16(p.v_buf);
    auto kern = vec ? decode_attend_kernel<scalar_t, true> : decode_attend_kernel<scalar_t, false>;
    if (smem > 40 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
    if (e == cudaSuccess) e = launch_link(kern, dim3(splits, BH), smem, 1, pdl, st, p);
    if (e == cudaSuccess)
      e = launch_link(decode_combine_kernel<scalar_t>, dim3(div_up(p.dv, 128), BH), 0, 1, pdl, st, p, splits);
  });
  return e == cudaSuccess ? 0 : -3;
}

int decode_layer_norm(const void* x, const void* w, const void* b, void* y, int rows, int D, float eps, int dtype,
                      bool pdl, cudaStream_t st) {
  if (rows == 0) return 0;
  cudaError_t e = cudaSuccess;
  MB_DISPATCH_16BIT(dtype, {
    auto kern = decode_layer_norm_kernel<scalar_t>;
    if (D * sizeof(float) > 40 * 1024)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess)
      e = launch_link(kern, dim3(rows), D * sizeof(float), 1, pdl, st, (const scalar_t*)x, (const scalar_t*)w,
                      (const scalar_t*)b, (scalar_t*)y, D, eps);
  });
  return e == cudaSuccess ? 0 : -3;
}

}  // namespace mb
