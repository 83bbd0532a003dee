// One token through a MEGA block with a fixed-shape state: everything between the matrix products.
//
//   decode_norm_ema   TimestepNorm step -> complex-EMA step -> RMSNorm, state updated in place (the RMSNorm's factor left
//                     to the products that follow, where groups of features can do without each other)
//   decode_attend     per-head RMSNorm of z, query / key affine and rotary, key / value appended to the
//                     buffers, attention of one query over the filled slots split over the keys
//   decode_combine    the partial results of the splits put together, times the gate; attention in one
//                     launch (`attend_plan`) does without it
//   decode_layer_norm LayerNorm of the feed-forward branch
//
// A step is bound by its chain of launches, not by bytes: per layer these three or four and four products
// (skinny_gemm.cu) replace some thirty-five launches.  All of them are written as links of a programmatic
// dependent launch chain: `pdl_wait` before the first access to anything another kernel writes.
#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

#include <type_traits>

namespace mb {

bool make_tmap_rows(CUtensorMap* out, const void* base, long long width, long long rows, int box_width, int box_rows,
                    int elem_dtype);

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

// The same step for a reader that applies the RMSNorm's factor itself: no CTA then needs the whole row, so a CTA owns
// one group (or enough of them for 32 features), nothing is exchanged, and a row's state comes through all SMs instead
// of the eight of a cluster.  Everything but x, the parameters of the norms included, is loaded ahead of the wait.
// The link alone, 16 states, cluster form / this one, us: 8 rows of 1024 features 6.9 / 4.7, 32 rows 7.8 / 8.1, 64 rows
// 14.7 / 11.7; 16 rows of 2048 10.7 / 7.8, 64 rows 21.6 / 19.2; 8 rows of 4096 11.6 / 5.7, 32 rows 18.6 / 15.3.  With one or
// two groups a row has as many CTAs as the cluster form and takes as long (8192 features in one group 119.7 / 119.3), from
// nine rows on less (102 / 65 us for 16 rows of 4096), where a cluster's CTAs have 256 threads too.
// A row's count of steps also counts the CTAs that have read it, from bit kArrivalBit on (there are 512 at the most: 16384
// features, 32 of them to a CTA); the last one takes them off and adds the step.
constexpr int kArrivalBit = 52;
template <typename T, int PER, int BATCH>      // PER: threads of a feature, two states each; BATCH: items of a thread whose
__global__ void __launch_bounds__(kDecThreads, BATCH == 1 ? 5 : 3)      // loads are in flight together
decode_norm_ema_wide_kernel(const __grid_constant__ DecodeNormEma p, int groups) {
  extern __shared__ float sm[];
  __shared__ float scratch[32];
  __shared__ double weight_old, weight_new;
  const int gs = p.D / p.G, nf = groups * gs, b = blockIdx.y, f0 = blockIdx.x * nf, g0 = blockIdx.x * groups;
  float* xs = sm;                 // nf: input
  float* ts = xs + nf;            // nf: normalised input as the products see it
  float* gm = ts + nf;            // means and reciprocal deviations of the groups
  float* gr = gm + groups;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long row0 = (long long)b * p.D + f0;
  const int total = nf * PER;
  constexpr int kBatch = BATCH;
  const long long c0 = (long long)f0 * PER;
  float4* hx = reinterpret_cast<float4*>(p.hx) + (long long)b * p.D * PER + c0;
  float4 h[kBatch], q[kBatch], ga[kBatch];
  float2 pp[kBatch];
  float om[kBatch], rw[kBatch];
  auto load_items = [&](int base) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = base + u * kDecThreads + tid;
      if (i >= total) continue;
      h[u] = hx[i];
      q[u] = __ldg(reinterpret_cast<const float4*>(p.q) + c0 + i);
      ga[u] = __ldg(reinterpret_cast<const float4*>(p.gamma) + c0 + i);
      pp[u] = __ldg(reinterpret_cast<const float2*>(p.p) + c0 + i);
      if (i % PER == 0) {
        om[u] = to_f(reinterpret_cast<const T*>(p.omega)[f0 + i / PER]);
        rw[u] = p.rms_w != nullptr ? to_f(reinterpret_cast<const T*>(p.rms_w)[f0 + i / PER]) + 1.f : 1.f;
      }
    }
  };
  load_items(0);
  float w0 = 0.f, b0 = 0.f, u_old = 0.f, v_old = 0.f;
  if (tid < nf) {
    w0 = to_f(reinterpret_cast<const T*>(p.w)[f0 + tid]) + 1.f;
    b0 = to_f(reinterpret_cast<const T*>(p.b)[f0 + tid]);
  }
  if (warp < groups) {             // of this warp's first group
    u_old = p.mean[(long long)b * p.G + g0 + warp];
    v_old = p.var[(long long)b * p.G + g0 + warp];
  }
  unsigned long long seen = 0;
  if (tid == 0) {
    seen = atomicAdd(reinterpret_cast<unsigned long long*>(p.count + b), 1ull << kArrivalBit);
    const double n0 = (double)(seen & ((1ull << kArrivalBit) - 1));
    weight_old = n0 / (n0 + 1.0);
    weight_new = 1.0 / (n0 + 1.0);
  }
  pdl_wait();
  pdl_launch_dependents();
  for (int i = tid; i < nf; i += kDecThreads) xs[i] = to_f(reinterpret_cast<const T*>(p.x)[row0 + i]);
  __syncthreads();
  for (int g = warp; g < groups; g += kDecThreads / 32) {
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
      const long long gi = (long long)b * p.G + g0 + g;
      const double u0 = g == warp ? u_old : p.mean[gi], v0 = g == warp ? v_old : p.var[gi], ud = u;
      const double mean = weight_old * u0 + weight_new * ud;
      const double var = fmax(weight_old * (v0 + u0 * u0) + weight_new * ((double)v + ud * ud) - mean * mean, 0.0);
      p.mean[gi] = (float)mean;
      p.var[gi] = (float)var;
      gm[g] = (float)mean;
      gr[g] = rsqrtf((float)var + p.eps);
    }
  }
  __syncthreads();
  for (int i = tid; i < nf; i += kDecThreads) {
    const int g = i / gs;
    if (i != tid) {
      w0 = to_f(reinterpret_cast<const T*>(p.w)[f0 + i]) + 1.f;
      b0 = to_f(reinterpret_cast<const T*>(p.b)[f0 + i]);
    }
    const T t = from_f<T>((xs[i] - gm[g]) * gr[g] * w0 + b0);
    reinterpret_cast<T*>(p.t_out)[row0 + i] = t;
    ts[i] = to_f(t);
  }
  __syncthreads();
  float sq = 0.f;
  for (int base = 0; base < total; base += kBatch * kDecThreads) {
    if (base > 0) load_items(base);
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = base + u * kDecThreads + tid;
      const bool on = i < total;
      float acc = 0.f;
      const float t = on ? ts[i / PER] : 0.f;
      if (on) {
        float4 n;
        n.x = fmaf(q[u].x, h[u].x, fmaf(-q[u].y, h[u].y, pp[u].x * t));
        n.y = fmaf(q[u].x, h[u].y, q[u].y * h[u].x);
        n.z = fmaf(q[u].z, h[u].z, fmaf(-q[u].w, h[u].w, pp[u].y * t));
        n.w = fmaf(q[u].z, h[u].w, q[u].w * h[u].z);
        hx[i] = n;
        acc = ga[u].x * n.x - ga[u].y * n.y + ga[u].z * n.z - ga[u].w * n.w;
      }
      acc = subwarp_sum<PER>(acc);
      if (on && i % PER == 0) {
        const float y = to_f(from_f<T>(fmaf(om[u], t, acc)));
        reinterpret_cast<T*>(p.mx_out)[row0 + i / PER] = from_f<T>(y * rw[u]);
        sq = fmaf(y, y, sq);
      }
    }
  }
  sq = block_sum(sq, scratch);
  // (a group of one or two features that has no small divisor to be bundled by: more groups than threads)
  for (int g = tid; g < groups; g += kDecThreads) p.sumsq[(long long)b * p.G + g0 + g] = g == 0 ? sq : 0.f;
  if (tid == 0 && (seen >> kArrivalBit) == gridDim.x - 1)
    atomicAdd(reinterpret_cast<unsigned long long*>(p.count + b), 1ull - ((unsigned long long)gridDim.x << kArrivalBit));
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
// A CTA a row; a thread keeps up to kPieces pieces of eight features and their parameters, loaded ahead of the wait, in
// registers (longer rows go through memory again).
template <typename T>
__global__ void __launch_bounds__(kDecThreads)
decode_layer_norm_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b, T* __restrict__ y,
                         int D, float eps) {
  constexpr int kPieces = 2, kStep = kDecThreads * 8;
  __shared__ float scratch[32];
  const long long row = (long long)blockIdx.x * D;
  const int first = threadIdx.x * 8;
  float v[kPieces][8], wv[kPieces][8], bv[kPieces][8];
  auto load_params = [&](int i, float (&wp)[8], float (&bp)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) { wp[j] = 0.f; bp[j] = 0.f; }
    if (w != nullptr) load8(w + i, wp);
    if (b != nullptr) load8(b + i, bp);
  };
#pragma unroll
  for (int u = 0; u < kPieces; ++u)
    if (first + u * kStep < D) load_params(first + u * kStep, wv[u], bv[u]);
  pdl_wait();
  pdl_launch_dependents();
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < kPieces; ++u) {
    if (first + u * kStep >= D) break;
    load8(x + row + first + u * kStep, v[u]);
  }
#pragma unroll
  for (int u = 0; u < kPieces; ++u) {
    if (first + u * kStep >= D) break;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += v[u][j];
  }
  for (int i = first + kPieces * kStep; i < D; i += kStep) {
    float t[8];
    load8(x + row + i, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += t[j];
  }
  const float mean = block_sum(s, scratch) / D;
  float q = 0.f;
#pragma unroll
  for (int u = 0; u < kPieces; ++u) {
    if (first + u * kStep >= D) break;
#pragma unroll
    for (int j = 0; j < 8; ++j) q = fmaf(v[u][j] - mean, v[u][j] - mean, q);
  }
  for (int i = first + kPieces * kStep; i < D; i += kStep) {
    float t[8];
    load8(x + row + i, t);
#pragma unroll
    for (int j = 0; j < 8; ++j) q = fmaf(t[j] - mean, t[j] - mean, q);
  }
  const float rstd = rsqrtf(block_sum(q, scratch) / D + eps);
  auto finish = [&](int i, const float (&t)[8], const float (&wp)[8], const float (&bp)[8]) {
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (t[j] - mean) * rstd * (w != nullptr ? wp[j] + 1.f : 1.f) + bp[j];
    store8(y + row + i, o);
  };
#pragma unroll
  for (int u = 0; u < kPieces; ++u)
    if (first + u * kStep < D) finish(first + u * kStep, v[u], wv[u], bv[u]);
  for (int i = first + kPieces * kStep; i < D; i += kStep) {
    float t[8], wp[8], bp[8];
    load8(x + row + i, t);
    load_params(i, wp, bp);
    finish(i, t, wp, bp);
  }
}

// ---------------------------------------------------------------- attention of one query, one launch
// CTA = (split of the keys, block of value columns, sequence x head); the splits of one block form a cluster, whose
// partial rows meet in distributed shared memory, so neither they nor a second launch go through global memory.
//   * Keys and values of a split stream through one ring of 16 KiB stages (bulk copies by a warp of its own): the
//     values follow the keys without a gap, and in the chain the ring is filled before the wait - the older slots were
//     written by launches long before the predecessor.
//   * With one or two heads in all the value columns are divided too, and every column block works out the scores again:
//     its keys come from L2.  Its rows of values are boxes of a tensor map (a copy a row is bound by the number of
//     copies: 2000 keys of one head 17.9 us, with boxes 14.6, in clusters of 8).
// One query is bound by bytes where there are many sequences (128 heads, 500 keys: 4.6 TB/s; 3.6 in two launches) and by
// latencies where there are few.
constexpr int kAttStage = 16384;
constexpr int kAttThreads = kDecThreads + 32;      // eight consumer warps and the producer
constexpr int kAttMaxStages = 8;
constexpr int kAttMaxSplits = 16;
constexpr int kAttMaxSmem = 220 * 1024;

struct AttendPlan {
  int splits, blocks, cw, stages, key_rows, val_rows;
  int bw;              // columns of one copy of values: whole rows (cw == dv), or the width of `vmap`'s box
};

__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kDecThreads) : "memory"); }
// sum / maximum over the consumer warps; `scratch` holds 8 floats
template <bool MAX>
__device__ __forceinline__ float consumer_reduce(float v, float* scratch) {
  v = MAX ? warp_max(v) : warp_sum(v);
  consumer_sync();                                 // (the scratch of the reduction before this one has been read)
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  consumer_sync();
  float t = scratch[0];
#pragma unroll
  for (int w = 1; w < kDecThreads / 32; ++w) t = MAX ? fmaxf(t, scratch[w]) : t + scratch[w];
  return t;
}

// d += a b^T for 16 x 16 of a (rows 8 to 15 zero) and 8 x 16 of b, bf16 with fp32 sums
__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, {%7, %8}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1));
}

// the score of one key by one thread
__device__ __noinline__ float fma_score(const float* q, const __nv_bfloat16* key, int dk) {
  float s = 0.f;
  for (int e = 0; e < dk; ++e) s = fmaf(q[e], to_f(key[e]), s);
  return s;
}

__global__ void __launch_bounds__(kAttThreads, 2)
decode_attend_cluster_kernel(const __grid_constant__ DecodeAttend p, const __grid_constant__ AttendPlan pl,
                             const __grid_constant__ CUtensorMap vmap) {
  using T = __nv_bfloat16;
  extern __shared__ uint8_t att_raw[];
  __shared__ float scratch[8];
  __shared__ float2 ml[kAttMaxSplits];
  __shared__ uint64_t full_bar[kAttMaxStages], empty_bar[kAttMaxStages];
  __shared__ int failed;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(att_raw) + 127) & ~uintptr_t(127));
  float* qs = reinterpret_cast<float*>(ring + pl.stages * kAttStage);   // dk: query
  float* kn = qs + p.dk;                                                // dk: this token's key
  T* qrow = reinterpret_cast<T*>(kn + p.dk);                            // 3 dk: the query as a sum of 16-bit rows
  float* red = kn + p.dk + (3 * p.dk + 7) / 8 * 4;                      // kDecThreads * 8: rows of the thread groups
  float* comb = red + kDecThreads * 8;                                  // cw: partial rows of all splits, own columns
  float* sc = comb + pl.cw;                                             // scores of this split
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = pl.splits, split = blockIdx.x;
  const int bh = blockIdx.z, h = bh % p.H, col0 = blockIdx.y * pl.cw;
  const bool fused = p.z != nullptr;
  if (tid == 0) {
    for (int i = 0; i < pl.stages; ++i) {
      mbar_init(full_bar + i, 1);
      mbar_init(empty_bar + i, kDecThreads / 32);
    }
    failed = 0;
    fence_barrier_init();
    if (pl.cw != p.dv) prefetch_tmap(&vmap);
  }
  __syncthreads();
  if (S > 1) cluster_arrive();     // awaited before the first store into another CTA: by then all have started
  if (!fused) pdl_wait();          // (nothing is known here about what wrote the position and the slots)
  const int at = (int)min(p.pos[0], (long long)p.C - 1);
  const int n = at + 1, per = (n + S - 1) / S;
  const int lo = min(n, split * per), hi = min(n, lo + per), cnt = hi - lo;
  const bool mine = fused && at >= lo && at < hi;           // this split has the new slot
  const int old = mine ? cnt - 1 : cnt;
  const T* kold = reinterpret_cast<const T*>(p.k_buf) + ((long long)bh * p.C + lo) * p.dk;
  const T* vold = reinterpret_cast<const T*>(p.v_buf) + ((long long)bh * p.C + lo) * p.dv + col0;
  const int key_stages = (old + pl.key_rows - 1) / pl.key_rows, val_stages = (old + pl.val_rows - 1) / pl.val_rows;

  if (warp == kDecThreads / 32) {
    // ------------------------------------------------------------ producer
    const int total = key_stages + val_stages;
    int i = 0, st = 0;
    uint32_t phase = 1;
    for (; i < total; ++i) {
      // (all lanes wait: one answer for the warp)
      const bool room = i < pl.stages || mbar_wait(empty_bar + st, phase);
      if (!__all_sync(0xffffffffu, room)) {
        failed = 1;
        break;
      }
      const uint32_t dst = smem_u32(ring + st * kAttStage);
      const bool keys = i < key_stages;
      const int per_stage = keys ? pl.key_rows : pl.val_rows, width = keys ? p.dk : pl.cw;
      const int j = (keys ? i : i - key_stages) * per_stage, rows = min(per_stage, old - j);
      if (lane == 0) {
        if (keys || pl.cw == p.dv) {
          mbar_expect_tx(full_bar + st, rows * width * sizeof(T));
          bulk_load(dst, keys ? kold + (long long)j * p.dk : vold + (long long)j * p.dv, rows * width * sizeof(T),
                    full_bar + st);
        } else {
          // (whole boxes: what lies behind the split's last key is not used)
          const int box = pl.val_rows * pl.bw * (int)sizeof(T);
          mbar_expect_tx(full_bar + st, box * (pl.cw / pl.bw));
          for (int k = 0; k < pl.cw / pl.bw; ++k)
            tma_load_4d(ring + st * kAttStage + k * box, &vmap, full_bar + st, col0 + k * pl.bw, bh * p.C + lo + j, 0, 0);
        }
      }
      __syncwarp();
      if (++st == pl.stages) { st = 0; phase ^= 1; }
    }
    for (int k = max(0, i - pl.stages); k < i; ++k)       // no copy is in flight when the CTA leaves
      if (!mbar_wait(full_bar + k % pl.stages, (k / pl.stages) & 1)) failed = 1;
    __syncwarp();
  } else {
    // ------------------------------------------------------------ consumers
    bool ok = true;
    // the query / key parameters and rotation of this thread's first pair
    const T *ga = reinterpret_cast<const T*>(p.gamma) + h * p.dk, *be = reinterpret_cast<const T*>(p.beta) + h * p.dk;
    const float2* freqs = reinterpret_cast<const float2*>(p.freqs) + (long long)at * (p.dk / 2);
    const int Z = p.H * p.dk;
    struct Pair { float2 f, gq, gk, bq, bk; };
    auto load_pair = [&](int i) {
      auto two = [](const T* s) { return make_float2(to_f(s[0]), to_f(s[1])); };
      return Pair{freqs[i], two(ga + 2 * i), two(ga + Z + 2 * i), two(be + 2 * i), two(be + Z + 2 * i)};
    };
    Pair pair{};
    if (fused && tid < p.dk / 2) pair = load_pair(tid);
    pdl_wait();
    pdl_launch_dependents();
    // columns of this thread (8 of the block), row groups, and the new value row's piece
    const int ct = pl.cw / 8, ng = kDecThreads / ct, grp = tid / ct, c = (tid - grp * ct) * 8;
    uint4 vnew = make_uint4(0u, 0u, 0u, 0u);
    const bool has_new = mine && grp == 0;
    if (has_new)
      vnew = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.v_new) + (long long)bh * p.dv + col0 + c);
    if (fused) {
      const T* zr = reinterpret_cast<const T*>(p.z) + (long long)bh * p.dk;
      float s = 0.f;
      for (int i = tid; i < p.dk; i += kDecThreads) {
        const float v = to_f(zr[i]);
        qs[i] = v;
        s = fmaf(v, v, s);
      }
      const float rstd = rsqrtf(consumer_reduce<false>(s, scratch) / p.dk + p.eps);
      const float inv = rsqrtf((float)p.dk);
      T* krow = reinterpret_cast<T*>(p.k_buf) + ((long long)bh * p.C + at) * p.dk;
      for (int i = tid; i < p.dk / 2; i += kDecThreads) {
        if (i != tid) pair = load_pair(i);
        const float2 f = pair.f;
        const float z0 = qs[2 * i] * rstd, z1 = qs[2 * i + 1] * rstd;
        const float a0 = z0 * (pair.gq.x + 1.f) * inv + pair.bq.x, a1 = z1 * (pair.gq.y + 1.f) * inv + pair.bq.y;
        const float c0 = z0 * (pair.gk.x + 1.f) * inv + pair.bk.x, c1 = z1 * (pair.gk.y + 1.f) * inv + pair.bk.y;
        qs[2 * i] = a0 * f.x - a1 * f.y;
        qs[2 * i + 1] = a0 * f.y + a1 * f.x;
        const T k0 = from_f<T>(c0 * f.x - c1 * f.y), k1 = from_f<T>(c0 * f.y + c1 * f.x);
        kn[2 * i] = to_f(k0);
        kn[2 * i + 1] = to_f(k1);
        if (mine && blockIdx.y == 0) {
          krow[2 * i] = k0;
          krow[2 * i + 1] = k1;
        }
      }
    } else {
      const T* qr = reinterpret_cast<const T*>(p.q) + (long long)bh * p.dk;
      for (int i = tid; i < p.dk; i += kDecThreads) qs[i] = to_f(qr[i]);
    }
    consumer_sync();
    for (int i = tid; i < p.dk; i += kDecThreads) {
      float rest = qs[i];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const T part = from_f<T>(rest);
        qrow[r * p.dk + i] = part;
        rest -= to_f(part);
      }
    }
    consumer_sync();
    int st = 0;
    uint32_t phase = 0;
    auto wait_stage = [&]() {
      if (ok && !mbar_wait(full_bar + st, phase)) {
        ok = false;
        failed = 1;
      }
    };
    auto free_stage = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_bar + st);
      if (++st == pl.stages) { st = 0; phase ^= 1; }
    };
    // Scores.  With a width that is a multiple of 32 eight keys of a warp at a time on the tensor cores, the query as the
    // sum of three bf16 rows of the other operand (its 24 bits; products and sums are fp32): some 40 instructions for
    // eight keys instead of 400, which with several column blocks bounded the link.  A fragment's places along the
    // contraction are dealt out so that a lane's part of a key, and of a query row, is 16 contiguous bytes.
    const bool mma = p.dk % 32 == 0;
    for (int i = 0; i < key_stages; ++i) {
      wait_stage();
      const T* keys = reinterpret_cast<const T*>(ring + st * kAttStage);
      const int base = i * pl.key_rows, rows = min(pl.key_rows, old - base);
      if (mma) {
        const int g = lane >> 2, t8 = (lane & 3) * 8;
        for (int j0 = warp * 8; j0 < rows; j0 += kDecThreads / 32 * 8) {
          const T* key = keys + min(j0 + g, rows - 1) * p.dk + t8;
          float d[4] = {0.f, 0.f, 0.f, 0.f}, d2[4] = {0.f, 0.f, 0.f, 0.f};
          for (int e = 0; e < p.dk; e += 32) {
            uint4 qa = make_uint4(0u, 0u, 0u, 0u);
            if (g < 3) qa = *reinterpret_cast<const uint4*>(qrow + g * p.dk + e + t8);
            const uint4 kb = *reinterpret_cast<const uint4*>(key + e);
            mma_m16n8k16(d, qa.x, qa.y, kb.x, kb.y);
            mma_m16n8k16(d2, qa.z, qa.w, kb.z, kb.w);
          }
          // rows 0 to 2 of the result, columns 2 (lane & 3) and the next
          float s0 = d[0] + d2[0], s1 = d[1] + d2[1];
          s0 += __shfl_down_sync(0xffffffffu, s0, 4) + __shfl_down_sync(0xffffffffu, s0, 8);
          s1 += __shfl_down_sync(0xffffffffu, s1, 4) + __shfl_down_sync(0xffffffffu, s1, 8);
          const int j = j0 + 2 * lane;
          if (lane < 4 && j < rows) sc[base + j] = s0 * p.scale;
          if (lane < 4 && j + 1 < rows) sc[base + j + 1] = s1 * p.scale;
        }
      } else {
        for (int j = warp; j < rows; j += kDecThreads / 32) {
          float s = 0.f;
          for (int e = lane * 8; e < p.dk; e += 256) {
            float q[8], kv[8];
            load8(qs + e, q);
            load8(keys + j * p.dk + e, kv);
#pragma unroll
            for (int k = 0; k < 8; ++k) s = fmaf(q[k], kv[k], s);
          }
          s = warp_sum(s);
          if (lane == 0) sc[base + j] = s * p.scale;
        }
      }
      free_stage();
    }
    if (mine && warp == 0) {
      float s = 0.f;
      for (int e = lane; e < p.dk; e += 32) s = fmaf(qs[e], kn[e], s);
      s = warp_sum(s);
      if (lane == 0) sc[old] = s * p.scale;
    }
    consumer_sync();
    float m = -INFINITY;
    for (int j = tid; j < cnt; j += kDecThreads) {
      float v = sc[j];
      // An infinity in a key is NaN after the products with the query's parts, one of which is zero or of the other sign.
      // (Where the products are, a look at them costs up to 8 % with many heads.)
      if (mma && isnan(v) && j < old) sc[j] = v = fma_score(qs, kold + (long long)j * p.dk, p.dk) * p.scale;
      m = fmaxf(m, v);
    }
    m = consumer_reduce<true>(m, scratch);
    const float ref = m == -INFINITY ? 0.f : m;      // a split without keys, or whose keys all have weight zero
    float sum = 0.f;
    for (int j = tid; j < cnt; j += kDecThreads) {
      const float e = __expf(sc[j] - ref);
      sc[j] = e;
      sum += e;
    }
    sum = consumer_reduce<false>(sum, scratch);      // (its barriers also publish the weights)
    // values
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < val_stages; ++i) {
      wait_stage();
      const T* vals = reinterpret_cast<const T*>(ring + st * kAttStage) + c / pl.bw * (pl.val_rows * pl.bw) + c % pl.bw;
      const int base = i * pl.val_rows, rows = min(pl.val_rows, old - base);
      if (grp < ng) {
#pragma unroll 4
        for (int r = grp; r < rows; r += ng) {
          float v[8];
          load8(vals + r * pl.bw, v);
          const float e = sc[base + r];
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] = fmaf(e, v[k], acc[k]);
        }
      }
      free_stage();
    }
    if (has_new) {
      *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.v_buf) + ((long long)bh * p.C + at) * p.dv + col0 + c) = vnew;
      float v[8];
      load8(reinterpret_cast<const T*>(&vnew), v);
      const float e = sc[old];
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] = fmaf(e, v[k], acc[k]);
    }
    if (ng > 1) {
      if (grp < ng) store8(red + tid * 8, acc);
      consumer_sync();
      if (grp == 0) {
        for (int g = 1; g < ng; ++g) {
          float v[8];
          load8(red + (g * ct * 8 + tid * 8), v);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += v[k];
        }
      }
    }
    if (S > 1) cluster_wait();
    // column k of the block is finished by split k / (cw / S)
    const int R = pl.cw / S;
    if (grp == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int owner = (c + k) / R, slot = split * R + (c + k) - owner * R;
        if (S > 1) st_cluster_f32(map_to_cta(smem_u32(comb + slot), owner), acc[k]);
        else comb[slot] = acc[k];
      }
    }
    if (tid < S) {
      if (failed) sum = __int_as_float(0x7fffffff);      // a copy that never came: the result is not a number
      if (S > 1) {
        const uint32_t dst = map_to_cta(smem_u32(ml + split), tid);
        st_cluster_f32(dst, m);
        st_cluster_f32(dst + 4, sum);
      } else {
        ml[0] = make_float2(m, sum);
      }
    }
  }
  if (S > 1) {
    if (warp == kDecThreads / 32) cluster_wait();          // (the consumers have come to theirs above)
    cluster_sync_all();
  } else {
    __syncthreads();
  }
  if (tid >= kDecThreads) return;
  float m = ml[0].x;
  for (int s = 1; s < S; ++s) m = fmaxf(m, ml[s].x);
  float l = 0.f;
  for (int s = 0; s < S; ++s) l += __expf(ml[s].x - m) * ml[s].y;
  const int R = pl.cw / S;
  for (int k = tid; k < R; k += kDecThreads) {
    float v = 0.f;
    for (int s = 0; s < S; ++s) v = fmaf(__expf(ml[s].x - m), comb[s * R + k], v);
    const long long o = (long long)bh * p.dv + col0 + split * R + k;
    v /= l;
    if (p.gate != nullptr) v *= to_f(reinterpret_cast<const T*>(p.gate)[o]);
    reinterpret_cast<T*>(p.out)[o] = from_f<T>(v);
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

static int decode_norm_ema_wide(const DecodeNormEma& p, int B, int dtype, bool pdl, cudaStream_t st) {
  const int gs = p.D / p.G;
  // Features of a CTA: 32, or 64 where that would be more CTAs than the five to an SM that run at once (us, 32 / 64:
  // 24 x 1024 8.1 / 7.6, 32 x 1024 8.5 / 8.1, 64 x 1024 12.8 / 11.7, 16 x 2048 8.7 / 7.8, 64 x 2048 23.4 / 19.2).
  const int least = (long long)B * p.D > 32 * 5 * 148 ? 64 : 32;
  int groups = 1;                                   // the fewest, dividing G evenly, with that many
  while (groups < p.G && (groups * gs < least || p.G % groups != 0)) ++groups;
  const size_t smem = sizeof(float) * (2 * groups * gs + 2 * groups);
  cudaError_t e = cudaSuccess;
  MB_DISPATCH_16BIT(dtype, {
    auto launch = [&](auto kern) {
      if (smem > 40 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
      if (e == cudaSuccess) e = launch_link(kern, dim3(p.G / groups, B), smem, 1, pdl, st, p, groups);
    };
    // One item a thread keeps five CTAs to an SM, which many rows need to start in one or two waves.
    auto pick = [&](auto per) {
      constexpr int P = decltype(per)::value;
      if (groups * gs * P <= kDecThreads) launch(decode_norm_ema_wide_kernel<scalar_t, P, 1>);
      else launch(decode_norm_ema_wide_kernel<scalar_t, P, 2>);
    };
    if (p.N == 2) pick(std::integral_constant<int, 1>());
    else if (p.N == 4) pick(std::integral_constant<int, 2>());
    else if (p.N == 8) pick(std::integral_constant<int, 4>());
    else if (p.N == 16) pick(std::integral_constant<int, 8>());
    else pick(std::integral_constant<int, 16>());
  });
  return e == cudaSuccess ? 0 : -3;
}

int decode_norm_ema(const DecodeNormEma& p, int B, int dtype, bool pdl, cudaStream_t st) {
  if (B == 0) return 0;
  if (p.hx != nullptr && p.sumsq != nullptr) return decode_norm_ema_wide(p, B, dtype, pdl, st);
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

// How one launch divides the work, if it takes the shapes and is the better form; bf16 only, since three 16-bit parts of a
// query are its 24 bits in bf16 alone (fp16 ones end at 2^-24), and with the scores as fp32 FMAs two launches are as fast.
//   * The column blocks of a head repeat its scores, so there are several of them only for one or two heads in all, 128
//     CTAs in clusters of 16.
//   * More heads: the largest cluster of 8, 4, 2 whose CTAs run at once - two to an SM, but clusters of four and eight leave
//     SMs of a GPC over: 264 CTAs of 296 fit in eights, 272 in fours - and fill the SMs.  A wave that is not full and one
//     CTA too many are what loses: us, two launches / one, d_qk 256, d_v 1024, 1000 keys: 19 heads 18.2 / 21.5,
//     24 22.5 / 22.5, 28 26.2 / 23.5, 32 28.6 / 24.5, 36 28.3 / 37.3, 48 36.0 / 36.4, 64 48.5 / 36.9, 72 1.18 times two
//     launches, 104 to 180 0.74 to 0.75 times.  Rows of at most 640 columns pay from one CTA an SM on: d_qk 64, d_v 256,
//     19 heads 0.71 times, 48 0.61; single CTAs do so at any width (150 heads 0.68 to 0.77).
//   * A width that is no multiple of 32 has its scores from FMAs, which only pairs and single CTAs keep up with: d_qk 72,
//     2000 keys, 32 heads 1.20 times two launches, 56 1.31, 104 0.91.
// One or two heads (d_qk 256, d_v 2048): 300 keys 8.9 / 7.5 and 9.0 / 7.9, 2000 keys 13.7 / 11.9 and 15.8 / 15.0.
static bool attend_plan(const DecodeAttend& p, int BH, int num_sms, int dtype, bool wide_clusters, AttendPlan& pl,
                        size_t& smem) {
  if (dtype != kBF16 || p.dv % 8 != 0 || !aligned16(p.v_buf) || !aligned16(p.k_buf) || p.dk > kAttStage / 2) return false;
  int most;                                             // CTAs up to which there are several column blocks
  if (BH <= 2 && wide_clusters) {
    pl.splits = kAttMaxSplits;
    most = 128;
  } else {
    pl.splits = p.dk % 32 == 0 ? 8 : 2;
    while (pl.splits > 1 && pl.splits * BH > (pl.splits == 2 ? 2 * num_sms : 7 * num_sms / 4)) pl.splits /= 2;
    const int least = pl.splits == 1 || p.dk + p.dv <= 640 ? num_sms : 29 * num_sms / 20;
    if (pl.splits * BH < least) return false;
    most = 0;
  }
  const int pieces = p.dv / 8;
  pl.blocks = 0;
  for (int b = 1; b <= pieces && b <= 64; ++b) {
    const int cw = p.dv / b;
    if (pieces % b != 0 || cw > 8 * kDecThreads || cw % pl.splits != 0 || (b > 1 && cw > 256 && cw % 256 != 0)) continue;
    if (pl.blocks != 0 && (cw < 128 || b * pl.splits * BH > most)) break;
    pl.blocks = b;
  }
  if (pl.blocks == 0) return false;
  pl.cw = p.dv / pl.blocks;
  pl.bw = pl.blocks == 1 || pl.cw < 256 ? pl.cw : 256;
  pl.key_rows = kAttStage / (p.dk * 2);
  pl.val_rows = kAttStage / (pl.cw * 2);
  if (pl.val_rows > 256) pl.val_rows = 256;             // (a copy's box)
  const size_t other = sizeof(float) * (2 * p.dk + (3 * p.dk + 7) / 8 * 4 + kDecThreads * 8 + pl.cw +
                                        div_up(p.C, pl.splits)) + 128;
  const size_t room = 112 * 1024;                       // two CTAs to an SM
  pl.stages = other + 2 * kAttStage > room ? 2 : (int)((room - other) / kAttStage);
  if (pl.stages > kAttMaxStages) pl.stages = kAttMaxStages;
  smem = other + (size_t)pl.stages * kAttStage;
  return smem <= kAttMaxSmem;
}

// Whether clusters of 16 of the kernel can run on the current device (a size that is not portable).
static bool attend_wide_clusters() {
  static std::atomic<unsigned long long> known{0}, can{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
  const unsigned long long bit = 1ull << dev;
  if ((known.load(std::memory_order_acquire) & bit) == 0) {
    auto kern = decode_attend_cluster_kernel;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kAttMaxSplits, 1, 1);
    cfg.blockDim = dim3(kAttThreads, 1, 1);
    cfg.dynamicSmemBytes = kAttMaxSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kAttMaxSplits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttMaxSmem) == cudaSuccess &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0)
      can.fetch_or(bit, std::memory_order_release);
    (void)cudaGetLastError();
    known.fetch_or(bit, std::memory_order_release);
  }
  return (can.load(std::memory_order_acquire) & bit) != 0;
}

int decode_attend_plan(int BH, int C, int dk, int dv, int dtype, int num_sms) {
  DecodeAttend p = {};
  p.C = C; p.dk = dk; p.dv = dv;
  AttendPlan pl;
  size_t bytes;
  return attend_plan(p, BH, num_sms, dtype, true, pl, bytes) ? pl.splits * pl.blocks : 0;
}

int decode_attend(const DecodeAttend& p, int B, int splits, int num_sms, int dtype, bool pdl, cudaStream_t st) {
  if (B == 0) return 0;
  cudaError_t e = cudaSuccess;
  AttendPlan pl;
  size_t bytes;
  CUtensorMap vmap = {};
  if (B * p.H <= 65535 && attend_plan(p, B * p.H, num_sms, dtype, B * p.H <= 2 && attend_wide_clusters(), pl, bytes) &&
      (pl.blocks == 1 || make_tmap_rows(&vmap, p.v_buf, p.dv, (long long)B * p.H * p.C, pl.bw, pl.val_rows, dtype))) {
    auto kern = decode_attend_cluster_kernel;
    static std::atomic<unsigned long long> configured{0};
    if (!allow_dynamic_smem(kern, kAttMaxSmem, configured)) return -2;
    e = launch_link<kAttThreads>(kern, dim3(pl.splits, pl.blocks, B * p.H), bytes, pl.splits, pdl, st, p, pl, vmap);
    return e == cudaSuccess ? 0 : -3;
  }
  if (p.z != nullptr && (p.dv % 8 != 0 || !aligned16(p.v_buf))) return -1;      // (the new value row leaves in pieces)
  const int BH = B * p.H;
  const int keys = div_up(p.C, splits) < 8 ? 8 : div_up(p.C, splits);
  const size_t smem = sizeof(float) * (2 * p.dk + kDecThreads * 8 + keys);
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
    e = launch_link(decode_layer_norm_kernel<scalar_t>, dim3(rows), 0, 1, pdl, st, (const scalar_t*)x,
                    (const scalar_t*)w, (const scalar_t*)b, (scalar_t*)y, D, eps);
  });
  return e == cudaSuccess ? 0 : -3;
}

}  // namespace mb
