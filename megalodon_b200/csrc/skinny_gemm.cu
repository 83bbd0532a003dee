// Linear layers for few rows (decoding, short prompts, the last position of a prefill):
//
//   y[m, n] = act(sum_k x[m, k] w[n, k] + bias[n]) + addend[m, n]              m < M <= 64
//
// One pass over the weights is what such a product costs, so the kernel is organised as a stream of
// weight tiles over all SMs.  The operands are swapped: 128 weight rows are the M side of the tcgen05.mma,
// the (padded) rows of x its N side, so a 64-deep stage is 16 KiB of weights and 2 KiB per 16 rows of x, and
// the accumulator holds output features in its lanes (stores of consecutive features coalesce).
// K is split over a cluster of 1..8 CTAs, so that N / 128 tiles fill the machine; the partial accumulators
// meet in distributed shared memory, each CTA adding up and finishing 128 / S of the tile's features.
// Up to four products over the same rows share a launch (the four projections of a MEGA layer), and a
// product may carry a second weight for SwiGLU: y = silu(x w^T) * (x w2^T).  Rows of x may come without their RMSNorm's
// factor, which is then applied to the sums (`row_sq`).
//
// In a chain of programmatic dependent launches the weight tiles of the first ring round are requested before the
// previous kernel has finished: weights do not depend on it, x does.  (Prefetching the rest into L2 as well gained
// nothing at 1024 features and cost the 4096-wide layers a tenth: 16 tokens 10.9 -> 12.0 ms.  So did one CTA per SM
// with twice the ring, 12.9 ms, and splitting until there are two CTAs per SM, 11.4 ms.)
//
// All waits are bounded; a timeout sets `*err` and the CTA unwinds.
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace mb {

bool make_tmap_4d(CUtensorMap* out, const void* base, long long inner, long long outer, long long batch,
                  long long batch2, long long row_stride, long long batch_stride, long long batch2_stride,
                  int box_inner, int box_outer, int elem_dtype);

namespace {

using namespace ptx;

constexpr int kSkThreads = 192;          // TMA producer, MMA issuer, four epilogue warps
constexpr int kSkBK = 64;
constexpr int kSkRows = 128;             // weight rows of a tile
constexpr int kSkMaxStages = 8;

struct SkinnyMaps {
  CUtensorMap w[kSkinnyJobs], w2[kSkinnyJobs], x[kSkinnyJobs];
};
struct SkinnyParams {
  SkinnyJob job[kSkinnyJobs];
  int tile0[kSkinnyJobs];                // first tile of each product
  int njobs, M, mpad, split, stages, stage_bytes, tmem_cols, fmt, red_bytes;
  int* err;
};

__device__ __forceinline__ bool sk_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0xff) == 0) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > kWaitTimeoutNs) return false;
    }
  }
  return true;
}

template <typename T>
__device__ __forceinline__ float sk_addend(const SkinnyJob& j, int m, int n) {
  return j.addend == nullptr ? 0.f : to_f(reinterpret_cast<const T*>(j.addend)[(long long)m * j.ld_add + n]);
}
template <typename T>
__device__ __forceinline__ void sk_finish(const SkinnyJob& j, int m, int n, float v, float v2, float bias, float addend) {
  v += bias;
  if (j.act == kSkinnySilu) v = silu_f(v);
  else if (j.act == kSkinnySwiGLU) v = silu_f(v) * v2;
  v += addend;
  if (j.out_f32) reinterpret_cast<float*>(j.y)[(long long)m * j.ldy + n] = v;
  else reinterpret_cast<T*>(j.y)[(long long)m * j.ldy + n] = from_f<T>(v);
}

__device__ __forceinline__ float sk_bias(const SkinnyJob& j, int n) {
  if (j.bias == nullptr) return 0.f;
  if (j.bias_dtype == kF32) return reinterpret_cast<const float*>(j.bias)[n];
  if (j.bias_dtype == kBF16) return to_f(reinterpret_cast<const __nv_bfloat16*>(j.bias)[n]);
  return to_f(reinterpret_cast<const __half*>(j.bias)[n]);
}

template <typename T>
__global__ void __launch_bounds__(kSkThreads)
skinny_gemm_kernel(const __grid_constant__ SkinnyMaps maps, const __grid_constant__ SkinnyParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + p.stages * p.stage_bytes + p.red_bytes);
  uint64_t* empty_bar = full_bar + kSkMaxStages;
  uint64_t* acc_bar = empty_bar + kSkMaxStages;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
  float* row_scale = reinterpret_cast<float*>(tmem_holder + 2);      // kSkinnyMaxRows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.split;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int tile = blockIdx.x / S;
  int ji = 0;
  while (ji + 1 < p.njobs && tile >= p.tile0[ji + 1]) ++ji;
  const SkinnyJob& job = p.job[ji];
  const int n0 = (tile - p.tile0[ji]) * kSkRows;
  const int nk = (job.K + kSkBK - 1) / kSkBK;
  const int kb0 = (int)((long long)rank * nk / S), kb1 = (int)((long long)(rank + 1) * nk / S);
  const bool dual = job.act == kSkinnySwiGLU;
  const uint32_t w_bytes = kSkRows * kSkBK * 2;
  const uint32_t x_off = dual ? 2 * w_bytes : w_bytes;
  const uint32_t tx_bytes = x_off + p.mpad * kSkBK * 2;

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(full_bar + i, 1);
      mbar_init(empty_bar + i, 1);
    }
    mbar_init(acc_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, p.tmem_cols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  if (S > 1) cluster_arrive();       // awaited before the first store into another CTA: by then all have started

  if (warp == 0) {
    if (elect_one()) {
      // (the descriptor of x as well: otherwise its fetch begins only when x is there)
      prefetch_tmap(&maps.w[ji]);
      if (dual) prefetch_tmap(&maps.w2[ji]);
      prefetch_tmap(&maps.x[ji]);
      const int total = kb1 - kb0;
      const int first = min(total, p.stages);
      for (int i = 0; i < first; ++i) {
        uint8_t* st = smem + i * p.stage_bytes;
        mbar_expect_tx(full_bar + i, tx_bytes);
        tma_load_4d(st, &maps.w[ji], full_bar + i, (kb0 + i) * kSkBK, n0, 0, 0);
        if (dual) tma_load_4d(st + w_bytes, &maps.w2[ji], full_bar + i, (kb0 + i) * kSkBK, n0, 0, 0);
      }
      pdl_wait();
      for (int i = 0; i < first; ++i)
        tma_load_4d(smem + i * p.stage_bytes + x_off, &maps.x[ji], full_bar + i, (kb0 + i) * kSkBK, 0, 0, 0);
      bool ok = true;
      int stage = 0, issued = first;
      uint32_t phase = 0;
      for (int i = first; i < total; ++i) {
        if (!sk_wait(empty_bar + stage, phase, abort_flag)) { ok = false; break; }
        uint8_t* st = smem + stage * p.stage_bytes;
        const int k = (kb0 + i) * kSkBK;
        mbar_expect_tx(full_bar + stage, tx_bytes);
        tma_load_4d(st, &maps.w[ji], full_bar + stage, k, n0, 0, 0);
        if (dual) tma_load_4d(st + w_bytes, &maps.w2[ji], full_bar + stage, k, n0, 0, 0);
        tma_load_4d(st + x_off, &maps.x[ji], full_bar + stage, k, 0, 0, 0);
        ++issued;
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (!ok) {
        *abort_flag = 1;
        atomicExch(p.err, 11);
        for (int i = max(0, issued - p.stages); i < issued; ++i)        // let the copies in flight land
          mbar_wait(full_bar + i % p.stages, (i / p.stages) & 1);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(kSkRows, p.mpad, p.fmt, 0, 0);
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!sk_wait(full_bar + stage, phase, abort_flag)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t sw = smem_u32(smem + stage * p.stage_bytes), sx = sw + x_off;
#pragma unroll
        for (int kk = 0; kk < kSkBK / 16; ++kk) {
          const uint64_t dx = make_smem_desc(sx + kk * 32, 16, 1024);
          const uint32_t on = (kb != kb0 || kk != 0) ? 1u : 0u;
          umma_f16(tmem_base, make_smem_desc(sw + kk * 32, 16, 1024), dx, idesc, on);
          if (dual) umma_f16(tmem_base + p.mpad, make_smem_desc(sw + w_bytes + kk * 32, 16, 1024), dx, idesc, on);
        }
        umma_commit(empty_bar + stage);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(acc_bar);
      else { *abort_flag = 1; atomicExch(p.err, 12); }
    }
  }
  __syncwarp();

  const int quarter = warp & 3;
  const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
  const int nl = quarter * 32 + lane;              // this thread's feature within the tile
  bool ok = true;
  // Biases (weights, so ahead of the wait) and addends of the first elements that a thread finishes come in while the
  // product is under way.
  constexpr int kPre = 2;
  const int R = kSkRows / S;                       // features finished by each CTA of a cluster
  float bias_pre[kPre], add_pre[kPre];
  auto finished = [&](int u, int& m, int& n) {     // element u of this thread; false if it has none
    const int idx = (int)threadIdx.x - 64 + u * (kSkThreads - 64);
    m = idx / R;
    n = n0 + rank * R + idx % R;
    return m < p.M && n < job.N;
  };
  if (warp >= 2) {
    int m, n;
#pragma unroll
    for (int u = 0; u < kPre; ++u) bias_pre[u] = S > 1 && finished(u, m, n) ? sk_bias(job, n) : 0.f;
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int u = 0; u < kPre; ++u) add_pre[u] = S > 1 && finished(u, m, n) ? sk_addend<T>(job, m, n) : 0.f;
    if (job.row_sq != nullptr) {
      // Eight lanes a row, all rows in flight: one row of a warp after the other costs a memory latency and a chain of
      // shuffles each (a product of 1024 x 1024 with 32 parts a row, without a factor / so / one by one: 16 rows 3.5 / 3.7 / 5.4 us,
      // 64 rows 7.3 / 7.5 / 15.1)
      constexpr int kPass = kSkinnyMaxRows / 16;
      const int l8 = lane & 7, first = (warp - 2) * 4 + (lane >> 3), parts = job.row_parts;
      float s[kPass] = {};
      if ((parts & 3) == 0 && (reinterpret_cast<uintptr_t>(job.row_sq) & 15) == 0) {
        for (int i = l8 * 4; i < parts; i += 32) {
          float4 v[kPass];
#pragma unroll
          for (int u = 0; u < kPass; ++u)
            if (16 * u < p.M) v[u] = *reinterpret_cast<const float4*>(job.row_sq + min(first + 16 * u, p.M - 1) * parts + i);
#pragma unroll
          for (int u = 0; u < kPass; ++u)
            if (16 * u < p.M) s[u] += (v[u].x + v[u].y) + (v[u].z + v[u].w);
        }
      } else {
        for (int i = l8; i < parts; i += 8) {
#pragma unroll
          for (int u = 0; u < kPass; ++u)
            if (16 * u < p.M) s[u] += job.row_sq[min(first + 16 * u, p.M - 1) * parts + i];
        }
      }
      float mine = 0.f;                            // lane u of a row's eight finishes its row of pass u
#pragma unroll
      for (int u = 0; u < kPass; ++u) {
        s[u] = subwarp_sum<8>(s[u]);
        if (l8 == u) mine = s[u];
      }
      const int row = first + 16 * l8;
      if (l8 < kPass && row < p.M) row_scale[row] = rsqrtf(mine / job.K + job.row_eps);
      asm volatile("bar.sync 1, %0;" ::"n"(kSkThreads - 64) : "memory");     // the four epilogue warps
    }
    ok = sk_wait(acc_bar, 0, abort_flag);
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 13); }
    tcgen05_fence_after();
  }
  auto scaled = [&](float v, int m) { return job.row_sq != nullptr ? v * row_scale[m] : v; };
  if (S == 1) {
    if (warp >= 2 && ok) {
      const int n = n0 + nl;
      const float bias = n < job.N ? sk_bias(job, n) : 0.f;
      for (int c = 0; c < p.mpad; c += 16) {
        uint32_t r[16], r2[16];
        tmem_ld_32x16(t_row + c, r);
        if (dual) tmem_ld_32x16(t_row + p.mpad + c, r2);
        tmem_ld_wait();
        if (n < job.N) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c + i < p.M)
              sk_finish<T>(job, c + i, n, scaled(__uint_as_float(r[i]), c + i),
                           dual ? scaled(__uint_as_float(r2[i]), c + i) : 0.f, bias, sk_addend<T>(job, c + i, n));
        }
      }
    }
  } else {
    cluster_wait();
    uint8_t* red_smem = smem + p.stages * p.stage_bytes;      // partial sums have memory of their own
    const uint32_t red = smem_u32(red_smem);
    const int plane = p.mpad * R;                  // floats of one (source, accumulator)
    const int naccs = dual ? 2 : 1;
    if (warp >= 2) {
      const uint32_t dst = map_to_cta(red, (uint32_t)(nl / R)) + (uint32_t)((rank * naccs * plane + nl % R) * 4);
      for (int c = 0; c < p.mpad; c += 16) {
        uint32_t r[16];
        for (int a = 0; a < naccs; ++a) {
          tmem_ld_32x16(t_row + a * p.mpad + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c + i < p.M) st_cluster_f32(dst + (uint32_t)((a * plane + (c + i) * R) * 4), __uint_as_float(r[i]));
        }
      }
    }
    cluster_sync_all();
    if (warp >= 2 && ok) {
      const float* part = reinterpret_cast<const float*>(red_smem);
      auto finish = [&](int m, int n, float bias, float addend) {
        const int fl = n - n0 - rank * R;
        float v = 0.f, v2 = 0.f;
        for (int s = 0; s < S; ++s) {
          v += part[s * naccs * plane + m * R + fl];
          if (dual) v2 += part[(s * 2 + 1) * plane + m * R + fl];
        }
        sk_finish<T>(job, m, n, scaled(v, m), scaled(v2, m), bias, addend);
      };
      int m, n;
#pragma unroll
      for (int u = 0; u < kPre; ++u)
        if (finished(u, m, n)) finish(m, n, bias_pre[u], add_pre[u]);
      for (int u = kPre; u * (kSkThreads - 64) < R * p.M; ++u)
        if (finished(u, m, n)) finish(m, n, sk_bias(job, n), sk_addend<T>(job, m, n));
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

template <typename T>
int launch_skinny(const SkinnyMaps& maps, const SkinnyParams& p, int tiles, size_t smem, bool pdl, cudaStream_t st) {
  auto kern = skinny_gemm_kernel<T>;
  static std::atomic<unsigned long long> configured{0};
  if (!allow_dynamic_smem(kern, 227 * 1024, configured)) return -2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles * p.split, 1, 1);
  cfg.blockDim = dim3(kSkThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (p.split > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.split;
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
  ++thread_launches();
  return cudaLaunchKernelEx(&cfg, kern, maps, p) == cudaSuccess ? 0 : -3;
}

}  // namespace

// Whether one product is inside what the kernel handles (16-bit operands, TMA strides and alignment).
bool skinny_gemm_ok(int M, int N, int K, long long ldx, long long ldw, const void* x, const void* w, int in_dtype) {
  return M >= 1 && M <= kSkinnyMaxRows && N >= 1 && K >= 8 && K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 &&
         aligned16(x) && aligned16(w) && (in_dtype == kBF16 || in_dtype == kF16);
}

int skinny_gemm(const SkinnyJob* jobs, int njobs, int M, int in_dtype, bool pdl, int* err, int num_sms,
                cudaStream_t st) {
  if (njobs < 1 || njobs > kSkinnyJobs || M < 1 || M > kSkinnyMaxRows) return -1;
  SkinnyMaps maps;
  SkinnyParams p{};
  p.njobs = njobs;
  p.M = M;
  p.mpad = (M + 15) / 16 * 16;
  p.fmt = in_dtype == kBF16 ? 1 : 0;
  p.err = err;
  int tiles = 0, min_nk = 1 << 30;
  bool dual = false;
  for (int i = 0; i < njobs; ++i) {
    const SkinnyJob& j = jobs[i];
    if (!skinny_gemm_ok(M, j.N, j.K, j.ldx, j.ldw, j.x, j.w, in_dtype)) return -1;
    p.job[i] = j;
    p.tile0[i] = tiles;
    tiles += div_up(j.N, kSkRows);
    min_nk = min_nk < div_up(j.K, kSkBK) ? min_nk : div_up(j.K, kSkBK);
    if (!make_tmap_4d(&maps.w[i], j.w, j.K, j.N, 1, 1, j.ldw, 0, 0, kSkBK, kSkRows, in_dtype)) return -4;
    if (j.act == kSkinnySwiGLU) {
      dual = true;
      if (!aligned16(j.w2) || !make_tmap_4d(&maps.w2[i], j.w2, j.K, j.N, 1, 1, j.ldw, 0, 0, kSkBK, kSkRows, in_dtype)) return -4;
    }
    if (!make_tmap_4d(&maps.x[i], j.x, j.K, M, 1, 1, j.ldx, 0, 0, kSkBK, p.mpad, in_dtype)) return -4;
  }
  p.stage_bytes = (dual ? 2 : 1) * kSkRows * kSkBK * 2 + p.mpad * kSkBK * 2;
  // K is split until the tiles cover every SM; at least two k-blocks are left to each CTA.  Two CTAs share an SM as
  // long as a ring of at least four stages fits half of its shared memory.  Where it does not (SwiGLU, whose stages
  // hold two weight tiles), the CTAs have to fit one per SM: a second wave of a few costs as much as the first
  // (2 x 2560 x 1024 weights: 160 CTAs 8.9 us, 80 CTAs 5.1 us).
  const int accs = dual ? 2 : 1, red_max = accs * p.mpad * kSkRows * 4;
  const bool shared_sm = 4 * p.stage_bytes <= 110 * 1024 - red_max;
  p.split = 1;
  while (p.split < 8 && min_nk >= 4 * p.split &&
         (shared_sm ? tiles * p.split < num_sms : 2 * tiles * p.split <= num_sms))
    p.split *= 2;
  p.red_bytes = p.split > 1 ? red_max : 0;
  p.stages = ((shared_sm ? 110 : 224) * 1024 - p.red_bytes) / p.stage_bytes;
  if (p.stages > kSkMaxStages) p.stages = kSkMaxStages;
  const int ring = p.stages * p.stage_bytes;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.mpad * (dual ? 2 : 1)) p.tmem_cols *= 2;
  const size_t smem = 1024 + ring + p.red_bytes + (2 * kSkMaxStages + 1) * 8 + 16 + 4 * kSkinnyMaxRows;
  if (in_dtype == kBF16) return launch_skinny<__nv_bfloat16>(maps, p, tiles, smem, pdl, st);
  return launch_skinny<__half>(maps, p, tiles, smem, pdl, st);
}

}  // namespace mb
