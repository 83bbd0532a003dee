// Persistent, warp-specialised tcgen05 GEMM for sm_100a.
//
//   C[M, N] = epilogue( A * B^T )       fp32 accumulation in tensor memory
//
// A supplies M rows, B supplies N rows, both reduced over K.  Each operand is
// either K-major (stored [rows, K], K contiguous) or MN-major (stored
// [K, rows], rows contiguous), so the three GEMMs of a linear layer need no
// transposed copies:
//   forward  y  = x  w^T      A = x  [M, K]  K-major,   B = w  [N, K]  K-major
//   dgrad    dx = dy w        A = dy [M, N'] K-major,   B = w  [N', K'] MN-major
//   wgrad    dw = dy^T x      A = dy [T, N'] MN-major,  B = x  [T, K'] MN-major
//
// CTA = 10 warps (6 for BN = 64): warp 0 issues TMA loads (128B-swizzled tiles, no multicast)
// into a shared-memory ring (4, 6 or 8 stages for BN = 256, 128, 64); warp 1 issues tcgen05.mma (128 x BN x 16)
// into one of two TMEM accumulators; the other warps drain the other accumulator
// with tcgen05.ld, apply bias / SiLU and store, so the epilogue of tile i
// overlaps the main loop of tile i+1.  Tiles are walked in bands of rows so that
// CTAs that run together share A and B tiles in L2 (see `row_band`).
//
// All mbarrier waits are bounded; a timeout sets `*err` and the CTA unwinds
// (releasing its TMEM) instead of hanging.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "common.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace mb {
namespace {

using namespace ptx;

constexpr int BM = 128;
constexpr int BK = 64;          // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int kEpiStageBytes = 32 * 64;   // staging buffer of an epilogue warp: 32 rows of 64 bytes
constexpr int kMaxPeers = 8;

// Ring of the single-CTA kernel: a tile that walks K alone is bound by one memory latency per ring round, so the
// narrow tiles spend their smaller stages on a deeper ring.
template <int BN>
struct SmemLayout {
  static constexpr int kStages = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int epi_warps = BN == 64 ? 4 : 8;
  static constexpr int threads = 64 + 32 * epi_warps;
  static constexpr int a_bytes = BM * BK * 2;       // 16 KiB
  static constexpr int b_bytes = BN * BK * 2;       // 32 KiB at BN = 256
  static constexpr int stage_bytes = a_bytes + b_bytes;
  static constexpr int bar_offset = kStages * stage_bytes;
  static constexpr int epi_offset = bar_offset + 256;    // barriers
  static constexpr int total = epi_offset + epi_warps * kEpiStageBytes + 1024;  // + alignment slack
};

// Triangular (causal) structure, used when the GEMM is one of the products of
// chunk-local causal attention (row index and contraction / column index count
// the same positions):
//   1  skip output tiles that lie entirely above the diagonal   (S = Q K^T, dP = dO V^T)
//   2  contract only over k <= last row of the tile             (O = P V, dQ = dS K;  A lower-triangular)
//   3  contract only over k >= first row of the tile            (dV = P^T dO, dK = dS^T Q; A^T lower-triangular)
struct GemmParams {
  int M, N, K;
  void* C;             // [M, N] with row stride ldc
  void* preact;        // optional [M, N]: value before the activation
  const void* bias;    // optional [N]
  int bias_dtype;      // DType
  int act;             // 0 none, 1 SiLU
  int* err;
  long long ldc;       // elements
  int mode;            // 0 dense, 1..3 see above
  int band;            // row tiles of a band of the tile walk (`row_band`)
  float alpha;         // C = alpha * acc (+ bias)
  int accumulate;      // 1: C += alpha * acc (+ bias); the old C is read in the epilogue
  int batch;           // independent problems sharing shapes (tensor maps carry their strides)
  int batch_in;        // problem i is (i / batch_in, i % batch_in): two batch strides per operand (sequence, head)
  long long c_batch_stride;   // elements between consecutive C (and preact) matrices of the inner batch index
  long long c_outer_stride;   // and of the outer one
  // all-gather -> GEMM: A is the concatenation along K of `a_parts` pieces of `a_part_k` columns, piece i
  // read through tensor map i (a peer GPU's memory); the walk over K starts at piece `a_first`
  int a_parts, a_part_k, a_first;
  // GEMM -> reduce-scatter: column block i of `c_part_cols` columns is stored to c_parts[i] (row stride
  // c_part_cols), a slot in the memory of the rank that owns those columns
  int c_nparts, c_part_cols;
  void* c_parts[kMaxPeers];
  // all-gather -> GEMM on the weight operand (B, K-major [N, K], rows sharded over `g_world` ranks in
  // blocks of N / g_world rows; pair kernel only).  g_src[r] is rank r's block (peer memory for r !=
  // g_rank), g_dst the local full matrix that tmap_b reads.  The copy warps of all CTAs move the matrix
  // in 128-row chunks (claimed 8 KiB at a time through g_flags[0], starting with this rank's own rows);
  // g_flags[1 + c] counts the finished 8 KiB units of chunk c, and a producer loads B rows of chunk c
  // only once all K / 32 of them are in.  The n-tile walk starts at this rank's own rows too.
  int g_world, g_rank;
  const void* g_src[kMaxPeers];
  void* g_dst;
  unsigned int* g_flags;
  // Softmax of chunk-local attention fused into the epilogues of its products (fp32 row vectors indexed
  // [batch, row]; column j of row i takes part iff j <= i + causal_off when mode == 1, always otherwise):
  //   1 row max     nothing is stored; row_out[i] = max(row_out[i], alpha * acc[i, j])        (S = Q K^T, pass 1)
  //   2 exp         C = exp(alpha * acc - row_in[i]) (0 where masked), row_out[i] += sum_j C  (S = Q K^T, pass 2)
  //   3 row scale   C = alpha * acc / row_in[i]  (0 for an empty row)                         (O = P V)
  //   4 dS          C = aux[i, j] / row_in[i] * (alpha * acc - row_in2[i])                    (dP = dO V^T -> dS)
  // `aux` has the layout of C and may be C itself.
  int epi;
  const float* row_in;
  const float* row_in2;
  float* row_out;
  const void* aux;
  int causal_off;
  // set by the launcher
  bool staged;         // C, preact and aux suit the 16-byte pieces of `epi_staged`
  bool bias_vec;       // bias may be read in 16-byte pieces
};

__device__ __forceinline__ long long c_base(const GemmParams& p, int bz) {
  const int bo = bz / p.batch_in;
  return bo * p.c_outer_stride + (bz - bo * p.batch_in) * p.c_batch_stride;
}

struct TmapArray {
  CUtensorMap m[kMaxPeers];
};

// Tile `t` of a problem, walked band after band of `band` row tiles and inside a band column by column.
__device__ __forceinline__ void banded_tile(int t, int num_m, int num_n, int band, int& mt, int& nt) {
  const int b = t / (band * num_n), r = t - b * band * num_n;
  const int rows = min(band, num_m - b * band);
  nt = r / rows;
  mt = b * band + (r - nt * rows);
}

struct TileCoord {
  int m0, n0, bz;
};
template <int BN>
__device__ __forceinline__ TileCoord decode_tile(int tile, int num_m, int num_n, int band) {
  const int tiles_per_batch = num_m * num_n;
  const int bz = tile / tiles_per_batch;
  int mt, nt;
  banded_tile(tile - bz * tiles_per_batch, num_m, num_n, band, mt, nt);
  return {mt * BM, nt * BN, bz};
}

template <int BN>
__device__ __forceinline__ bool tile_skipped(const GemmParams& p, int m0, int n0) {
  return p.mode == 1 && n0 > m0 + BM - 1;
}

__device__ __forceinline__ void k_range(const GemmParams& p, int m0, int num_k, int& kb0, int& kb1) {
  kb0 = 0;
  kb1 = num_k;
  if (p.mode == 2) kb1 = min(num_k, (m0 + BM + BK - 1) / BK);
  if (p.mode == 3) kb0 = min(num_k - 1, m0 / BK);
}

__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
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

template <typename OutT>
__device__ __forceinline__ void store_row32(OutT* dst, const float (&v)[32], int ncols_valid);

template <>
__device__ __forceinline__ void store_row32<__nv_bfloat16>(__nv_bfloat16* dst, const float (&v)[32], int nvalid) {
  if (nvalid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 pk;
      __nv_bfloat162 t0 = __floats2bfloat162_rn(v[8 * i + 0], v[8 * i + 1]);
      __nv_bfloat162 t1 = __floats2bfloat162_rn(v[8 * i + 2], v[8 * i + 3]);
      __nv_bfloat162 t2 = __floats2bfloat162_rn(v[8 * i + 4], v[8 * i + 5]);
      __nv_bfloat162 t3 = __floats2bfloat162_rn(v[8 * i + 6], v[8 * i + 7]);
      pk.x = *reinterpret_cast<uint32_t*>(&t0);
      pk.y = *reinterpret_cast<uint32_t*>(&t1);
      pk.z = *reinterpret_cast<uint32_t*>(&t2);
      pk.w = *reinterpret_cast<uint32_t*>(&t3);
      reinterpret_cast<uint4*>(dst)[i] = pk;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)      // (unrolled: an index that is not a constant would move v to local memory)
      if (i < nvalid) dst[i] = __float2bfloat16_rn(v[i]);
  }
}

template <>
__device__ __forceinline__ void store_row32<__half>(__half* dst, const float (&v)[32], int nvalid) {
  if (nvalid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 pk;
      __half2 t0 = __floats2half2_rn(v[8 * i + 0], v[8 * i + 1]);
      __half2 t1 = __floats2half2_rn(v[8 * i + 2], v[8 * i + 3]);
      __half2 t2 = __floats2half2_rn(v[8 * i + 4], v[8 * i + 5]);
      __half2 t3 = __floats2half2_rn(v[8 * i + 6], v[8 * i + 7]);
      pk.x = *reinterpret_cast<uint32_t*>(&t0);
      pk.y = *reinterpret_cast<uint32_t*>(&t1);
      pk.z = *reinterpret_cast<uint32_t*>(&t2);
      pk.w = *reinterpret_cast<uint32_t*>(&t3);
      reinterpret_cast<uint4*>(dst)[i] = pk;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid) dst[i] = __float2half_rn(v[i]);
  }
}

template <>
__device__ __forceinline__ void store_row32<float>(float* dst, const float (&v)[32], int nvalid) {
  if (nvalid >= 32) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid) dst[i] = v[i];
  }
}

// v[i] += dst[i] for the first nvalid of 32 consecutive elements (accumulating epilogue)
template <typename OutT>
__device__ __forceinline__ void add_row32(const OutT* src, float (&v)[32], int nvalid) {
  if (nvalid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float t[8];
      load8(src + 8 * i, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[8 * i + j] += t[j];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid) v[i] += to_f(src[i]);
  }
}

enum EpiMode : int { kEpiStd = 0, kEpiRowMax = 1, kEpiExp = 2, kEpiRowScale = 3, kEpiDS = 4 };

__device__ __forceinline__ void atomic_max_float(float* addr, float v) {
  if (v >= 0.f) atomicMax(reinterpret_cast<int*>(addr), __float_as_int(v));
  else atomicMin(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

// Per-row state of the fused-softmax epilogues: one thread owns one output row of the tile.
struct EpiRow {
  float a, b, acc;       // a, b: row scalars read once per tile; acc: running max / sum over the tile
};
__device__ __forceinline__ void epi_row_begin(const GemmParams& p, long long ridx, bool row_ok, EpiRow& r) {
  r.a = r.b = 0.f;
  r.acc = p.epi == kEpiRowMax ? -INFINITY : 0.f;
  if (!row_ok) return;
  if (p.epi == kEpiExp) r.a = p.row_in[ridx];
  else if (p.epi == kEpiRowScale || p.epi == kEpiDS) {
    const float s = p.row_in[ridx];
    r.a = s > 0.f ? 1.f / s : 0.f;
    if (p.epi == kEpiDS) r.b = p.row_in2[ridx];
  }
}
__device__ __forceinline__ void epi_row_end(const GemmParams& p, long long ridx, bool row_ok, const EpiRow& r) {
  if (!row_ok) return;
  if (p.epi == kEpiRowMax) { if (r.acc > -INFINITY) atomic_max_float(p.row_out + ridx, r.acc); }
  else if (p.epi == kEpiExp) atomicAdd(p.row_out + ridx, r.acc);
}
// One 32-column chunk of row `row` (v = alpha * acc).
template <typename OutT>
__device__ __forceinline__ void epi_chunk(const GemmParams& p, float (&v)[32], int row, int col0, int nvalid,
                                          long long off, OutT* C, EpiRow& r) {
  const int last = p.mode == 1 ? row + p.causal_off : 0x7fffffff;      // last column that takes part
  if (p.epi == kEpiRowMax) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nvalid && col0 + i <= last) r.acc = fmaxf(r.acc, v[i]);
    return;
  }
  if (p.epi == kEpiExp) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float e = (i < nvalid && col0 + i <= last) ? __expf(v[i] - r.a) : 0.f;
      e = to_f(from_f<OutT>(e));                 // the sum is taken over the values as they are stored
      r.acc += e;
      v[i] = e;
    }
    store_row32<OutT>(C + off, v, nvalid);
    return;
  }
  if (p.epi == kEpiRowScale) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] *= r.a;
    store_row32<OutT>(C + off, v, nvalid);
    return;
  }
  // kEpiDS
  float pt[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) pt[i] = 0.f;
  add_row32<OutT>(reinterpret_cast<const OutT*>(p.aux) + off, pt, nvalid);
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = (i < nvalid && col0 + i <= last) ? pt[i] * r.a * (v[i] - r.b) : 0.f;
  store_row32<OutT>(C + off, v, nvalid);
}

// bias[col, col + 32) added to a thread's 32 columns; columns beyond the last are not read
__device__ __forceinline__ void add_bias32(const GemmParams& p, int col, float (&v)[32]) {
  if (p.bias_vec && col + 32 <= p.N) {
    auto add = [&](auto* bias) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float t[8];
        load8(bias + col + 8 * i, t);      // the same address in every lane
#pragma unroll
        for (int j = 0; j < 8; ++j) v[8 * i + j] += t[j];
      }
    };
    if (p.bias_dtype == kF32) add(reinterpret_cast<const float*>(p.bias));
    else if (p.bias_dtype == kBF16) add(reinterpret_cast<const __nv_bfloat16*>(p.bias));
    else add(reinterpret_cast<const __half*>(p.bias));
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (col + i < p.N) {
      if (p.bias_dtype == kF32) v[i] += reinterpret_cast<const float*>(p.bias)[col + i];
      else if (p.bias_dtype == kBF16) v[i] += __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[col + i]);
      else v[i] += __half2float(reinterpret_cast<const __half*>(p.bias)[col + i]);
    }
  }
}
// SiLU of the epilogues: x / (1 + e^-x) with the quotient from a reciprocal and one step of Newton's iteration on its
// residual (Markstein's correction), which leaves the rounding of the last fused multiply-add: the bits of a division
// without its branch.  The reciprocal is taken of a quarter of the denominator, so that it is normal up to where e^-x
// overflows; there, and for an infinite x, the residual is NaN and the first quotient is the result.  6216 x 1024 -> 2048
// with bias and SiLU 31.0 us, with the division 45.0; 29.6 with a quotient of two units in the last place, which is zero
// below -87.3.
__device__ __forceinline__ float silu_quotient(float x) {
  const float d = 1.f + __expf(-x);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(0.25f * d));
  r *= 0.25f;
  const float q = x * r, e = fmaf(-q, d, x);
  return e == e ? fmaf(e, r, q) : q;
}
__device__ __forceinline__ void silu32(float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = silu_quotient(v[i]);
}

// ---- epilogue through staging buffers.  A thread owns one row of the accumulator, so writing its columns straight to
// global memory makes every warp store touch 32 different lines, 16 bytes each: the load/store unit, not DRAM, then
// bounds products with short k loops.  Instead a warp collects 64 bytes of each of its 32 rows in shared memory and
// moves them with instructions that each cover 8 whole segments of 64 bytes; inputs of the epilogue (the accumulated
// C, an addend, the stored probabilities of the dS epilogue) come in the same way.  Pieces of 16 bytes are
// XOR-swizzled by the row, which makes both directions conflict-free.  Eight warps, two on each quarter
// of the accumulator's lanes, so that two instruction streams per scheduler cover one another's latencies; 2 KiB a warp leave the ring of stages as it is and room for a small kernel beside the CTA.
// us, back to back, before (four warps, bias and pre-activation from scalar accesses in the threads' own rows, the
// whole tile in local memory where a column index was not a constant; pairs alone staged) and after:
//   bias + SiLU   6216 x 1024 -> 2048  99 / 34, 6216 x 1024 -> 1024  68 / 26, 4096 x 4096 -> 8192  286 / 212
//   neither       6216 x 1024 -> 2048  27 / 27, 4096 x 4096 -> 8192  208 / 203
//   scores of a 4096-token chunk, 4 heads of 256: maxima 36 / 31, exponentials 54 / 45
__device__ __forceinline__ uint32_t epi_stage_addr(uint32_t base, int row, int piece) {
  return base + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4);
}
__device__ __forceinline__ void lds128(uint32_t addr, uint4& v) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
template <typename OutT>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  __half2 t = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
template <typename OutT>
__device__ __forceinline__ void unpack2(uint32_t w, float& a, float& b);
template <>
__device__ __forceinline__ void unpack2<__nv_bfloat16>(uint32_t w, float& a, float& b) {
  a = __uint_as_float(w << 16);
  b = __uint_as_float(w & 0xffff0000u);
}
template <>
__device__ __forceinline__ void unpack2<__half>(uint32_t w, float& a, float& b) {
  const __half2 t = *reinterpret_cast<__half2*>(&w);
  a = __low2float(t);
  b = __high2float(t);
}
// 64 bytes of each of 32 rows, global <-> a warp's staging buffer: lane -> piece (lane & 3) of rows (lane >> 2) + 8 j.
// Rows from rows_valid and elements from cols_valid on are left alone.  `vec`: the pieces lie on 16-byte boundaries.
template <typename T>
__device__ __forceinline__ void epi_load(uint4 (&raw)[4], const T* src, long long ld, int rows_valid, int cols_valid,
                                         bool vec, int lane) {
  constexpr int kPiece = 16 / sizeof(T);
  const int c = (lane & 3) * kPiece;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = 8 * j + (lane >> 2);
    raw[j] = make_uint4(0u, 0u, 0u, 0u);
    if (r >= rows_valid) continue;
    const T* s = src + (long long)r * ld + c;
    if (vec && c + kPiece <= cols_valid) {
      raw[j] = *reinterpret_cast<const uint4*>(s);
    } else if (sizeof(T) == 2) {
      uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c + i < cols_valid) w[i / 2] |= (uint32_t)reinterpret_cast<const unsigned short*>(s)[i] << (16 * (i & 1));
      raw[j] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}
__device__ __forceinline__ void epi_stage_in(uint32_t stg, const uint4 (&raw)[4], int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j) sts128(epi_stage_addr(stg, 8 * j + (lane >> 2), lane & 3), raw[j]);
}
template <typename T>
__device__ __forceinline__ void epi_stage_out(uint32_t stg, T* dst, long long ld, int rows_valid, int cols_valid,
                                              bool vec, int lane) {
  constexpr int kPiece = 16 / sizeof(T);
  const int c = (lane & 3) * kPiece;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = 8 * j + (lane >> 2);
    uint4 v;
    lds128(epi_stage_addr(stg, r, lane & 3), v);
    if (r >= rows_valid) continue;
    T* d = dst + (long long)r * ld + c;
    if (vec && c + kPiece <= cols_valid) {
      *reinterpret_cast<uint4*>(d) = v;
    } else if (sizeof(T) == 2) {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c + i < cols_valid) reinterpret_cast<unsigned short*>(d)[i] = (unsigned short)(w[i / 2] >> (16 * (i & 1)));
    } else {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (c + i < cols_valid) reinterpret_cast<uint32_t*>(d)[i] = w[i];
    }
  }
}
// the thread's own row: 32 columns as floats
template <typename OutT>
__device__ __forceinline__ void epi_stage_get(uint32_t stg, int lane, float (&v)[32]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 w;
    lds128(epi_stage_addr(stg, lane, i), w);
    unpack2<OutT>(w.x, v[8 * i + 0], v[8 * i + 1]);
    unpack2<OutT>(w.y, v[8 * i + 2], v[8 * i + 3]);
    unpack2<OutT>(w.z, v[8 * i + 4], v[8 * i + 5]);
    unpack2<OutT>(w.w, v[8 * i + 6], v[8 * i + 7]);
  }
}
// the thread's 32 columns -> row segments of `dst` (first row and column of the warp's block)
template <typename OutT>
__device__ __forceinline__ void epi_store32(uint32_t stg, const float (&v)[32], OutT* dst, long long ld, int rows_valid,
                                            int cols_valid, bool vec, int lane) {
  if constexpr (sizeof(OutT) == 2) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      sts128(epi_stage_addr(stg, lane, i),
             make_uint4(pack2<OutT>(v[8 * i + 0], v[8 * i + 1]), pack2<OutT>(v[8 * i + 2], v[8 * i + 3]),
                        pack2<OutT>(v[8 * i + 4], v[8 * i + 5]), pack2<OutT>(v[8 * i + 6], v[8 * i + 7])));
    __syncwarp();
    epi_stage_out<OutT>(stg, dst, ld, rows_valid, cols_valid, vec, lane);
    __syncwarp();
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        sts128(epi_stage_addr(stg, lane, i),
               make_uint4(__float_as_uint(v[16 * h + 4 * i]), __float_as_uint(v[16 * h + 4 * i + 1]),
                          __float_as_uint(v[16 * h + 4 * i + 2]), __float_as_uint(v[16 * h + 4 * i + 3])));
      __syncwarp();
      epi_stage_out<OutT>(stg, dst + 16 * h, ld, rows_valid, cols_valid - 16 * h, vec, lane);
      __syncwarp();
    }
  }
}
// Per-row constants of the fused epilogues, folded so that an element costs one FMA plus the operation
// itself: exp(alpha s - m) = 2^(s * alpha log2e - m log2e); dS = p~ (s * alpha / l - delta / l).
struct EpiFold {
  float k1, k2;
};
__device__ __forceinline__ EpiFold epi_fold(const GemmParams& p, const EpiRow& er) {
  if (p.epi == kEpiExp) return {p.alpha * 1.4426950408889634f, er.a * 1.4426950408889634f};
  if (p.epi == kEpiRowScale) return {p.alpha * er.a, 0.f};
  if (p.epi == kEpiDS) return {p.alpha * er.a, er.a * er.b};
  return {p.alpha, 0.f};
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 32 columns of the thread's row: raw accumulator `r` -> values to store in `v`.  MASKED: the tile touches
// the diagonal or the last column, and columns beyond `last` give zero (and take no part in maxima / sums); other
// tiles skip the comparison.  The row sum of kEpiExp adds the values before they are rounded to the
// output type.
template <bool MASKED>
__device__ __forceinline__ void epi_compute(const GemmParams& p, const uint32_t (&r)[32], const float (&pt)[32],
                                            float (&v)[32], int last, int col0, const EpiFold& f, EpiRow& er) {
  if (p.epi == kEpiRowMax) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (!MASKED || col0 + i <= last) er.acc = fmaxf(er.acc, __uint_as_float(r[i]) * f.k1);
  } else if (p.epi == kEpiExp) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float e = ex2_approx(fmaf(__uint_as_float(r[i]), f.k1, -f.k2));
      if (MASKED && col0 + i > last) e = 0.f;
      er.acc += e;
      v[i] = e;
    }
  } else if (p.epi == kEpiRowScale) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * f.k1;
  } else {   // kEpiDS
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float d = pt[i] * fmaf(__uint_as_float(r[i]), f.k1, -f.k2);
      v[i] = (MASKED && col0 + i > last) ? 0.f : d;
    }
  }
}

// 32 columns from `col` on of a warp's 32 rows, whose first one lies `off` elements into C.  The read of tensor memory
// and all global reads are under way before the first wait.  SOFTMAX: one of the fused-softmax epilogues (their kernels
// are instances of their own: one kernel for both spills registers).
template <typename OutT, bool SOFTMAX>
__device__ __forceinline__ void epi_staged(const GemmParams& p, uint32_t t_addr, uint32_t stg, long long off,
                                           int rows_valid, int col, int row, int lane, const EpiFold& fold, EpiRow& er) {
  OutT* C = reinterpret_cast<OutT*>(p.C) + off;
  const int cols_valid = p.N - col;
  uint32_t r[32];
  tmem_ld_32x32(t_addr, r);
  const bool need_in = sizeof(OutT) == 2 && (SOFTMAX ? p.epi == kEpiDS : p.accumulate || p.aux != nullptr);
  uint4 in[4];
  if (need_in)
    epi_load<OutT>(in, !SOFTMAX && p.accumulate ? C : reinterpret_cast<const OutT*>(p.aux) + off, p.ldc, rows_valid,
                   cols_valid, !SOFTMAX || p.staged, lane);
  tmem_ld_wait_for(r);
  float v[32], pt[32];
  if (need_in) {
    epi_stage_in(stg, in, lane);
    __syncwarp();
    if constexpr (sizeof(OutT) == 2) epi_stage_get<OutT>(stg, lane, pt);
  }
  if constexpr (!SOFTMAX) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
    if (p.bias != nullptr) add_bias32(p, col, v);
    if (need_in) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] += pt[i];
    }
    if (p.preact != nullptr)
      epi_store32<OutT>(stg, v, reinterpret_cast<OutT*>(p.preact) + off, p.ldc, rows_valid, cols_valid, true, lane);
    if (p.act == 1) silu32(v);
  } else {
    const int last = p.mode == 1 ? min(row + p.causal_off, p.N - 1) : p.N - 1;
    // does any row of this warp end inside these columns?  (warp-uniform)
    if (min(p.mode == 1 ? row - lane + p.causal_off : p.N - 1, p.N - 1) < col + 31)
      epi_compute<true>(p, r, pt, v, last, col, fold, er);
    else
      epi_compute<false>(p, r, pt, v, last, col, fold, er);
    if (p.epi == kEpiRowMax) return;
  }
  epi_store32<OutT>(stg, v, C, p.ldc, rows_valid, cols_valid, !SOFTMAX || p.staged, lane);
}

// 32 columns written straight from the registers: a C that is split over ranks, rows that start off a 16-byte
// boundary, fp32 results with inputs, the softmax epilogues of fp32 results and of the single-CTA kernel
template <typename OutT, bool SOFTMAX>
__device__ __forceinline__ void epi_direct(const GemmParams& p, uint32_t t_addr, int row, int col0, long long cb,
                                           EpiRow& er) {
  OutT* C = reinterpret_cast<OutT*>(p.C);
  OutT* P = reinterpret_cast<OutT*>(p.preact);
  uint32_t r[32];
  tmem_ld_32x32(t_addr, r);
  tmem_ld_wait_for(r);
  if (col0 >= p.N || row >= p.M) return;
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
  const int nvalid = min(32, p.N - col0);
  const long long off = cb + (long long)row * p.ldc + col0;
  if constexpr (SOFTMAX) {
    epi_chunk<OutT>(p, v, row, col0, nvalid, off, C, er);
    return;
  }
  if (p.bias != nullptr) add_bias32(p, col0, v);
  if (p.c_nparts > 1) {
    // push this 32-column chunk into the slot of the rank that owns these columns
    const int owner = col0 / p.c_part_cols;
    OutT* slot = reinterpret_cast<OutT*>(p.c_parts[owner]);
    store_row32<OutT>(slot + (long long)row * p.c_part_cols + (col0 - owner * p.c_part_cols), v, nvalid);
    return;
  }
  if (p.accumulate) add_row32<OutT>(C + off, v, nvalid);
  if (p.aux != nullptr) add_row32<OutT>(reinterpret_cast<const OutT*>(p.aux) + off, v, nvalid);   // + addend
  if (P != nullptr) store_row32<OutT>(P + off, v, nvalid);
  if (p.act == 1) silu32(v);
  store_row32<OutT>(C + off, v, nvalid);
}

template <int BN, bool A_MN, bool B_MN, typename OutT>
__global__ void __launch_bounds__(SmemLayout<BN>::threads, 1)
gemm_tcgen05_kernel(const __grid_constant__ TmapArray tmaps_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ GemmParams p, int in_fmt) {
  using L = SmemLayout<BN>;
  constexpr int kStages = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::bar_offset);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* tmem_full = empty_bar + kStages;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_m = (p.M + BM - 1) / BM;
  const int num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n * p.batch;
  const int num_k = (p.K + BK - 1) / BK;
  constexpr uint32_t kTmemCols = 2 * BN;     // two accumulators (a power of two)

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full_bar + i, 1);
      mbar_init(empty_bar + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tmem_full + i, 1);
      mbar_init(tmem_empty + i, p.epi != kEpiStd ? 4 : L::epi_warps);    // epilogue warps of a tile
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_holder, kTmemCols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  begin_dependent();        // barriers and tensor memory are set up under the end of the kernel before

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      for (int i = 0; i < p.a_parts; ++i) prefetch_tmap(&tmaps_a.m[i]);
      prefetch_tmap(&tmap_b);
      const int kb_shift = p.a_parts > 1 ? p.a_first * (p.a_part_k / BK) : 0;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const TileCoord tc = decode_tile<BN>(tile, num_m, num_n, p.band);
        const int m0 = tc.m0, n0 = tc.n0, bo = tc.bz / p.batch_in, bi = tc.bz - bo * p.batch_in;
        if (tile_skipped<BN>(p, m0, n0)) continue;
        int kb0, kb1;
        k_range(p, m0, num_k, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(empty_bar + stage, phase ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + stage * L::stage_bytes;
          uint8_t* sb = sa + L::a_bytes;
          mbar_expect_tx(full_bar + stage, L::stage_bytes);
          // with a gathered A the K walk is rotated so that every rank starts on its own piece
          const int kbr = p.a_parts > 1 ? (kb + kb_shift) % num_k : kb;
          const int k0 = kbr * BK;
          const int part = p.a_parts > 1 ? k0 / p.a_part_k : 0;
          const int ka = p.a_parts > 1 ? k0 - part * p.a_part_k : k0;     // column inside the piece
          const CUtensorMap* tmap_a = &tmaps_a.m[part];
          if constexpr (!A_MN) {
            tma_load_4d(sa, tmap_a, full_bar + stage, ka, m0, bi, bo);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_4d(sa + j * 8192, tmap_a, full_bar + stage, m0 + 64 * j, ka, bi, bo);
          }
          if constexpr (!B_MN) {
            tma_load_4d(sb, &tmap_b, full_bar + stage, k0, n0, bi, bo);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_4d(sb + j * 8192, &tmap_b, full_bar + stage, n0 + 64 * j, k0, bi, bo);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.err, 1); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(BM, BN, in_fmt, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const TileCoord tc = decode_tile<BN>(tile, num_m, num_n, p.band);
        const int m0 = tc.m0, n0 = tc.n0;
        if (tile_skipped<BN>(p, m0, n0)) continue;
        int kb0, kb1;
        k_range(p, m0, num_k, kb0, kb1);
        if (!wait_or_abort(tmem_empty + acc, acc_phase ^ 1, abort_flag)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(full_bar + stage, phase, abort_flag)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t sa = smem_u32(smem + stage * L::stage_bytes);
          const uint32_t sb = sa + L::a_bytes;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            const uint64_t da = A_MN ? make_smem_desc(sa + kk * 2048, 8192, 1024)
                                     : make_smem_desc(sa + kk * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + kk * 2048, 8192, 1024)
                                     : make_smem_desc(sb + kk * 32, 16, 1024);
            umma_f16(d_tmem, da, db, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
          }
          umma_commit(empty_bar + stage);      // stage reusable once these MMAs have read it
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(tmem_full + acc);          // accumulator complete
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.err, 2); }
    }
  } else {
    // ------------------------------------------------------------ epilogue (the other warps)
    const int quarter = warp & 3;              // TMEM lanes [32 * quarter, +32) belong to this warp
    // Eight warps share a tile's columns; with a softmax epilogue each four take every other tile, whole rows of it, so
    // that a row's maximum and sum get one contribution from a tile.
    constexpr int kGroups = L::epi_warps / 4;
    const bool by_tile = p.epi != kEpiStd;
    const int group = (warp - 2) / 4;
    const int cols = by_tile ? BN : BN / kGroups, col_off = by_tile ? 0 : group * cols;
    const uint32_t stage_buf = smem_u32(smem + L::epi_offset + (warp - 2) * kEpiStageBytes);
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      const TileCoord tc = decode_tile<BN>(tile, num_m, num_n, p.band);
      const int m0 = tc.m0, n0 = tc.n0 + col_off;
      if (tile_skipped<BN>(p, m0, tc.n0)) continue;
      if (kGroups == 2 && by_tile && acc != group) {
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      if (!wait_or_abort(tmem_full + acc, acc_phase, abort_flag)) { ok = false; break; }
      tcgen05_fence_after();
      const int row_base = m0 + quarter * 32, row = row_base + lane;
      const uint32_t t_row = tmem_base + acc * BN + col_off + ((uint32_t)(quarter * 32) << 16);
      const long long ridx = (long long)tc.bz * p.M + row;
      const long long cb = c_base(p, tc.bz);
      EpiRow er;
      if (p.epi != kEpiStd) epi_row_begin(p, ridx, row < p.M, er);
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        const int col = n0 + c;
        if (col >= p.N) break;                // warp-uniform
        if (p.epi != kEpiStd) {
          epi_direct<OutT, true>(p, t_row + c, row, col, cb, er);
        } else if (p.staged) {
          epi_staged<OutT, false>(p, t_row + c, stage_buf, cb + (long long)row_base * p.ldc + col, p.M - row_base, col,
                                  row, lane, EpiFold{}, er);
        } else {
          epi_direct<OutT, false>(p, t_row + c, row, col, cb, er);
        }
      }
      if (p.epi != kEpiStd) epi_row_end(p, ridx, row < p.M, er);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty + acc);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 3); }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------- CTA-pair variant
// Same roles and pipeline, but two CTAs of a 2-CTA cluster share one 256 x 256 output tile through
// tcgen05.mma.cta_group::2: CTA r stages rows [m0 + 128 r, +128) of A and rows [n0 + 128 r, +128) of
// B, so each SM streams 32 KiB per k-block instead of 48 KiB and the ring is 6 stages deep.  The even
// CTA issues the MMAs; every "stage consumed" and "accumulator ready" signal is committed once to
// each CTA's barrier, and both CTAs' epilogue warps release the accumulator on the even CTA's barrier.
constexpr int kPairStages = 6;
constexpr int kPairBM = 256;      // rows of the pair's tile
constexpr int kPairBN = 256;
constexpr int kPairTile = 512;    // name of this variant among the tiles (the others go by their width)

struct PairSmem {
  static constexpr int a_bytes = BM * BK * 2;                 // this CTA's 128 rows of A
  static constexpr int b_bytes = (kPairBN / 2) * BK * 2;      // this CTA's 128 rows of B
  static constexpr int stage_bytes = a_bytes + b_bytes;       // 32 KiB
  static constexpr int bar_offset = kPairStages * stage_bytes;
  static constexpr int epi_offset = bar_offset + 256;
  static constexpr int total = epi_offset + 8 * kEpiStageBytes + 1024;
};
// Epilogue warps; the gathering variant keeps its other four for the copies.
constexpr int pair_epi_warps(bool gather) { return gather ? 4 : 8; }

__device__ __forceinline__ bool pair_tile_skipped(const GemmParams& p, int m0, int n0) {
  return p.mode == 1 && n0 > m0 + kPairBM - 1;
}

__device__ __forceinline__ void pair_k_range(const GemmParams& p, int m0, int num_k, int& kb0, int& kb1) {
  kb0 = 0;
  kb1 = num_k;
  if (p.mode == 2) kb1 = min(num_k, (m0 + kPairBM + BK - 1) / BK);
  if (p.mode == 3) kb0 = min(num_k - 1, m0 / BK);
}

constexpr int kGatherWarps = 4;                 // copy warps of the gathering variant
constexpr int kPairThreads = 64 + 32 * 8;       // producer, MMA issuer and eight epilogue (and copy) warps
static_assert(pair_epi_warps(true) + kGatherWarps == pair_epi_warps(false), "both variants have ten warps");
constexpr int kGatherUnitBytes = 8192;          // one claim: 32 lanes x 16 loads of 16 bytes

// Tiles of one batch element that the kernel computes: with mode 1 (causal scores) only those on or below
// the diagonal.
__device__ __forceinline__ int pair_tiles_per_batch(const GemmParams& p, int num_m, int num_n) {
  if (p.mode != 1) return num_m * num_n;
  int t = 0;
  for (int mt = 0; mt < num_m; ++mt) t += min(mt + 1, num_n);
  return t;
}

// Tile -> (m0, n0, batch).  With a gathered B the n-tiles are walked starting at this rank's own rows,
// whose chunks are copied first.  The causal modes hand every CTA pair tiles `pair, pair + P, ...` of an
// ORDER chosen for balance: mode 1 numbers only the tiles it computes (the plain order left a pair with up
// to 10 of them against a mean of 7.4); modes 2 and 3, whose k loop grows with the distance from the
// diagonal, order all tiles of all batch elements from the longest k loop to the shortest and deal them
// out in alternating direction (the plain order: 0.84 of the mean on the busiest pair, this one 0.97).
__device__ __forceinline__ void pair_tile_coords(const GemmParams& p, int tile, int num_m, int num_n,
                                                 int tiles_per_batch, int num_pairs, int& m0, int& n0, int& bz) {
  if (p.mode >= 1 && p.mode <= 3 && p.g_world == 0) {
    const int num_tiles = tiles_per_batch * p.batch;
    const int round = tile / num_pairs;
    int pos = tile - round * num_pairs;
    if (round & 1) pos = min(num_pairs, num_tiles - round * num_pairs) - 1 - pos;
    const int i = round * num_pairs + pos;
    int mt, nt;
    if (p.mode == 1) {
      bz = i / tiles_per_batch;
      int t = i - bz * tiles_per_batch;
      mt = 0;
      while (t >= min(mt + 1, num_n)) {
        t -= min(mt + 1, num_n);
        ++mt;
      }
      nt = t;
    } else {
      const int per_m = num_n * p.batch;
      const int q = i / per_m, rem = i - q * per_m;
      mt = p.mode == 2 ? num_m - 1 - q : q;       // longest k loop first
      bz = rem / num_n;
      nt = rem - bz * num_n;
    }
    m0 = mt * kPairBM;
    n0 = nt * kPairBN;
    return;
  }
  bz = tile / tiles_per_batch;
  const int t = tile - bz * tiles_per_batch;
  int mt, nt;
  banded_tile(t, num_m, num_n, p.band, mt, nt);
  if (p.g_world > 0) {
    nt += (int)(((long long)p.g_rank * (p.N / p.g_world)) / kPairBN);
    if (nt >= num_n) nt -= num_n;
  }
  m0 = mt * kPairBM;
  n0 = nt * kPairBN;
}

__device__ __forceinline__ unsigned int ld_acquire_gpu_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Bounded wait until chunk `chunk` of the gathered matrix is complete in local memory.
__device__ __forceinline__ bool wait_chunk(const GemmParams& p, int chunk, volatile int* abort_flag) {
  const unsigned int need = (unsigned int)(p.K / 32);
  const unsigned int* flag = p.g_flags + 1 + chunk;
  if (ld_acquire_gpu_u32(flag) < need) {
    const unsigned long long t0 = globaltimer_ns();
    uint32_t spins = 0;
    while (ld_acquire_gpu_u32(flag) < need) {
      if ((++spins & 0x3f) == 0) {
        if (*abort_flag) return false;
        if (globaltimer_ns() - t0 > kWaitTimeoutNs) return false;
      }
      __nanosleep(64);
    }
  }
  fence_proxy_async_all();        // the copy warps wrote through the generic proxy, TMA reads through the async one
  return true;
}

// Body of one copy warp: claim 8 KiB units until none is left.  Never waits for anything.
__device__ __forceinline__ void gather_copy_warp(const GemmParams& p, int lane) {
  const int nchunks = p.N / 128;
  const int upc = p.K / 32;                              // 8 KiB units per 128-row chunk (K * 256 B / 8192)
  const int total = nchunks * upc;
  const int rows_per_rank = p.N / p.g_world;
  const int first_chunk = (int)(((long long)p.g_rank * rows_per_rank) / 128);
  while (true) {
    unsigned int u = 0;
    if (lane == 0) u = atomicAdd(p.g_flags, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= (unsigned int)total) break;
    const int oc = (int)u / upc, sub = (int)u - oc * upc;
    int chunk = oc + first_chunk;
    if (chunk >= nchunks) chunk -= nchunks;
    const int row0 = chunk * 128;
    const int owner = row0 / rows_per_rank;
    const long long src_byte = (long long)(row0 - owner * rows_per_rank) * p.K * 2 + (long long)sub * kGatherUnitBytes;
    const long long dst_byte = (long long)row0 * p.K * 2 + (long long)sub * kGatherUnitBytes;
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p.g_src[owner]) + src_byte);
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<char*>(p.g_dst) + dst_byte);
    uint4 v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __ldcv(src + lane + 32 * i);
#pragma unroll
    for (int i = 0; i < 16; ++i) dst[lane + 32 * i] = v[i];
    fence_proxy_async_all();
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(p.g_flags + 1 + chunk, 1u);
  }
}

template <bool A_MN, bool B_MN, typename OutT, bool GATHER = false, bool SOFTMAX = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ TmapArray tmaps_a, const __grid_constant__ CUtensorMap tmap_b,
                         const __grid_constant__ GemmParams p, int in_fmt) {
  using L = PairSmem;
  constexpr int kEpi = pair_epi_warps(GATHER);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::bar_offset);     // used in the even CTA only
  uint64_t* empty_bar = full_bar + kPairStages;                               // one set per CTA
  uint64_t* tmem_full = empty_bar + kPairStages;                              // one set per CTA
  uint64_t* tmem_empty = tmem_full + 2;                                       // used in the even CTA only
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();          // 0 = even CTA (issues the MMAs), 1 = its peer
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int num_m = (p.M + kPairBM - 1) / kPairBM;
  const int num_n = (p.N + kPairBN - 1) / kPairBN;
  const int tiles_per_batch = pair_tiles_per_batch(p, num_m, num_n);
  const int num_tiles = tiles_per_batch * p.batch;
  const int num_k = (p.K + BK - 1) / BK;
  constexpr uint32_t kTmemCols = 2 * kPairBN;       // two accumulators of 256 columns

  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairStages; ++i) {
      mbar_init(full_bar + i, 2);                   // one arrive.expect_tx from each CTA's producer
      mbar_init(empty_bar + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(tmem_full + i, 1);
      mbar_init(tmem_empty + i, SOFTMAX ? 8 : 2 * kEpi);   // epilogue warps of a tile in both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_holder, kTmemCols);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                               // the peer's barriers exist before anything signals them
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  begin_dependent();        // barriers and tensor memory are set up under the end of the kernel before

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      for (int i = 0; i < p.a_parts; ++i) prefetch_tmap(&tmaps_a.m[i]);
      prefetch_tmap(&tmap_b);
      const int kb_shift = p.a_parts > 1 ? p.a_first * (p.a_part_k / BK) : 0;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        int m0, n0, bz;
        pair_tile_coords(p, tile, num_m, num_n, tiles_per_batch, num_pairs, m0, n0, bz);
        if (pair_tile_skipped(p, m0, n0)) continue;
        const int my_m = m0 + (int)rank * BM;
        const int bo = bz / p.batch_in, bi = bz - bo * p.batch_in;
        const int my_n = n0 + (int)rank * (kPairBN / 2);
        int kb0, kb1;
        pair_k_range(p, m0, num_k, kb0, kb1);
        if constexpr (GATHER) {
          // this CTA's 128 rows of B are exactly one chunk of the gathered matrix
          if (my_n < p.N && !wait_chunk(p, my_n / 128, abort_flag)) { ok = false; break; }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(empty_bar + stage, phase ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* sa = smem + stage * L::stage_bytes;
          uint8_t* sb = sa + L::a_bytes;
          const uint32_t full0 = map_to_cta(smem_u32(full_bar + stage), 0);
          mbar_expect_tx_cluster(full0, L::stage_bytes);
          const int kbr = p.a_parts > 1 ? (kb + kb_shift) % num_k : kb;
          const int k0 = kbr * BK;
          const int part = p.a_parts > 1 ? k0 / p.a_part_k : 0;
          const int ka = p.a_parts > 1 ? k0 - part * p.a_part_k : k0;
          const CUtensorMap* tmap_a = &tmaps_a.m[part];
          if constexpr (!A_MN) {
            tma_load_4d_pair(sa, tmap_a, full0, ka, my_m, bi, bo);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_4d_pair(sa + j * 8192, tmap_a, full0, my_m + 64 * j, ka, bi, bo);
          }
          if constexpr (!B_MN) {
            tma_load_4d_pair(sb, &tmap_b, full0, k0, my_n, bi, bo);
          } else {
#pragma unroll
            for (int j = 0; j < kPairBN / 128; ++j)
              tma_load_4d_pair(sb + j * 8192, &tmap_b, full0, my_n + 64 * j, k0, bi, bo);
          }
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.err, 1); }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA only)
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_f16(kPairBM, kPairBN, in_fmt, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        int m0, n0, bz;
        pair_tile_coords(p, tile, num_m, num_n, tiles_per_batch, num_pairs, m0, n0, bz);
        if (pair_tile_skipped(p, m0, n0)) continue;
        int kb0, kb1;
        pair_k_range(p, m0, num_k, kb0, kb1);
        if (!wait_or_abort(tmem_empty + acc, acc_phase ^ 1, abort_flag)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kPairBN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(full_bar + stage, phase, abort_flag)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t sa = smem_u32(smem + stage * L::stage_bytes);
          const uint32_t sb = sa + L::a_bytes;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            const uint64_t da = A_MN ? make_smem_desc(sa + kk * 2048, 8192, 1024)
                                     : make_smem_desc(sa + kk * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + kk * 2048, 8192, 1024)
                                     : make_smem_desc(sb + kk * 32, 16, 1024);
            umma_f16_pair(d_tmem, da, db, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
          }
          // the stage is reusable in both CTAs once these MMAs have read it
          const uint32_t e = smem_u32(empty_bar + stage);
          umma_commit_pair(e);
          umma_commit_pair(map_to_cta(e, 1));
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        const uint32_t f = smem_u32(tmem_full + acc);
        umma_commit_pair(f);
        umma_commit_pair(map_to_cta(f, 1));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok) { *abort_flag = 1; atomicExch(p.err, 2); }
    }
  } else if (GATHER && warp >= 2 + kEpi) {
    // ------------------------------------------------------------ copy warps (gathering variant)
    gather_copy_warp(p, lane);
  } else {
    // ------------------------------------------------------------ epilogue (the other warps, both CTAs)
    const int quarter = warp & 3;
    // Eight warps share a tile's columns.  With a softmax epilogue each four take every other tile, whole rows of it, so
    // that a row's maximum and sum get one contribution from a tile.
    constexpr int kGroups = kEpi / 4;
    constexpr int kCols = SOFTMAX ? kPairBN : kPairBN / kGroups;
    constexpr bool kAlways = SOFTMAX && sizeof(OutT) == 2;
    const int group = (warp - 2) / 4;
    const int col_off = SOFTMAX ? 0 : group * kCols;
    const uint32_t stage_buf = smem_u32(smem + L::epi_offset + (warp - 2) * kEpiStageBytes);
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int m0, n0, bz;
      pair_tile_coords(p, tile, num_m, num_n, tiles_per_batch, num_pairs, m0, n0, bz);
      if (pair_tile_skipped(p, m0, n0)) continue;
      if (SOFTMAX && kGroups == 2 && acc != group) {
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      if (!wait_or_abort(tmem_full + acc, acc_phase, abort_flag)) { ok = false; break; }
      tcgen05_fence_after();
      n0 += col_off;
      const int row_base = m0 + (int)rank * BM + quarter * 32, row = row_base + lane;
      const uint32_t t_row = tmem_base + acc * kPairBN + col_off + ((uint32_t)(quarter * 32) << 16);
      const long long ridx = (long long)bz * p.M + row;
      const long long cb = c_base(p, bz);
      EpiRow er;
      if constexpr (SOFTMAX) epi_row_begin(p, ridx, row < p.M, er);
      const EpiFold fold = SOFTMAX ? epi_fold(p, er) : EpiFold{};
#pragma unroll 1
      for (int c = 0; c < kCols; c += 32) {
        const int col = n0 + c;
        if (col >= p.N) break;                // warp-uniform
        if (kAlways || p.staged) {
          epi_staged<OutT, SOFTMAX>(p, t_row + c, stage_buf, cb + (long long)row_base * p.ldc + col,
                                    p.M - row_base, col, row, lane, fold, er);
        } else {
          epi_direct<OutT, SOFTMAX>(p, t_row + c, row, col, cb, er);
        }
      }
      if constexpr (SOFTMAX) epi_row_end(p, ridx, row < p.M, er);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(tmem_empty + acc), 0));
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (!ok && lane == 0) { *abort_flag = 1; atomicExch(p.err, 3); }
  }

  // Neither CTA may leave (or free tensor memory) while the other can still signal its barriers,
  // read its shared memory or write its accumulator.
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// ---------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

}  // namespace

// 4-D bf16/fp16 tensor map [outer batch, batch, outer, inner] (inner contiguous) with a {1, 1, box_outer,
// box_inner} box.  Strides are in elements and must be multiples of 8 (16 bytes).
static bool encode_tmap(CUtensorMap* out, const void* base, long long inner, long long outer, long long batch,
                        long long batch2, long long row_stride, long long batch_stride, long long batch2_stride,
                        int box_inner, int box_outer, int elem_dtype, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return false;
  // The encoder is a driver entry point and needs a current context; a thread that has made no
  // runtime call yet (the autograd engine's worker on its first backward) has none bound.
  static thread_local bool context_bound = false;
  if (!context_bound) {
    cudaFree(nullptr);
    context_bound = true;
  }
  if (batch <= 1) batch_stride = row_stride * outer;      // unused, but must be a valid stride
  if (batch2 <= 1) batch2_stride = batch_stride;
  const cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)(batch < 1 ? 1 : batch),
                              (cuuint64_t)(batch2 < 1 ? 1 : batch2)};
  const cuuint64_t strides[3] = {(cuuint64_t)row_stride * 2, (cuuint64_t)batch_stride * 2, (cuuint64_t)batch2_stride * 2};
  const cuuint32_t box[4] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = elem_dtype == kBF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const CUresult res = fn(out, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS)
    fprintf(stderr,
            "tensor map encode failed (CUresult %d): base %p dims {%llu, %llu, %llu, %llu} strides {%llu, %llu, %llu} B "
            "box {%u, %u}\n",
            (int)res, base, (unsigned long long)dims[0], (unsigned long long)dims[1], (unsigned long long)dims[2],
            (unsigned long long)dims[3], (unsigned long long)strides[0], (unsigned long long)strides[1],
            (unsigned long long)strides[2], box[0], box[1]);
  return res == CUDA_SUCCESS;
}

// ... with 128-byte swizzle
bool make_tmap_4d(CUtensorMap* out, const void* base, long long inner, long long outer, long long batch,
                  long long batch2, long long row_stride, long long batch_stride, long long batch2_stride,
                  int box_inner, int box_outer, int elem_dtype) {
  return encode_tmap(out, base, inner, outer, batch, batch2, row_stride, batch_stride, batch2_stride, box_inner, box_outer,
                     elem_dtype, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Map of a contiguous 16-bit matrix [rows, width], box [box_rows, box_width] row by row without swizzle.
bool make_tmap_rows(CUtensorMap* out, const void* base, long long width, long long rows, int box_width, int box_rows,
                    int elem_dtype) {
  return encode_tmap(out, base, width, rows, 1, 1, width, width * rows, width * rows, box_width, box_rows, elem_dtype,
                     CU_TENSOR_MAP_SWIZZLE_NONE);
}

template <int BN, bool A_MN, bool B_MN, typename OutT>
static int launch_gemm(const TmapArray& ta, const CUtensorMap& tb, const GemmParams& p, int in_fmt, int sms,
                       cudaStream_t st) {
  using L = SmemLayout<BN>;
  auto kern = gemm_tcgen05_kernel<BN, A_MN, B_MN, OutT>;
  static std::atomic<unsigned long long> configured{0};
  if (!allow_dynamic_smem(kern, L::total, configured)) return -2;
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN) * p.batch;
  const int grid = tiles < sms ? tiles : sms;
  return launch_dependent(kern, grid, L::threads, L::total, st, ta, tb, p, in_fmt) == cudaSuccess ? 0 : -3;
}

// Pair kernel with copy warps that gather the K-major weight operand from its owners while the tensor
// cores work (see GemmParams::g_*).  The claim counter and the chunk flags are cleared on the stream first.
template <typename OutT>
static int launch_gemm_pair_gather(const TmapArray& ta, const CUtensorMap& tb, const GemmParams& p, int in_fmt,
                                   int sms, cudaStream_t st) {
  using L = PairSmem;
  auto kern = gemm_tcgen05_pair_kernel<false, false, OutT, true>;
  static std::atomic<unsigned long long> configured{0};
  if (!allow_dynamic_smem(kern, L::total, configured)) return -2;
  if (cudaMemsetAsync(p.g_flags, 0, sizeof(unsigned int) * (1 + p.N / 128), st) != cudaSuccess) return -8;
  const int tiles = ((p.M + kPairBM - 1) / kPairBM) * ((p.N + kPairBN - 1) / kPairBN) * p.batch;
  const int pairs = sms / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  kern<<<grid, kPairThreads, L::total, st>>>(ta, tb, p, in_fmt);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <bool A_MN, bool B_MN, typename OutT, bool SOFTMAX>
static int launch_gemm_pair(const TmapArray& ta, const CUtensorMap& tb, const GemmParams& p, int in_fmt, int sms,
                            cudaStream_t st) {
  using L = PairSmem;
  auto kern = gemm_tcgen05_pair_kernel<A_MN, B_MN, OutT, false, SOFTMAX>;
  static std::atomic<unsigned long long> configured{0};
  if (!allow_dynamic_smem(kern, L::total, configured)) return -2;
  const int tiles = ((p.M + kPairBM - 1) / kPairBM) * ((p.N + kPairBN - 1) / kPairBN) * p.batch;
  const int pairs = sms / 2;
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  return launch_dependent(kern, grid, kPairThreads, L::total, st, ta, tb, p, in_fmt) == cudaSuccess ? 0 : -3;
}

static bool g_use_pair = true;

// Which tile a product runs on: the one whose estimate is lowest,
//   (waves - 1) * max(k-blocks * t, e) + k-blocks * t + c,   t = max(latency, bytes of the resident tiles / rate).
// Constants fitted to back-to-back launches (each beginning under the end of the one before) of 849 products: 64 to 20000
// rows, 64 to 32000 columns, K from 64 to 65536, in three layouts; the choice is 0.1 % off the best tile over all of them and
// 9 % at the worst (constants fitted to K up to 4864 alone: 2.2 and 29 %):
//   latency per k-block   0.280 us as a CTA pair, 0.320 as 128 x 256, 0.189 as 128 x 128 and 128 x 64 (what a ring of
//                         6, 4, 6, 8 stages leaves of a memory latency)
//   epilogue e            2.85 / 5.08 / 2.30 / 1.91 us a tile, hidden behind the next tile's loop except at the end
//   start and end c       7.30 / 4.71 / 4.39 / 3.80 us
//   rate                  19.6 TB/s out of L2 and memory together, which the narrow tiles reach first
// Few wide tiles leave most SMs without work: 1024 x 512 x 512 takes 9.6 us in 8 pair tiles and 6.1 us in 64 tiles of
// 128 x 64, 2000 x 1024 x 2560 19.4 us in pairs and 13.4 us as 128 x 128; 4000 x 2048 x 4096 48 us in pairs, 59 as
// 128 x 128 and 87 as 128 x 64; with a long sum pairs lose least to a k-block: 513 x 4096 x 16384 84 us in pairs, 101 as
// 128 x 256, 111 as 128 x 128.
static int pick_tile(const GemmParams& p, int num_sms) {
  const bool pair_ok = g_use_pair && p.M > BM && num_sms >= 2;
  if (p.a_parts > 1 || p.c_nparts > 1) return pair_ok ? kPairTile : 256;
  // The causal products of one attention write and read the same scores at the granularity of their row tiles:
  // what Q K^T skips above the diagonal P V must not contract.  All of them see the same number of rows, so the row
  // tile may depend on nothing else.
  if (p.mode != 0 && pair_ok) return kPairTile;
  const double nk = (p.K + BK - 1) / BK, rate = 19.6e6;      // bytes per us
  struct Tile { int name, bm, bn; double lat, bytes, e, c; };
  const Tile tiles[] = {{kPairTile, kPairBM, kPairBN, 0.280, 65536, 2.85, 7.30},
                        {256, BM, 256, 0.320, 49152, 5.08, 4.71},
                        {128, BM, 128, 0.189, 32768, 2.30, 4.39},
                        {64, BM, 64, 0.189, 24576, 1.91, 3.80}};
  int best = 256;
  double best_us = 1e30;
  for (const Tile& t : tiles) {
    if (t.name == kPairTile && !pair_ok) continue;
    const long long n = (long long)((p.M + t.bm - 1) / t.bm) * ((p.N + t.bn - 1) / t.bn) * p.batch;
    const int slots = t.name == kPairTile ? num_sms / 2 : num_sms;
    const double resident = n < slots ? (double)n : (double)slots;
    const double loop = nk * (t.lat > t.bytes * resident / rate ? t.lat : t.bytes * resident / rate);
    const double us = (double)((n + slots - 1) / slots - 1) * (loop > t.e ? loop : t.e) + loop + t.c;
    if (us < best_us) {
      best_us = us;
      best = t.name;
    }
  }
  return best;
}

// Row tiles (of `bm` rows) of a band of the tile walk: equal bands of at most 4096 rows.  What runs together reads a
// band of A and the few column tiles of B next to each other in the walk.  Without bands, 16384 rows of A (134 MB at
// K = 4096) pass through L2 once per column of tiles: 4 GB out of memory for a product of 0.4 GB of operands, and the
// energy of it comes out of the tensor cores' clock.  16384 x 4096 -> 8192, back to back under the power cap: 1057 us
// at 915 MHz without bands, 875 with bands of 1024 rows, 850 of 2304, 831 of 4096, 839 of 6144; 16384 x 11264 -> 4096
// 1469 -> 1208; 4096 rows are 2 to 3 % slower in two bands than in one.
static int row_band(int M, int bm) {
  const int num_m = (M + bm - 1) / bm, most = 4096 / bm;
  const int bands = (num_m + most - 1) / most;
  return (num_m + bands - 1) / bands;
}

int gemm_tile(int M, int N, int K, int batch, int num_sms) {
  GemmParams p = {};
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.a_parts = p.c_nparts = 1;
  return pick_tile(p, num_sms);
}

// Returns 0 on success, negative on a host-side failure.  `err` is a device int
// that the kernel sets non-zero if one of its bounded waits gives up.
int gemm_bf16_tcgen05(const void* A, const void* B, void* C, void* preact, const void* bias, int bias_dtype,
                      int act, int M, int N, int K, long long lda, long long ldb, long long ldc, bool a_mn,
                      bool b_mn, int mode, float alpha, int batch, long long a_bs, long long b_bs, long long c_bs,
                      int in_dtype, int out_dtype, int* err, int num_sms, cudaStream_t st,
                      const GemmPeerSpec* peers, bool accumulate, const GemmGatherSpec* gather,
                      const GemmSoftmaxSpec* softmax, const GemmOuterBatch* outer, int tile) {
  const int nb2 = outer != nullptr ? outer->count : 1;
  if (M <= 0 || N <= 0 || batch <= 0 || nb2 <= 0) return 0;
  if (K <= 0) return -12;      // (an empty sum is the caller's: no tile would write it)
  // TMA wants 16-byte strides; the vectorised epilogue wants 16-byte aligned rows of C
  if (lda % 8 != 0 || ldb % 8 != 0 || ldc % 8 != 0) return -1;
  if (batch > 1 && (a_bs % 8 != 0 || b_bs % 8 != 0 || c_bs % 8 != 0)) return -1;
  const long long a_bs2 = outer != nullptr ? outer->a_stride : 0, b_bs2 = outer != nullptr ? outer->b_stride : 0;
  if (nb2 > 1 && (a_bs2 % 8 != 0 || b_bs2 % 8 != 0 || outer->c_stride % 8 != 0)) return -1;
  TmapArray ta;
  CUtensorMap tb;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.C = C; p.preact = preact; p.bias = bias; p.bias_dtype = bias_dtype; p.act = act;
  p.err = err; p.ldc = ldc; p.mode = mode; p.alpha = alpha; p.batch = batch * nb2; p.batch_in = batch;
  p.c_batch_stride = c_bs; p.c_outer_stride = outer != nullptr ? outer->c_stride : 0;
  p.a_parts = 1; p.a_part_k = K; p.a_first = 0; p.c_nparts = 1; p.c_part_cols = N;
  p.accumulate = accumulate ? 1 : 0;
  if (softmax != nullptr && softmax->kind == 0 && softmax->aux != nullptr) {
    if (peers != nullptr && peers->c_nparts > 1) return -10;
    p.aux = softmax->aux;              // standard epilogue with an addend of C's layout
  }
  if (softmax != nullptr && softmax->kind != 0) {
    if (softmax->kind < 1 || softmax->kind > 4 || bias != nullptr || act != 0 || preact != nullptr || accumulate ||
        peers != nullptr)
      return -10;
    p.epi = softmax->kind; p.row_in = softmax->row_in; p.row_in2 = softmax->row_in2; p.row_out = softmax->row_out;
    p.aux = softmax->aux; p.causal_off = softmax->causal_off;
  }
  bool ok = true;
  if (peers != nullptr && peers->a_parts > 1) {
    // gathered A: K-major pieces [M, K / parts] living on different GPUs
    if (a_mn || p.batch != 1 || peers->a_parts > kMaxPeers || K % peers->a_parts != 0) return -6;
    p.a_parts = peers->a_parts;
    p.a_part_k = K / peers->a_parts;
    p.a_first = peers->a_first;
    if (p.a_part_k % BK != 0) return -6;
    for (int i = 0; i < p.a_parts; ++i)
      ok = ok && make_tmap_4d(&ta.m[i], peers->a_ptrs[i], p.a_part_k, M, 1, 1, lda, 0, 0, BK, BM, in_dtype);
  } else {
    ok = a_mn ? make_tmap_4d(&ta.m[0], A, M, K, batch, nb2, lda, a_bs, a_bs2, 64, 64, in_dtype)
              : make_tmap_4d(&ta.m[0], A, K, M, batch, nb2, lda, a_bs, a_bs2, BK, BM, in_dtype);
  }
  if (peers != nullptr && peers->c_nparts > 1) {
    if (p.batch != 1 || peers->c_nparts > kMaxPeers || N % peers->c_nparts != 0) return -7;
    p.c_nparts = peers->c_nparts;
    p.c_part_cols = N / peers->c_nparts;
    if (p.c_part_cols % 32 != 0) return -7;
    for (int i = 0; i < p.c_nparts; ++i) p.c_parts[i] = peers->c_ptrs[i];
  }
  if (!ok) return -41;
  {
    const bool f32 = out_dtype == kF32;
    const long long strides = ldc | (batch > 1 ? c_bs : 0) | (nb2 > 1 ? outer->c_stride : 0);
    const uintptr_t bases = reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(preact) |
                            reinterpret_cast<uintptr_t>(p.aux);
    p.staged = p.c_nparts == 1 && (strides & (f32 ? 3 : 7)) == 0 && (bases & 15) == 0 &&
               !(f32 && (p.epi != kEpiStd || p.accumulate || p.aux != nullptr)) &&
               !(p.epi == kEpiStd && p.accumulate && p.aux != nullptr);
    p.bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
  }
  if (gather != nullptr && gather->world > 0) tile = kPairTile;
  if (tile == 0) tile = pick_tile(p, num_sms);
  if (tile != kPairTile && tile != 64 && tile != 128 && tile != 256) return -11;
  const bool pair = tile == kPairTile && g_use_pair;
  p.band = row_band(M, pair ? kPairBM : BM);
  if (gather != nullptr && gather->world > 0) {
    // B must be the whole K-major weight, contiguous, its row blocks whole 128-row chunks
    if (!gemm_gather_supported(M, N, K, gather->world) || !pair || a_mn || b_mn || p.batch != 1 || mode != 0 ||
        p.a_parts != 1 || ldb != K || gather->world > kMaxPeers || gather->flags == nullptr || B != gather->dst)
      return -9;
    // (the rows of a chunk are wanted by all row tiles as soon as it has come in)
    p.band = (M + kPairBM - 1) / kPairBM;
    p.g_world = gather->world; p.g_rank = gather->rank; p.g_dst = gather->dst; p.g_flags = gather->flags;
    for (int i = 0; i < gather->world; ++i) p.g_src[i] = gather->src[i];
  }
  ok = ok && (b_mn ? make_tmap_4d(&tb, B, N, K, batch, nb2, ldb, b_bs, b_bs2, 64, 64, in_dtype)
                   : make_tmap_4d(&tb, B, K, N, batch, nb2, ldb, b_bs, b_bs2, BK, pair ? kPairBN / 2 : tile, in_dtype));
  if (!ok) return -4;
  const int fmt = in_dtype == kBF16 ? 1 : 0;
  if (p.g_world > 0) {
    if (out_dtype == kBF16) return launch_gemm_pair_gather<__nv_bfloat16>(ta, tb, p, fmt, num_sms, st);
    if (out_dtype == kF16) return launch_gemm_pair_gather<__half>(ta, tb, p, fmt, num_sms, st);
    return launch_gemm_pair_gather<float>(ta, tb, p, fmt, num_sms, st);
  }
  if (pair) {
#define GEMM_PAIR_CASE(AMN, BMN, SM)                                                                        \
  if (a_mn == AMN && b_mn == BMN && (p.epi != kEpiStd) == SM) {                                             \
    if (out_dtype == kBF16) return launch_gemm_pair<AMN, BMN, __nv_bfloat16, SM>(ta, tb, p, fmt, num_sms, st); \
    if (out_dtype == kF16) return launch_gemm_pair<AMN, BMN, __half, SM>(ta, tb, p, fmt, num_sms, st);      \
    return launch_gemm_pair<AMN, BMN, float, SM>(ta, tb, p, fmt, num_sms, st);                              \
  }
#define GEMM_PAIR_CASES(SM)        \
  GEMM_PAIR_CASE(false, false, SM) \
  GEMM_PAIR_CASE(false, true, SM)  \
  GEMM_PAIR_CASE(true, true, SM)   \
  GEMM_PAIR_CASE(true, false, SM)
    GEMM_PAIR_CASES(false)
    GEMM_PAIR_CASES(true)
#undef GEMM_PAIR_CASES
#undef GEMM_PAIR_CASE
    return -5;
  }
#define GEMM_CASE(BNV, AMN, BMN)                                                                         \
  if (tile == BNV && a_mn == AMN && b_mn == BMN) {                                                       \
    if (out_dtype == kBF16) return launch_gemm<BNV, AMN, BMN, __nv_bfloat16>(ta, tb, p, fmt, num_sms, st); \
    if (out_dtype == kF16) return launch_gemm<BNV, AMN, BMN, __half>(ta, tb, p, fmt, num_sms, st);       \
    return launch_gemm<BNV, AMN, BMN, float>(ta, tb, p, fmt, num_sms, st);                               \
  }
#define GEMM_CASES(BNV)         \
  GEMM_CASE(BNV, false, false)  \
  GEMM_CASE(BNV, false, true)   \
  GEMM_CASE(BNV, true, true)    \
  GEMM_CASE(BNV, true, false)
  GEMM_CASES(64)
  GEMM_CASES(128)
  GEMM_CASES(256)
#undef GEMM_CASES
#undef GEMM_CASE
  return -5;
}

void gemm_set_cta_pairs(bool on) { g_use_pair = on; }

bool gemm_gather_supported(int M, int N, int K, int world) {
  return g_use_pair && M > BM && world > 1 && world <= kMaxPeers && N % (world * 128) == 0 && K % 64 == 0;
}
int gemm_gather_flag_words(int N) { return 1 + N / 128; }

// How many CTA pairs of the pair kernel the device can hold at once (diagnostic).
int gemm_pair_max_active_clusters() {
  auto kern = gemm_tcgen05_pair_kernel<false, false, __nv_bfloat16>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairSmem::total) != cudaSuccess) return -1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(148, 1, 1);
  cfg.blockDim = dim3(kPairThreads, 1, 1);
  cfg.dynamicSmemBytes = PairSmem::total;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = -1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) return -2;
  return n;
}

}  // namespace mb
