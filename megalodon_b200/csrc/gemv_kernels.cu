// Linear layer for one row (the last position of a prefill, a single token):
//
//   y[n] = act(sum_k x[k] w[n, k] + bias[n])
//
// The work is one pass over the weight matrix, so the kernel is organised around that stream: a warp owns
// NR consecutive weight rows and walks K in chunks of 256 elements, every lane holding one 16-byte piece of
// each row (NR * KU loads in flight per lane); the matching pieces of x come from L1/L2.  Partial sums are
// reduced over the warp with shuffles.  From two rows on, and for long rows, skinny_gemm.cu takes over: here
// every further row costs as much arithmetic as the first (1 / 4 / 16 rows of a 4096 x 2048 weight: 12.3 / 24.6 /
// 69.6 us here, 13.3 / 13.3 / 15.4 us there).
#include "common.cuh"
#include "kernels.h"

namespace mb {
namespace {

constexpr int kGemvThreads = 128;   // 4 warps
constexpr int kGemvNR = 4;          // weight rows per warp
constexpr int kGemvKU = 4;          // 256-element chunks of K per loop trip

template <typename T, typename OutT>
__global__ void __launch_bounds__(kGemvThreads)
gemv_kernel(const T* __restrict__ x, const T* __restrict__ w, const void* __restrict__ bias, int bias_dtype,
            OutT* __restrict__ y, int N, int K, long long ldw, int act) {
  begin_dependent();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int n0 = (blockIdx.x * (kGemvThreads / 32) + warp) * kGemvNR;
  if (n0 >= N) return;
  float acc[kGemvNR];
#pragma unroll
  for (int r = 0; r < kGemvNR; ++r) acc[r] = 0.f;

  // kGemvKU chunks of 256 elements per trip: NR * KU 16-byte weight loads in flight per lane, kept raw
  // (4 registers each) until they are used
  for (int k0 = lane * 8; k0 < K; k0 += 256 * kGemvKU) {
    uint4 raw[kGemvKU][kGemvNR];
#pragma unroll
    for (int u = 0; u < kGemvKU; ++u) {
      const int k = k0 + u * 256;
#pragma unroll
      for (int r = 0; r < kGemvNR; ++r) {
        if (k < K && n0 + r < N) raw[u][r] = __ldg(reinterpret_cast<const uint4*>(w + (long long)(n0 + r) * ldw + k));
        else raw[u][r] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
#pragma unroll
    for (int u = 0; u < kGemvKU; ++u) {
      const int k = k0 + u * 256;
      if (k >= K) break;
      float xv[8];
      load8(x + k, xv);
#pragma unroll
      for (int r = 0; r < kGemvNR; ++r) {
        float wv[8];
        load8(reinterpret_cast<const T*>(&raw[u][r]), wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[r] = fmaf(xv[j], wv[j], acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kGemvNR; ++r) acc[r] = warp_sum(acc[r]);
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < kGemvNR; ++r) {
      const int n = n0 + r;
      if (n >= N) break;
      float b = 0.f;
      if (bias != nullptr) {
        if (bias_dtype == kF32) b = reinterpret_cast<const float*>(bias)[n];
        else if (bias_dtype == kBF16) b = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[n]);
        else b = __half2float(reinterpret_cast<const __half*>(bias)[n]);
      }
      float v = acc[r] + b;
      if (act == 1) v = silu_f(v);
      y[n] = from_f<OutT>(v);
    }
  }
}

template <typename T, typename OutT>
void launch_gemv(const void* x, const void* w, const void* bias, int bias_dtype, void* y, int N, int K, long long ldw,
                 int act, cudaStream_t st) {
  const int grid = div_up(N, (kGemvThreads / 32) * kGemvNR);
  launch_dependent(gemv_kernel<T, OutT>, grid, kGemvThreads, 0, st, (const T*)x, (const T*)w, bias, bias_dtype, (OutT*)y, N, K, ldw,
                                                      act);
}

}  // namespace

// Returns false when the shapes / alignment are outside what the kernel handles.
bool gemv(const void* x, const void* w, const void* bias, int bias_dtype, void* y, int N, int K, long long ldw, int act,
          int in_dtype, int out_dtype, cudaStream_t st) {
  if (K % 8 != 0 || ldw % 8 != 0 || in_dtype == kF32) return false;
  if (!aligned16(x) || !aligned16(w)) return false;
  if (in_dtype == kBF16) {
    if (out_dtype == kBF16) launch_gemv<__nv_bfloat16, __nv_bfloat16>(x, w, bias, bias_dtype, y, N, K, ldw, act, st);
    else if (out_dtype == kF32) launch_gemv<__nv_bfloat16, float>(x, w, bias, bias_dtype, y, N, K, ldw, act, st);
    else return false;
  } else {
    if (out_dtype == kF16) launch_gemv<__half, __half>(x, w, bias, bias_dtype, y, N, K, ldw, act, st);
    else if (out_dtype == kF32) launch_gemv<__half, float>(x, w, bias, bias_dtype, y, N, K, ldw, act, st);
    else return false;
  }
  return true;
}

}  // namespace mb
