// Shared device helpers for the sm_100a kernels: type conversion, warp/block
// reductions, vector loads.  Everything here is header-only and torch-free so
// the kernel translation units compile in seconds.
#pragma once

#include "kernels.h"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace mb {

constexpr int kWarp = 32;

// Lets a kernel use `bytes` of dynamic shared memory.  A function attribute belongs to the device that is current
// when it is set, so `done` (one per kernel) keeps a bit for each device.
template <typename Kernel>
inline bool allow_dynamic_smem(Kernel kern, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if ((done.load(std::memory_order_acquire) & bit) != 0) return true;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return false;
  done.fetch_or(bit, std::memory_order_release);
  return true;
}

enum DType : int { kF32 = 0, kBF16 = 1, kF16 = 2 };

template <typename T> struct TypeTag;
template <> struct TypeTag<float> { static constexpr int value = kF32; };
template <> struct TypeTag<__nv_bfloat16> { static constexpr int value = kBF16; };
template <> struct TypeTag<__half> { static constexpr int value = kF16; };

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float to_f(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

// 8 consecutive elements as floats.  16-bit types move as one 16-byte access, fp32 as two;
// the pointer must be aligned to 8 elements of T.
template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&v)[8]);
template <>
__device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <>
__device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
template <>
__device__ __forceinline__ void load8<__half>(const __half* p, float (&v)[8]) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&v)[8]);
template <>
__device__ __forceinline__ void store8<float>(float* p, const float (&v)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
template <>
__device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16* p, const float (&v)[8]) {
  uint4 r;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = r;
}
template <>
__device__ __forceinline__ void store8<__half>(__half* p, const float (&v)[8]) {
  uint4 r;
  __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = r;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the first `width` lanes groups (width a power of two <= 32).
template <int WIDTH>
__device__ __forceinline__ float subwarp_sum(float v) {
#pragma unroll
  for (int o = WIDTH / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum; every thread gets the result.  `scratch` holds >= 32 floats.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? scratch[lane] : 0.f;
  t = warp_sum(t);
  return t;
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarp = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? scratch[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }
__device__ __forceinline__ float silu_grad_f(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  return s * (1.f + x * (1.f - s));
}

struct cfloat {
  float re, im;
};
__device__ __forceinline__ cfloat cmul(cfloat a, cfloat b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
__device__ __forceinline__ cfloat cconj(cfloat a) { return {a.re, -a.im}; }
__device__ __forceinline__ cfloat cadd(cfloat a, cfloat b) { return {a.re + b.re, a.im + b.im}; }

#define MB_DISPATCH_DTYPE(dtype, ...)                         \
  do {                                                        \
    if ((dtype) == mb::kF32) {                                \
      using scalar_t = float;                                 \
      __VA_ARGS__;                                            \
    } else if ((dtype) == mb::kBF16) {                        \
      using scalar_t = __nv_bfloat16;                         \
      __VA_ARGS__;                                            \
    } else {                                                  \
      using scalar_t = __half;                                \
      __VA_ARGS__;                                            \
    }                                                         \
  } while (0)

#define MB_DISPATCH_16BIT(dtype, ...)                         \
  do {                                                        \
    if ((dtype) == mb::kBF16) {                               \
      using scalar_t = __nv_bfloat16;                         \
      __VA_ARGS__;                                            \
    } else {                                                  \
      using scalar_t = __half;                                \
      __VA_ARGS__;                                            \
    }                                                         \
  } while (0)

// element i of a vector whose type is known at run time
__device__ __forceinline__ float load_any(const void* p, int dtype, int i) {
  return dtype == kF32 ? static_cast<const float*>(p)[i]
                       : dtype == kBF16 ? to_f(static_cast<const __nv_bfloat16*>(p)[i]) : to_f(static_cast<const __half*>(p)[i]);
}

// An ordinary launch: for kernels whose grid fills the chip about once, or not at all, with CTAs that take long (scans,
// column sums).  Placed while the kernel before them drains, their CTAs crowd on the SMs that came free first.  us, ordinary
// / dependent: TimestepNorm backward 1 x 12000 x 1024 138 / 329, 1 x 16384 x 4096 310 / 446, 2 x 2048 x 2048 37.3 / 41.4, its
// forward 64 x 16 x 512 5.9 / 7.9; column sums of 8192 x 4096 18.2 / 21.4; RMSNorm backward 2 x 2048 x 2048 16.8 / 18.3.
template <typename... KArgs, typename... Args>
inline void launch_plain(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  ++thread_launches();
  kern<<<grid, block, smem, st>>>(KArgs(args)...);
}

// ---- launches that begin under the end of the kernel before them
// A kernel launched with `launch_dependent` calls `begin_dependent` before anything else: it returns when every kernel
// ahead of it in the stream is complete and its writes are visible (at once for an ordinary launch), and lets the next
// such kernel be placed on the SMs as they come free.  What the pair saves is the time from the last CTA of one kernel to
// the first of the next, some 1.5 us of it a launch: graph-replayed products of 512 features 8.6 -> 6.9 us.
__device__ __forceinline__ void begin_dependent() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                    Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ++thread_launches();
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace mb
