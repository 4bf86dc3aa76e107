// Shared helpers for the libb200lmk kernels: error reporting, dtype conversion, small device utilities.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>
#include <math.h>
#include "../../include/b200lmk.h"

namespace lmk {

// Per-thread error text returned by lmk_last_error().
char* error_buffer();
int fail(int code, const char* fmt, ...);

// Multiprocessors of the current device (asked for once per device); a status code.
int sm_count(int* n);

#define LMK_CHECK_ARG(cond, ...)                                   \
  do {                                                             \
    if (!(cond)) return lmk::fail(LMK_ERR_INVALID, __VA_ARGS__);   \
  } while (0)

#define LMK_CUDA(call)                                                                        \
  do {                                                                                        \
    cudaError_t e__ = (call);                                                                 \
    if (e__ != cudaSuccess)                                                                   \
      return lmk::fail(LMK_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e__));       \
  } while (0)

template <typename T> __device__ __forceinline__ float to_f32(T x);
template <> __device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

static inline int dtype_size(int dtype) { return dtype == LMK_F32 ? 4 : 2; }

// Launch with the programmatic-stream-serialization attribute: the kernel's CTAs may start, and its launch be processed, while the
// kernel in front of it in the stream drains.  Such a kernel executes griddepcontrol.wait (ptx::grid_dep_wait) before it
// touches global memory, has no __restrict__ pointer among its parameters and uses no __ldg: both promise memory that no other
// kernel writes meanwhile, and allow the compiler to read it in front of the wait.
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace lmk
