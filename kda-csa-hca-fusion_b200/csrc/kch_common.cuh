// Shared device/host helpers for the kch_b200 kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/kch_b200.h"

#define KCH_SMS 148            // of the chip that these kernels are for: the unit of the dispatch rules that were measured on it

// ---- error reporting -----------------------------------------------------------------
void kch_set_error(const char* fmt, ...);
void kch_note_launch(int n);   // host-side count of kernels launched by this library

#define KCH_REQUIRE(cond, ...)            \
  do {                                    \
    if (!(cond)) {                        \
      kch_set_error(__VA_ARGS__);         \
      return KCH_ERR_INVALID;             \
    }                                     \
  } while (0)

#define KCH_CUDA_OK(expr)                                                        \
  do {                                                                           \
    cudaError_t _e = (expr);                                                     \
    if (_e != cudaSuccess) {                                                     \
      kch_set_error("%s failed: %s", #expr, cudaGetErrorString(_e));             \
      return KCH_ERR_CUDA;                                                       \
    }                                                                            \
  } while (0)

#define KCH_LAUNCH_OK()                                                          \
  do {                                                                           \
    kch_note_launch(1);                                                          \
    cudaError_t _e = cudaGetLastError();                                         \
    if (_e != cudaSuccess) {                                                     \
      kch_set_error("kernel launch failed at %s:%d: %s", __FILE__, __LINE__,     \
                    cudaGetErrorString(_e));                                     \
      return KCH_ERR_CUDA;                                                       \
    }                                                                            \
  } while (0)

static inline cudaStream_t kch_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ---- typed loads / stores ---------------------------------------------------------------
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float ldf(const float* p) { return *p; }
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void stf(float* p, float v) { *p = v; }
__device__ __forceinline__ void stf(bf16* p, float v) { *p = __float2bfloat16_rn(v); }

// round a float through the storage type T (identity for float)
template <typename T>
__device__ __forceinline__ float round_to(float v);
template <>
__device__ __forceinline__ float round_to<float>(float v) { return v; }
template <>
__device__ __forceinline__ float round_to<bf16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

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

// the activations of the projections, in fp32
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// generic load by runtime dtype tag (slow path helpers)
__device__ __forceinline__ float ld_any(const void* p, int64_t i, int dtype) {
  return dtype == KCH_BF16 ? __bfloat162float(((const bf16*)p)[i]) : ((const float*)p)[i];
}

// ---- chained launches (the kernels of a decode step) ------------------------------------------------------------------
// A step is ~30 short kernels in a row, each a few microseconds long: launch latency and set-up between two of them cost
// as much as some of them.  kch_launch_chained lets a kernel start while the one before it drains.  Such a kernel calls
// chain_wait() in every thread before it touches anything an earlier launch may still write or read: the call returns
// when all earlier launches have completed and their stores are visible.  chain_trigger() (after the wait, so that a
// kernel's start implies that everything before its predecessor is complete) lets the next one start.  A kernel that takes
// tensor memory triggers after it holds it: the next kernel may take its own before its wait, and a CTA still waiting for
// columns that the next kernel holds, which in turn waits for that CTA, would wait for good.  Both are no-ops in
// a kernel launched the ordinary way.  Inputs are not `const __restrict__` there: such loads could be moved above the wait.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... K, typename... A>
static inline cudaError_t kch_launch_chained(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, unsigned cluster_x, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster_x; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cfg.attrs = attr; cfg.numAttrs = cluster_x > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}

static inline int64_t ceil_div64(int64_t a, int64_t b) { return (a + b - 1) / b; }

#define KCH_DISPATCH_FLOAT(dtype, T, ...)                       \
  do {                                                          \
    if ((dtype) == KCH_F32) {                                   \
      typedef float T;                                          \
      __VA_ARGS__;                                              \
    } else if ((dtype) == KCH_BF16) {                           \
      typedef bf16 T;                                           \
      __VA_ARGS__;                                              \
    } else {                                                    \
      kch_set_error("unsupported dtype tag %d", (int)(dtype));  \
      return KCH_ERR_INVALID;                                   \
    }                                                           \
  } while (0)
