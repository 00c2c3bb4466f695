// Shared helpers for the sm_100a kernels of libmoe_b200.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <stdio.h>
#include <utility>
#include "../../include/moe_b200.h"

// per-thread error message, set by every failing entry point
void moe_set_error(const char* fmt, ...);

#define MOE_CHECK_ARG(cond, ...)                 \
  do {                                           \
    if (!(cond)) {                               \
      moe_set_error(__VA_ARGS__);                \
      return MOE_ERR_ARG;                        \
    }                                            \
  } while (0)

#define MOE_CHECK_CUDA(expr)                                                              \
  do {                                                                                    \
    cudaError_t _e = (expr);                                                              \
    if (_e != cudaSuccess) {                                                              \
      moe_set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
      return MOE_ERR_CUDA;                                                                \
    }                                                                                     \
  } while (0)

void moe_count_launch();   // one kernel launch (api.cu keeps the process-wide counter)
#define MOE_CHECK_LAUNCH()              \
  do {                                  \
    moe_count_launch();                 \
    MOE_CHECK_CUDA(cudaGetLastError()); \
  } while (0)

// ---- programmatic dependent launch ---------------------------------------------------------------------------
// Kernels of the short chains (routing, layer step) are launched with the programmatic-stream-serialization attribute: the
// next kernel of the stream may start once every block of this one has passed pdl_launch_dependents() or left, and whatever it
// reads or writes comes after its own pdl_wait(), which returns when its predecessors have completed and their writes are
// visible (so those kernels take their pointers without __restrict__: a load through such a pointer may move ahead of the
// wait).  Launch and prologue of a kernel then overlap the tail of the one before.  A kernel waits, with all its threads, before
// it lets its dependents go, so at most one kernel is ahead of a running one.  It reads nothing of device memory ahead of the wait,
// not even what kernels further back wrote: that they have completed orders nothing for a kernel that has not waited.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() { pdl_wait(); pdl_launch_dependents(); }

// What a kernel may do ahead of its wait is to ask L2 for memory it expects to need: a hint that is wrong, or older than the memory, is
// without effect on what is loaded later.  Words that steer it are read past L1, where an early copy would stay, and are read again
// behind the wait for all else.
__device__ __forceinline__ int ld_hint(const int32_t* a) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ void l2_hint(const void* a, uint32_t bytes) {       // 16-byte aligned, a multiple of 16
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(bytes) : "memory");
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
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
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

static inline int64_t cdiv64(int64_t a, int64_t b) { return (a + b - 1) / b; }

int moe_sm_count();  // SMs of the current device (cached per device)

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Dispatch a generic lambda on one of the three float element types.
#define MOE_DISPATCH_FLOAT(dtype, T, ...)                                   \
  switch (dtype) {                                                          \
    case MOE_F32: { using T = float; __VA_ARGS__; break; }                  \
    case MOE_F16: { using T = __half; __VA_ARGS__; break; }                 \
    case MOE_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }         \
    default: moe_set_error("unsupported dtype %d", (int)(dtype)); return MOE_ERR_ARG; \
  }

// 32 contiguous bytes (aligned to 32), a whole sector, in one store
__device__ __forceinline__ void st_v8(void* p, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x),
               "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}
