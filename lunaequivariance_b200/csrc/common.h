// Shared host-side helpers: thread-local error text, CUDA call checking, dtype dispatch.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/luna_b200.h"

namespace luna {

// Stores a printf-formatted message for luna_last_error() and returns `code`.
int fail(int code, const char* format, ...);
void clear_error();

#define LUNA_CUDA_CHECK(expr)                                                                          \
  do {                                                                                                 \
    cudaError_t luna_err_ = (expr);                                                                    \
    if (luna_err_ != cudaSuccess) {                                                                    \
      return ::luna::fail(LUNA_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(luna_err_), \
                          __FILE__, __LINE__);                                                         \
    }                                                                                                  \
  } while (0)

#define LUNA_LAUNCH_CHECK(name)                                                                          \
  do {                                                                                                   \
    cudaError_t luna_err_ = cudaGetLastError();                                                          \
    if (luna_err_ != cudaSuccess) {                                                                      \
      return ::luna::fail(LUNA_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(luna_err_)); \
    }                                                                                                    \
  } while (0)

inline bool aligned_to(const void* p, size_t bytes) { return (reinterpret_cast<uintptr_t>(p) % bytes) == 0; }

template <typename T>
struct dtype_of;
template <>
struct dtype_of<float> {
  static constexpr int value = LUNA_F32;
};
template <>
struct dtype_of<double> {
  static constexpr int value = LUNA_F64;
};

#ifdef __CUDACC__
// Launches that overlap the end of the one before them (programmatic dependent launch).  A kernel calls let_next_start at once
// and wait_for_previous before it touches anything that an earlier kernel has written or reads: by then that kernel, and so
// everything before it, is complete and visible.  What is hidden is the launch itself and the kernel's start, some two us each
// time: the five launches of a new neighbour list 105 -> 93 us (20,000 nodes), a force step of 2,083 nodes 2 % of 184.  Only for kernels
// that fill an SM with one CTA or have far more CTAs than fit: the CTAs of the harmonics, exactly as many as fit, came to lie unevenly
// where SMs were free first (4 M vectors, forward and backward 296 -> 358 us), so they let others start early and start late.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
inline void launch_early(void (*kernel)(P...), dim3 grid, unsigned threads, size_t shared, cudaStream_t stream, A... arguments) {
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = shared;
  config.stream = stream;
  config.attrs = &early;
  config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, static_cast<P>(arguments)...);  // LUNA_LAUNCH_CHECK reports
}
#endif

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace luna
