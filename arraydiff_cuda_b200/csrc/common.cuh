// Shared helpers for the sm_100a kernels: status codes, launch accounting, dtype access.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "arraydiff_b200.h"

namespace adk {

// Every kernel launch of the library goes through this counter so that callers can
// report how many of OUR kernels ran inside a timed region.
extern unsigned long long g_launch_count;
inline void count_launch(unsigned long long n = 1) { __atomic_fetch_add(&g_launch_count, n, __ATOMIC_RELAXED); }

// Which kernel family the calling thread's most recent ad_conv2d_* call launched (ad_conv2d_last_kernel).
enum { kConvNone = 0, kConvDirectF32 = 1, kConvTcGeneral = 2, kConvTcRow = 3 };
extern thread_local int g_last_conv_kernel;

inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? AD_OK : AD_ERR_CUDA;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int elem_size(int dtype) { return dtype == AD_F32 ? 4 : (dtype == AD_BF16 ? 2 : 0); }

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs

inline unsigned grid_for(size_t work_items, unsigned per_block, unsigned max_blocks_per_sm = 8) {
  size_t b = (work_items + per_block - 1) / per_block;
  size_t cap = (size_t)kNumSMs * max_blocks_per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// ---- typed element access (device) ----
template <typename T> __device__ __forceinline__ float ld_f(const T* p);
template <> __device__ __forceinline__ float ld_f<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ld_f<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void st_f(T* p, float v);
template <> __device__ __forceinline__ void st_f<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void st_f<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

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

// Launches that overlap their set-up with the end of the kernel in front of them in the stream (programmatic dependent
// launch): blocks may become resident once every block of that kernel has passed its own grid_dependency(), and stop in
// theirs until it has completed and its stores are visible.  So every kernel that is launched this way calls
// grid_dependency() in all threads, before its first access to global memory (set-up of shared and tensor memory may
// come first), and results are those of plain launches.  Measured: batch norm (5 kernels) 202 -> 191 us, the three passes
// of a small strided convolution 103 -> 88, a training step of 118 launches 1.29 -> 1.21 ms.  A kernel whose blocks share the
// machine evenly must not let them pile up on the SMs that are free first: see LoadRing::kSmem, and conv_f32.cu, which
// launches plainly (early, its large blocks made an 18-layer step 10 % slower).
// Off (LateLaunch) for work on a stream beside the critical one: blocks that only wait would take the room of the kernels
// of the other stream.
__device__ __forceinline__ void grid_dependency() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}
extern thread_local bool g_early_launch;
struct LateLaunch {
  bool old = g_early_launch;
  LateLaunch() { g_early_launch = false; }
  ~LateLaunch() { g_early_launch = old; }
};
inline void launch_attr(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at) {   // appends the attribute
  cfg.attrs = at;
  if (!g_early_launch) return;
  at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
  ++cfg.numAttrs;
}
template <typename... K, typename... A>
void launch(void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  launch_attr(cfg, at);
  cudaLaunchKernelEx(&cfg, kernel, K(args)...);   // an error is what launch_status() returns
}

// A ring of 16-byte loads in flight, D per thread and stream, in shared memory: each thread copies its own next elements
// (cp.async) and reads only what it copied, so no barrier is needed and the loads in flight cost no registers.  For
// streaming kernels of 256 threads, two blocks per SM: with 8 x 4 KB per stream the batch normalisation passes measured
// 5.0-6.5 TB/s where batches of 4 loads in registers reached 4.1-5.4.
constexpr int kRingThreads = 256;
template <int S, int D>
struct LoadRing {
  static constexpr int kBytes = S * D * kRingThreads * 16;
  // What a launch asks for: no third block fits on an SM.  Blocks that become resident early (launch) would pile up on the
  // SMs that are free first, and the rest of the machine would have one or none.
  static constexpr int kSmem = kBytes > 77 * 1024 ? kBytes : 77 * 1024;
  uint4* base;   // this thread's slots
  int put_at, get_at;
  __device__ __forceinline__ explicit LoadRing(void* smem) : base((uint4*)smem + threadIdx.x), put_at(0), get_at(0) {}
  __device__ __forceinline__ void copy(int stream, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(base + (put_at * S + stream) * kRingThreads)),
                 "l"(src) : "memory");
  }
  // after the copies of one element of every stream (or none, past the end)
  __device__ __forceinline__ void commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++put_at == D) put_at = 0;
  }
  // D - 1 elements are committed ahead of the one that is waited for
  __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory"); }
  __device__ __forceinline__ uint4 get(int stream) const { return base[(get_at * S + stream) * kRingThreads]; }
  __device__ __forceinline__ void next() { if (++get_at == D) get_at = 0; }
};

// Dispatch a callable templated on the element type.
#define AD_DISPATCH_DTYPE(dtype, ...)                                   \
  do {                                                                  \
    if ((dtype) == AD_F32) { using T = float; __VA_ARGS__; }            \
    else if ((dtype) == AD_BF16) { using T = __nv_bfloat16; __VA_ARGS__; } \
    else return AD_ERR_UNSUPPORTED;                                     \
  } while (0)

}  // namespace adk
