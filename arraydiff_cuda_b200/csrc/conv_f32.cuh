// Shared by the fp32 convolution kernels: packed FMAs, asynchronous gathers, parameters, cluster launches.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "conv_f32_plan.h"

namespace cg = cooperative_groups;

namespace adk {

typedef unsigned long long u64;

__device__ __forceinline__ void ffma2(u64& d, u64 a, u64 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ u64 dup2(float v) {
  u64 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float2 unpack2(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
// 4 bytes global -> shared asynchronously where all bits of `need` are in `have`, else a zero (source size 0: not read)
__device__ __forceinline__ void gather4(uint32_t dst, const float* src, uint32_t have, uint32_t need) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"((have & need) == need ? 4u : 0u) : "memory");
}
// the same with a condition that is at hand as a predicate: one instruction
__device__ __forceinline__ void gather4_if(uint32_t dst, const float* src, bool have) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\tcp.async.ca.shared.global [%0], [%1], 4, p;\n\t}" ::"r"(dst), "l"(src), "r"((uint32_t)have)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void fadd2(u64& d, u64 a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }

// Sum of four neighbouring floats of the tiles of all CTAs of the cluster, in rank order; all loads are in flight together
template <int MOST>
__device__ __forceinline__ float4 cluster_total4(cg::cluster_group& cluster, float* sm, uint32_t cs, size_t at) {
  if (cs == 1) return *(const float4*)(sm + at);
  float4 v[MOST];
#pragma unroll
  for (uint32_t q = 0; q < MOST; ++q)
    v[q] = q < cs ? *(const float4*)((cs > 1 ? cluster.map_shared_rank(sm, q) : sm) + at) : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 t = v[0];
#pragma unroll
  for (uint32_t q = 1; q < MOST; ++q)
    if (q < cs) { t.x += v[q].x; t.y += v[q].y; t.z += v[q].z; t.w += v[q].w; }
  return t;
}

constexpr int kF32Most = 16;             // CTAs of a cluster, forward and data gradient
constexpr uint32_t kF32Never = 1u << 31; // a bit no pixel has

// Forward and data gradient: `in` is the tensor that is read (x, dy), M the output channels of the pass, CR the channels summed over
struct GemmF32 {
  const float *in, *w, *bias;
  float* out;
  uint32_t M, CR, NI;
  uint32_t IH, IW;                    // extent of `in`
  long long in_pitch, in_plane, in_img;
  uint32_t OH, OW;                    // full output extent
  long long out_pitch, out_plane, out_img;
  long long w_m, w_c;                 // filter strides of m and of the reduction channel (taps are contiguous)
  uint32_t kh, kw, sh, sw, dh, dw;
  int ph, pw;
  int relu, accumulate;
};
// Filter and bias gradient
struct WgradF32 {
  const float *x, *dy;
  float *dw, *db, *part;
  uint32_t K, C, N, P, Q, H, W, kh, kw, sh, sw, dh, dw_;
  int ph, pw;
  long long dy_pitch, dy_plane;
  int accumulate;
  uint32_t slices;
};

// What the launches of one kernel share: on which devices (a bit each) its limits are raised, and how many clusters of
// 1, 2, 4, 8, 16 CTAs the machine holds at a time, plus one (0: not asked yet).  That is less than CTAs per SM x 148 / size:
// a cluster stays within one group of SMs.
struct F32Launch { unsigned raised = 0; uint32_t held[5] = {}; };

template <typename Params>
inline cudaLaunchConfig_t f32_config(void (*)(Params), dim3 grid, int threads, int smem, uint32_t cs, cudaLaunchAttribute* at, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.numAttrs = cs > 1 ? 1 : 0;
  cfg.attrs = at;
  return cfg;
}
template <typename Params>
inline int raise_f32(void (*k)(Params), int smem, F32Launch& l) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (l.raised & (1u << (dev & 31))) return AD_OK;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return AD_ERR_CUDA;
  }
  l.raised |= 1u << (dev & 31);
  return AD_OK;
}
template <typename Params>
inline int launch_f32(void (*k)(Params), dim3 grid, int threads, int smem, uint32_t cs, const Params& p, F32Launch& l, cudaStream_t s) {
  if (int rc = raise_f32(k, smem, l)) return rc;
  cudaLaunchAttribute at[1];
  const cudaLaunchConfig_t cfg = f32_config(k, grid, threads, smem, cs, at, s);
  if (cudaLaunchKernelEx(&cfg, k, p) != cudaSuccess) { cudaGetLastError(); return AD_ERR_CUDA; }
  count_launch();
  return launch_status();
}
// 0: not one such cluster fits (part of a GPU, a size above what the device allows)
template <typename Params>
inline uint32_t f32_held(void (*k)(Params), int threads, int smem, uint32_t cs, F32Launch& l) {
  uint32_t i = 0;
  while ((1u << i) < cs) ++i;
  if (!l.held[i]) {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = f32_config(k, dim3(cs), threads, smem, cs, at, nullptr);
    cfg.numAttrs = 1;
    int n = 0;
    if (raise_f32(k, smem, l) != AD_OK || cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess || n < 0) { cudaGetLastError(); n = 0; }
    l.held[i] = (uint32_t)n + 1;
  }
  return l.held[i] - 1;
}

// 3x3 (conv_f32_k3.cu): forward of stride 1 under any dilation or of stride 2, data gradient of stride 1 under any dilation
template <bool DGRAD> int f32_k3_gemm(const GemmF32& p, cudaStream_t s);
// 1x1 without padding (conv_f32_k1.cu)
template <bool DGRAD> int f32_k1_gemm(const GemmF32& p, cudaStream_t s);
// filter and bias gradient, as the forward pass
F32Split f32_k3_wgrad_split(uint32_t K, uint32_t C, uint32_t N, uint32_t P, uint32_t Q, uint32_t stride, uint32_t dil);
int f32_k3_wgrad(const WgradF32& p, uint32_t cs, cudaStream_t s);

}  // namespace adk
