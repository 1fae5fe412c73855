// Bias gradients of the tensor-core convolutions: partial sums per block, added up by blocks of their own in the kernel that
// reduces the filter gradient's partials (a launch of their own cost 2 - 3 us behind every filter gradient with a bias).
#pragma once

#include "common.cuh"

namespace adk {
namespace tc {

struct BiasParts {
  const float* part;            // [rows][pitch]
  uint32_t rows, pitch, K;
  float* db;                    // NULL: none
  uint32_t blocks;              // of the launch, in front of its others (the rows are a longer chain of loads than theirs)
};
// In one of the first b.blocks blocks: db[32 channels] (+)= the rows' sums, in order, by up to 8 lanes of rows.  true: this was one.
__device__ __forceinline__ bool bias_finish_blocks(const BiasParts& b, int accumulate) {
  if (blockIdx.x >= b.blocks) return false;
  __shared__ float red[8][33];
  const uint32_t lanes = blockDim.x / 32 < 8 ? blockDim.x / 32 : 8, tx = threadIdx.x & 31, ty = threadIdx.x >> 5, k = blockIdx.x * 32 + tx;
  float t = 0.f;
  if (k < b.K && ty < lanes) {
    for (uint32_t r0 = ty; r0 < b.rows; r0 += 16 * lanes) {
      float v[16];                // in flight together
#pragma unroll
      for (uint32_t u = 0; u < 16; ++u) {
        const uint32_t r = r0 + u * lanes;
        v[u] = r < b.rows ? b.part[(size_t)r * b.pitch + k] : 0.f;
      }
#pragma unroll
      for (uint32_t u = 0; u < 16; ++u) t += v[u];
    }
  }
  if (ty < lanes) red[ty][tx] = t;
  __syncthreads();
  if (ty == 0 && k < b.K) {
    for (uint32_t w = 1; w < lanes; ++w) t += red[w][tx];
    b.db[k] = accumulate ? b.db[k] + t : t;
  }
  return true;
}

size_t bias_grad_bytes(size_t pixels, uint32_t K);
BiasParts bias_grad_parts(size_t pixels, uint32_t K, const void* dy, float* db, float* part, size_t part_bytes, cudaStream_t s);

}  // namespace tc
}  // namespace adk
