// NLL loss on probabilities (the reference's two small kernels) and the fused per-pixel
// softmax cross-entropy.  HBM-bound: logits are read once per pass and kept in registers or shared memory.
//   NCHW: one thread per pixel, the C strided reads of neighbouring threads coalesce; up to 32 classes stay in registers.
//   NHWC: up to 32 classes a block stages 256 pixels in shared memory by 16-byte vectors, a thread per pixel; up to 256
//   classes a warp holds several pixels in registers; more: a warp per pixel.
// A map of one position is the same memory in both layouts (a classifier's [batch][classes]) and takes the NHWC kernels.
// A label that is no class (255 for "void", -1) is compared, never used as an index: its pixel's loss is logsumexp(logits), whose
// gradient is dloss * softmax, zero under a weight of zero.
#include "common.cuh"

namespace adk {

__global__ void nll_fwd_kernel(uint32_t C, uint32_t B, const float* __restrict__ y, const uint32_t* __restrict__ label,
                               float* loss) {
  grid_dependency();
  uint32_t b = threadIdx.x + blockDim.x * blockIdx.x;
  if (b < B) loss[b] = -logf(y[label[b] + (size_t)C * b]);
}

__global__ void nll_bwd_kernel(uint32_t C, uint32_t B, const float* __restrict__ y, const uint32_t* __restrict__ label,
                               const float* __restrict__ dloss, float* dx) {
  grid_dependency();
  size_t idx = threadIdx.x + (size_t)blockDim.x * blockIdx.x;
  if (idx >= (size_t)C * B) return;
  uint32_t c = (uint32_t)(idx % C), b = (uint32_t)(idx / C);
  // Integer label compare (the reference converts the label to float first, which is the
  // same for labels below 2^24: src/kernels/softmax.cu:70-72).
  float yi = y[idx], d = dloss[b];
  float t = label[b] == c ? __fsub_rn(yi, 1.0f) : yi;
  dx[idx] = fmaf(d, t, dx[idx]);
}

// NCHW, C <= CM classes held in registers (more than 32 classes: ce_fwd_nchw / ce_bwd_nchw below read them again)
template <typename T, int CM, bool BWD>
__global__ void __launch_bounds__(256) ce_nchw_reg(uint32_t N, uint32_t C, uint32_t HW, const T* __restrict__ x, const uint32_t* __restrict__ label,
                                                   float* loss, unsigned long long* picked, const float* __restrict__ dloss, T* dx, int accumulate) {
  grid_dependency();
  const size_t total = (size_t)N * HW;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t n = i / HW, t = i - n * HW;
    const T* px = x + n * C * HW + t;
    float v[CM];
#pragma unroll
    for (int c = 0; c < CM; ++c) v[c] = c < (int)C ? ld_f(px + (size_t)c * HW) : -INFINITY;
    const uint32_t l = label[i];
    float m = -INFINITY;
#pragma unroll
    for (int c = 0; c < CM; ++c) m = fmaxf(m, v[c]);
    float z = 0.f;
    if (!BWD) {
      float vl = 0.f;
#pragma unroll
      for (int c = 0; c < CM; ++c)
        if (c < (int)C) { z += expf(v[c] - m); if ((uint32_t)c == l) vl = v[c]; }
      loss[i] = (logf(z) + m) - vl;
      if (picked) picked[i] = (n * C + l) * HW + t;
    } else {
#pragma unroll
      for (int c = 0; c < CM; ++c)
        if (c < (int)C) { v[c] = expf(v[c] - m); z += v[c]; }
      const float rz = 1.f / z, d = dloss[i];
      T* pdx = dx + n * C * HW + t;
#pragma unroll
      for (int c = 0; c < CM; ++c)
        if (c < (int)C) {
          float g = d * (v[c] * rz - ((uint32_t)c == l ? 1.f : 0.f));
          if (accumulate) g += ld_f(pdx + (size_t)c * HW);
          st_f(pdx + (size_t)c * HW, g);
        }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) ce_fwd_nchw(uint32_t N, uint32_t C, uint32_t HW, const T* __restrict__ x,
                                                    const uint32_t* __restrict__ label, float* loss,
                                                    unsigned long long* picked) {
  grid_dependency();
  const size_t total = (size_t)N * HW;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t n = i / HW, t = i % HW;
    const T* px = x + n * C * HW + t;
    float m = -INFINITY;
    for (uint32_t c = 0; c < C; ++c) m = fmaxf(m, ld_f(px + (size_t)c * HW));
    float z = 0.f;
    for (uint32_t c = 0; c < C; ++c) z += expf(ld_f(px + (size_t)c * HW) - m);
    const uint32_t l = label[i];
    const size_t li = (n * C + l) * HW + t;
    loss[i] = (logf(z) + m) - (l < C ? ld_f(x + li) : 0.f);
    if (picked) picked[i] = li;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) ce_bwd_nchw(uint32_t N, uint32_t C, uint32_t HW, const T* __restrict__ x,
                                                    const uint32_t* __restrict__ label,
                                                    const float* __restrict__ dloss, T* dx, int accumulate) {
  grid_dependency();
  const size_t total = (size_t)N * HW;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t n = i / HW, t = i % HW;
    const T* px = x + n * C * HW + t;
    T* pdx = dx + n * C * HW + t;
    float m = -INFINITY;
    for (uint32_t c = 0; c < C; ++c) m = fmaxf(m, ld_f(px + (size_t)c * HW));
    float z = 0.f;
    for (uint32_t c = 0; c < C; ++c) z += expf(ld_f(px + (size_t)c * HW) - m);
    const float rz = 1.f / z, d = dloss[i];
    const uint32_t l = label[i];
    for (uint32_t c = 0; c < C; ++c) {
      float pr = expf(ld_f(px + (size_t)c * HW) - m) * rz;
      float g = d * (pr - (c == l ? 1.f : 0.f));
      if (accumulate) g += ld_f(pdx + (size_t)c * HW);
      st_f(pdx + (size_t)c * HW, g);
    }
  }
}

template <typename T, bool BWD>
__global__ void __launch_bounds__(256) ce_nhwc(uint32_t C, size_t pixels, const T* __restrict__ x,
                                                const uint32_t* __restrict__ label, float* loss,
                                                unsigned long long* picked, const float* __restrict__ dloss, T* dx,
                                                int accumulate) {
  grid_dependency();
  const int lane = threadIdx.x & 31;
  const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t i = warp; i < pixels; i += nw) {
    const T* px = x + i * C;
    float m = -INFINITY;
    for (uint32_t c = lane; c < C; c += 32) m = fmaxf(m, ld_f(px + c));
    m = warp_max(m);
    float z = 0.f;
    for (uint32_t c = lane; c < C; c += 32) z += expf(ld_f(px + c) - m);
    z = warp_sum(z);
    const uint32_t l = label[i];
    if (!BWD) {
      if (lane == 0) {
        loss[i] = (logf(z) + m) - (l < C ? ld_f(px + l) : 0.f);
        if (picked) picked[i] = i * C + l;
      }
    } else {
      const float rz = 1.f / z, d = dloss[i];
      for (uint32_t c = lane; c < C; c += 32) {
        float g = d * (expf(ld_f(px + c) - m) * rz - (c == l ? 1.f : 0.f));
        if (accumulate) g += ld_f(dx + i * C + c);
        st_f(dx + i * C + c, g);
      }
    }
  }
}

// 33 to 256 classes, NHWC: a warp holds PX pixels, K = ceil(C / 32) classes of each per lane, read once
template <typename T, int K, bool BWD>
__global__ void __launch_bounds__(256) ce_nhwc_reg(uint32_t C, size_t pixels, const T* __restrict__ x, const uint32_t* __restrict__ label,
                                                   float* loss, unsigned long long* picked, const float* __restrict__ dloss, T* dx, int accumulate) {
  grid_dependency();
  constexpr int PX = K <= 2 ? 4 : 2;
  const int lane = threadIdx.x & 31;
  const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t i0 = warp * PX; i0 < pixels; i0 += nw * PX) {
    float v[PX][K], m[PX], z[PX];
#pragma unroll
    for (int q = 0; q < PX; ++q)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t c = lane + k * 32;
        v[q][k] = c < C && i0 + q < pixels ? ld_f(x + (i0 + q) * C + c) : -INFINITY;
      }
#pragma unroll
    for (int q = 0; q < PX; ++q) {
      m[q] = v[q][0];
#pragma unroll
      for (int k = 1; k < K; ++k) m[q] = fmaxf(m[q], v[q][k]);
      m[q] = warp_max(m[q]);
    }
#pragma unroll
    for (int q = 0; q < PX; ++q) {
      if (i0 + q >= pixels) break;
      const size_t i = i0 + q;
      const uint32_t l = label[i], lc = l < C ? l : 0xffffffffu;   // no class's number: a test of c < C per class took 72 us for 63 (150 classes)
      float vl = 0.f;
      z[q] = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t c = lane + k * 32;
        if (c == lc) vl = v[q][k];
        v[q][k] = c < C ? expf(v[q][k] - m[q]) : 0.f;
        z[q] += v[q][k];
      }
      z[q] = warp_sum(z[q]);
      if (!BWD) {
        vl = __shfl_sync(0xffffffffu, vl, l & 31u);
        if (lane == 0) {
          loss[i] = (logf(z[q]) + m[q]) - vl;
          if (picked) picked[i] = i * C + l;
        }
      } else {
        const float rz = 1.f / z[q], d = dloss[i];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t c = lane + k * 32;
          if (c < C) {
            float g = d * (v[q][k] * rz - (c == l ? 1.f : 0.f));
            if (accumulate) g += ld_f(dx + i * C + c);
            st_f(dx + i * C + c, g);
          }
        }
      }
    }
  }
}

// Few classes, bf16: a thread takes two neighbouring pixels, whose 2 C values are C aligned words of shared memory -- a stride
// that is free of bank conflicts for odd C -- and keeps them in registers.  Tiles of 512 pixels in two buffers: the next
// tile's copy is in flight while this one is worked on.  Bound by its instructions (an exponential per class).
// 4,194,304 pixels of 19 classes: 45 us forward, 68 backward; one pixel per thread by 2-byte accesses took 63 and 104 with
// two buffers, 87 and 117 with one.  The label's class is taken out of the loops over the classes (a comparison, a selection
// and a subtraction for each, and the addend's test: 46 and 87 us): its value is worked out by itself and replaces the one
// that the loop wrote.  Its bounds cost 0.3 and 2 us of 1,766,016 pixels' 21 and 32 (as selections instead of branches 0.8 and 4).
template <int C, bool BWD>
__global__ void __launch_bounds__(256) ce_nhwc_pair(size_t pixels, int vec, const __nv_bfloat16* __restrict__ x,
                                                    const uint32_t* __restrict__ label, float* loss, unsigned long long* picked,
                                                    const float* __restrict__ dloss, __nv_bfloat16* dx, int accumulate) {
  grid_dependency();
  extern __shared__ __align__(16) uint32_t ce_words[];   // [2][256 pairs][C]
  const size_t tiles = (pixels + 511) / 512;
  auto fetch = [&](size_t tile, uint32_t buf) {
    if (tile < tiles) {
      const size_t p0 = tile * 512;
      const uint32_t np = pixels - p0 < 512 ? (uint32_t)(pixels - p0) : 512u, ne = np * C, nv = vec ? ne / 8 : 0;
      const __nv_bfloat16* xb = x + p0 * C;
      uint32_t* sm = ce_words + buf * 256 * C;
      for (uint32_t q = threadIdx.x; q < nv; q += 256)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared((uint4*)sm + q)), "l"((const uint4*)xb + q) : "memory");
      for (uint32_t q = nv * 8 + threadIdx.x; q < ne; q += 256) ((__nv_bfloat16*)sm)[q] = xb[q];
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(blockIdx.x, 0);
  uint32_t buf = 0;
  for (size_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1u) {
    const size_t p0 = tile * 512, i = p0 + 2 * threadIdx.x;
    const uint32_t np = pixels - p0 < 512 ? (uint32_t)(pixels - p0) : 512u, ne = np * C, nv = vec ? ne / 8 : 0;
    uint32_t l[2];
    float d[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool mine = 2 * threadIdx.x + h < np;
      l[h] = mine ? label[i + h] : 0;
      d[h] = BWD && mine ? dloss[i + h] : 0.f;
    }
    fetch(tile + gridDim.x, buf ^ 1u);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    uint32_t *sm = ce_words + buf * 256 * C, *px = sm + threadIdx.x * C;
    if (2 * threadIdx.x < np) {
      float v[2 * C], m[2], xl[2];
      uint32_t top[2] = {0xff80ff80u, 0xff80ff80u};   // packed maxima of the words that lie in one pixel (from -infinity)
      __nv_bfloat16* pe = (__nv_bfloat16*)px;
#pragma unroll
      for (int h = 0; h < 2; ++h) xl[h] = l[h] < C ? ld_f(pe + h * C + l[h]) : 0.f;
#pragma unroll
      for (int k = 0; k < C; ++k) {   // an odd last pixel leaves half of its pair's words undefined: computed, not written
        const uint32_t w = px[k];
        v[2 * k] = __uint_as_float(w << 16);
        v[2 * k + 1] = __uint_as_float(w & 0xffff0000u);
        if (2 * k + 1 < C || 2 * k >= C) {
          uint32_t& t = top[2 * k >= C];
          const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&t), *reinterpret_cast<const __nv_bfloat162*>(&w));
          t = *reinterpret_cast<const uint32_t*>(&r);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        m[h] = fmaxf(__uint_as_float(top[h] << 16), __uint_as_float(top[h] & 0xffff0000u));
        if (C & 1) m[h] = fmaxf(m[h], v[C - 1 + h]);   // the word that both pixels share
        float z = 0.f;
        if (!BWD) {
#pragma unroll
          for (int c = 0; c < C; ++c) z += expf(v[h * C + c] - m[h]);
          if (2 * threadIdx.x + h < np) {
            loss[i + h] = (logf(z) + m[h]) - xl[h];
            if (picked) picked[i + h] = (i + h) * C + l[h];
          }
        } else {
#pragma unroll
          for (int c = 0; c < C; ++c) { v[h * C + c] = expf(v[h * C + c] - m[h]); z += v[h * C + c]; }
          const float rz = 1.f / z;
#pragma unroll
          for (int c = 0; c < C; ++c) v[h * C + c] = d[h] * (v[h * C + c] * rz);
          xl[h] = d[h] * (expf(xl[h] - m[h]) * rz - 1.f);   // the label's class, whose value replaces the one above
        }
      }
      if (BWD && accumulate) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (2 * threadIdx.x + h < np) {
            const __nv_bfloat16* old = dx + (i + h) * C;
#pragma unroll
            for (int c = 0; c < C; ++c) v[h * C + c] += ld_f(old + c);
            if (l[h] < C) xl[h] += ld_f(old + l[h]);
          }
      }
      if (BWD) {
#pragma unroll
        for (int k = 0; k < C; ++k) {
          const __nv_bfloat162 g = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
          px[k] = *reinterpret_cast<const uint32_t*>(&g);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (l[h] < C) st_f(pe + h * C + l[h], xl[h]);
      }
    }
    if (BWD) {
      __syncthreads();
      __nv_bfloat16* db = dx + p0 * C;
      for (uint32_t q = threadIdx.x; q < nv; q += 256) ((uint4*)db)[q] = ((const uint4*)sm)[q];
      for (uint32_t q = nv * 8 + threadIdx.x; q < ne; q += 256) db[q] = ((const __nv_bfloat16*)sm)[q];
    }
    __syncthreads();   // the buffer is free for the tile after the next
  }
}
template <bool BWD, int C = 1, typename... A>
static int launch_ce_pair(uint32_t classes, size_t pixels, cudaStream_t s, A... args) {
  if constexpr (C <= 32) {
    if (classes != (uint32_t)C) return launch_ce_pair<BWD, C + 1>(classes, pixels, s, args...);
    constexpr int smem = 2 * 256 * C * 4;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(ce_nhwc_pair<C, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    launch(ce_nhwc_pair<C, BWD>, grid_for((pixels + 511) / 512, 1, 5), 256, smem, s, pixels, args...);
    return AD_OK;
  } else return AD_ERR_UNSUPPORTED;
}

// Few classes (C <= 32), fp32: a thread owns one pixel of a tile in shared memory, results leave by vectors again.
// CM: C rounded up to a multiple of 4 (the class loops are unrolled; a class past C is -inf and adds nothing).
template <typename T, int CM, bool BWD>
__global__ void __launch_bounds__(256) ce_nhwc_small(uint32_t C, size_t pixels, int vec, const T* __restrict__ x,
                                                      const uint32_t* __restrict__ label, float* loss,
                                                      unsigned long long* picked, const float* __restrict__ dloss, T* dx,
                                                      int accumulate) {
  grid_dependency();
  // Tiles of 256 pixels, two buffers: the next tile's copy is in flight while this one is worked on (one tile per block
  // waited for memory most of the time)
  extern __shared__ __align__(16) uint8_t ce_raw[];   // [2][256][C]
  constexpr uint32_t V = 16 / sizeof(T);
  const size_t tiles = (pixels + 255) / 256;
  uint32_t l = 0, ln = 0;
  float d = 0.f, dn = 0.f;
  auto fetch = [&](size_t tile, uint32_t buf) {
    if (tile < tiles) {
      const size_t p0 = tile * 256;
      const uint32_t np = pixels - p0 < 256 ? (uint32_t)(pixels - p0) : 256u, ne = np * C, nv = vec ? ne / V : 0;
      const T* xb = x + p0 * C;
      T* sm = (T*)ce_raw + buf * 256 * C;
      for (uint32_t q = threadIdx.x; q < nv; q += 256)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared((uint4*)sm + q)), "l"((const uint4*)xb + q) : "memory");
      for (uint32_t q = nv * V + threadIdx.x; q < ne; q += 256) sm[q] = xb[q];
      ln = threadIdx.x < np ? label[p0 + threadIdx.x] : 0;
      dn = BWD && threadIdx.x < np ? dloss[p0 + threadIdx.x] : 0.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(blockIdx.x, 0);
  uint32_t buf = 0;
  for (size_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, buf ^= 1u) {
    l = ln; d = dn;
    fetch(tile + gridDim.x, buf ^ 1u);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    T* sm = (T*)ce_raw + buf * 256 * C;
    const size_t p0 = tile * 256, i = p0 + threadIdx.x;
    const uint32_t np = pixels - p0 < 256 ? (uint32_t)(pixels - p0) : 256u, ne = np * C, nv = vec ? ne / V : 0;
    const bool mine = threadIdx.x < np;
    if (mine) {
      T* px = sm + threadIdx.x * C;
      float m = -INFINITY, v[CM];
  #pragma unroll
      for (uint32_t c = 0; c < CM; ++c) {
        v[c] = c + 4 < CM || c < C ? ld_f(px + c) : -INFINITY;
        m = fmaxf(m, v[c]);
      }
      float z = 0.f;
      if (!BWD) {
        const float vl = l < C ? ld_f(px + l) : 0.f;
  #pragma unroll
        for (uint32_t c = 0; c < CM; ++c) z += expf(v[c] - m);
        loss[i] = (logf(z) + m) - vl;
        if (picked) picked[i] = i * C + l;
      } else {
  #pragma unroll
        for (uint32_t c = 0; c < CM; ++c) { v[c] = expf(v[c] - m); z += v[c]; }
        const float rz = 1.f / z;
        const T* old = dx + i * C;
  #pragma unroll
        for (uint32_t c = 0; c < CM; ++c)
          if (c + 4 < CM || c < C) {
            float g = d * (v[c] * rz - (c == l ? 1.f : 0.f));
            if (accumulate) g += ld_f(old + c);
            st_f(px + c, g);
          }
      }
    }
    if (BWD) {
      __syncthreads();
      T* db = dx + p0 * C;
      for (uint32_t q = threadIdx.x; q < nv; q += 256) ((uint4*)db)[q] = ((const uint4*)sm)[q];
      for (uint32_t q = nv * V + threadIdx.x; q < ne; q += 256) db[q] = sm[q];
    }
    __syncthreads();   // the buffer is free for the tile after the next
  }
}

// Picks the kernel for a layout, class count and direction
template <typename T, bool BWD>
static int launch_ce(int32_t layout, uint32_t N, uint32_t C, uint32_t HW, const T* x, const uint32_t* label, float* loss, unsigned long long* picked,
                     const float* dloss, T* dx, int accumulate, cudaStream_t s) {
  const size_t pixels = (size_t)N * HW;
  if (layout != AD_NCHW && layout != AD_NHWC) return AD_ERR_UNSUPPORTED;
  if (layout == AD_NCHW && HW > 1) {
    if (C <= 8) launch(ce_nchw_reg<T, 8, BWD>, grid_for(pixels, 256), 256, 0, s, N, C, HW, x, label, loss, picked, dloss, dx, accumulate);
    else if (C <= 32) launch(ce_nchw_reg<T, 32, BWD>, grid_for(pixels, 256), 256, 0, s, N, C, HW, x, label, loss, picked, dloss, dx, accumulate);
    else if (BWD) launch(ce_bwd_nchw<T>, grid_for(pixels, 256), 256, 0, s, N, C, HW, x, label, dloss, dx, accumulate);
    else launch(ce_fwd_nchw<T>, grid_for(pixels, 256), 256, 0, s, N, C, HW, x, label, loss, picked);
  } else if (C <= 32 && pixels <= (1ull << 31) * 256 - 256) {
    const int vec = ((uintptr_t)x & 15u) == 0 && (!BWD || ((uintptr_t)dx & 15u) == 0);
    if constexpr (sizeof(T) == 2) {
      const int rc = launch_ce_pair<BWD>(C, pixels, s, vec, x, label, loss, picked, dloss, dx, accumulate);
      if (rc != AD_OK) return rc;
    } else {
      const int smem = (int)(2 * 256 * C * sizeof(T)), most = (int)(2 * 256 * ((C + 3) / 4 * 4) * sizeof(T));
      bool ok = true;
      auto go = [&](auto kernel) {
        // the limit belongs to the function: the most that it takes, whatever other threads' class counts
        if (smem > 48 * 1024) ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
        if (ok) launch(kernel, grid_for((pixels + 255) / 256, 1, 6), 256, smem, s, C, pixels, vec, x, label, loss, picked, dloss, dx, accumulate);
      };
      switch ((C + 3) / 4) {
        case 1: go(ce_nhwc_small<T, 4, BWD>); break;
        case 2: go(ce_nhwc_small<T, 8, BWD>); break;
        case 3: go(ce_nhwc_small<T, 12, BWD>); break;
        case 4: go(ce_nhwc_small<T, 16, BWD>); break;
        case 5: go(ce_nhwc_small<T, 20, BWD>); break;
        case 6: go(ce_nhwc_small<T, 24, BWD>); break;
        case 7: go(ce_nhwc_small<T, 28, BWD>); break;
        default: go(ce_nhwc_small<T, 32, BWD>); break;
      }
      if (!ok) { cudaGetLastError(); return AD_ERR_CUDA; }
    }
  } else if (C <= 64) {
    launch(ce_nhwc_reg<T, 2, BWD>, grid_for(pixels, 32), 256, 0, s, C, pixels, x, label, loss, picked, dloss, dx, accumulate);
  } else if (C <= 128) {
    launch(ce_nhwc_reg<T, 4, BWD>, grid_for(pixels, 16), 256, 0, s, C, pixels, x, label, loss, picked, dloss, dx, accumulate);
  } else if (C <= 256) {
    launch(ce_nhwc_reg<T, 8, BWD>, grid_for(pixels, 16), 256, 0, s, C, pixels, x, label, loss, picked, dloss, dx, accumulate);
  } else {
    launch(ce_nhwc<T, BWD>, grid_for(pixels, 8), 256, 0, s, C, pixels, x, label, loss, picked, dloss, dx, accumulate);
  }
  count_launch();
  return launch_status();
}

}  // namespace adk

using namespace adk;

extern "C" int ad_softmax_nll_loss_fwd(uint32_t C, uint32_t B, const float* y, const uint32_t* label, float* loss,
                                       void* stream) {
  if (B == 0) return AD_OK;
  if (!y || !label || !loss || C == 0) return AD_ERR_BAD_ARG;
  launch(nll_fwd_kernel, (B + 255) / 256, 256, 0, as_stream(stream), C, B, y, label, loss);
  count_launch();
  return launch_status();
}

extern "C" int ad_softmax_nll_loss_bwd(uint32_t C, uint32_t B, const float* y, const uint32_t* label,
                                       const float* dloss, float* dx, void* stream) {
  if (B == 0 || C == 0) return AD_OK;
  if (!y || !label || !dloss || !dx) return AD_ERR_BAD_ARG;
  size_t total = (size_t)C * B;
  launch(nll_bwd_kernel, (unsigned)((total + 255) / 256), 256, 0, as_stream(stream), C, B, y, label, dloss, dx);
  count_launch();
  return launch_status();
}

extern "C" int ad_softmax_ce_pixel_fwd(int32_t dtype, int32_t layout, uint32_t N, uint32_t C, uint32_t HW,
                                       const void* logits, const uint32_t* label, float* loss, uint64_t* picked,
                                       void* stream) {
  if ((size_t)N * HW == 0) return AD_OK;
  if (!logits || !label || !loss || C == 0 || C > 1024) return AD_ERR_BAD_ARG;
  AD_DISPATCH_DTYPE(dtype, return (launch_ce<T, false>(layout, N, C, HW, (const T*)logits, label, loss, (unsigned long long*)picked, nullptr, nullptr, 0,
                                                       as_stream(stream))));
}

extern "C" int ad_softmax_ce_pixel_bwd(int32_t dtype, int32_t layout, uint32_t N, uint32_t C, uint32_t HW,
                                       const void* logits, const uint32_t* label, const float* dloss, void* dlogits,
                                       int32_t accumulate, void* stream) {
  if ((size_t)N * HW == 0) return AD_OK;
  if (!logits || !label || !dloss || !dlogits || C == 0 || C > 1024) return AD_ERR_BAD_ARG;
  AD_DISPATCH_DTYPE(dtype, return (launch_ce<T, true>(layout, N, C, HW, (const T*)logits, label, nullptr, nullptr, dloss, (T*)dlogits, accumulate,
                                                      as_stream(stream))));
}
