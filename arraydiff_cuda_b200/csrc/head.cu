// Classifier head after the spatial stages: average pooling (global or windowed) and the fully connected
// layer.  Small, HBM- / latency-bound kernels: the head works on [batch][channels] vectors.
//   average pool:  CudnnPool2DOp with kAveragePool (reference src/op.cc:3346-3633; zoo.cc:1843-1852)
//   linear:        CublasLinearOp (reference src/op.cc:1199-1340: cublasSgemm + bias add)
#include <algorithm>

#include "common.cuh"

namespace adk {

struct HView { char* base; long long sn, sc, sy, sx; };
static HView hview(const ad_tensor4* t) { return HView{(char*)t->base, t->sn, t->sc, t->sy, t->sx}; }

struct AvgP {
  HView x, y;
  uint32_t N, C, H, W, P, Q, kh, kw, sh, sw;
  int c_fastest, accumulate;
};

// one thread per output element; the window mean is accumulated in row-major order
template <typename T>
__global__ void __launch_bounds__(256) avgpool_fwd_kernel(AvgP p) {
  grid_dependency();
  const uint32_t total = p.N * p.C * p.P * p.Q, nt = gridDim.x * blockDim.x;
  const float inv = 1.0f / (float)(p.kh * p.kw);
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {   // past 2^32 on the last step
    uint32_t n, c, q, s, r = (uint32_t)i;
    if (p.c_fastest) { c = r % p.C; r /= p.C; s = r % p.Q; r /= p.Q; q = r % p.P; n = r / p.P; }
    else { s = r % p.Q; r /= p.Q; q = r % p.P; r /= p.P; c = r % p.C; n = r / p.C; }
    const T* X = (const T*)p.x.base + n * p.x.sn + c * p.x.sc;
    float acc = 0.f;
    for (uint32_t a = 0; a < p.kh; ++a)
      for (uint32_t b = 0; b < p.kw; ++b) acc += ld_f(X + (q * p.sh + a) * p.x.sy + (s * p.sw + b) * p.x.sx);
    st_f((T*)p.y.base + n * p.y.sn + c * p.y.sc + q * p.y.sy + s * p.y.sx, acc * inv);
  }
}
// one thread per input element gathers from the windows over it
template <typename T>
__global__ void __launch_bounds__(256) avgpool_bwd_kernel(AvgP p) {
  grid_dependency();
  const uint32_t total = p.N * p.C * p.H * p.W, nt = gridDim.x * blockDim.x;
  const float inv = 1.0f / (float)(p.kh * p.kw);
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {   // past 2^32 on the last step
    uint32_t n, c, y, x, r = (uint32_t)i;
    if (p.c_fastest) { c = r % p.C; r /= p.C; x = r % p.W; r /= p.W; y = r % p.H; n = r / p.H; }
    else { x = r % p.W; r /= p.W; y = r % p.H; r /= p.H; c = r % p.C; n = r / p.C; }
    const uint32_t q_lo = y + 1 > p.kh ? (y + 1 - p.kh + p.sh - 1) / p.sh : 0;
    const uint32_t s_lo = x + 1 > p.kw ? (x + 1 - p.kw + p.sw - 1) / p.sw : 0;
    const T* G = (const T*)p.y.base + n * p.y.sn + c * p.y.sc;
    float acc = 0.f;
    for (uint32_t q = q_lo; q < p.P && q * p.sh <= y; ++q)
      for (uint32_t s = s_lo; s < p.Q && s * p.sw <= x; ++s) acc += ld_f(G + q * p.y.sy + s * p.y.sx);
    acc *= inv;
    T* o = (T*)p.x.base + n * p.x.sn + c * p.x.sc + y * p.x.sy + x * p.x.sx;
    st_f(o, p.accumulate ? ld_f(o) + acc : acc);
  }
}

// Global pool (the window is the whole map): what the classifier head does.
//   channel-fastest bf16 in 16-byte groups: a thread per group of 8 channels adds up to 256 pixels in order (8 in flight);
//   larger maps: a block owns (image, up to 32 groups), its remaining lanes split the pixels and meet in shared memory;
//   planes: a warp per plane, lanes over the pixels.
// 32 x 2048 channels of 7 x 7: forward 16 us, gradient 54 -> 5 us.
template <typename T>
__global__ void __launch_bounds__(256) avgpool_global_plane_fwd(AvgP p) {
  grid_dependency();
  const uint32_t planes = p.N * p.C, lane = threadIdx.x & 31, hw = p.H * p.W;
  const uint32_t plane = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const uint32_t n = plane / p.C, c = plane - n * p.C;
  const T* X = (const T*)p.x.base + n * p.x.sn + c * p.x.sc;
  float acc = 0.f;
#pragma unroll 4
  for (uint32_t i = lane; i < hw; i += 32) {
    const uint32_t y = i / p.W, x = i - y * p.W;
    acc += ld_f(X + y * p.x.sy + x * p.x.sx);
  }
  acc = warp_sum(acc);
  if (lane == 0) st_f((T*)p.y.base + n * p.y.sn + c * p.y.sc, acc * (1.0f / (float)hw));
}
template <typename T>
__global__ void __launch_bounds__(256) avgpool_global_plane_bwd(AvgP p) {
  grid_dependency();
  const uint32_t planes = p.N * p.C, lane = threadIdx.x & 31, hw = p.H * p.W;
  const uint32_t plane = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const uint32_t n = plane / p.C, c = plane - n * p.C;
  const float g = ld_f((const T*)p.y.base + n * p.y.sn + c * p.y.sc) * (1.0f / (float)hw);
  T* X = (T*)p.x.base + n * p.x.sn + c * p.x.sc;
  for (uint32_t i = lane; i < hw; i += 32) {
    const uint32_t y = i / p.W, x = i - y * p.W;
    T* o = X + y * p.x.sy + x * p.x.sx;
    st_f(o, p.accumulate ? ld_f(o) + g : g);
  }
}
__device__ __forceinline__ void un8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 t = __bfloat1622float2(h[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}
__device__ __forceinline__ uint4 pk8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
  return v;
}
__global__ void __launch_bounds__(64) avgpool_global_nhwc_seq(AvgP p) {
  grid_dependency();
  const uint32_t g = blockIdx.x * 64 + threadIdx.x, n = blockIdx.y;
  if (g >= p.C / 8) return;
  const __nv_bfloat16* X = (const __nv_bfloat16*)p.x.base + n * p.x.sn + g * 8;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  // 16 pixels in flight, added in their order
  const uint32_t px = p.H * p.W;
  uint32_t y = 0, x = 0;
  for (uint32_t i = 0; i < px; i += 16) {
    uint4 q[16];
#pragma unroll
    for (uint32_t u = 0; u < 16; ++u) {
      if (i + u < px) q[u] = *(const uint4*)(X + y * p.x.sy + x * p.x.sx);
      if (++x == p.W) { x = 0; ++y; }
    }
#pragma unroll
    for (uint32_t u = 0; u < 16; ++u) {
      if (i + u >= px) break;
      float v[8];
      un8(q[u], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
  const float inv = 1.0f / (float)(p.H * p.W);
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] *= inv;
  *(uint4*)((__nv_bfloat16*)p.y.base + n * p.y.sn + g * 8) = pk8(acc);
}
// gb: groups of 8 channels per block (a power of two up to 32)
__global__ void __launch_bounds__(256) avgpool_global_nhwc_fwd(AvgP p, uint32_t gb) {
  grid_dependency();
  __shared__ float sm[256][9];
  const uint32_t G = p.C / 8, gl = threadIdx.x % gb, pl = threadIdx.x / gb, PL = 256 / gb, g = blockIdx.x * gb + gl, n = blockIdx.y;
  const uint32_t hw = p.H * p.W;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (g < G) {
    const __nv_bfloat16* X = (const __nv_bfloat16*)p.x.base + n * p.x.sn + g * 8;
#pragma unroll 4
    for (uint32_t i = pl; i < hw; i += PL) {
      const uint32_t y = i / p.W, x = i - y * p.W;
      float v[8];
      un8(*(const uint4*)(X + y * p.x.sy + x * p.x.sx), v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[threadIdx.x][j] = acc[j];
  __syncthreads();
  const float inv = 1.0f / (float)hw;
  for (uint32_t t = threadIdx.x; t < gb * 8; t += 256) {
    const uint32_t tg = t >> 3, j = t & 7;
    if (blockIdx.x * gb + tg >= G) continue;
    float v = 0.f;
    for (uint32_t q = 0; q < PL; ++q) v += sm[q * gb + tg][j];
    st_f((__nv_bfloat16*)p.y.base + n * p.y.sn + (blockIdx.x * gb + tg) * 8 + j, v * inv);
  }
}
__global__ void __launch_bounds__(256) avgpool_global_nhwc_bwd(AvgP p, uint32_t gb) {
  grid_dependency();
  const uint32_t G = p.C / 8, gl = threadIdx.x % gb, pl = threadIdx.x / gb, PL = 256 / gb, g = blockIdx.x * gb + gl, n = blockIdx.y;
  if (g >= G) return;
  const uint32_t hw = p.H * p.W;
  const float inv = 1.0f / (float)hw;
  float v[8];
  un8(*(const uint4*)((const __nv_bfloat16*)p.y.base + n * p.y.sn + g * 8), v);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] *= inv;
  const uint4 q = pk8(v);
  __nv_bfloat16* X = (__nv_bfloat16*)p.x.base + n * p.x.sn + g * 8;
#pragma unroll 4
  for (uint32_t i = pl; i < hw; i += PL) {
    const uint32_t y = i / p.W, x = i - y * p.W;
    uint4* o = (uint4*)(X + y * p.x.sy + x * p.x.sx);
    if (p.accumulate) {
      float old[8];
      un8(*o, old);
#pragma unroll
      for (int j = 0; j < 8; ++j) old[j] += v[j];
      *o = pk8(old);
    } else {
      *o = q;
    }
  }
}
static bool avg_vec_ok(const ad_tensor4* t) {
  return t->dtype == AD_BF16 && t->sc == 1 && (t->C & 7u) == 0 && !((uintptr_t)t->base & 15u) && !(t->sn & 7) && !(t->sy & 7) && !(t->sx & 7);
}
// Launches the global form if the call is one; `launched` says so
static int launch_global(const AvgP& p, const ad_tensor4* x, const ad_tensor4* y, bool bwd, bool& launched, cudaStream_t s) {
  launched = p.kh == p.H && p.kw == p.W && p.N <= 65535;
  if (!launched) return AD_OK;
  if (avg_vec_ok(x) && avg_vec_ok(y)) {
    // few (image, channel) pairs: fewer groups per block leave more lanes to split the pixels
    uint32_t gb = 32;
    while (gb > 1 && (unsigned long long)((p.C / 8 + gb - 1) / gb) * p.N < 2ull * kNumSMs && 256 / gb < p.H * p.W) gb >>= 1;
    while (gb > 1 && gb / 2 >= p.C / 8) gb >>= 1;
    const dim3 grid((p.C / 8 + gb - 1) / gb, p.N);
    if (bwd) launch(avgpool_global_nhwc_bwd, grid, 256, 0, s, p, gb);
    else if (p.H * p.W <= 256) launch(avgpool_global_nhwc_seq, dim3((p.C / 8 + 63) / 64, p.N), 64, 0, s, p);
    else launch(avgpool_global_nhwc_fwd, grid, 256, 0, s, p, gb);
  } else if (x->sc != 1 || x->C == 1) {
    const unsigned grid = (unsigned)(((size_t)p.N * p.C + 7) / 8);
    if (bwd) AD_DISPATCH_DTYPE(x->dtype, (launch(avgpool_global_plane_bwd<T>, grid, 256, 0, s, p)));
    else AD_DISPATCH_DTYPE(x->dtype, (launch(avgpool_global_plane_fwd<T>, grid, 256, 0, s, p)));
  } else {
    launched = false;
    return AD_OK;
  }
  count_launch();
  return launch_status();
}

static int avg_params(const ad_tensor4* x, const ad_tensor4* y, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, AvgP& p) {
  if (!x || !y || !x->base || !y->base || kh == 0 || kw == 0 || sh == 0 || sw == 0) return AD_ERR_BAD_ARG;
  if (x->H < kh || x->W < kw) return AD_ERR_BAD_ARG;
  const uint32_t P = (x->H - kh) / sh + 1, Q = (x->W - kw) / sw + 1;
  if (y->N != x->N || y->C != x->C || y->H != P || y->W != Q || y->dtype != x->dtype) return AD_ERR_BAD_ARG;
  if ((size_t)x->N * x->C * x->H * x->W >= (1ull << 32)) return AD_ERR_LIMIT;
  p.x = hview(x); p.y = hview(y);
  p.N = x->N; p.C = x->C; p.H = x->H; p.W = x->W; p.P = P; p.Q = Q; p.kh = kh; p.kw = kw; p.sh = sh; p.sw = sw;
  return AD_OK;
}

// ------------------------------------------------------------------ fully connected
// Each kernel reads the fp32 weights for 8 images (the weight gradient x for 8 rows) at a time, four features per thread and
// load: a warp meets 128 products with every 12 loads forward, 32 with 3 in the gradients, so that neither loads nor
// shared memory bound them but the latency of a chain of loads, which more warps and loads in flight cut.  With a product per
// read of shared memory (forward), one chain over all rows per column (data gradient) and one load at a time (weight
// gradient), 64 x 2048 -> 1000 took 37, 40 and 19 us, 4 x 512 -> 1000 6, 39 and 6; now 15, 15 and 12, 5, 13 and 5 (5 of them the
// launch).  Sums over 62 rows and 16 warps are also closer than a chain over 1000: 5.7e-7 -> 1.6e-7 against 64 bits.
// VEC: rows are multiples of four elements and aligned: 16-byte loads of weights; else a thread's four features are 32 apart.
constexpr uint32_t kLinB = 8;
static unsigned lin_groups(uint32_t n, uint32_t per) { const uint32_t g = n / per + (n % per != 0); return g > 65535 ? 65535 : g; }
// a thread's four features of the 128 from c0 on
template <bool VEC> __device__ __forceinline__ uint32_t lin_col(uint32_t c0, uint32_t lane, uint32_t e) { return c0 + (VEC ? lane * 4 + e : lane + e * 32); }
template <typename T, bool VEC>
__device__ __forceinline__ void lin_ld4(const T* row, uint32_t c0, uint32_t lane, uint32_t I, bool have, float (&v)[4]) {
  if (VEC) {
    const uint32_t c = c0 + lane * 4;
    if (sizeof(T) == 4) {
      const float4 q = have && c < I ? *(const float4*)(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
      const uint2 q = have && c < I ? *(const uint2*)(row + c) : make_uint2(0u, 0u);
      v[0] = __uint_as_float(q.x << 16); v[1] = __uint_as_float(q.x & 0xffff0000u);
      v[2] = __uint_as_float(q.y << 16); v[3] = __uint_as_float(q.y & 0xffff0000u);
    }
  } else {
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) { const uint32_t c = lin_col<false>(c0, lane, e); v[e] = have && c < I ? ld_f(row + c) : 0.f; }
  }
}
// y[b][o] = bias[o] + sum_i x[b][i] * w[o][i]: a warp for four outputs and 8 images, its lanes along i; the 32 sums over the
// lanes in 31 exchanges, after which a lane holds one
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) linear_fwd_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
                                                         const float* __restrict__ w, const float* __restrict__ bias, T* y) {
  grid_dependency();
  const uint32_t o0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 4, lane = threadIdx.x & 31;
  if (o0 >= O) return;
  for (uint32_t b0 = blockIdx.y * kLinB; b0 < B; b0 += gridDim.y * kLinB) {
    const uint32_t nb = B - b0 < kLinB ? B - b0 : kLinB;
    float acc[32];                      // [output][image]
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k] = 0.f;
#pragma unroll 2
    for (uint32_t c0 = 0; c0 < I; c0 += 128) {
      float wv[4][4], xv[kLinB][4];
#pragma unroll
      for (uint32_t o = 0; o < 4; ++o) lin_ld4<float, VEC>(w + (size_t)(o0 + o) * I, c0, lane, I, o0 + o < O, wv[o]);
#pragma unroll
      for (uint32_t j = 0; j < kLinB; ++j) lin_ld4<T, VEC>(x + (size_t)(b0 + j) * I, c0, lane, I, j < nb, xv[j]);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int o = 0; o < 4; ++o)
#pragma unroll
          for (uint32_t j = 0; j < kLinB; ++j) acc[o * 8 + j] = fmaf(xv[j][e], wv[o][e], acc[o * 8 + j]);
    }
#pragma unroll
    for (int n = 16; n >= 1; n >>= 1) {
      const bool up = lane & n;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        const float other = __shfl_xor_sync(0xffffffffu, up ? acc[k] : acc[k + n], n);
        acc[k] = (up ? acc[k + n] : acc[k]) + other;
      }
    }
    const uint32_t o = o0 + lane / 8, j = lane % 8;
    if (o < O && j < nb) st_f(y + (size_t)(b0 + j) * O + o, acc[0] + (bias ? bias[o] : 0.f));
  }
}
// The same with a warp per output, the 8 images as fp32 in shared memory (1024 features at a time): rows of bf16 that no 8-byte load
// reaches
constexpr uint32_t kFwdI = 1024;
template <typename T>
__global__ void __launch_bounds__(256) linear_fwd_staged_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
                                                                const float* __restrict__ w, const float* __restrict__ bias, T* y) {
  grid_dependency();
  __shared__ float xs[kLinB][kFwdI];
  const uint32_t o = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  for (uint32_t b0 = blockIdx.y * kLinB; b0 < B; b0 += gridDim.y * kLinB) {
    const uint32_t nb = B - b0 < kLinB ? B - b0 : kLinB;
    float acc[kLinB];
#pragma unroll
    for (uint32_t j = 0; j < kLinB; ++j) acc[j] = 0.f;
    for (uint32_t i0 = 0; i0 < I; i0 += kFwdI) {
      const uint32_t ni = I - i0 < kFwdI ? I - i0 : kFwdI;
      __syncthreads();
      for (uint32_t j = 0; j < kLinB; ++j)
        for (uint32_t i = threadIdx.x; i < ni; i += 256) xs[j][i] = j < nb ? ld_f(x + (size_t)(b0 + j) * I + i0 + i) : 0.f;
      __syncthreads();
      if (o < O) {
        const float* wr = w + (size_t)o * I + i0;
        uint32_t i = lane;
        for (; i + 7 * 32 < ni; i += 8 * 32) {
          float wv[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) wv[u] = wr[i + u * 32];
#pragma unroll
          for (int u = 0; u < 8; ++u)
#pragma unroll
            for (uint32_t j = 0; j < kLinB; ++j) acc[j] = fmaf(xs[j][i + u * 32], wv[u], acc[j]);
        }
        for (; i < ni; i += 32) {
          const float wv = wr[i];
#pragma unroll
          for (uint32_t j = 0; j < kLinB; ++j) acc[j] = fmaf(xs[j][i], wv, acc[j]);
        }
      }
    }
    if (o < O) {
#pragma unroll
      for (uint32_t j = 0; j < kLinB; ++j) {
        const float v = warp_sum(acc[j]);
        if (lane == 0 && j < nb) st_f(y + (size_t)(b0 + j) * O + o, v + (bias ? bias[o] : 0.f));
      }
    }
  }
}
// Single loads of bf16 features bound the kernel of four outputs per warp, which reads each image's once for every four outputs
// (64 x 2046 -> 100 33 us with the images in shared memory, 66; 256 x 2046 -> 4096 482, 610); short rows and, up to 1023 features,
// many outputs run it all the same (1024 x 65 -> 4096 390, 170; 1024 x 511 -> 4096 682, 587).
static bool lin_fwd_staged(bool vec, size_t es, uint32_t B, uint32_t I, uint32_t O) {
  return !vec && es == 2 && B > 1 && (I >= 1024 || (I >= 256 && O < 1000));
}
// dx[b][i] (+)= sum_o dy[b][o] * w[o][i]: W warps share the rows o of 128 columns and 8 images, every W-th each; their sums are
// added in order.  The gradients of the 8 images lie in shared memory, 1024 rows at a time.  W is 16, but where few rows in many
// blocks leave a warp with less to sum than the W sums of the others (lin_dx_warps).
constexpr uint32_t kDxMaxO = 1024;
template <typename T, bool VEC, uint32_t W>
__global__ void __launch_bounds__(W * 32) linear_dx_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ dy,
                                                                  const float* __restrict__ w, T* dx, int accumulate) {
  grid_dependency();
  extern __shared__ __align__(16) float lin_sm[];
  float* const part = lin_sm;                                      // [warp][image, column of four][lane]
  float* const g = lin_sm + W * 32 * 32;                           // [row][image]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = blockIdx.x * 128;
  for (uint32_t b0 = blockIdx.y * kLinB; b0 < B; b0 += gridDim.y * kLinB) {
    const uint32_t nb = B - b0 < kLinB ? B - b0 : kLinB;
    float acc[kLinB][4];
#pragma unroll
    for (uint32_t j = 0; j < kLinB; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    for (uint32_t oc = 0; oc < O; oc += kDxMaxO) {
      const uint32_t no = O - oc < kDxMaxO ? O - oc : kDxMaxO;
      __syncthreads();
#pragma unroll
      for (uint32_t j = 0; j < kLinB; ++j)
        for (uint32_t o = threadIdx.x; o < no; o += W * 32) g[o * kLinB + j] = j < nb ? ld_f(dy + (size_t)(b0 + j) * O + oc + o) : 0.f;
      __syncthreads();
#pragma unroll 8
      for (uint32_t o = warp; o < no; o += W) {
        float wv[4];
        lin_ld4<float, VEC>(w + (size_t)(oc + o) * I, c0, lane, I, true, wv);
        const float4 g0 = *(const float4*)(g + o * kLinB), g1 = *(const float4*)(g + o * kLinB + 4);
        const float gv[kLinB] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
        for (uint32_t j = 0; j < kLinB; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] = fmaf(gv[j], wv[e], acc[j][e]);
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < kLinB; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) part[(warp * 32 + j * 4 + e) * 32 + lane] = acc[j][e];
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < 32 * 32; t += W * 32) {
      const uint32_t j = t >> 7, e = (t >> 5) & 3, i = lin_col<VEC>(c0, t & 31, e);
      if (j >= nb || i >= I) continue;
      float v = 0.f;
#pragma unroll
      for (uint32_t q = 0; q < W; ++q) v += part[q * 32 * 32 + t];
      T* d = dx + (size_t)(b0 + j) * I + i;
      st_f(d, accumulate ? ld_f(d) + v : v);
    }
  }
}
// dw[o][i] (+)= sum_b dy[b][o] * x[b][i]; db[o] (+)= sum_b dy[b][o]: a thread for 8 rows o and four columns i, batch in order; the 8
// rows' gradients of 64 images at a time in shared memory
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) linear_dw_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
                                                        const T* __restrict__ dy, float* dw, float* db, int accumulate) {
  grid_dependency();
  __shared__ __align__(16) float g[64][8];
  const uint32_t lane = threadIdx.x & 31, c0 = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 128;
  for (uint32_t o0 = blockIdx.y * 8; o0 < O; o0 += gridDim.y * 8) {
    const uint32_t no = O - o0 < 8 ? O - o0 : 8;
    float acc[8][4], accb = 0.f;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[k][e] = 0.f;
    for (uint32_t b0 = 0; b0 < B; b0 += 64) {
      const uint32_t nb = B - b0 < 64 ? B - b0 : 64;
      __syncthreads();
      for (uint32_t t = threadIdx.x; t < nb * 8; t += 128) g[t >> 3][t & 7] = (t & 7) < no ? ld_f(dy + (size_t)(b0 + (t >> 3)) * O + o0 + (t & 7)) : 0.f;
      __syncthreads();
      if (db && blockIdx.x == 0 && threadIdx.x < 8) {
#pragma unroll 8
        for (uint32_t b = 0; b < nb; ++b) accb += g[b][threadIdx.x];
      }
      for (uint32_t b = 0; b < nb; b += 8) {
        float xv[8][4];
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {
          const T* row = x + (size_t)(b0 + (b + r < nb ? b + r : b)) * I;      // past the last image and feature: others, not used
          if (VEC) {
            lin_ld4<T, VEC>(row, c0, lane, I, true, xv[r]);
          } else {
#pragma unroll
            for (uint32_t e = 0; e < 4; ++e) xv[r][e] = ld_f(row + min(lin_col<false>(c0, lane, e), I - 1));
          }
        }
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {
          if (b + r >= nb) break;
          const float4 g0 = *(const float4*)&g[b + r][0], g1 = *(const float4*)&g[b + r][4];
          const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[k][e] = fmaf(gv[k], xv[r][e], acc[k][e]);
        }
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      if (k >= no) break;
      float* d = dw + (size_t)(o0 + k) * I;
      if (VEC) {
        const uint32_t c = lin_col<true>(c0, lane, 0);
        if (c < I) {
          float4 v = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
          if (accumulate) { const float4 old = *(const float4*)(d + c); v = make_float4(old.x + v.x, old.y + v.y, old.z + v.z, old.w + v.w); }
          *(float4*)(d + c) = v;
        }
      } else {
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
          const uint32_t c = lin_col<false>(c0, lane, e);
          if (c < I) d[c] = accumulate ? d[c] + acc[k][e] : acc[k][e];
        }
      }
    }
    if (db && blockIdx.x == 0 && threadIdx.x < no) db[o0 + threadIdx.x] = accumulate ? db[o0 + threadIdx.x] + accb : accb;
  }
}
// The same by a thread per column: rows that no 16-byte load reaches
template <typename T>
__global__ void __launch_bounds__(256) linear_dw_column_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
                                                               const T* __restrict__ dy, float* dw, float* db, int accumulate) {
  grid_dependency();
  __shared__ __align__(16) float g[64][8];
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  for (uint32_t o0 = blockIdx.y * 8; o0 < O; o0 += gridDim.y * 8) {
    const uint32_t no = O - o0 < 8 ? O - o0 : 8;
    float acc[8], accb[8], old[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
      acc[j] = accb[j] = 0.f;
      old[j] = accumulate && j < no && i < I ? dw[(size_t)(o0 + j) * I + i] : 0.f;
    }
    for (uint32_t b0 = 0; b0 < B; b0 += 64) {
      const uint32_t nb = B - b0 < 64 ? B - b0 : 64;
      __syncthreads();
      for (uint32_t t = threadIdx.x; t < nb * 8; t += 256) g[t >> 3][t & 7] = (t & 7) < no ? ld_f(dy + (size_t)(b0 + (t >> 3)) * O + o0 + (t & 7)) : 0.f;
      __syncthreads();
      if (i < I) {
#pragma unroll 8
        for (uint32_t b = 0; b < nb; ++b) {
          const float xv = ld_f(x + (size_t)(b0 + b) * I + i);
          const float4 g0 = *(const float4*)&g[b][0], g1 = *(const float4*)&g[b][4];
          const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) { acc[j] = fmaf(gv[j], xv, acc[j]); accb[j] += gv[j]; }
        }
      }
    }
    if (i < I) {
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j)
        if (j < no) {
          dw[(size_t)(o0 + j) * I + i] = accumulate ? old[j] + acc[j] : acc[j];
          if (db && i == 0) db[o0 + j] = accumulate ? db[o0 + j] + accb[j] : accb[j];
        }
    }
  }
}
// rows of four elements per load: x and dx of `es` bytes each
static bool lin_vec(uint32_t I, const void* w, const void* x, size_t es) {
  return I % 4 == 0 && ((uintptr_t)w & 15u) == 0 && ((uintptr_t)x & (4 * es - 1)) == 0;
}
// Filter gradient with a thread per column.  Four columns per thread leave a quarter of the warps, which without 16-byte loads wait
// three times as long (1024 x 2046 -> 100 fp32 181 us by columns, 478; 64 x 511 -> 1000 bf16 16, 33), but for a few images and
// many outputs, where the stores count (1 x 2046 -> 4096: 18, 14).  Of 64 features in bf16 half a warp has work: 1024 x 64 ->
// 4096 135, 161.
static bool lin_dw_by_columns(bool vec, size_t es, uint32_t B, uint32_t I, uint32_t O) {
  return vec ? es == 2 && I <= 64 && O >= 2048 : I < 512 || B > (O < 512 ? 0u : O < 2048 ? 4u : 16u);
}

}  // namespace adk

using namespace adk;

extern "C" int ad_avgpool2d_fwd(const ad_tensor4* x, const ad_tensor4* y, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw,
                                void* stream) {
  AvgP p{};
  int st = avg_params(x, y, kh, kw, sh, sw, p);
  if (st != AD_OK) return st;
  const size_t total = (size_t)p.N * p.C * p.P * p.Q;
  if (total == 0) return AD_OK;
  bool launched = false;
  st = launch_global(p, x, y, false, launched, as_stream(stream));
  if (launched || st != AD_OK) return st;
  p.c_fastest = y->sc == 1 && y->C > 1;
  AD_DISPATCH_DTYPE(x->dtype, (launch(avgpool_fwd_kernel<T>, grid_for(total, 256, 16), 256, 0, as_stream(stream), p)));
  count_launch();
  return launch_status();
}

extern "C" int ad_avgpool2d_bwd(const ad_tensor4* dy, const ad_tensor4* dx, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw,
                                int32_t accumulate, void* stream) {
  AvgP p{};
  int st = avg_params(dx, dy, kh, kw, sh, sw, p);
  if (st != AD_OK) return st;
  const size_t total = (size_t)p.N * p.C * p.H * p.W;
  if (total == 0) return AD_OK;
  p.c_fastest = dx->sc == 1 && dx->C > 1;
  p.accumulate = accumulate;
  bool launched = false;
  st = launch_global(p, dx, dy, true, launched, as_stream(stream));
  if (launched || st != AD_OK) return st;
  AD_DISPATCH_DTYPE(dx->dtype, (launch(avgpool_bwd_kernel<T>, grid_for(total, 256, 16), 256, 0, as_stream(stream), p)));
  count_launch();
  return launch_status();
}

extern "C" int ad_linear_fwd(int32_t dtype, uint32_t batch, uint32_t in_features, uint32_t out_features, const void* x,
                             const float* w, const float* bias, void* y, void* stream) {
  if (!x || !w || !y) return AD_ERR_BAD_ARG;
  if ((size_t)batch * out_features >= (1ull << 31) || (size_t)batch * in_features >= (1ull << 31)) return AD_ERR_LIMIT;
  if (batch == 0 || out_features == 0) return AD_OK;
  AD_DISPATCH_DTYPE(dtype, {
    const bool vec = lin_vec(in_features, w, x, sizeof(T)), staged = lin_fwd_staged(vec, sizeof(T), batch, in_features, out_features);
    const unsigned per = staged ? 8 : 32;
    launch(staged ? linear_fwd_staged_kernel<T> : vec ? linear_fwd_kernel<T, true> : linear_fwd_kernel<T, false>,
           dim3((unsigned)(((size_t)out_features + per - 1) / per), lin_groups(batch, kLinB)), 256, 0, as_stream(stream), batch, in_features, out_features,
           (const T*)x, w, bias, (T*)y);
  });
  count_launch();
  return launch_status();
}

// Warps that share a block's rows.  16 x 4 KB of sums for 128 rows and fewer cost more than their products where the blocks fill the
// machine (fp32, 1024 x 8192 -> 10 207 us with 16 warps, 43 with 4, -> 100 323, 145 with 8); fewer blocks are one chain of rows each.
static uint32_t lin_dx_warps(uint32_t B, uint32_t I, uint32_t O) {
  if (O > 128 || (unsigned long long)((I + 127) / 128) * lin_groups(B, kLinB) <= kNumSMs) return 16;
  return O > 32 ? 8 : 4;
}
template <typename T, bool VEC, uint32_t W>
static int launch_linear_dx(uint32_t B, uint32_t I, uint32_t O, const T* dy, const float* w, T* dx, int accumulate, cudaStream_t s) {
  if (lin_dx_warps(B, I, O) != W) {
    if constexpr (W > 4) return launch_linear_dx<T, VEC, W / 2>(B, I, O, dy, w, dx, accumulate, s);
  }
  constexpr uint32_t most = (kDxMaxO * kLinB + W * 32 * 32) * 4;
  static unsigned attr_done = 0;       // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_done & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(linear_dx_kernel<T, VEC, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    attr_done |= 1u << (dev & 31);
  }
  const uint32_t smem = (std::min(O, kDxMaxO) * kLinB + W * 32 * 32) * 4;
  launch(linear_dx_kernel<T, VEC, W>, dim3((I + 127) / 128, lin_groups(B, kLinB)), W * 32, smem, s, B, I, O, dy, w, dx, accumulate);
  return AD_OK;
}

extern "C" int ad_linear_bwd(int32_t dtype, uint32_t batch, uint32_t in_features, uint32_t out_features, const void* x,
                             const float* w, const void* dy, void* dx, float* dw, float* db, int32_t accumulate_dx,
                             int32_t accumulate_dw, void* stream) {
  if (!x || !w || !dy) return AD_ERR_BAD_ARG;
  if ((size_t)batch * out_features >= (1ull << 31) || (size_t)batch * in_features >= (1ull << 31) ||
      (size_t)in_features * out_features >= (1ull << 31))
    return AD_ERR_LIMIT;
  if (batch == 0) return AD_OK;
  cudaStream_t s = as_stream(stream);
  if (dx && in_features) {
    AD_DISPATCH_DTYPE(dtype, {
      const int st = lin_vec(in_features, w, w, sizeof(T)) ? launch_linear_dx<T, true, 16>(batch, in_features, out_features, (const T*)dy, w, (T*)dx, accumulate_dx, s)
                                                           : launch_linear_dx<T, false, 16>(batch, in_features, out_features, (const T*)dy, w, (T*)dx, accumulate_dx, s);
      if (st != AD_OK) return st;
    });
    count_launch();
  }
  if (dw && in_features && out_features) {
    AD_DISPATCH_DTYPE(dtype, {
      const bool vec = lin_vec(in_features, dw, x, sizeof(T));
      const unsigned groups = lin_groups(out_features, 8);
      if (lin_dw_by_columns(vec, sizeof(T), batch, in_features, out_features))
        launch(linear_dw_column_kernel<T>, dim3((in_features + 255) / 256, groups), 256, 0, s, batch, in_features, out_features, (const T*)x, (const T*)dy, dw, db,
               accumulate_dw);
      else
        launch(vec ? linear_dw_kernel<T, true> : linear_dw_kernel<T, false>, dim3((in_features + 511) / 512, groups), 128, 0, s, batch, in_features, out_features,
               (const T*)x, (const T*)dy, dw, db, accumulate_dw);
    });
    count_launch();
  }
  return launch_status();
}
