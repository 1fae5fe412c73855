// Classifier head after the spatial stages: average pooling (global or windowed) and the fully connected
// layer.  Small, HBM- / latency-bound kernels: the head works on [batch][channels] vectors.
//   average pool:  CudnnPool2DOp with kAveragePool (reference src/op.cc:3346-3633; zoo.cc:1843-1852)
//   linear:        CublasLinearOp (reference src/op.cc:1199-1340: cublasSgemm + bias add)
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
// The weights (fp32) are the traffic: every kernel reads them for 8 images at a time.  64 x 2048 -> 1000: forward 73 -> 49,
// data gradient 75 -> 53, weight gradient 116 -> 25 us (beside the other strip's, which reads the same memory system).
constexpr uint32_t kLinB = 8;
static unsigned lin_groups(uint32_t n, uint32_t per) { const uint32_t g = n / per + (n % per != 0); return g > 65535 ? 65535 : g; }
// y[b][o] = bias[o] + sum_i x[b][i] * w[o][i]: one warp per output and 8 images, lanes stride over i, shuffle sums; the 8
// images lie in shared memory as fp32 (1024 features at a time), read by the 8 warps of the block
constexpr uint32_t kFwdI = 1024;
template <typename T>
__global__ void __launch_bounds__(256) linear_fwd_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
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
// dx[b][i] (+)= sum_o dy[b][o] * w[o][i]: a thread owns a column i and 8 images and adds the rows o in order; weights come
// through a ring of asynchronous copies (96 rows ahead), the gradients of the 8 images from shared memory
constexpr uint32_t kDxCols = 128, kDxRows = 32, kDxStages = 4, kDxMaxO = 1024;
template <typename T>
__global__ void __launch_bounds__(kDxCols) linear_dx_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ dy,
                                                            const float* __restrict__ w, T* dx, int accumulate) {
  grid_dependency();
  extern __shared__ __align__(16) float lin_sm[];
  float* const ring = lin_sm;                                      // [stage][row][column]
  float* const g = lin_sm + kDxStages * kDxRows * kDxCols;         // [row][image]
  const uint32_t tx = threadIdx.x, i = blockIdx.x * kDxCols + tx;
  const uint32_t bytes = i < I ? 4u : 0u;
  for (uint32_t b0 = blockIdx.y * kLinB; b0 < B; b0 += gridDim.y * kLinB) {
    const uint32_t nb = B - b0 < kLinB ? B - b0 : kLinB;
    float acc[kLinB];
#pragma unroll
    for (uint32_t j = 0; j < kLinB; ++j) acc[j] = 0.f;
    for (uint32_t oc = 0; oc < O; oc += kDxMaxO) {
      const uint32_t no = O - oc < kDxMaxO ? O - oc : kDxMaxO, steps = (no + kDxRows - 1) / kDxRows;
      __syncthreads();
      auto load = [&](uint32_t st) {
        float* d = ring + (st % kDxStages) * kDxRows * kDxCols + tx;
#pragma unroll 8
        for (uint32_t r = 0; r < kDxRows; ++r) {
          const uint32_t o = st * kDxRows + r;
          const float* src = w + (size_t)(oc + (o < no ? o : 0)) * I + (i < I ? i : 0);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(d + r * kDxCols)), "l"(src),
                       "r"(o < no ? bytes : 0u) : "memory");
        }
      };
      for (uint32_t st = 0; st < kDxStages - 1; ++st) {
        if (st < steps) load(st);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      for (uint32_t j = 0; j < kLinB; ++j)
        for (uint32_t o = tx; o < steps * kDxRows; o += kDxCols)
          g[o * kLinB + j] = j < nb && o < no ? ld_f(dy + (size_t)(b0 + j) * O + oc + o) : 0.f;
      for (uint32_t st = 0; st < steps; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kDxStages - 2) : "memory");
        __syncthreads();
        if (st + kDxStages - 1 < steps) load(st + kDxStages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* wr = ring + (st % kDxStages) * kDxRows * kDxCols + tx;
        const float* gr = g + st * kDxRows * kLinB;
        const uint32_t rows = no - st * kDxRows < kDxRows ? no - st * kDxRows : kDxRows;
#pragma unroll 8
        for (uint32_t r = 0; r < rows; ++r) {
          const float wv = wr[r * kDxCols];
          const float4 g0 = *(const float4*)(gr + r * kLinB), g1 = *(const float4*)(gr + r * kLinB + 4);
          const float gv[kLinB] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
          for (uint32_t j = 0; j < kLinB; ++j) acc[j] = fmaf(gv[j], wv, acc[j]);
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    if (i < I) {
#pragma unroll
      for (uint32_t j = 0; j < kLinB; ++j)
        if (j < nb) {
          T* d = dx + (size_t)(b0 + j) * I + i;
          st_f(d, accumulate ? ld_f(d) + acc[j] : acc[j]);
        }
    }
  }
}
constexpr int kDxSmem = (kDxStages * kDxRows * kDxCols + kDxMaxO * kLinB) * 4;
// dw[o][i] (+)= sum_b dy[b][o] * x[b][i]; db[o] (+)= sum_b dy[b][o]: one thread per (8 rows o, i), batch in order; the 8
// rows' gradients of 64 images at a time in shared memory
template <typename T>
__global__ void __launch_bounds__(256) linear_dw_kernel(uint32_t B, uint32_t I, uint32_t O, const T* __restrict__ x,
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
  const dim3 grid((unsigned)(((size_t)out_features + 7) / 8), lin_groups(batch, kLinB));
  AD_DISPATCH_DTYPE(dtype, (launch(linear_fwd_kernel<T>, grid, 256, 0, as_stream(stream), batch, in_features, out_features, (const T*)x, w, bias, (T*)y)));
  count_launch();
  return launch_status();
}

template <typename T>
static int launch_linear_dx(uint32_t B, uint32_t I, uint32_t O, const T* dy, const float* w, T* dx, int accumulate, cudaStream_t s) {
  static unsigned attr_done = 0;       // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_done & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(linear_dx_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDxSmem) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    attr_done |= 1u << (dev & 31);
  }
  launch(linear_dx_kernel<T>, dim3((I + kDxCols - 1) / kDxCols, lin_groups(B, kLinB)), kDxCols, kDxSmem, s, B, I, O, dy, w, dx, accumulate);
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
    AD_DISPATCH_DTYPE(dtype, { const int st = launch_linear_dx<T>(batch, in_features, out_features, (const T*)dy, w, (T*)dx, accumulate_dx, s); if (st != AD_OK) return st; });
    count_launch();
  }
  if (dw && in_features && out_features) {
    const dim3 grid((in_features + 255) / 256, lin_groups(out_features, 8));
    AD_DISPATCH_DTYPE(dtype, (launch(linear_dw_kernel<T>, grid, 256, 0, s, batch, in_features, out_features, (const T*)x, (const T*)dy, dw, db, accumulate_dw)));
    count_launch();
  }
  return launch_status();
}
