// Packed fp32 array arithmetic, the fused SGD update, and strided ReLU / add / convert.
// All HBM-bound: one read of each input and one write of each output, 16-byte vectors
// where the pointers allow, grid-stride loops sized from the SM count.
#include <algorithm>

#include "common.cuh"

namespace adk {

unsigned long long g_launch_count = 0;
thread_local bool g_early_launch = true;
thread_local int g_last_conv_kernel = kConvNone;

// ---------------------------------------------------------------- packed fp32 arrays
// The rounding of each expression is written out (explicit fmaf / __fmul_rn) so that the
// result does not depend on compiler contraction and matches the reference kernels, which
// nvcc compiles with fused multiply-add (src/kernels/array.cu:58-150).
enum ArrOp { kSet, kAdd, kAddScaled, kAddOnline, kScale, kScaleAdd };

template <int OP>
__device__ __forceinline__ float arr_apply(float a, float b, float x, float y) {
  switch (OP) {
    case kSet: return a;
    case kAdd: return __fadd_rn(x, y);
    case kAddScaled: return fmaf(b, y, __fmul_rn(a, x));
    case kAddOnline: return fmaf(a, __fsub_rn(x, y), y);
    case kScale: return __fmul_rn(a, x);
    default: return fmaf(a, x, y);
  }
}

template <int OP>
__global__ void __launch_bounds__(256) arr_kernel(size_t n, float a, float b, const float* __restrict__ x, float* y) {
  grid_dependency();
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
  const bool vec = (((uintptr_t)y | (uintptr_t)(OP == kSet ? (const float*)y : x)) & 15u) == 0;
  if (vec) {
    const size_t n4 = n / 4;
    for (size_t i = tid; i < n4; i += nt) {
      float4 xv = OP == kSet ? make_float4(0, 0, 0, 0) : reinterpret_cast<const float4*>(x)[i];
      float4 yv = (OP == kSet || OP == kScale) ? make_float4(0, 0, 0, 0) : reinterpret_cast<float4*>(y)[i];
      yv.x = arr_apply<OP>(a, b, xv.x, yv.x); yv.y = arr_apply<OP>(a, b, xv.y, yv.y);
      yv.z = arr_apply<OP>(a, b, xv.z, yv.z); yv.w = arr_apply<OP>(a, b, xv.w, yv.w);
      reinterpret_cast<float4*>(y)[i] = yv;
    }
    for (size_t i = n4 * 4 + tid; i < n; i += nt)
      y[i] = arr_apply<OP>(a, b, OP == kSet ? 0.f : x[i], (OP == kSet || OP == kScale) ? 0.f : y[i]);
  } else {
    for (size_t i = tid; i < n; i += nt)
      y[i] = arr_apply<OP>(a, b, OP == kSet ? 0.f : x[i], (OP == kSet || OP == kScale) ? 0.f : y[i]);
  }
}

template <int OP>
static int arr_launch(size_t n, float a, float b, const float* x, float* y, void* stream) {
  if (n == 0) return AD_OK;
  if (!y || (OP != kSet && !x)) return AD_ERR_BAD_ARG;
  launch(arr_kernel<OP>, grid_for((n + 3) / 4, 256), 256, 0, as_stream(stream), n, a, b, x, y);
  count_launch();
  return launch_status();
}

// ---------------------------------------------------------------- fused SGD
__global__ void __launch_bounds__(256) sgd_kernel(size_t n, float* theta, float* g, float* m, float l2, float mu,
                                                  float alpha, float alpha_next, int nesterov,
                                                  __nv_bfloat16* shadow, const int32_t* guard) {
  grid_dependency();
  // a step whose bounded waits ran out worked on stale halo rows or gradients: leave the parameters alone
  if (guard && *guard != 0) return;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
  const float nmu = __fmul_rn(-alpha_next, mu);
  for (size_t i = tid; i < n; i += nt) {
    float gi = g[i], th = theta[i], mi = m[i];
    // each line is add_scaled(alpha, x, beta): y = fma(beta, y, round(alpha * x))
    if (l2 != 0.f) gi = fmaf(1.0f, gi, __fmul_rn(l2, th));
    mi = fmaf(mu, mi, __fmul_rn(1.0f, gi));
    if (nesterov) {
      th = fmaf(1.0f, th, __fmul_rn(-alpha, gi));
      th = fmaf(1.0f, th, __fmul_rn(nmu, mi));
    } else {
      th = fmaf(1.0f, th, __fmul_rn(-alpha, mi));
    }
    g[i] = gi; m[i] = mi; theta[i] = th;
    if (shadow) shadow[i] = __float2bfloat16_rn(th);
  }
}

// ---------------------------------------------------------------- strided views
struct View {
  char* base;
  long long sn, sc, sy, sx;
};
static View view_of(const ad_tensor4* t) { return View{(char*)t->base, t->sn, t->sc, t->sy, t->sx}; }

// Linear index -> (n,c,y,x) in the order that makes the OUTPUT view's fastest axis the
// fastest thread index (channel-fastest if sc == 1, else x-fastest).
struct Dims { uint32_t N, C, H, W; int c_fastest; };
__device__ __forceinline__ void unpack(const Dims& d, size_t i, uint32_t& n, uint32_t& c, uint32_t& y, uint32_t& x) {
  if (d.c_fastest) {
    c = (uint32_t)(i % d.C); i /= d.C;
    x = (uint32_t)(i % d.W); i /= d.W;
    y = (uint32_t)(i % d.H); n = (uint32_t)(i / d.H);
  } else {
    x = (uint32_t)(i % d.W); i /= d.W;
    y = (uint32_t)(i % d.H); i /= d.H;
    c = (uint32_t)(i % d.C); n = (uint32_t)(i / d.C);
  }
}
__device__ __forceinline__ long long voff(const View& v, uint32_t n, uint32_t c, uint32_t y, uint32_t x) {
  return n * v.sn + c * v.sc + y * v.sy + x * v.sx;
}

enum EwOp { kRelu, kReluBwd, kAdd2, kConvert };

template <int OP, typename TA, typename TB, typename TY>
__global__ void __launch_bounds__(256) ew_kernel(Dims d, View a, View b, View yv, int accumulate) {
  grid_dependency();
  const size_t total = (size_t)d.N * d.C * d.H * d.W;
  const size_t nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t n, c, y, x;
    unpack(d, i, n, c, y, x);
    TY* yp = (TY*)yv.base + voff(yv, n, c, y, x);
    float av = ld_f((const TA*)a.base + voff(a, n, c, y, x));
    float r;
    if (OP == kRelu) r = fmaxf(av, 0.f);
    else if (OP == kConvert) r = av;
    else {
      float bv = ld_f((const TB*)b.base + voff(b, n, c, y, x));
      r = OP == kAdd2 ? av + bv : (av > 0.f ? bv : 0.f);
    }
    if (accumulate) r += ld_f(yp);
    st_f(yp, r);
  }
}


// bf16 channel-fastest views with 8-element-aligned strides: 8 channels (16 bytes) per thread.
__device__ __forceinline__ void ew_unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) { float2 t = __bfloat1622float2(h[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}
// Element offset of channel group cg of pixel i; evenly spaced pixels need no division.
__device__ __forceinline__ long long ew_pix_off(const View& v, uint32_t i, uint32_t H, uint32_t W) {
  if (v.sy == (long long)W * v.sx && v.sn == (long long)H * v.sy) return (long long)i * v.sx;
  const uint32_t r = i / W, x = i - r * W, n = r / H, y = r - n * H;
  return n * v.sn + y * v.sy + x * v.sx;
}
// G = C/8 channel groups; the launcher guarantees N*H*W*G < 2^31.  HBM-bound: kEwDepth loads per thread and operand in flight.
constexpr int kEwDepth = 8;
template <int OP>
__global__ void __launch_bounds__(256, 2) ew_vec_kernel(Dims d, View a, View b, View yv, int accumulate) {
  grid_dependency();
  constexpr bool kTwo = OP == kAdd2 || OP == kReluBwd;
  extern __shared__ __align__(128) uint4 ring_smem[];
  LoadRing<2 + kTwo, kEwDepth> ring(ring_smem);
  const uint32_t G = d.C / 8;
  const uint32_t total = d.N * d.H * d.W * G, nt = gridDim.x * blockDim.x;
  auto issue = [&](uint32_t i) {
    if (i < total) {
      const uint32_t pix = i / G, cg = i - pix * G;
      ring.copy(0, (const __nv_bfloat16*)a.base + ew_pix_off(a, pix, d.H, d.W) + cg * 8);
      if (accumulate) ring.copy(1, (const __nv_bfloat16*)yv.base + ew_pix_off(yv, pix, d.H, d.W) + cg * 8);
      if (kTwo) ring.copy(1 + kTwo, (const __nv_bfloat16*)b.base + ew_pix_off(b, pix, d.H, d.W) + cg * 8);
    }
    ring.commit();
  };
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
  for (int u = 0; u < kEwDepth - 1; ++u) issue(i + u * nt);
  for (; i < total; i += nt) {
    ring.wait();
    float av[8], bv[8], o[8], old[8];
    ew_unpack8(ring.get(0), av);
    if (kTwo) ew_unpack8(ring.get(1 + kTwo), bv);
    if (accumulate) ew_unpack8(ring.get(1), old);
    ring.next();
    issue(i + (kEwDepth - 1) * nt);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v;
      if (OP == kRelu) v = fmaxf(av[j], 0.f);
      else if (OP == kConvert) v = av[j];
      else if (OP == kAdd2) v = av[j] + bv[j];
      else v = av[j] > 0.f ? bv[j] : 0.f;
      o[j] = accumulate ? v + old[j] : v;
    }
    uint4 pk;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
    const uint32_t pix = i / G, cg = i - pix * G;
    *(uint4*)((__nv_bfloat16*)yv.base + ew_pix_off(yv, pix, d.H, d.W) + cg * 8) = pk;
  }
}
static bool ew_vec_ok(const ad_tensor4* t) {
  return t->dtype == AD_BF16 && t->sc == 1 && (t->C & 7u) == 0 && !((uintptr_t)t->base & 15u) && !(t->sn & 7) &&
         !(t->sy & 7) && !(t->sx & 7);
}

// fp32 planes -> bf16 pixels of C <= 4 channels (a host image on its way into a tensor-core net): four pixels per thread, 16-byte
// loads from each plane and C 8-byte stores where rows are aligned (VEC).  Element by element, each 2-byte store and 4-byte
// load on its own with three divisions, 2 x 3 x 1024 x 2048 took 67 us (12 us of memory).
template <int C, bool VEC>
__global__ void __launch_bounds__(256) planes_to_pixels_kernel(Dims d, View a, View yv) {
  grid_dependency();
  const uint32_t quads = (d.W + 3) / 4, total = d.N * d.H * quads;
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    const uint32_t q = i % quads, r = i / quads, y = r % d.H, n = r / d.H, x = q * 4;
    const float* src = (const float*)a.base + n * a.sn + y * a.sy + x;
    __nv_bfloat16* dst = (__nv_bfloat16*)yv.base + n * yv.sn + y * yv.sy + (long long)x * C;
    float v[C][4];
    if (VEC) {
#pragma unroll
      for (int c = 0; c < C; ++c) *(float4*)v[c] = *(const float4*)(src + c * a.sc);
      uint2 w[C];
      __nv_bfloat162* h = (__nv_bfloat162*)w;
#pragma unroll
      for (int k = 0; k < 2 * C; ++k) h[k] = __floats2bfloat162_rn(v[2 * k % C][2 * k / C], v[(2 * k + 1) % C][(2 * k + 1) / C]);
#pragma unroll
      for (int k = 0; k < C; ++k) ((uint2*)dst)[k] = w[k];
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < d.W)
#pragma unroll
          for (int c = 0; c < C; ++c) v[c][j] = src[c * a.sc + j];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < d.W)
#pragma unroll
          for (int c = 0; c < C; ++c) dst[j * C + c] = __float2bfloat16_rn(v[c][j]);
    }
  }
}
template <int C = 1>
static void launch_planes_to_pixels(const Dims& d, const View& a, const View& y, bool vec, cudaStream_t s) {
  if constexpr (C <= 4) {
    if (d.C != C) return launch_planes_to_pixels<C + 1>(d, a, y, vec, s);
    launch(vec ? planes_to_pixels_kernel<C, true> : planes_to_pixels_kernel<C, false>, grid_for((size_t)d.N * d.H * ((d.W + 3) / 4), 256, 8), 256, 0, s, d, a, y);
  }
}

static int same_dims(const ad_tensor4* a, const ad_tensor4* b) {
  return a->N == b->N && a->C == b->C && a->H == b->H && a->W == b->W;
}

template <int OP>
static int ew_launch(const ad_tensor4* a, const ad_tensor4* b, const ad_tensor4* y, int accumulate, void* stream) {
  if (!a || !y || !a->base || !y->base || (OP != kRelu && OP != kConvert && (!b || !b->base))) return AD_ERR_BAD_ARG;
  if (!same_dims(a, y) || (b && !same_dims(b, y))) return AD_ERR_BAD_ARG;
  const size_t total = (size_t)y->N * y->C * y->H * y->W;
  if (total == 0) return AD_OK;
  Dims d{y->N, y->C, y->H, y->W, y->sc == 1 && y->C > 1};
  View va = view_of(a), vb = b ? view_of(b) : View{nullptr, 0, 0, 0, 0}, vy = view_of(y);
  cudaStream_t s = as_stream(stream);
  if (total / 8 < (1ull << 31) && ew_vec_ok(a) && ew_vec_ok(y) && (!b || ew_vec_ok(b))) {
    constexpr int smem = LoadRing<2 + (OP == kAdd2 || OP == kReluBwd), kEwDepth>::kSmem;
    // the attribute is per function and per device; setting it is cheap enough to do per launch
    if (cudaFuncSetAttribute(ew_vec_kernel<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    launch(ew_vec_kernel<OP>, grid_for(total / 8, 256, 2), 256, smem, s, d, va, vb, vy, accumulate);
    count_launch();
    return launch_status();
  }
  if (OP == kConvert && !accumulate && a->dtype == AD_F32 && y->dtype == AD_BF16 && y->C <= 4 && a->sx == 1 && y->sc == 1 && y->sx == (int64_t)y->C &&
      (size_t)y->N * y->H * ((y->W + 3) / 4) < (1ull << 31)) {
    auto in4 = [](int64_t v) { return v % 4 == 0; };
    const bool vec = in4(y->W) && in4(a->sn) && in4(a->sc) && in4(a->sy) && in4(y->sn) && in4(y->sy) && !((uintptr_t)a->base & 15u) && !((uintptr_t)y->base & 7u);
    launch_planes_to_pixels(d, va, vy, vec, s);
    count_launch();
    return launch_status();
  }
  const unsigned grid = grid_for(total, 256, 16);
  const int da = a->dtype, db = b ? b->dtype : a->dtype, dy = y->dtype;
#define EW_CASE(TA_, TB_, TY_) launch(ew_kernel<OP, TA_, TB_, TY_>, grid, 256, 0, s, d, va, vb, vy, accumulate)
  using bf = __nv_bfloat16;
  if (da == AD_F32 && db == AD_F32 && dy == AD_F32) EW_CASE(float, float, float);
  else if (da == AD_BF16 && db == AD_BF16 && dy == AD_BF16) EW_CASE(bf, bf, bf);
  else if (da == AD_F32 && db == AD_F32 && dy == AD_BF16) EW_CASE(float, float, bf);
  else if (da == AD_BF16 && db == AD_BF16 && dy == AD_F32) EW_CASE(bf, bf, float);
  else return AD_ERR_UNSUPPORTED;
#undef EW_CASE
  count_launch();
  return launch_status();
}

}  // namespace adk

using namespace adk;

extern "C" const char* ad_status_string(int status) {
  switch (status) {
    case AD_OK: return "ok";
    case AD_ERR_BAD_ARG: return "bad argument";
    case AD_ERR_UNSUPPORTED: return "unsupported dtype/layout/shape";
    case AD_ERR_CUDA: return "CUDA launch error";
    case AD_ERR_TIMEOUT: return "bounded device wait timed out";
    case AD_ERR_ALIGN: return "misaligned pointer or pitch";
    case AD_ERR_SCRATCH: return "scratch buffer too small";
    case AD_ERR_LIMIT: return "size exceeds a limit built into the entry point";
    default: return "unknown status";
  }
}

extern "C" int32_t ad_conv2d_last_kernel(void) { return g_last_conv_kernel; }
extern "C" uint64_t ad_launch_count(void) { return __atomic_load_n(&g_launch_count, __ATOMIC_RELAXED); }

extern "C" int ad_array_set_constant(size_t n, float c, float* x, void* stream) {
  return arr_launch<kSet>(n, c, 0.f, nullptr, x, stream);
}
extern "C" int ad_array_add(size_t n, const float* x, float* y, void* stream) {
  return arr_launch<kAdd>(n, 0.f, 0.f, x, y, stream);
}
extern "C" int ad_array_add_scaled(size_t n, float alpha, float beta, const float* x, float* y, void* stream) {
  return arr_launch<kAddScaled>(n, alpha, beta, x, y, stream);
}
extern "C" int ad_array_add_online(size_t n, float alpha, const float* x, float* y, void* stream) {
  return arr_launch<kAddOnline>(n, alpha, 0.f, x, y, stream);
}
extern "C" int ad_array_scale(size_t n, float scale, const float* x, float* y, void* stream) {
  return arr_launch<kScale>(n, scale, 0.f, x, y, stream);
}
extern "C" int ad_array_scale_add(size_t n, float scale, const float* x, float* y, void* stream) {
  return arr_launch<kScaleAdd>(n, scale, 0.f, x, y, stream);
}

extern "C" int ad_fill_zero(void* x, size_t bytes, void* stream) {
  if (bytes == 0) return AD_OK;
  if (!x) return AD_ERR_BAD_ARG;
  // A memset node: runs on the copy/fill path at full HBM write bandwidth, no kernel needed.
  return cudaMemsetAsync(x, 0, bytes, as_stream(stream)) == cudaSuccess ? AD_OK : AD_ERR_CUDA;
}

extern "C" int ad_sgd_step(size_t n, float* theta, float* g, float* m, float l2, float mu, float alpha,
                           float alpha_next, int32_t nesterov, void* bf16_shadow, void* stream) {
  if (n == 0) return AD_OK;
  if (!theta || !g || !m) return AD_ERR_BAD_ARG;
  launch(sgd_kernel, grid_for(n, 256), 256, 0, as_stream(stream), n, theta, g, m, l2, mu, alpha, alpha_next, nesterov,
                                                               (__nv_bfloat16*)bf16_shadow, nullptr);
  count_launch();
  return launch_status();
}
extern "C" int ad_sgd_step_guarded(size_t n, float* theta, float* g, float* m, float l2, float mu, float alpha,
                                   float alpha_next, int32_t nesterov, void* bf16_shadow, const int32_t* status_word,
                                   void* stream) {
  if (n == 0) return AD_OK;
  if (!theta || !g || !m) return AD_ERR_BAD_ARG;
  launch(sgd_kernel, grid_for(n, 256), 256, 0, as_stream(stream), n, theta, g, m, l2, mu, alpha, alpha_next, nesterov,
                                                               (__nv_bfloat16*)bf16_shadow, status_word);
  count_launch();
  return launch_status();
}

extern "C" int ad_relu_fwd(const ad_tensor4* x, const ad_tensor4* y, void* stream) {
  return ew_launch<kRelu>(x, nullptr, y, 0, stream);
}
extern "C" int ad_relu_bwd(const ad_tensor4* x, const ad_tensor4* dy, const ad_tensor4* dx, int32_t accumulate,
                           void* stream) {
  return ew_launch<kReluBwd>(x, dy, dx, accumulate, stream);
}
extern "C" int ad_add(const ad_tensor4* a, const ad_tensor4* b, const ad_tensor4* y, void* stream) {
  return ew_launch<kAdd2>(a, b, y, 0, stream);
}
extern "C" int ad_convert(const ad_tensor4* src, const ad_tensor4* dst, int32_t accumulate, void* stream) {
  return ew_launch<kConvert>(src, nullptr, dst, accumulate, stream);
}

// ---------------------------------------------------------------- patch matrix for C_in < 8 layers
namespace adk {
template <typename T>
__global__ void __launch_bounds__(256) im2col_kernel(View x, uint32_t N, uint32_t C, uint32_t H, uint32_t W, uint32_t kh,
                                                     uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw,
                                                     uint32_t P, uint32_t Q, __nv_bfloat16* out, uint32_t ldo) {
  grid_dependency();
  const uint32_t cols = kh * kw * C;
  const size_t total = (size_t)N * P * Q * cols, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    const uint32_t col = (uint32_t)(i % cols);
    const size_t pix = i / cols;
    const uint32_t c = col % C, tap = col / C, s = tap % kw, r = tap / kw;
    const uint32_t q = (uint32_t)(pix % Q);
    const size_t rest = pix / Q;
    const uint32_t p = (uint32_t)(rest % P), n = (uint32_t)(rest / P);
    const uint32_t yy = p * sh + r * dh, xx = q * sw + s * dw;
    float v = 0.f;
    if (yy < H && xx < W) v = ld_f((const T*)x.base + voff(x, n, c, yy, xx));
    out[pix * ldo + col] = __float2bfloat16_rn(v);
  }
}
// Same matrix, 8 output columns (one 16-byte store) per thread; columns past kh*kw*C are written as zeros.
template <typename T>
__global__ void __launch_bounds__(256) im2col_vec_kernel(View x, uint32_t N, uint32_t C, uint32_t H, uint32_t W, uint32_t kh,
                                                         uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw,
                                                         uint32_t P, uint32_t Q, __nv_bfloat16* out, uint32_t ldo) {
  grid_dependency();
  const uint32_t cols = kh * kw * C, groups = ldo / 8;
  const size_t total = (size_t)N * P * Q * groups, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    const uint32_t gcol = (uint32_t)(i % groups) * 8;
    const size_t pix = i / groups;
    const uint32_t q = (uint32_t)(pix % Q);
    const size_t rest = pix / Q;
    const uint32_t p = (uint32_t)(rest % P), n = (uint32_t)(rest / P);
    uint32_t c = gcol % C, tap = gcol / C;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = 0.f;
      if (gcol + j < cols) {
        const uint32_t s = tap % kw, r = tap / kw;
        const uint32_t yy = p * sh + r * dh, xx = q * sw + s * dw;
        if (yy < H && xx < W) v[j] = ld_f((const T*)x.base + voff(x, n, c, yy, xx));
      }
      if (++c == C) { c = 0; ++tap; }
    }
    uint4 pk;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *(uint4*)(out + pix * ldo + gcol) = pk;
  }
}
// Same matrix built one output row per block: the kh input rows the row's patches touch are staged in
// shared memory as bf16 (zeros past the tensor's edge), a table maps each column to its offset inside the
// staged rows, and every thread then assembles 16-byte pieces of the output from shared memory.  Each input
// element is fetched from global memory once per output row instead of once per patch that holds it.
template <typename T, bool EVEN>
__global__ void __launch_bounds__(512) im2col_row_kernel(View x, uint32_t C, uint32_t H, uint32_t W, uint32_t kh, uint32_t kw,
                                                         uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw, uint32_t P,
                                                         uint32_t Q, __nv_bfloat16* out, uint32_t ldo, uint32_t rowlen, uint32_t qseg) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char im2col_smem[];
  __nv_bfloat16* rows = (__nv_bfloat16*)im2col_smem;                                    // [kh][rowlen]
  const uint32_t segs = (Q + qseg - 1) / qseg, q0 = blockIdx.x % segs * qseg, row = blockIdx.x / segs;
  const uint32_t p = row % P, n = row / P, cols = kh * kw * C, nq = Q - q0 < qseg ? Q - q0 : qseg;
  const bool packed = x.sc == 1 && x.sx == (long long)C;
  const T* src = (const T*)x.base + n * x.sn + (long long)p * sh * x.sy + (long long)q0 * sw * x.sx;
  const uint32_t left = q0 * sw < W ? W - q0 * sw : 0u;   // input columns from the segment's first on
  const uint32_t have = packed ? (left * C < rowlen ? left * C : rowlen) : 0u;
  // eight rows at a time, so that a thread's loads are in flight together
  for (uint32_t r0 = 0; r0 < kh; r0 += 8)
    for (uint32_t e = threadIdx.x; e < rowlen; e += blockDim.x) {
      float v[8];
      const uint32_t xx = packed ? 0u : e / C, c = packed ? e : e - xx * C;
      const T* at = src + (long long)(r0 * dh) * x.sy + (packed ? (long long)e : xx * x.sx + c * x.sc);
      const bool ok = packed ? e < have : xx < left;
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r) {
        v[r] = ok && r0 + r < kh && p * sh + (r0 + r) * dh < H ? ld_f(at) : 0.f;
        at += (long long)dh * x.sy;
      }
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r)
        if (r0 + r < kh) rows[(r0 + r) * rowlen + e] = __float2bfloat16_rn(v[r]);
    }
  __syncthreads();
  // A thread stays with a pair of columns and walks the pixels, so where the pair lies in the rows is in registers; a warp
  // writes 128 contiguous bytes from 32 adjacent words of shared memory.  EVEN: the first of a pair is always at an even
  // element, so that one 32-bit load brings both unless they are in different rows.  Bound by the stores:
  // 7x7 x 3 stem, 1,048,576 pixels x 192: 147 us; with 8 columns per thread, a table of offsets in shared memory and a whole
  // output row per block 183.
  const uint32_t pairs = ldo / 2, pb = pairs < blockDim.x ? pairs : blockDim.x, lanes = blockDim.x / pb, step = sw * C;
  uint32_t* orow = (uint32_t*)(out + (((size_t)n * P + p) * Q + q0) * ldo);
  const unsigned short* rs = (const unsigned short*)rows;
  if (threadIdx.x >= pb * lanes) return;
  for (uint32_t pr = threadIdx.x % pb; pr < pairs; pr += pb) {
    uint32_t e[2], mask = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t t = pr * 2 + h, c = t % C, tap = t / C, s = tap % kw, r = tap / kw;
      e[h] = t < cols ? r * rowlen + s * dw * C + c : 0u;
      if (t < cols) mask |= 0xffffu << (16 * h);
    }
    const bool split = !EVEN || (mask == 0xffffffffu && e[1] != e[0] + 1);
#pragma unroll 4
    for (uint32_t q = threadIdx.x / pb; q < nq; q += lanes) {
      uint32_t w = EVEN ? *(const uint32_t*)(rs + e[0] + q * step) : rs[e[0] + q * step];
      if (split) w = (w & 0xffffu) | ((uint32_t)rs[e[1] + q * step] << 16);
      orow[(size_t)q * pairs + pr] = w & mask;
    }
  }
}
// Rows of packed bf16 pixels behind a 16-byte aligned base (the input of a tensor-core net), as a pipeline: a block works through
// segments of one output row; while it assembles one (two words and a permutation of bytes for a pair of columns), the input rows of the next come by 16-byte asynchronous copies
// (from the aligned element in front of the segment on, so that each row has a phase of its own), and the part of the matrix
// that it assembled before, one run of memory, leaves by a bulk copy.  Bound by instructions: a block per segment with a branch
// for the pairs that lie in two rows (im2col_row_kernel) spent 47 per word and warp on a 7x7 x 3 stem of 1,048,576 pixels x
// 192, 141 us; 90 now (57 at the rate of a fill).  Segments of 64 pixels with two tiles took 104: what is worked out once per
// segment counts.
__global__ void __launch_bounds__(384) im2col_pipe_kernel(View x, uint32_t C, uint32_t H, uint32_t W, uint32_t kh, uint32_t kw, uint32_t sh,
                                                          uint32_t sw, uint32_t dh, uint32_t dw, uint32_t P, uint32_t Q, __nv_bfloat16* out,
                                                          uint32_t ldo, uint32_t rowlen, uint32_t qseg, uint32_t total) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char im2col_smem[];
  const uint32_t pairs = ldo / 2, rows_bytes = kh * rowlen * 2 + 16, segs = (Q + qseg - 1) / qseg, cols = kh * kw * C, step = sw * C;
  unsigned char* const tiles = im2col_smem + 2 * rows_bytes;
  // a segment's place, moved on by the grid's size without divisions
  struct Place { uint32_t q, p, n; };              // segment of the row, row, image
  const uint32_t hop_q = gridDim.x % segs, hop_p = gridDim.x / segs % P, hop_n = gridDim.x / segs / P;
  auto advance = [&](Place t) {
    t.q += hop_q; t.p += hop_p; t.n += hop_n;
    if (t.q >= segs) { t.q -= segs; ++t.p; }
    if (t.p >= P) { t.p -= P; ++t.n; }
    return t;
  };
  auto first_of = [&](const Place& t) { return t.n * x.sn + (long long)(t.p * sh) * x.sy + (long long)(t.q * qseg * sw) * x.sx; };   // element
  const uint32_t per_row = rowlen / 8, r0 = threadIdx.x / per_row, k0 = threadIdx.x - r0 * per_row;
  auto fetch = [&](const Place& t, bool any, uint32_t buf) {
    if (any) {
      const uint32_t x0 = t.q * qseg * sw, left = x0 < W ? (W - x0) * C : 0u, have = left < rowlen ? left : rowlen;   // none: a segment past the last column
      const long long base = first_of(t);
      __nv_bfloat16* rows = (__nv_bfloat16*)(im2col_smem + buf * rows_bytes);
      for (uint32_t i = threadIdx.x, r = r0, k = k0; i < kh * per_row; i += blockDim.x, r = i / per_row, k = i - r * per_row) {
        const long long first = base + (long long)(r * dh) * x.sy;
        const uint32_t phase = (uint32_t)first & 7u, end = t.p * sh + r * dh < H ? phase + have : 0u;   // elements of the copy that exist
        const __nv_bfloat16* from = (const __nv_bfloat16*)x.base + (first - phase) + k * 8;
        __nv_bfloat16* to = rows + r * rowlen + k * 8;
        if (k * 8 + 8 <= end)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
        else
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) to[j] = k * 8 + j >= phase && k * 8 + j < end ? from[j] : __float2bfloat16_rn(0.f);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // a thread's pair of columns: which rows and elements of a row of taps it lies in
  const uint32_t lanes = blockDim.x / pairs, pr = threadIdx.x % pairs;
  uint32_t row[2], off[2], mask = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t t = pr * 2 + h, c = t % C, tap = t / C, s = tap % kw, r = tap / kw;
    row[h] = t < cols ? r : 0u;
    off[h] = t < cols ? s * dw * C + c : 0u;
    if (t < cols) mask |= 0xffffu << (16 * h);
  }
  Place now{blockIdx.x % segs, blockIdx.x / segs % P, blockIdx.x / segs / P}, next;
  fetch(now, blockIdx.x < total, 0);
  uint32_t buf = 0;
  for (uint32_t seg = blockIdx.x; seg < total; seg += gridDim.x, buf ^= 1u, now = next) {
    next = advance(now);
    fetch(next, seg + gridDim.x < total, buf ^ 1u);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the tile before has left
    __syncthreads();
    const uint32_t q0 = now.q * qseg, nq = Q - q0 < qseg ? Q - q0 : qseg;
    const long long base = first_of(now);
    uint32_t* const tile = (uint32_t*)tiles;
    const unsigned char* rows = im2col_smem + buf * rows_bytes;
    if (threadIdx.x < pairs * lanes) {
      uint32_t e[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) e[h] = row[h] * rowlen + off[h] + ((uint32_t)(base + (long long)(row[h] * dh) * x.sy) & 7u);
      // the halves of two words (of one, or neighbours, or in two rows); the step from pixel to pixel is even, so which halves stays
      const uint32_t sel = (e[0] & 1u ? 0x32u : 0x10u) | (e[1] & 1u ? 0x7600u : 0x5400u), q1 = threadIdx.x / pairs, hop = lanes * (step / 2);
      const uint32_t *a = (const uint32_t*)rows + e[0] / 2 + q1 * (step / 2), *b = (const uint32_t*)rows + e[1] / 2 + q1 * (step / 2);
      uint32_t* o = tile + q1 * pairs + pr;
#pragma unroll 4
      for (uint32_t q = q1; q < nq; q += lanes, a += hop, b += hop, o += lanes * pairs) *o = __byte_perm(*a, *b, sel) & mask;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(out + (((size_t)now.n * P + now.p) * Q + q0) * ldo),
                   "r"((uint32_t)__cvta_generic_to_shared(tile)), "r"(nq * pairs * 4) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// The limit belongs to the function, so every call sets the most that its path takes: of two threads with calls of different
// sizes, one would lower it between the other's setting and its launch.
constexpr size_t kIm2colPipeMost = 96 * 1024, kIm2colRowMost = 100 * 1024;
template <typename K>
static bool im2col_limit(K kernel, size_t most) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}
template <typename T>
static int launch_im2col_row(const View& v, const ad_tensor4* x, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh,
                             uint32_t dw, uint32_t P, uint32_t Q, __nv_bfloat16* out, uint32_t ldo, uint32_t rowlen, uint32_t qseg, size_t smem,
                             cudaStream_t s) {
  const bool even = dw == 1 && ((sw * x->C) & 1u) == 0;   // and the row pitch has the parity of a row of taps
  auto kern = even ? im2col_row_kernel<T, true> : im2col_row_kernel<T, false>;
  const uint32_t pairs = ldo / 2, threads = pairs > 256 ? 256 : 384 / pairs * pairs > 384 ? 384 : (384 / pairs * pairs + 31) / 32 * 32;
  if (smem > 48 * 1024 && !im2col_limit(kern, kIm2colRowMost)) return AD_ERR_CUDA;
  launch(kern, x->N * P * ((Q + qseg - 1) / qseg), threads, smem, s, v, x->C, x->H, x->W, kh, kw, sh, sw, dh, dw, P, Q, out, ldo, rowlen, qseg);
  return AD_OK;
}
}  // namespace adk

extern "C" int ad_im2col(const ad_tensor4* x, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw,
                         uint32_t P, uint32_t Q, void* out_bf16, uint32_t ldo, void* stream) {
  if (!x || !x->base || !out_bf16 || kh == 0 || kw == 0 || sh == 0 || sw == 0 || dh == 0 || dw == 0) return AD_ERR_BAD_ARG;
  if (ldo < kh * kw * x->C) return AD_ERR_BAD_ARG;
  const size_t total = (size_t)x->N * P * Q * kh * kw * x->C;
  if (total == 0) return AD_OK;
  adk::View v = adk::view_of(x);
  if ((ldo & 7u) == 0 && ((uintptr_t)out_bf16 & 15u) == 0) {
    // staged-row form when the rows of one output row fit shared memory
    // of the parity of a row of taps, so that (dilation 1) a pair of columns starts at an even element in every row
    const uint32_t pairs = ldo / 2, reach = (kw - 1) * dw + 1;
    if (x->dtype == AD_BF16 && x->sc == 1 && x->sx == (int64_t)x->C && !((uintptr_t)x->base & 15u) && x->sn >= 0 && x->sy >= 0 && pairs <= 384 &&
        (sw * x->C) % 2 == 0) {
      // two stages of input rows and a tile of 48 KB at most; as many blocks per SM as fit, four at most
      const uint32_t qs = std::max(1u, std::min(Q, 24576u / ldo)), len = (((qs - 1) * sw + reach) * x->C + 14) / 8 * 8;
      const size_t need = 2 * ((size_t)kh * len * 2 + 16) + (size_t)qs * ldo * 2, segs = (size_t)x->N * P * ((Q + qs - 1) / qs);
      if (need <= adk::kIm2colPipeMost && segs < (1ull << 31)) {
        if (need > 48 * 1024 && !adk::im2col_limit(adk::im2col_pipe_kernel, adk::kIm2colPipeMost)) return AD_ERR_CUDA;
        const uint32_t per_sm = std::min(4u, (uint32_t)(220 * 1024 / (need + 1024)));
        launch(adk::im2col_pipe_kernel, (unsigned)std::min<size_t>(segs, adk::kNumSMs * per_sm), 384 / pairs * pairs > 32 ? (384 / pairs * pairs + 31) / 32 * 32 : 32,
               need, adk::as_stream(stream), v, x->C, x->H, x->W, kh, kw, sh, sw, dh, dw, P, Q, (__nv_bfloat16*)out_bf16, ldo, len, qs, (uint32_t)segs);
        adk::count_launch();
        return adk::launch_status();
      }
    }
    const uint32_t qseg = Q < 128 ? Q : 128;   // output pixels per block: enough blocks per SM to keep the stores going
    uint32_t rowlen = ((qseg - 1) * sw + (kw - 1) * dw + 1) * x->C;
    rowlen += (rowlen ^ (kw * x->C)) & 1u;
    const size_t smem = (((size_t)kh * rowlen * 2 + 15) & ~(size_t)15) + 16;   // a masked pair may read past the last element
    if (smem <= adk::kIm2colRowMost && (size_t)x->N * P * Q < (1ull << 31) && (size_t)Q * (ldo / 8) < (1ull << 31)) {
      int st = AD_OK;
      AD_DISPATCH_DTYPE(x->dtype, (st = adk::launch_im2col_row<T>(v, x, kh, kw, sh, sw, dh, dw, P, Q, (__nv_bfloat16*)out_bf16, ldo,
                                                                  rowlen, qseg, smem, adk::as_stream(stream))));
      if (st != AD_OK) return st;
      adk::count_launch();
      return adk::launch_status();
    }
    const size_t tv = (size_t)x->N * P * Q * (ldo / 8);
    AD_DISPATCH_DTYPE(x->dtype, (launch(adk::im2col_vec_kernel<T>, adk::grid_for(tv, 256, 16), 256, 0, adk::as_stream(stream), v, x->N, x->C, x->H, x->W, kh, kw, sh, sw, dh, dw, P, Q, (__nv_bfloat16*)out_bf16, ldo)));
    adk::count_launch();
    return adk::launch_status();
  }
  AD_DISPATCH_DTYPE(x->dtype, (launch(adk::im2col_kernel<T>, adk::grid_for(total, 256, 16), 256, 0, adk::as_stream(stream), v, x->N, x->C, x->H, x->W, kh, kw, sh, sw, dh, dw, P, Q, (__nv_bfloat16*)out_bf16, ldo)));
  adk::count_launch();
  return adk::launch_status();
}
