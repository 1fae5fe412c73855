// fp32 NCHW convolution with fp32 FMA accumulate: the exact-precision path (max-relative 1e-5 against a
// double-accumulating CPU result).  The tiled kernels of conv_f32.cu serve every geometry within their limits
// (f32_gemm_ok: 32-bit offsets, at most 64 taps) but the smallest calls (direct_wins); the one-thread-per-output kernels
// here take those and what is left.
#include <cstdlib>

#include "common.cuh"

namespace adk {

struct ConvG {
  uint32_t N, C, H, W, K, kh, kw, sh, sw, dh, dw, ph, pw, P, Q;
  long long y_pitch, y_plane;
  int relu, accumulate;
};

__global__ void __launch_bounds__(256) conv_fprop_f32(ConvG g, const float* __restrict__ x, const float* __restrict__ w,
                                                      const float* __restrict__ bias, float* y) {
  const size_t total = (size_t)g.N * g.K * g.P * g.Q, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += nt) {
    uint32_t s = (uint32_t)(idx % g.Q);
    size_t r = idx / g.Q;
    uint32_t q = (uint32_t)(r % g.P); r /= g.P;
    uint32_t k = (uint32_t)(r % g.K), n = (uint32_t)(r / g.K);
    float acc = bias ? bias[k] : 0.f;
    for (uint32_t c = 0; c < g.C; ++c) {
      float part = 0.f;  // per-channel partial keeps the running sum short
      const float* xp = x + ((size_t)n * g.C + c) * g.H * g.W;
      const float* wp = w + ((size_t)k * g.C + c) * g.kh * g.kw;
      for (uint32_t i = 0; i < g.kh; ++i) {
        int yy = (int)(q * g.sh + i * g.dh) - (int)g.ph;
        if (yy < 0 || yy >= (int)g.H) continue;
        for (uint32_t j = 0; j < g.kw; ++j) {
          int xx = (int)(s * g.sw + j * g.dw) - (int)g.pw;
          if (xx < 0 || xx >= (int)g.W) continue;
          part = fmaf(xp[(size_t)yy * g.W + xx], wp[i * g.kw + j], part);
        }
      }
      acc += part;
    }
    if (g.relu) acc = fmaxf(acc, 0.f);
    y[((size_t)n * g.K + k) * g.y_plane + (size_t)q * g.y_pitch + s] = acc;
  }
}

__global__ void __launch_bounds__(256) conv_dgrad_f32(ConvG g, const float* __restrict__ dy, const float* __restrict__ w,
                                                      float* dx) {
  const size_t total = (size_t)g.N * g.C * g.H * g.W, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += nt) {
    uint32_t xx = (uint32_t)(idx % g.W);
    size_t r = idx / g.W;
    uint32_t yy = (uint32_t)(r % g.H); r /= g.H;
    uint32_t c = (uint32_t)(r % g.C), n = (uint32_t)(r / g.C);
    float acc = 0.f;
    for (uint32_t i = 0; i < g.kh; ++i) {
      int t = (int)(yy + g.ph) - (int)(i * g.dh);
      if (t < 0 || t % (int)g.sh) continue;
      uint32_t q = (uint32_t)t / g.sh;
      if (q >= g.P) continue;
      for (uint32_t j = 0; j < g.kw; ++j) {
        int u = (int)(xx + g.pw) - (int)(j * g.dw);
        if (u < 0 || u % (int)g.sw) continue;
        uint32_t s = (uint32_t)u / g.sw;
        if (s >= g.Q) continue;
        float part = 0.f;
        for (uint32_t k = 0; k < g.K; ++k)
          part = fmaf(dy[((size_t)n * g.K + k) * g.y_plane + (size_t)q * g.y_pitch + s],
                      w[(((size_t)k * g.C + c) * g.kh + i) * g.kw + j], part);
        acc += part;
      }
    }
    if (g.accumulate) acc += dx[idx];
    dx[idx] = acc;
  }
}

// One block per (k, c): every thread sums a strided share of the (n, q, s) positions for all
// kh*kw taps (at most 49 here), then a fixed-order tree reduction.
template <int MAXT>
__global__ void __launch_bounds__(256) conv_wgrad_f32(ConvG g, const float* __restrict__ x, const float* __restrict__ dy,
                                                      float* dw) {
  const uint32_t k = blockIdx.x / g.C, c = blockIdx.x % g.C;
  const uint32_t taps = g.kh * g.kw;
  float acc[MAXT];
#pragma unroll
  for (int t = 0; t < MAXT; ++t) acc[t] = 0.f;
  const size_t per = (size_t)g.N * g.P * g.Q;
  for (size_t idx = threadIdx.x; idx < per; idx += blockDim.x) {
    uint32_t s = (uint32_t)(idx % g.Q);
    size_t r = idx / g.Q;
    uint32_t q = (uint32_t)(r % g.P), n = (uint32_t)(r / g.P);
    const float d = dy[((size_t)n * g.K + k) * g.y_plane + (size_t)q * g.y_pitch + s];
    const float* xp = x + ((size_t)n * g.C + c) * g.H * g.W;
#pragma unroll
    for (int t = 0; t < MAXT; ++t) {
      if (t < (int)taps) {
        uint32_t i = t / g.kw, j = t % g.kw;
        int yy = (int)(q * g.sh + i * g.dh) - (int)g.ph, xx = (int)(s * g.sw + j * g.dw) - (int)g.pw;
        if (yy >= 0 && yy < (int)g.H && xx >= 0 && xx < (int)g.W) acc[t] = fmaf(d, xp[(size_t)yy * g.W + xx], acc[t]);
      }
    }
  }
  __shared__ float red[8];
#pragma unroll
  for (int t = 0; t < MAXT; ++t) {
    if (t < (int)taps) {
      float v = warp_sum(acc[t]);
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
      __syncthreads();
      if (threadIdx.x == 0) {
        float tot = 0.f;
        for (int wv = 0; wv < 8; ++wv) tot += red[wv];
        float* o = dw + ((size_t)k * g.C + c) * taps + t;
        *o = g.accumulate ? *o + tot : tot;
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(256) conv_bgrad_f32(ConvG g, const float* __restrict__ dy, float* db) {
  const uint32_t k = blockIdx.x;
  float acc = 0.f;
  const size_t per = (size_t)g.N * g.P * g.Q;
  for (size_t idx = threadIdx.x; idx < per; idx += blockDim.x) {
    uint32_t s = (uint32_t)(idx % g.Q);
    size_t r = idx / g.Q;
    uint32_t q = (uint32_t)(r % g.P), n = (uint32_t)(r / g.P);
    acc += dy[((size_t)n * g.K + k) * g.y_plane + (size_t)q * g.y_pitch + s];
  }
  __shared__ float red[8];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int wv = 0; wv < 8; ++wv) tot += red[wv];
    db[k] = g.accumulate ? db[k] + tot : tot;
  }
}

static int geometry(const ad_conv2d_args* a, ConvG& g) {
  if (!a) return AD_ERR_BAD_ARG;
  if (a->N == 0 || a->C == 0 || a->H == 0 || a->W == 0 || a->K == 0 || a->kh == 0 || a->kw == 0) return AD_ERR_BAD_ARG;
  if (a->stride_h == 0 || a->stride_w == 0 || a->dil_h == 0 || a->dil_w == 0) return AD_ERR_BAD_ARG;
  const long long eh = (long long)a->H + 2ll * a->pad_h - (long long)a->dil_h * (a->kh - 1) - 1;
  const long long ew = (long long)a->W + 2ll * a->pad_w - (long long)a->dil_w * (a->kw - 1) - 1;
  if (eh < 0 || ew < 0) return AD_ERR_BAD_ARG;
  g = ConvG{a->N, a->C, a->H, a->W, a->K, a->kh, a->kw, a->stride_h, a->stride_w, a->dil_h, a->dil_w, a->pad_h, a->pad_w,
            (uint32_t)(eh / a->stride_h + 1), (uint32_t)(ew / a->stride_w + 1), 0, 0, a->relu, a->accumulate};
  g.y_pitch = a->y_pitch ? a->y_pitch : g.Q;
  g.y_plane = a->y_plane ? a->y_plane : (long long)g.P * g.Q;
  return AD_OK;
}

bool f32_gemm_ok(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane);
int f32_gemm_fprop(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s);
int f32_gemm_dgrad(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s);
int f32_gemm_wgrad(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s);
size_t f32_wgrad_scratch(const ad_conv2d_args* a, uint32_t P, uint32_t Q);
size_t f32_dgrad_scratch(const ad_conv2d_args* a, uint32_t P, uint32_t Q);

// A tiled kernel takes 16 - 27 us (a filter gradient 25 - 45) however little there is to do: tables, the fill of its ring,
// the sums over the cluster.  A thread per output is bound by its chain of loads (0.36 us per term of a 1x1 filter, whose
// terms are planes apart, 0.14 of a larger one, 0.06 per term of a data gradient), by the number of terms in all, and as a
// filter gradient by the rounds of 256 pixels of a block.  These times come within a quarter of 60 measured layers of up to
// 25 M multiplications; of those the smallest ran three times faster this way.  (The 3x3 kernels of conv_f32_k3.cu would take
// 10 - 19 us for the smallest calls too; but these sums of 9 terms and of channels are the more precise ones, 0.75e-7 against
// 0.85 - 1.2e-7, and the calls stay here.)
static bool direct_wins(const ConvG& g, int pass) {
  if (const char* t = getenv("ARRAYDIFF_B200_F32_TILES")) return t[0] == '0';   // the parity tests: "1" tiled, "2" 3x3 kernels first (conv_f32.cu), "0" direct
  const double taps = (double)g.kh * g.kw, px = (double)g.N * g.P * g.Q, mmac = px * g.K * g.C * taps * 1e-6;
  const bool one = g.kh * g.kw == 1;
  auto most = [](double x, double y) { return x > y ? x : y; };
  if (pass == 0) return 4 + (one ? 0.36 : 0.14) * most(g.C * taps, 9 * mmac) < 25;
  if (pass == 1) return 4 + most(0.06 * g.K * taps, 2 * mmac * g.sh * g.sw) < 25;
  return taps <= 49 && 6 + most(px / 256 * (one ? 0.9 : 0.25 * taps), mmac * (one ? 7.8 : 2.6)) < 40;
}

int conv_direct_fprop(const ad_conv2d_args* a, cudaStream_t s) {
  ConvG g;
  int st = geometry(a, g);
  if (st != AD_OK) return st;
  if (!a->x || !a->w || !a->y) return AD_ERR_BAD_ARG;
  if (a->out_row_count) return AD_ERR_UNSUPPORTED;   // row ranges: tensor-core path only
  if (!direct_wins(g, 0) && f32_gemm_ok(a, g.P, g.Q, g.y_pitch, g.y_plane)) return f32_gemm_fprop(a, g.P, g.Q, g.y_pitch, g.y_plane, s);
  const size_t total = (size_t)g.N * g.K * g.P * g.Q;
  conv_fprop_f32<<<grid_for(total, 256, 16), 256, 0, s>>>(g, (const float*)a->x, (const float*)a->w, a->bias, (float*)a->y);
  count_launch();
  return launch_status();
}

int conv_direct_dgrad(const ad_conv2d_args* a, cudaStream_t s) {
  ConvG g;
  int st = geometry(a, g);
  if (st != AD_OK) return st;
  if (!a->y || !a->w || !a->dx) return AD_ERR_BAD_ARG;
  if (a->dx_col_count) return AD_ERR_UNSUPPORTED;   // column ranges: tensor-core path only
  if (!direct_wins(g, 1) && f32_gemm_ok(a, g.P, g.Q, g.y_pitch, g.y_plane)) return f32_gemm_dgrad(a, g.P, g.Q, g.y_pitch, g.y_plane, s);
  const size_t total = (size_t)g.N * g.C * g.H * g.W;
  conv_dgrad_f32<<<grid_for(total, 256, 16), 256, 0, s>>>(g, (const float*)a->y, (const float*)a->w, (float*)a->dx);
  count_launch();
  return launch_status();
}

// Scratch with which a filter gradient of few outputs and many pixels is split further, or a data gradient into few
// channels takes its two-step form (optional: less or none is fine)
size_t conv_direct_scratch_bytes(const ad_conv2d_args* a, int pass) {
  ConvG g;
  if (geometry(a, g) != AD_OK || direct_wins(g, pass) || !f32_gemm_ok(a, g.P, g.Q, g.y_pitch, g.y_plane)) return 0;
  if (pass == 1) return f32_dgrad_scratch(a, g.P, g.Q);
  if (pass != 2 || g.kh * g.kw > 49) return 0;
  return f32_wgrad_scratch(a, g.P, g.Q);
}

int conv_direct_wgrad(const ad_conv2d_args* a, cudaStream_t s) {
  ConvG g;
  int st = geometry(a, g);
  if (st != AD_OK) return st;
  if (!a->x || !a->y || !a->dw) return AD_ERR_BAD_ARG;
  const uint32_t taps = g.kh * g.kw;
  if (taps <= 49 && !direct_wins(g, 2) && f32_gemm_ok(a, g.P, g.Q, g.y_pitch, g.y_plane)) return f32_gemm_wgrad(a, g.P, g.Q, g.y_pitch, g.y_plane, s);
  if (taps <= 9) conv_wgrad_f32<9><<<g.K * g.C, 256, 0, s>>>(g, (const float*)a->x, (const float*)a->y, (float*)a->dw);
  else if (taps <= 49) conv_wgrad_f32<49><<<g.K * g.C, 256, 0, s>>>(g, (const float*)a->x, (const float*)a->y, (float*)a->dw);
  else return AD_ERR_UNSUPPORTED;
  count_launch();
  if (a->db) {
    conv_bgrad_f32<<<g.K, 256, 0, s>>>(g, (const float*)a->y, a->db);
    count_launch();
  }
  return launch_status();
}

}  // namespace adk
