// Spatial batch normalisation (training statistics, optional fused ReLU) and max pooling
// on strided 4-D views.  HBM-bound.
//
// Statistics are a two-stage, order-fixed reduction: stage 1 writes per-split partial sums
// to caller scratch, stage 2 combines them in double.  No atomics, so results are
// reproducible run to run.  Threads walk the tensor along its fastest axis (x for
// NCHW-like views, channel for NHWC-like views) so that warps read whole sectors.
#include <algorithm>
#include <atomic>

#include "common.cuh"

namespace adk {

constexpr int kBnMaxSplits = 128;
// Partial-sum rows a reduction may use for C channels: as many as fit the scratch of the widest layer
// ((128 + 1) rows of 2 * 2048 floats) beside the two trailing rows (combined sums, their means), at
// most 1024 -- narrow layers get more blocks in flight.
__host__ __device__ inline int bn_max_splits(uint32_t C) {
  long long s = (long long)(kBnMaxSplits + 1) * 2 * 2048 / (2ll * (C ? C : 1)) - 2;
  return (int)(s > 1024 ? 1024 : (s < 1 ? 1 : s));
}

struct BView { const char* base; long long sn, sc, sy, sx; };
static BView bview(const ad_tensor4* t) { return BView{(const char*)t->base, t->sn, t->sc, t->sy, t->sx}; }

// partial[split][0..C) = sum a, partial[split][C..2C) = sum b, where (a, b) is
//   MODE 0: (x, x^2)                      -- forward statistics
//   MODE 1: (g, g * xhat), g = dy masked   -- backward reductions
struct BnRed {
  BView x, dy;
  uint32_t N, C, H, W;
  int relu;
  const float *gamma, *beta, *mean, *invstd;
  int dual;               // forward sums of an x-fastest view: in double too
};

template <typename T, int MODE>
__device__ __forceinline__ float bn_term(const BnRed& p, uint32_t n, uint32_t c, uint32_t y, uint32_t x, float& a, float& b) {
  const long long ox = n * p.x.sn + c * p.x.sc + y * p.x.sy + x * p.x.sx;
  const float xv = ld_f((const T*)p.x.base + ox);
  if (MODE == 0) {
    a += xv;
    b = fmaf(xv, xv, b);
  } else {
    const long long od = n * p.dy.sn + c * p.dy.sc + y * p.dy.sy + x * p.dy.sx;
    float g = ld_f((const T*)p.dy.base + od);
    const float xhat = (xv - p.mean[c]) * p.invstd[c];
    if (p.relu && fmaf(p.gamma[c], xhat, p.beta[c]) <= 0.f) g = 0.f;
    a += g;
    b = fmaf(g, xhat, b);
  }
  return xv;
}
// Views whose planes are runs of floats that 16-byte loads reach
static bool planes_vec_ok(const ad_tensor4* t) {
  return t->dtype == AD_F32 && t->sx == 1 && t->sy == (int64_t)t->W && !((uintptr_t)t->base & 15u) && !(t->sn & 3) && !(t->sc & 3) &&
         ((unsigned long long)t->H * t->W) % 4 == 0 && (unsigned long long)t->H * t->W < (1ull << 31);
}

// NCHW-like: block (256) per (channel, split); threads stride over (n, y, x); the backward sums take 4 pixels at a time where the
// planes of x and dy allow it (VEC), the forward ones always one.
// The forward statistics are summed in fp32, one pixel after the other, and beside that in double, which a split writes as two
// more rows of floats, high and low parts; bn_finish takes the double ones where the two differ (bn_statistics).  The
// conversions and double additions are a tenth of what the SM can do in the time of the loads.
template <typename T, int MODE, bool VEC>
__global__ void __launch_bounds__(256) bn_reduce_xfast(BnRed p, float* partial) {
  grid_dependency();
  const uint32_t c = blockIdx.x, split = blockIdx.y, nsplit = gridDim.y;
  float a = 0.f, b = 0.f;
  double da = 0.0, db = 0.0;
  // the position moves on by the same (images, rows, columns) each time: no division per element
  const size_t first = (size_t)split * 256 + threadIdx.x, hop = (size_t)nsplit * 256;
  if constexpr (VEC) {       // MODE 1
    const uint32_t hw = p.H * p.W / 4, hi = (uint32_t)(hop % hw), hn = (uint32_t)(hop / hw);
    uint32_t i = (uint32_t)(first % hw), n = (uint32_t)(first / hw);
    const float *xb = (const float*)p.x.base + c * p.x.sc, *gb = (const float*)p.dy.base + c * p.dy.sc;
    const float mean = p.mean[c], invstd = p.invstd[c], gam = p.gamma[c], bet = p.beta[c];
#pragma unroll 4
    for (; n < p.N;) {
      const float4 v = *(const float4*)(xb + n * p.x.sn + (size_t)i * 4);
      const float xv[4] = {v.x, v.y, v.z, v.w};
      const float4 w = *(const float4*)(gb + n * p.dy.sn + (size_t)i * 4);
      const float gv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float xhat = (xv[j] - mean) * invstd;
        const float g = p.relu && fmaf(gam, xhat, bet) <= 0.f ? 0.f : gv[j];
        a += g;
        b = fmaf(g, xhat, b);
      }
      i += hi; n += hn;
      if (i >= hw) { i -= hw; ++n; }
    }
  } else {
    const size_t per = (size_t)p.N * p.H * p.W;
    const uint32_t hx = (uint32_t)(hop % p.W), hy = (uint32_t)(hop / p.W % p.H), hn = (uint32_t)(hop / p.W / p.H);
    uint32_t x = (uint32_t)(first % p.W), y = (uint32_t)(first / p.W % p.H), n = (uint32_t)(first / p.W / p.H);
#pragma unroll 4
    for (size_t i = first; i < per; i += hop) {
      const float v = bn_term<T, MODE>(p, n, c, y, x, a, b);
      if (MODE == 0) { da += (double)v; db = fma((double)v, (double)v, db); }
      x += hx; y += hy; n += hn;
      if (x >= p.W) { x -= p.W; ++y; }
      if (y >= p.H) { y -= p.H; ++n; }
    }
  }
  __shared__ float sa[8], sb[8];
  __shared__ double sd[2][8];
  a = warp_sum(a); b = warp_sum(b);
  if (MODE == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { da += __shfl_xor_sync(0xffffffffu, da, o); db += __shfl_xor_sync(0xffffffffu, db, o); }
  }
  if ((threadIdx.x & 31) == 0) { sa[threadIdx.x >> 5] = a; sb[threadIdx.x >> 5] = b; sd[0][threadIdx.x >> 5] = da; sd[1][threadIdx.x >> 5] = db; }
  __syncthreads();
  if (threadIdx.x < 2) {
    float t = 0.f;
    for (int w = 0; w < 8; ++w) t += threadIdx.x ? sb[w] : sa[w];
    float* out = partial + (size_t)split * 2 * p.C + threadIdx.x * p.C + c;
    *out = t;
    if (MODE == 0 && p.dual) {
      double d = 0.0;
      for (int w = 0; w < 8; ++w) d += sd[threadIdx.x][w];
      out = partial + (size_t)(nsplit + 2 * split) * 2 * p.C + threadIdx.x * p.C + c;
      *out = (float)d;
      out[2 * p.C] = isfinite((float)d) ? (float)(d - (double)(float)d) : 0.f;
    }
  }
}

// NHWC-like: block (32 channels x 8 pixel lanes) per (channel group, split).
template <typename T, int MODE>
__global__ void __launch_bounds__(256) bn_reduce_cfast(BnRed p, float* partial) {
  grid_dependency();
  const uint32_t c = blockIdx.x * 32 + threadIdx.x, split = blockIdx.y, nsplit = gridDim.y;
  const size_t per = (size_t)p.N * p.H * p.W;
  float a = 0.f, b = 0.f;
  if (c < p.C)
    for (size_t i = (size_t)split * 8 + threadIdx.y; i < per; i += (size_t)nsplit * 8) {
      uint32_t x = (uint32_t)(i % p.W);
      size_t r = i / p.W;
      uint32_t y = (uint32_t)(r % p.H), n = (uint32_t)(r / p.H);
      bn_term<T, MODE>(p, n, c, y, x, a, b);
    }
  __shared__ float sa[8][33], sb[8][33];
  sa[threadIdx.y][threadIdx.x] = a;
  sb[threadIdx.y][threadIdx.x] = b;
  __syncthreads();
  if (threadIdx.y == 0 && c < p.C) {
    float ta = 0.f, tb = 0.f;
    for (int w = 0; w < 8; ++w) { ta += sa[w][threadIdx.x]; tb += sb[w][threadIdx.x]; }
    partial[(size_t)split * 2 * p.C + c] = ta;
    partial[(size_t)split * 2 * p.C + p.C + c] = tb;
  }
}

// Stage 2 of the statistics: the partial rows are added in double.
//   kind 0: mean / invstd / var from (sum x, sum x^2); double arithmetic for the cancellation in E[x^2]-E[x]^2
//   kind 1: sums[0..2C) = (sum g, sum g*xhat), sums[2C..4C) = those over count; dbeta, dgamma (+)= those sums
//   kind 2: sums[0..2C) only
struct BnFin {
  int kind;
  uint32_t C;
  double count;
  float eps;
  float *mean, *invstd, *var, *sums, *dgamma, *dbeta;
  int accumulate;     // kind 1: add to dgamma / dbeta (else overwrite)
  double rows;        // pixels behind the sums
};
// The sums that statistics are made of: those in fp32 (s, ss), or where the mean or the variance made of them is more than 1e-6 of
// the spread or the variance off, those in double.  The variance is the small difference of E[x^2] and E[x]^2: with fp32
// sums throughout, the gradients of a small net in strips differed from a double-precision one by 8e-4 (18 layers, 16
// pixels per channel at the end), now by 4e-5.  Statistics that agree keep their last digit from call to call of either form: one
// rounding moves pixels across the edge of the ReLU behind (2e-4 of the gradient of 10 M pixels).
__device__ __forceinline__ void bn_statistics(double count, double& s, double& ss, double ds, double dss) {
  const double m = s / count, v = ss / count - m * m, dm = ds / count, dv = dss / count - dm * dm;
  if (!(fabs(v - dv) <= 1e-6 * dv && (m - dm) * (m - dm) <= 1e-12 * dv)) { s = ds; ss = dss; }
}
__device__ __forceinline__ void bn_finish_channel(const BnFin& f, uint32_t c, double s, double ss) {
  if (f.kind == 0) {
    double m = s / f.count, v = ss / f.count - m * m;
    if (v < 0.0) v = 0.0;
    if (f.mean) f.mean[c] = (float)m;
    if (f.invstd) f.invstd[c] = (float)(1.0 / sqrt(v + (double)f.eps));
    if (f.var) f.var[c] = (float)v;
    return;
  }
  const float fs = (float)s, fss = (float)ss;
  f.sums[c] = fs;
  f.sums[f.C + c] = fss;
  if (f.kind == 1) {
    f.sums[2 * f.C + c] = (float)((double)fs / f.count);
    f.sums[3 * f.C + c] = (float)((double)fss / f.count);
    if (f.dbeta) f.dbeta[c] = f.accumulate ? f.dbeta[c] + fs : fs;
    if (f.dgamma) f.dgamma[c] = f.accumulate ? f.dgamma[c] + fss : fss;
  }
}
// 8 channels per block (a row's 32-byte sector), 32 row lanes of 16 values: a thread has its rows (10 of the usual 296) in
// flight at once, so the kernel is one trip to L2 and a short tree.  As 32 channels per block with 8 rows in flight and a
// serial sum of 32 lanes it took 5.6 us, this form 3.3 us at 256 channels.
constexpr uint32_t kFinishThreads = 512, kFinishRows = 10;
__device__ __forceinline__ double bn_finish_rows(const BnFin& f, uint32_t nsplit, const float* __restrict__ partial) {
  const uint32_t v = threadIdx.x & 15, rl = threadIdx.x >> 4, which = v >> 3, c = blockIdx.x * 8 + (v & 7);
  double t = 0.0;
  if (c < f.C) {
    const float* src = partial + which * f.C + c;
    for (uint32_t k0 = rl; k0 < nsplit; k0 += 32 * kFinishRows) {
      float r[kFinishRows];
#pragma unroll
      for (uint32_t u = 0; u < kFinishRows; ++u) {
        const uint32_t k = k0 + u * 32;
        r[u] = k < nsplit ? src[(size_t)k * 2 * f.C] : 0.f;
      }
#pragma unroll
      for (uint32_t u = 0; u < kFinishRows; ++u) t += (double)r[u];
    }
  }
  t += __shfl_xor_sync(0xffffffffu, t, 16);
  __shared__ double sh[16][17];
  if ((threadIdx.x & 31) < 16) sh[threadIdx.x >> 5][v] = t;
  __syncthreads();
  if (threadIdx.x < 32) {
    // lane: value v, half of the 16 warps' sums
    const uint32_t h = threadIdx.x >> 4;
    t = 0.0;
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w) t += sh[h * 8 + w][v];
    t += __shfl_xor_sync(0xffffffffu, t, 16);
  }
  return t;                   // of the first warp: lanes 0 .. 7 the first sum of channel c, 8 .. 15 the second
}
// DUAL: behind the rows of fp32 sums lie twice as many of double ones
template <bool DUAL>
__global__ void __launch_bounds__(kFinishThreads) bn_finish(BnFin f, int nsplit, const float* __restrict__ partial) {
  grid_dependency();
  double t = bn_finish_rows(f, (uint32_t)nsplit, partial), d = 0.0;
  if constexpr (DUAL) {
    __syncthreads();
    d = bn_finish_rows(f, 2u * nsplit, partial + (size_t)nsplit * 2 * f.C);
  }
  if (threadIdx.x >= 32) return;
  double ss = __shfl_down_sync(0xffffffffu, t, 8), dss = 0.0;
  if constexpr (DUAL) dss = __shfl_down_sync(0xffffffffu, d, 8);
  const uint32_t c = blockIdx.x * 8 + threadIdx.x;
  if (threadIdx.x >= 8 || c >= f.C) return;
  if constexpr (DUAL) bn_statistics(f.kind == 0 ? f.count : f.rows, t, ss, d, dss);
  bn_finish_channel(f, c, t, ss);
}

struct BnApply {
  BView x, dy, out, add;   // add: what the backward form adds to its result (accumulate), of out's dims
  uint32_t N, C, H, W;
  int c_fastest, relu, accumulate;
  const float *gamma, *beta, *mean, *invstd;
  const float* partial;  // backward: combined sums [2C], then (vector path) those over count [2C]
  int nsplit;
  double count;
};

// MODE 0: y = relu?(gamma*(x-mean)*invstd+beta)
// MODE 1: dx (+)= gamma*invstd*(g - mean(g) - xhat*mean(g*xhat))
template <typename T, int MODE>
__global__ void __launch_bounds__(256) bn_apply(BnApply p) {
  grid_dependency();
  const size_t total = (size_t)p.N * p.C * p.H * p.W, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t n, c, y, x;
    size_t r = i;
    if (p.c_fastest) {
      c = (uint32_t)(r % p.C); r /= p.C; x = (uint32_t)(r % p.W); r /= p.W; y = (uint32_t)(r % p.H); n = (uint32_t)(r / p.H);
    } else {
      x = (uint32_t)(r % p.W); r /= p.W; y = (uint32_t)(r % p.H); r /= p.H; c = (uint32_t)(r % p.C); n = (uint32_t)(r / p.C);
    }
    const float xv = ld_f((const T*)p.x.base + (n * p.x.sn + c * p.x.sc + y * p.x.sy + x * p.x.sx));
    T* op = (T*)p.out.base + (n * p.out.sn + c * p.out.sc + y * p.out.sy + x * p.out.sx);
    const float xhat = (xv - p.mean[c]) * p.invstd[c];
    if (MODE == 0) {
      float v = fmaf(p.gamma[c], xhat, p.beta[c]);
      if (p.relu) v = fmaxf(v, 0.f);
      st_f(op, v);
    } else {
      float g = ld_f((const T*)p.dy.base + (n * p.dy.sn + c * p.dy.sc + y * p.dy.sy + x * p.dy.sx));
      if (p.relu && fmaf(p.gamma[c], xhat, p.beta[c]) <= 0.f) g = 0.f;
      const float m1 = (float)((double)p.partial[c] / p.count), m2 = (float)((double)p.partial[p.C + c] / p.count);
      float v = p.gamma[c] * p.invstd[c] * (g - m1 - xhat * m2);
      if (p.accumulate) v += ld_f((const T*)p.add.base + (n * p.add.sn + c * p.add.sc + y * p.add.sy + x * p.add.sx));
      st_f(op, v);
    }
  }
}
// The same for views that are not channel-fastest: a block serves part of one (image, channel) plane, so that the channel's
// constants are read once and a pixel's place costs one 32-bit division (VEC: none, 4 pixels per load).  Element by element
// over the whole tensor (bn_apply, with 64-bit divisions and the sums divided by the count for each) the 34 normalisations
// of an 18-layer net on 4 x 224 x 224 took 527 us, so 205; with the sums 867 -> 372.
// Small planes: several per block, 2^shift threads each.  Fixed statistics, us element by element, with a block per plane, so: 64 x
// 2048 x 7 x 7 44, 239, 30; 64 x 1024 x 14 x 14 81, 75, 24; backward 97, 306, 73 and 196, 130, 60.
constexpr uint32_t kPlaneApply = 1024, kPlaneApplyVec = 2048;   // pixels per block
template <typename T, int MODE, bool VEC>
__global__ void __launch_bounds__(256) bn_apply_planes(BnApply p, uint32_t chunks, uint32_t shift) {
  grid_dependency();
  const uint32_t lanes = 1u << shift, lane = threadIdx.x & (lanes - 1), unit = (blockIdx.x << (8 - shift)) + (threadIdx.x >> shift);
  const uint32_t plane = unit / chunks, chunk = unit - plane * chunks, n = plane / p.C, c = plane - n * p.C, hw = p.H * p.W;
  if (n >= p.N) return;
  const float mean = p.mean[c], invstd = p.invstd[c], gam = p.gamma[c], bet = p.beta[c];
  const float m1 = MODE ? p.partial[2 * p.C + c] : 0.f, m2 = MODE ? p.partial[3 * p.C + c] : 0.f, scale = gam * invstd;
  const T *xb = (const T*)p.x.base + n * p.x.sn + c * p.x.sc, *db = (const T*)p.dy.base + n * p.dy.sn + c * p.dy.sc;
  const T* ab = (const T*)p.add.base + n * p.add.sn + c * p.add.sc;
  T* ob = (T*)p.out.base + n * p.out.sn + c * p.out.sc;
  auto value = [&](float xv, float g, float old) {
    const float xhat = (xv - mean) * invstd;
    if (MODE == 0) {
      const float v = fmaf(gam, xhat, bet);
      return p.relu ? fmaxf(v, 0.f) : v;
    }
    if (p.relu && fmaf(gam, xhat, bet) <= 0.f) g = 0.f;
    const float v = scale * (g - m1 - xhat * m2);
    return p.accumulate ? v + old : v;
  };
  if constexpr (VEC) {
    constexpr int U = kPlaneApplyVec / 1024;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xv[U], g[U], old[U];
    const uint32_t i0 = chunk * kPlaneApplyVec + lane * 4;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = i0 + u * lanes * 4;
      xv[u] = g[u] = old[u] = zero;
      if (i < hw) {
        xv[u] = *(const float4*)(xb + i);
        if (MODE == 1) g[u] = *(const float4*)(db + i);
        if (MODE == 1 && p.accumulate) old[u] = *(const float4*)(ab + i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = i0 + u * lanes * 4;
      if (i < hw)
        *(float4*)(ob + i) = make_float4(value(xv[u].x, g[u].x, old[u].x), value(xv[u].y, g[u].y, old[u].y), value(xv[u].z, g[u].z, old[u].z),
                                         value(xv[u].w, g[u].w, old[u].w));
    }
  } else {
    constexpr int U = kPlaneApply / 256;
    float xv[U], g[U], old[U];
    long long at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t i = chunk * kPlaneApply + u * lanes + lane, y = i / p.W, x = i - y * p.W;
      xv[u] = g[u] = old[u] = 0.f;
      at[u] = y * p.out.sy + x * p.out.sx;
      if (i < hw) {
        xv[u] = ld_f(xb + (y * p.x.sy + x * p.x.sx));
        if (MODE == 1) g[u] = ld_f(db + (y * p.dy.sy + x * p.dy.sx));
        if (MODE == 1 && p.accumulate) old[u] = ld_f(ab + (y * p.add.sy + x * p.add.sx));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (chunk * kPlaneApply + u * lanes + lane < hw) st_f(ob + at[u], value(xv[u], g[u], old[u]));
  }
}


// ------------------------------------------------------------------ NHWC bf16 fast paths
// Channel-fastest bf16 views whose strides are multiples of 8 elements: a thread owns 8 adjacent
// channels (one 16-byte load / store per pixel) of a fixed channel group, so the per-channel
// constants sit in registers and every warp access is a run of whole 128-byte lines.  A block holds
// 256 / (C / 8) pixel lanes; up to C / 8 - 1 threads are over when C / 8 is no power of two.
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) { float2 t = __bfloat1622float2(h[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
  return v;
}
// Element offset of pixel i (n, y, x flattened).  Views whose pixels are evenly spaced need no division;
// others decode with 32-bit arithmetic (the launchers require N*H*W < 2^31).
__device__ __forceinline__ long long pix_off(const BView& v, uint32_t i, uint32_t H, uint32_t W) {
  if (v.sy == (long long)W * v.sx && v.sn == (long long)H * v.sy) return (long long)i * v.sx;
  const uint32_t r = i / W, x = i - r * W, n = r / H, y = r - n * H;
  return n * v.sn + y * v.sy + x * v.sx;
}
__device__ __forceinline__ const void* at16(const BView& v, long long off) { return (const __nv_bfloat16*)v.base + off; }

constexpr int kBnUnroll = 4;      // pixels per thread below which a smaller grid would do (vec_grid)
constexpr int kBnDepth = 8;       // loads in flight per thread and stream
// of the gradient with an addend: three streams that fit beside a filter gradient's CTA
constexpr int bn_depth(bool add) { return add ? 6 : kBnDepth; }

// HBM-bound.  131,072 x 512 bf16 inside a net: 34 -> 27 us (MODE 0), 60 -> 53 us (MODE 1) against batches of 4 loads in
// registers; 16 in flight gained nothing more.
template <int MODE>
__global__ void __launch_bounds__(256, 2) bn_reduce_vec(BnRed p, float* partial) {
  grid_dependency();
  extern __shared__ __align__(128) uint4 ring_smem[];
  LoadRing<MODE + 1, kBnDepth> ring(ring_smem);
  const uint32_t G = p.C / 8, cg = threadIdx.x % G, pl = threadIdx.x / G, PL = 256 / G;
  const uint32_t per = p.N * p.H * p.W, stride = gridDim.x * PL;
  float a[8], b[8], mean[8], invstd[8], gam[8], bet[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    a[j] = b[j] = 0.f;
    if (MODE == 1) { mean[j] = p.mean[cg * 8 + j]; invstd[j] = p.invstd[cg * 8 + j]; gam[j] = p.gamma[cg * 8 + j]; bet[j] = p.beta[cg * 8 + j]; }
  }
  // Pixels are walked from the last to the first: the tensor was just written front to back by its producer, so its
  // tail is what the L2 still holds; the apply pass that follows walks front to back and meets what this pass read last.
  auto issue = [&](uint32_t k) {
    if (k < per) {
      const uint32_t i = per - 1u - k;
      ring.copy(0, at16(p.x, pix_off(p.x, i, p.H, p.W) + cg * 8));
      if (MODE == 1) ring.copy(MODE, at16(p.dy, pix_off(p.dy, i, p.H, p.W) + cg * 8));
    }
    ring.commit();
  };
  uint32_t k = pl < PL ? blockIdx.x * PL + pl : per;
#pragma unroll
  for (int d = 0; d < kBnDepth - 1; ++d) issue(k + d * stride);
  for (; k < per; k += stride) {
    ring.wait();
    float xv[8], g[8];
    unpack8(ring.get(0), xv);
    if (MODE == 1) unpack8(ring.get(MODE), g);
    ring.next();
    issue(k + (kBnDepth - 1) * stride);
    if (MODE == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) { a[j] += xv[j]; b[j] = fmaf(xv[j], xv[j], b[j]); }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = (xv[j] - mean[j]) * invstd[j];
        float gj = g[j];
        if (p.relu && fmaf(gam[j], xhat, bet[j]) <= 0.f) gj = 0.f;
        a[j] += gj;
        b[j] = fmaf(gj, xhat, b[j]);
      }
    }
  }
  // the ring's memory is free once every thread has read its last element
  float (*sa)[9] = (float (*)[9])ring_smem, (*sb)[9] = sa + 256;
  static_assert(LoadRing<1, kBnDepth>::kBytes >= 2 * 256 * 9 * 4, "the sums of the lanes fit the ring");
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) { sa[threadIdx.x][j] = a[j]; sb[threadIdx.x][j] = b[j]; }
  __syncthreads();
  // thread t < 2C sums one of the block's 2C outputs over the pixel lanes, in lane order
  for (uint32_t t = threadIdx.x; t < 2 * p.C; t += 256) {
    const uint32_t which = t / p.C, c = t - which * p.C, g = c >> 3, j = c & 7;
    float acc = 0.f;
#pragma unroll 8
    for (uint32_t q = 0; q < PL; ++q) acc += which ? sb[q * G + g][j] : sa[q * G + g][j];
    partial[(size_t)blockIdx.x * 2 * p.C + t] = acc;
  }
}

// ADD: the backward form adds *add to what it writes.  HBM-bound: 131,072 x 512 bf16 50 -> 42 us (MODE 0, 6.4 TB/s) and
// 78 -> 62 us (MODE 1, 6.5 TB/s) against batches of 3-4 loads in registers.
template <int MODE, bool ADD>
__global__ void __launch_bounds__(256, 2) bn_apply_vec(BnApply p) {
  grid_dependency();
  extern __shared__ __align__(128) uint4 ring_smem[];
  LoadRing<MODE + 1 + ADD, bn_depth(ADD)> ring(ring_smem);
  const uint32_t G = p.C / 8, cg = threadIdx.x % G, pl = threadIdx.x / G, PL = 256 / G;
  const uint32_t per = p.N * p.H * p.W, stride = gridDim.x * PL;
  float sc[8], sh[8], mean[8], invstd[8], m1[8], m2[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t c = cg * 8 + j;
    mean[j] = p.mean[c]; invstd[j] = p.invstd[c];
    sc[j] = p.gamma[c]; sh[j] = p.beta[c];
    if (MODE == 1) { m1[j] = p.partial[2 * p.C + c]; m2[j] = p.partial[3 * p.C + c]; }
  }
  auto issue = [&](uint32_t i) {
    if (i < per) {
      ring.copy(0, at16(p.x, pix_off(p.x, i, p.H, p.W) + cg * 8));
      if (MODE == 1) ring.copy(MODE, at16(p.dy, pix_off(p.dy, i, p.H, p.W) + cg * 8));
      if (ADD) ring.copy(MODE + ADD, at16(p.add, pix_off(p.add, i, p.H, p.W) + cg * 8));
    }
    ring.commit();
  };
  uint32_t i = pl < PL ? blockIdx.x * PL + pl : per;
#pragma unroll
  for (int d = 0; d < bn_depth(ADD) - 1; ++d) issue(i + d * stride);
  for (; i < per; i += stride) {
    ring.wait();
    float xv[8], g[8], old[8], o[8];
    unpack8(ring.get(0), xv);
    if (MODE == 1) unpack8(ring.get(MODE), g);
    if (ADD) unpack8(ring.get(MODE + ADD), old);
    ring.next();
    issue(i + (bn_depth(ADD) - 1) * stride);
    if (MODE == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = (xv[j] - mean[j]) * invstd[j];
        float v = fmaf(sc[j], xhat, sh[j]);
        o[j] = p.relu ? fmaxf(v, 0.f) : v;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = (xv[j] - mean[j]) * invstd[j];
        float gj = g[j];
        if (p.relu && fmaf(sc[j], xhat, sh[j]) <= 0.f) gj = 0.f;
        float v = sc[j] * invstd[j] * (gj - m1[j] - xhat * m2[j]);
        o[j] = ADD ? v + old[j] : v;
      }
    }
    *(uint4*)((__nv_bfloat16*)p.out.base + pix_off(p.out, i, p.H, p.W) + cg * 8) = pack8(o);
  }
}

static bool vec_view_ok(const ad_tensor4* t) {
  if (t->dtype != AD_BF16 || t->sc != 1 || (t->C & 7u) || t->C < 8 || t->C > 2048) return false;
  if ((size_t)t->N * t->H * t->W >= (1ull << 31)) return false;
  return !((uintptr_t)t->base & 15u) && !(t->sn & 7) && !(t->sy & 7) && !(t->sx & 7);
}
// blocks of the vector reduction = partial rows: enough to fill the machine, each thread with
// at least one batch of pixels, within the rows the scratch holds
static unsigned vec_grid(const ad_tensor4* t) {
  const size_t per = (size_t)t->N * t->H * t->W, PL = 256 / (t->C / 8);
  size_t g = (per + PL * kBnUnroll - 1) / (PL * kBnUnroll);
  if (g > (size_t)kNumSMs * 2) g = (size_t)kNumSMs * 2;   // two resident blocks per SM keep ~5 MB of loads in flight
  if (g > (size_t)bn_max_splits(t->C)) g = bn_max_splits(t->C);
  return (unsigned)(g < 1 ? 1 : g);
}

static int ring_smem_failed() { cudaGetLastError(); return AD_ERR_CUDA; }
template <int MODE, bool ADD>
static int launch_apply_vec(const BnApply& a, cudaStream_t s) {
  constexpr int smem = LoadRing<MODE + 1 + ADD, bn_depth(ADD)>::kSmem;
  if (cudaFuncSetAttribute(bn_apply_vec<MODE, ADD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return ring_smem_failed();
  const uint32_t PL = 256 / (a.C / 8), per = a.N * a.H * a.W;
  launch(bn_apply_vec<MODE, ADD>, grid_for(per, PL * kBnUnroll, 2), 256, smem, s, a);
  return AD_OK;
}

static int pick_splits(const ad_tensor4* x, bool cfast) {
  const size_t per = (size_t)x->N * x->H * x->W;
  const size_t groups = cfast ? (x->C + 31) / 32 : x->C;
  size_t want = ((size_t)kNumSMs * 4 + groups - 1) / groups;  // ~4 blocks per SM overall
  size_t maxs = (per + (cfast ? 8 : 256) * 4 - 1) / ((cfast ? 8 : 256) * 4);
  if (want > maxs) want = maxs;
  if (want > (size_t)kBnMaxSplits) want = kBnMaxSplits;
  if (want > (size_t)bn_max_splits(x->C)) want = bn_max_splits(x->C);
  if (want < 1) want = 1;
  return (int)want;
}

static void launch_finish(const BnFin& f, int nsplit, int dual, const float* partial, cudaStream_t s) {
  launch(dual ? bn_finish<true> : bn_finish<false>, (f.C + 7) / 8, kFinishThreads, 0, s, f, nsplit, partial);
  count_launch();
}
// Both stages of the statistics of x (MODE 0) or of the backward sums (MODE 1) into what `f` names
template <int MODE>
static int launch_reduce(const BnRed& p, const ad_tensor4* x, const BnFin& f, float* partial, cudaStream_t s, bool vec = false) {   // vec: MODE 1
  const bool cfast = x->sc == 1 && x->C > 1;
  int nsplit, dual = 0;
  BnFin fin = f;
  fin.rows = (double)x->N * x->H * x->W;
  if (vec_view_ok(x) && (MODE == 0 || (p.dy.sc == 1 && !((uintptr_t)p.dy.base & 15u) && !(p.dy.sn & 7) && !(p.dy.sy & 7) && !(p.dy.sx & 7)))) {
    nsplit = (int)vec_grid(x);
    constexpr int smem = LoadRing<MODE + 1, kBnDepth>::kSmem;
    // the attribute is per function and per device; setting it is cheap enough to do per launch
    if (cudaFuncSetAttribute(bn_reduce_vec<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return ring_smem_failed();
    launch(bn_reduce_vec<MODE>, nsplit, 256, smem, s, p, partial);
  } else {
    nsplit = pick_splits(x, cfast);
    if (cfast) {
      dim3 grid((x->C + 31) / 32, nsplit), block(32, 8);
      AD_DISPATCH_DTYPE(x->dtype, (launch(bn_reduce_cfast<T, MODE>, grid, block, 0, s, p, partial)));
    } else {
      BnRed r = p;
      r.dual = dual = MODE == 0 && 3 * nsplit <= bn_max_splits(x->C);
      const dim3 grid(x->C, nsplit);
      if (MODE == 1 && vec) launch(bn_reduce_xfast<float, 1, true>, grid, 256, 0, s, r, partial);
      else AD_DISPATCH_DTYPE(x->dtype, (launch(bn_reduce_xfast<T, MODE, false>, grid, 256, 0, s, r, partial)));
    }
  }
  count_launch();
  launch_finish(fin, nsplit, dual, partial, s);
  return launch_status();
}

static bool dims_eq(const ad_tensor4* a, const ad_tensor4* b) {
  return a->N == b->N && a->C == b->C && a->H == b->H && a->W == b->W && a->dtype == b->dtype;
}

// ------------------------------------------------------------------ max pooling
struct PoolP {
  BView x, y, dy, dx;
  uint32_t N, C, H, W, P, Q, kh, kw, sh, sw;
  int c_fastest, accumulate;
};

template <typename T>
__device__ __forceinline__ uint32_t window_argmax(const PoolP& p, uint32_t n, uint32_t c, uint32_t q, uint32_t s, float& best) {
  uint32_t bi = 0;
  best = -INFINITY;
  for (uint32_t i = 0; i < p.kh; ++i)
    for (uint32_t j = 0; j < p.kw; ++j) {
      const uint32_t yy = q * p.sh + i, xx = s * p.sw + j;
      const float v = ld_f((const T*)p.x.base + (n * p.x.sn + c * p.x.sc + yy * p.x.sy + xx * p.x.sx));
      if (v > best || (i == 0 && j == 0)) { best = v; bi = yy * p.W + xx; }
    }
  return bi;
}

template <typename T>
__global__ void __launch_bounds__(256) maxpool_fwd_kernel(PoolP p) {
  grid_dependency();
  const size_t total = (size_t)p.N * p.C * p.P * p.Q, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t n, c, q, s;
    size_t r = i;
    if (p.c_fastest) {
      c = (uint32_t)(r % p.C); r /= p.C; s = (uint32_t)(r % p.Q); r /= p.Q; q = (uint32_t)(r % p.P); n = (uint32_t)(r / p.P);
    } else {
      s = (uint32_t)(r % p.Q); r /= p.Q; q = (uint32_t)(r % p.P); r /= p.P; c = (uint32_t)(r % p.C); n = (uint32_t)(r / p.C);
    }
    float best;
    window_argmax<T>(p, n, c, q, s, best);
    st_f((T*)p.y.base + (n * p.y.sn + c * p.y.sc + q * p.y.sy + s * p.y.sx), best);
  }
}

// One thread per INPUT element gathers from the windows that contain it; a window
// contributes iff its first maximum is this element.  No atomics -> reproducible.
template <typename T>
__global__ void __launch_bounds__(256) maxpool_bwd_kernel(PoolP p) {
  grid_dependency();
  const size_t total = (size_t)p.N * p.C * p.H * p.W, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t n, c, y, x;
    size_t r = i;
    if (p.c_fastest) {
      c = (uint32_t)(r % p.C); r /= p.C; x = (uint32_t)(r % p.W); r /= p.W; y = (uint32_t)(r % p.H); n = (uint32_t)(r / p.H);
    } else {
      x = (uint32_t)(r % p.W); r /= p.W; y = (uint32_t)(r % p.H); r /= p.H; c = (uint32_t)(r % p.C); n = (uint32_t)(r / p.C);
    }
    float acc = 0.f;
    // windows q with q*sh <= y <= q*sh + kh - 1
    const uint32_t q_lo = y + 1 > p.kh ? (y + 1 - p.kh + p.sh - 1) / p.sh : 0;
    const uint32_t s_lo = x + 1 > p.kw ? (x + 1 - p.kw + p.sw - 1) / p.sw : 0;
    for (uint32_t q = q_lo; q < p.P && q * p.sh <= y; ++q)
      for (uint32_t s = s_lo; s < p.Q && s * p.sw <= x; ++s) {
        float best;
        if (window_argmax<T>(p, n, c, q, s, best) == y * p.W + x)
          acc += ld_f((const T*)p.dy.base + (n * p.dy.sn + c * p.dy.sc + q * p.dy.sy + s * p.dy.sx));
      }
    T* op = (T*)p.dx.base + (n * p.dx.sn + c * p.dx.sc + y * p.dx.sy + x * p.dx.sx);
    if (p.accumulate) acc += ld_f(op);
    st_f(op, acc);
  }
}


// NHWC bf16 pooling, 8 channels per thread: comparisons and selections on packed pairs.  Same first-maximum rule as the
// scalar kernels.
__device__ __forceinline__ uint32_t gt2(uint32_t a, uint32_t b) {
  return __hgt2_mask(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
}
// best = v where v > best (per 16-bit half); pos likewise takes `at`
__device__ __forceinline__ void max8(uint4& best, const uint4& v) {
  uint32_t* b = &best.x;
  const uint32_t* w = &v.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) { const uint32_t m = gt2(w[j], b[j]); b[j] = (w[j] & m) | (b[j] & ~m); }
}
__device__ __forceinline__ void argmax8(uint4& best, uint4& pos, const uint4& v, uint32_t at) {
  uint32_t *b = &best.x, *q = &pos.x;
  const uint32_t* w = &v.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t m = gt2(w[j], b[j]);
    b[j] = (w[j] & m) | (b[j] & ~m);
    q[j] = (at & m) | (q[j] & ~m);
  }
}
// K x K windows, or any extents (K = 0)
template <int K>
__global__ void __launch_bounds__(256) maxpool_fwd_vec(PoolP p) {
  grid_dependency();
  const uint32_t G = p.C / 8, kh = K ? K : p.kh, kw = K ? K : p.kw;
  const size_t total = (size_t)p.N * p.P * p.Q * G, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t cg, s, q, n;
    if (total < (1ull << 32)) {
      uint32_t r = (uint32_t)i;
      cg = r % G; r /= G; s = r % p.Q; r /= p.Q; q = r % p.P; n = r / p.P;
    } else {
      size_t r = i / G;
      cg = (uint32_t)(i % G); s = (uint32_t)(r % p.Q); r /= p.Q; q = (uint32_t)(r % p.P); n = (uint32_t)(r / p.P);
    }
    const __nv_bfloat16* xb = (const __nv_bfloat16*)p.x.base + n * p.x.sn + (long long)(q * p.sh) * p.x.sy + (long long)(s * p.sw) * p.x.sx + cg * 8;
    uint4 best;
    if constexpr (K != 0) {
      uint4 v[K * K];                  // the whole window in flight
#pragma unroll
      for (int a = 0; a < K; ++a)
#pragma unroll
        for (int b = 0; b < K; ++b) v[a * K + b] = *(const uint4*)(xb + a * p.x.sy + b * p.x.sx);
      best = v[0];
#pragma unroll
      for (int t = 1; t < K * K; ++t) max8(best, v[t]);
    } else {
      best = *(const uint4*)xb;
      for (uint32_t a = 0; a < kh; ++a)
        for (uint32_t b = 0; b < kw; ++b)
          if (a | b) max8(best, *(const uint4*)(xb + a * p.x.sy + b * p.x.sx));
    }
    *(uint4*)((__nv_bfloat16*)p.y.base + n * p.y.sn + q * p.y.sy + s * p.y.sx + cg * 8) = best;
  }
}
// one thread per input pixel x 8 channels; gathers from the (at most ceil(kh/sh) x ceil(kw/sw)) windows over it
__global__ void __launch_bounds__(256) maxpool_bwd_vec(PoolP p) {
  grid_dependency();
  const uint32_t G = p.C / 8;
  const size_t total = (size_t)p.N * p.H * p.W * G, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    const uint32_t cg = (uint32_t)(i % G);
    size_t r = i / G;
    const uint32_t x = (uint32_t)(r % p.W); r /= p.W;
    const uint32_t y = (uint32_t)(r % p.H), n = (uint32_t)(r / p.H);
    const __nv_bfloat16* xb = (const __nv_bfloat16*)p.x.base + n * p.x.sn + cg * 8;
    float acc[8], me[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    unpack8(*(const uint4*)(xb + y * p.x.sy + x * p.x.sx), me);
    const uint32_t q_lo = y + 1 > p.kh ? (y + 1 - p.kh + p.sh - 1) / p.sh : 0;
    const uint32_t s_lo = x + 1 > p.kw ? (x + 1 - p.kw + p.sw - 1) / p.sw : 0;
    for (uint32_t q = q_lo; q < p.P && q * p.sh <= y; ++q)
      for (uint32_t s = s_lo; s < p.Q && s * p.sw <= x; ++s) {
        // this element is the window's first maximum iff no earlier element (scan order) is >= it
        // and no later element is > it
        uint32_t win = 0xffu;   // bit j: channel j of this element is still the window's first maximum
        for (uint32_t a = 0; a < p.kh; ++a)
          for (uint32_t b = 0; b < p.kw; ++b) {
            const uint32_t yy = q * p.sh + a, xx = s * p.sw + b;
            if (yy == y && xx == x) continue;
            float v[8];
            unpack8(*(const uint4*)(xb + yy * p.x.sy + xx * p.x.sx), v);
            const bool earlier = yy < y || (yy == y && xx < x);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (!(earlier ? v[j] < me[j] : v[j] <= me[j])) win &= ~(1u << j);
          }
        float g[8];
        unpack8(*(const uint4*)((const __nv_bfloat16*)p.dy.base + n * p.dy.sn + q * p.dy.sy + s * p.dy.sx + cg * 8), g);
#pragma unroll
        for (int j = 0; j < 8; ++j) if (win & (1u << j)) acc[j] += g[j];
      }
    uint4* op = (uint4*)((__nv_bfloat16*)p.dx.base + n * p.dx.sn + y * p.dx.sy + x * p.dx.sx + cg * 8);
    if (p.accumulate) {
      float old[8];
      unpack8(*op, old);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += old[j];
    }
    *op = pack8(acc);
  }
}
// Tiled backward for NHWC bf16: a block owns a 16 x 16 patch of input pixels for up to 8 channel groups.
// Phase 1, once per window that touches the patch: the position of the window's first maximum (a small bf16 number per
// channel, so that packed comparisons serve it) and its gradient go to shared memory; phase 2 lets every input pixel pick
// its gradients there.  Same first-maximum rule and the same summation order (q, then s, ascending) as the kernels above.
// The bound is HBM (x, dy and dx once) for windows that do not overlap much; packed 16-bit comparisons keep the arithmetic
// near it.  Gradient of 2 x 64 x 514 x 1026 (46 us at the copy rate for 2 x 2 / 2): 2 x 2 / 2 132 -> 56 us, 3 x 3 / 3 142 -> 99,
// 3 x 3 / 1 560 -> 296, 5 x 5 / 2 6650 -> 278; 3 x 3 / 2 goes to maxpool_bwd_quads.
constexpr uint32_t kPoolTile = 16, kPoolMaxWin = 400;
// K x K windows of stride S, or any extents (K = 0)
template <int K, int S>
__global__ void __launch_bounds__(256) maxpool_bwd_tile(PoolP p, uint32_t gchunks) {
  grid_dependency();
  extern __shared__ uint4 win[];       // [window][8 groups][position, gradient]
  __shared__ uint32_t codes[256];      // position t < kh * kw as a bf16 in both halves
  const uint32_t kh = K ? K : p.kh, kw = K ? K : p.kw, sh = K ? S : p.sh, sw = K ? S : p.sw;
  const uint32_t G = p.C / 8, gc = blockIdx.x % gchunks, tx = blockIdx.x / gchunks, ty = blockIdx.y, n = blockIdx.z;
  const uint32_t g0 = gc * 8, gcnt = G - g0 < 8 ? G - g0 : 8;
  const uint32_t y0 = ty * kPoolTile, x0 = tx * kPoolTile;
  const uint32_t y1 = y0 + kPoolTile < p.H ? y0 + kPoolTile : p.H, x1 = x0 + kPoolTile < p.W ? x0 + kPoolTile : p.W;
  const uint32_t q_lo = y0 + 1 > kh ? (y0 + 1 - kh + sh - 1) / sh : 0;
  const uint32_t s_lo = x0 + 1 > kw ? (x0 + 1 - kw + sw - 1) / sw : 0;
  const uint32_t q_hi = (y1 - 1) / sh < p.P - 1 ? (y1 - 1) / sh : p.P - 1;   // inclusive
  const uint32_t s_hi = (x1 - 1) / sw < p.Q - 1 ? (x1 - 1) / sw : p.Q - 1;
  const uint32_t nq = q_hi >= q_lo ? q_hi - q_lo + 1 : 0, ns = s_hi >= s_lo ? s_hi - s_lo + 1 : 0;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)p.x.base + n * p.x.sn + g0 * 8;
  const __nv_bfloat16* gb = (const __nv_bfloat16*)p.dy.base + n * p.dy.sn + g0 * 8;
  auto code = [](uint32_t t) {         // t <= 256 as a bf16 in both halves
    const __nv_bfloat162 h = __float2bfloat162_rn((float)t);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  if (threadIdx.x < kh * kw) codes[threadIdx.x] = code(threadIdx.x);
  const uint32_t gsh = gcnt > 4 ? 3 : (gcnt > 2 ? 2 : (gcnt > 1 ? 1 : 0));   // lanes per pixel, a power of two
  for (uint32_t it = threadIdx.x; it < (nq * ns) << gsh; it += 256) {
    const uint32_t cg = it & ((1u << gsh) - 1u), w = it >> gsh, s = s_lo + w % ns, q = q_lo + w / ns;
    if (cg >= gcnt) continue;
    const __nv_bfloat16* xw = xb + (long long)(q * sh) * p.x.sy + (long long)(s * sw) * p.x.sx + cg * 8;
    uint4 best, pos = make_uint4(0u, 0u, 0u, 0u);
    const uint4 g = *(const uint4*)(gb + q * p.dy.sy + s * p.dy.sx + cg * 8);
    if constexpr (K != 0) {
      uint4 v[K * K];
#pragma unroll
      for (int a = 0; a < K; ++a)
#pragma unroll
        for (int b = 0; b < K; ++b) v[a * K + b] = *(const uint4*)(xw + a * p.x.sy + b * p.x.sx);
      best = v[0];
#pragma unroll
      for (int t = 1; t < K * K; ++t) argmax8(best, pos, v[t], code(t));
    } else {
      best = *(const uint4*)xw;
      for (uint32_t a = 0; a < kh; ++a)
        for (uint32_t b = 0; b < kw; ++b)
          if (a | b) argmax8(best, pos, *(const uint4*)(xw + a * p.x.sy + b * p.x.sx), code(a * kw + b));
    }
    win[(w * 8 + cg) * 2] = pos;
    win[(w * 8 + cg) * 2 + 1] = g;
  }
  __syncthreads();
  // a thread keeps its column and channel group and walks down the patch: 256 >> gsh lanes are whole rows of 16
  const uint32_t cg = threadIdx.x & ((1u << gsh) - 1u), pix0 = threadIdx.x >> gsh, x = x0 + pix0 % kPoolTile;
  if (x >= p.W || cg >= gcnt) return;
  const uint32_t sa = x + 1 > kw ? (x + 1 - kw + sw - 1) / sw : 0, sb = x / sw < p.Q - 1 ? x / sw : p.Q - 1;
  __nv_bfloat16* ob = (__nv_bfloat16*)p.dx.base + n * p.dx.sn + x * p.dx.sx + (g0 + cg) * 8;
  for (uint32_t y = y0 + pix0 / kPoolTile; y < y1; y += (256u >> gsh) / kPoolTile) {
    const uint32_t qa = y + 1 > kh ? (y + 1 - kh + sh - 1) / sh : 0, qb = y / sh < p.P - 1 ? y / sh : p.P - 1;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (uint32_t q = qa; q <= qb; ++q)
      for (uint32_t s = sa; s <= sb; ++s) {
        const uint32_t w = ((q - q_lo) * ns + (s - s_lo)) * 8 + cg, me = codes[(y - q * sh) * kw + (x - s * sw)];
        const uint4 pos = win[w * 2], g = win[w * 2 + 1];
        const uint32_t *pp = &pos.x, *gp = &g.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t m = gp[j] & __heq2_mask(*reinterpret_cast<const __nv_bfloat162*>(&pp[j]), *reinterpret_cast<const __nv_bfloat162*>(&me));
          acc[2 * j] += __uint_as_float(m << 16);
          acc[2 * j + 1] += __uint_as_float(m & 0xffff0000u);
        }
      }
    uint4* op = (uint4*)(ob + y * p.dx.sy);
    if (p.accumulate) {
      float old[8];
      unpack8(*op, old);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += old[j];
    }
    *op = pack8(acc);
  }
}
// The same for 3 x 3 windows of stride 2 (every net's stem): a thread takes the 2 x 2 pixels that start at an even row and
// column.  They lie in four windows at nine places known in advance, so it reads four table entries instead of nine and
// has no index arithmetic; windows outside the output are in the table with a zero gradient.  Bound by instructions
// before (2 x 64 x 514 x 1026: 92 us, 77 M instructions), 62 us and 44 M now; 46 us at the copy rate.
__global__ void __launch_bounds__(256) maxpool_bwd_quads(PoolP p, uint32_t gchunks) {
  grid_dependency();
  constexpr uint32_t kW = kPoolTile / 2 + 1;   // windows over the patch, each way
  __shared__ uint4 wpos[kW * kW * 8], wgrad[kW * kW * 8];   // [window][8 groups]
  const uint32_t G = p.C / 8, gc = blockIdx.x % gchunks, tx = blockIdx.x / gchunks, n = blockIdx.z;
  const uint32_t g0 = gc * 8, gcnt = G - g0 < 8 ? G - g0 : 8;
  const uint32_t y0 = blockIdx.y * kPoolTile, x0 = tx * kPoolTile;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)p.x.base + n * p.x.sn + g0 * 8;
  const __nv_bfloat16* gb = (const __nv_bfloat16*)p.dy.base + n * p.dy.sn + g0 * 8;
  auto code = [](uint32_t t) {         // t as a bf16 in both halves
    const __nv_bfloat162 h = __float2bfloat162_rn((float)t);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  const uint32_t gsh = gcnt > 4 ? 3 : (gcnt > 2 ? 2 : (gcnt > 1 ? 1 : 0));   // lanes per pixel, a power of two
  const uint32_t cg = threadIdx.x & ((1u << gsh) - 1u);
  if (cg < gcnt)
    for (uint32_t w = threadIdx.x >> gsh; w < kW * kW; w += 256u >> gsh) {
      const int q = (int)(y0 / 2 + w / kW) - 1, s = (int)(x0 / 2 + w % kW) - 1;
      uint4 pos = make_uint4(0u, 0u, 0u, 0u), g = pos;
      if (q >= 0 && s >= 0 && q < (int)p.P && s < (int)p.Q) {
        const __nv_bfloat16* xw = xb + (long long)(2 * q) * p.x.sy + (long long)(2 * s) * p.x.sx + cg * 8;
        g = *(const uint4*)(gb + (long long)q * p.dy.sy + (long long)s * p.dy.sx + cg * 8);
        uint4 v[9];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) v[a * 3 + b] = *(const uint4*)(xw + a * p.x.sy + b * p.x.sx);
        uint4 best = v[0];
#pragma unroll
        for (int t = 1; t < 9; ++t) argmax8(best, pos, v[t], code(t));
      }
      wpos[w * 8 + cg] = pos;
      wgrad[w * 8 + cg] = g;
    }
  __syncthreads();
  if (cg >= gcnt) return;
  for (uint32_t i = threadIdx.x >> gsh; i < kPoolTile * kPoolTile / 4; i += 256u >> gsh) {
    const uint32_t wy = i / (kPoolTile / 2), wx = i % (kPoolTile / 2), y = y0 + 2 * wy, x = x0 + 2 * wx;
    if (y >= p.H || x >= p.W) continue;
    const uint32_t w = (wy * kW + wx) * 8 + cg;   // the windows up and left: 00, 01, 10, 11
    const uint4 pos00 = wpos[w], pos01 = wpos[w + 8], pos10 = wpos[w + kW * 8], pos11 = wpos[w + kW * 8 + 8];
    const uint4 g00 = wgrad[w], g01 = wgrad[w + 8], g10 = wgrad[w + kW * 8], g11 = wgrad[w + kW * 8 + 8];
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    auto take = [&](const uint4& pos, const uint4& g, uint32_t t) {
      const uint32_t me = code(t);
      const uint32_t *pp = &pos.x, *gp = &g.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t m = gp[j] & __heq2_mask(*reinterpret_cast<const __nv_bfloat162*>(&pp[j]), *reinterpret_cast<const __nv_bfloat162*>(&me));
        acc[2 * j] += __uint_as_float(m << 16);
        acc[2 * j + 1] += __uint_as_float(m & 0xffff0000u);
      }
    };
    __nv_bfloat16* ob = (__nv_bfloat16*)p.dx.base + n * p.dx.sn + (long long)y * p.dx.sy + (long long)x * p.dx.sx + (g0 + cg) * 8;
    auto put = [&](__nv_bfloat16* at) {
      uint4* op = (uint4*)at;
      if (p.accumulate) {
        float old[8];
        unpack8(*op, old);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += old[j];
      }
      *op = pack8(acc);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    };
    take(pos00, g00, 8); take(pos01, g01, 6); take(pos10, g10, 2); take(pos11, g11, 0);
    put(ob);
    if (x + 1 < p.W) { take(pos01, g01, 7); take(pos11, g11, 1); put(ob + p.dx.sx); }
    if (y + 1 >= p.H) continue;
    take(pos10, g10, 5); take(pos11, g11, 3);
    put(ob + p.dx.sy);
    if (x + 1 < p.W) { take(pos11, g11, 4); put(ob + p.dx.sy + p.dx.sx); }
  }
}
// windows over a patch of `th` x `tw` pixels, at most
static uint32_t pool_windows(const PoolP& p, uint32_t th, uint32_t tw) {
  const uint32_t mq = (th + p.kh - 2) / p.sh + 1, ms = (tw + p.kw - 2) / p.sw + 1;
  return (mq < p.P ? mq : p.P) * (ms < p.Q ? ms : p.Q);
}
// the tile kernel's limits: positions are bf16 whole numbers, the windows over a patch fit its table
static bool pool_tile_ok(const PoolP& p) {
  if (p.kh > 16 || p.kw > 16 || p.N > 65535) return false;
  return pool_windows(p, kPoolTile, kPoolTile) <= kPoolMaxWin && (p.H + kPoolTile - 1) / kPoolTile <= 65535;
}
template <int K, int S>
static int launch_pool_bwd_tile(const PoolP& p, cudaStream_t s) {
  const uint32_t gchunks = (p.C / 8 + 7) / 8;
  const dim3 grid((p.W + kPoolTile - 1) / kPoolTile * gchunks, (p.H + kPoolTile - 1) / kPoolTile, p.N);
  static unsigned attr_done = 0;       // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_done & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(maxpool_bwd_tile<K, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPoolMaxWin * 256) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    attr_done |= 1u << (dev & 31);
  }
  launch(maxpool_bwd_tile<K, S>, grid, 256, pool_windows(p, kPoolTile, kPoolTile) * 256, s, p, gchunks);
  count_launch();
  return launch_status();
}

// Planes (x fastest): a block owns a 32 x 32 patch of one plane.  Forward: a thread per output.  Backward: first the
// position and the gradient of every window that touches the patch, then every input element gathers.
// 4 x 64 planes of 226 x 226 fp32, 3x3 / 2: forward 41 -> 33 us, gradient 475 -> 94 us.
constexpr uint32_t kPlaneTile = 32, kPlaneMaxWin = 2400;
template <typename T>
__global__ void __launch_bounds__(256) maxpool_fwd_plane(PoolP p) {
  grid_dependency();
  const uint32_t tq = (p.P + 7) / 8, ts = (p.Q + 31) / 32;
  uint32_t r = blockIdx.x;
  const uint32_t s = r % ts * 32 + (threadIdx.x & 31); r /= ts;
  const uint32_t q = r % tq * 8 + (threadIdx.x >> 5); r /= tq;
  const uint32_t c = r % p.C, n = r / p.C;
  if (q >= p.P || s >= p.Q) return;
  const T* xb = (const T*)p.x.base + n * p.x.sn + c * p.x.sc + (long long)(q * p.sh) * p.x.sy + s * p.sw;
  float best = ld_f(xb);
  for (uint32_t a = 0; a < p.kh; ++a)
    for (uint32_t b = 0; b < p.kw; ++b) {
      const float v = ld_f(xb + a * p.x.sy + b);
      if (v > best) best = v;
    }
  st_f((T*)p.y.base + n * p.y.sn + c * p.y.sc + q * p.y.sy + s, best);
}
template <typename T, int K, int S>
__global__ void __launch_bounds__(256) maxpool_bwd_plane(PoolP p) {
  grid_dependency();
  extern __shared__ float2 wpl[];      // per window: position (whole number), gradient
  const uint32_t kh = K ? K : p.kh, kw = K ? K : p.kw, sh = K ? S : p.sh, sw = K ? S : p.sw;
  const uint32_t ty = (p.H + kPlaneTile - 1) / kPlaneTile, tx = (p.W + kPlaneTile - 1) / kPlaneTile;
  uint32_t r = blockIdx.x;
  const uint32_t x0 = r % tx * kPlaneTile; r /= tx;
  const uint32_t y0 = r % ty * kPlaneTile; r /= ty;
  const uint32_t c = r % p.C, n = r / p.C, lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const uint32_t y1 = y0 + kPlaneTile < p.H ? y0 + kPlaneTile : p.H, x1 = x0 + kPlaneTile < p.W ? x0 + kPlaneTile : p.W;
  const uint32_t q_lo = y0 + 1 > kh ? (y0 + 1 - kh + sh - 1) / sh : 0;
  const uint32_t s_lo = x0 + 1 > kw ? (x0 + 1 - kw + sw - 1) / sw : 0;
  const uint32_t q_hi = (y1 - 1) / sh < p.P - 1 ? (y1 - 1) / sh : p.P - 1;   // inclusive
  const uint32_t s_hi = (x1 - 1) / sw < p.Q - 1 ? (x1 - 1) / sw : p.Q - 1;
  const uint32_t nq = q_hi >= q_lo ? q_hi - q_lo + 1 : 0, ns = s_hi >= s_lo ? s_hi - s_lo + 1 : 0;
  const T* xb = (const T*)p.x.base + n * p.x.sn + c * p.x.sc;
  const T* gb = (const T*)p.dy.base + n * p.dy.sn + c * p.dy.sc;
  for (uint32_t wq = row; wq < nq; wq += 8)
    for (uint32_t ws = lane; ws < ns; ws += 32) {
      const uint32_t q = q_lo + wq, s = s_lo + ws;
      const T* xw = xb + (long long)(q * sh) * p.x.sy + s * sw;
      const float g = ld_f(gb + q * p.dy.sy + s);
      uint32_t at = 0;
      if constexpr (K != 0) {
        float v[K * K];
#pragma unroll
        for (int a = 0; a < K; ++a)
#pragma unroll
          for (int b = 0; b < K; ++b) v[a * K + b] = ld_f(xw + a * p.x.sy + b);
        float best = v[0];
#pragma unroll
        for (int t = 1; t < K * K; ++t) if (v[t] > best) { best = v[t]; at = t; }
      } else {
        float best = ld_f(xw);
        for (uint32_t a = 0; a < kh; ++a)
          for (uint32_t b = 0; b < kw; ++b) {
            const float v = ld_f(xw + a * p.x.sy + b);
            if (v > best) { best = v; at = a * kw + b; }
          }
      }
      wpl[wq * ns + ws] = make_float2((float)at, g);
    }
  __syncthreads();
  const uint32_t x = x0 + lane;
  if (x >= x1) return;
  const uint32_t sa = x + 1 > kw ? (x + 1 - kw + sw - 1) / sw : 0;
#pragma unroll 4
  for (uint32_t y = y0 + row; y < y1; y += 8) {
    const uint32_t qa = y + 1 > kh ? (y + 1 - kh + sh - 1) / sh : 0;
    float acc = 0.f;
    for (uint32_t q = qa; q < p.P && q * sh <= y; ++q)
      for (uint32_t s = sa; s < p.Q && s * sw <= x; ++s) {
        const float2 w = wpl[(q - q_lo) * ns + (s - s_lo)];
        if (w.x == (float)((y - q * sh) * kw + (x - s * sw))) acc += w.y;
      }
    T* o = (T*)p.dx.base + n * p.dx.sn + c * p.dx.sc + y * p.dx.sy + x;
    if (p.accumulate) acc += ld_f(o);
    st_f(o, acc);
  }
}
// The plane kernels' limits: contiguous rows, positions exact as floats, the windows over a patch in 19 KB
static bool pool_plane_ok(const PoolP& p, const ad_tensor4* a, const ad_tensor4* b, const ad_tensor4* c, bool bwd) {
  if (a->sx != 1 || b->sx != 1 || (c && c->sx != 1)) return false;
  const unsigned long long planes = (unsigned long long)p.N * p.C;
  if (!bwd) return planes * ((p.P + 7) / 8) * ((p.Q + 31) / 32) < (1ull << 31);
  if (p.kh > 4096 || p.kw > 4096 || pool_windows(p, kPlaneTile, kPlaneTile) > kPlaneMaxWin) return false;
  return planes * ((p.H + kPlaneTile - 1) / kPlaneTile) * ((p.W + kPlaneTile - 1) / kPlaneTile) < (1ull << 31);
}
static bool pool_vec_ok(const ad_tensor4* t) {
  return t->dtype == AD_BF16 && t->sc == 1 && (t->C & 7u) == 0 && !((uintptr_t)t->base & 15u) && !(t->sn & 7) &&
         !(t->sy & 7) && !(t->sx & 7);
}

}  // namespace adk

using namespace adk;

extern "C" size_t ad_bn_scratch_bytes(uint32_t C) { return (size_t)(bn_max_splits(C) + 2) * 2 * C * sizeof(float); }

// y = the normalised x with the statistics a.mean / a.invstd, or the backward pass over them
template <int MODE>
static int launch_apply(const BnApply& a, const ad_tensor4* x, bool vec, bool planes_vec, cudaStream_t s) {
  if (vec) {
    const int rc = MODE == 1 && a.accumulate ? launch_apply_vec<MODE, MODE == 1>(a, s) : launch_apply_vec<MODE, false>(a, s);
    if (rc != AD_OK) return rc;
  } else {
    const size_t total = (size_t)x->N * x->C * x->H * x->W;
    const unsigned long long hw = (unsigned long long)x->H * x->W, chunks = planes_vec ? (hw + kPlaneApplyVec - 1) / kPlaneApplyVec : (hw + kPlaneApply - 1) / kPlaneApply;
    if (total && !a.c_fastest && hw < (1ull << 31) && (unsigned long long)x->N * x->C * chunks < (1ull << 31)) {
      // as many threads per plane as its pixels take, eight (VEC) or four each
      uint32_t shift = 0;
      while (shift < 8 && ((unsigned long long)(planes_vec ? kPlaneApplyVec : kPlaneApply) >> (8 - shift)) < hw) ++shift;
      const unsigned grid = (unsigned)((x->N * x->C * chunks + (256u >> shift) - 1) >> (8 - shift));
      if (planes_vec) launch(bn_apply_planes<float, MODE, true>, grid, 256, 0, s, a, (uint32_t)chunks, shift);
      else AD_DISPATCH_DTYPE(x->dtype, (launch(bn_apply_planes<T, MODE, false>, grid, 256, 0, s, a, (uint32_t)chunks, shift)));
    } else AD_DISPATCH_DTYPE(x->dtype, (launch(bn_apply<T, MODE>, grid_for(total, 256, 16), 256, 0, s, a)));
  }
  count_launch();
  return launch_status();
}

extern "C" int ad_bn_partial_stats(const ad_tensor4* x, float* sums, void* scratch, size_t scratch_bytes, void* stream) {
  if (!x || !x->base || !sums || !scratch) return AD_ERR_BAD_ARG;
  if (scratch_bytes < ad_bn_scratch_bytes(x->C)) return AD_ERR_SCRATCH;
  BnRed p{bview(x), bview(x), x->N, x->C, x->H, x->W, 0, nullptr, nullptr, nullptr, nullptr};
  return launch_reduce<0>(p, x, BnFin{2, x->C, 1.0, 0.f, nullptr, nullptr, nullptr, sums, nullptr, nullptr, 0}, (float*)scratch, as_stream(stream));
}

extern "C" int ad_bn_finalize_apply(const ad_tensor4* x, const ad_tensor4* y, const float* sums, double count,
                                    const float* gamma, const float* beta, float* save_mean, float* save_invstd,
                                    float* batch_var, float eps, int32_t relu, void* stream) {
  if (!x || !y || !x->base || !y->base || !sums || !gamma || !beta || !save_mean || !save_invstd) return AD_ERR_BAD_ARG;
  if (!dims_eq(x, y) || count <= 0.0) return AD_ERR_BAD_ARG;
  cudaStream_t s = as_stream(stream);
  launch_finish(BnFin{0, x->C, count, eps, save_mean, save_invstd, batch_var, nullptr, nullptr, nullptr, 0}, 1, 0, sums, s);
  BnApply a{bview(x), bview(x), bview(y), bview(y), x->N, x->C, x->H, x->W, y->sc == 1 && y->C > 1, relu, 0,
            gamma, beta, save_mean, save_invstd, nullptr, 1, count};
  return launch_apply<0>(a, x, vec_view_ok(x) && vec_view_ok(y), planes_vec_ok(x) && planes_vec_ok(y), s);
}

extern "C" int ad_bn_fwd_train(const ad_tensor4* x, const ad_tensor4* y, const float* gamma, const float* beta,
                               float* save_mean, float* save_invstd, float* batch_var, float eps, int32_t relu,
                               void* scratch, size_t scratch_bytes, void* stream) {
  if (!x || !y || !x->base || !y->base || !gamma || !beta || !save_mean || !save_invstd || !scratch) return AD_ERR_BAD_ARG;
  if (!dims_eq(x, y)) return AD_ERR_BAD_ARG;
  if (scratch_bytes < ad_bn_scratch_bytes(x->C)) return AD_ERR_SCRATCH;
  const size_t total = (size_t)x->N * x->C * x->H * x->W;
  if (total == 0) return AD_OK;
  cudaStream_t s = as_stream(stream);
  BnRed p{bview(x), bview(x), x->N, x->C, x->H, x->W, 0, nullptr, nullptr, nullptr, nullptr};
  const double count = (double)x->N * x->H * x->W;
  int st = launch_reduce<0>(p, x, BnFin{0, x->C, count, eps, save_mean, save_invstd, batch_var, nullptr, nullptr, nullptr, 0}, (float*)scratch, s);
  if (st != AD_OK) return st;
  BnApply a{bview(x), bview(x), bview(y), bview(y), x->N, x->C, x->H, x->W, y->sc == 1 && y->C > 1, relu, 0,
            gamma, beta, save_mean, save_invstd, nullptr, 1, count};
  return launch_apply<0>(a, x, vec_view_ok(x) && vec_view_ok(y), planes_vec_ok(x) && planes_vec_ok(y), s);
}

// invstd[c] = 1 / sqrt(var[c] + eps), in double as the training path does
__global__ void bn_invstd_kernel(uint32_t C, const float* __restrict__ var, float eps, float* __restrict__ invstd) {
  grid_dependency();
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < C) invstd[c] = (float)(1.0 / sqrt((double)var[c] + (double)eps));
}

extern "C" int ad_bn_fwd_inference(const ad_tensor4* x, const ad_tensor4* y, const float* gamma, const float* beta,
                                   const float* mean, const float* var, float* invstd_out, float eps, int32_t relu,
                                   void* stream) {
  if (!x || !y || !x->base || !y->base || !gamma || !beta || !mean || !var || !invstd_out) return AD_ERR_BAD_ARG;
  if (!dims_eq(x, y)) return AD_ERR_BAD_ARG;
  const size_t total = (size_t)x->N * x->C * x->H * x->W;
  if (total == 0) return AD_OK;
  cudaStream_t s = as_stream(stream);
  launch(bn_invstd_kernel, (x->C + 255) / 256, 256, 0, s, x->C, var, eps, invstd_out);
  count_launch();
  BnApply a{bview(x), bview(x), bview(y), bview(y), x->N, x->C, x->H, x->W, y->sc == 1 && y->C > 1, relu, 0,
            gamma, beta, mean, invstd_out, nullptr, 1, (double)x->N * x->H * x->W};
  return launch_apply<0>(a, x, vec_view_ok(x) && vec_view_ok(y), planes_vec_ok(x) && planes_vec_ok(y), s);
}

extern "C" int ad_bn_bwd_add(const ad_tensor4* x, const ad_tensor4* dy, const ad_tensor4* addend, const ad_tensor4* dx, const float* gamma,
                             const float* beta, const float* save_mean, const float* save_invstd, float* dgamma,
                             float* dbeta, int32_t relu, int32_t accumulate_params, void* scratch, size_t scratch_bytes,
                             void* stream) {
  if (!x || !dy || !dx || !x->base || !dy->base || !dx->base || !gamma || !beta || !save_mean || !save_invstd || !scratch)
    return AD_ERR_BAD_ARG;
  if (addend && !addend->base) return AD_ERR_BAD_ARG;
  if (!dims_eq(x, dy) || !dims_eq(x, dx) || (addend && !dims_eq(x, addend))) return AD_ERR_BAD_ARG;
  if (scratch_bytes < ad_bn_scratch_bytes(x->C)) return AD_ERR_SCRATCH;
  const size_t total = (size_t)x->N * x->C * x->H * x->W;
  if (total == 0) return AD_OK;
  cudaStream_t s = as_stream(stream);
  BnRed p{bview(x), bview(dy), x->N, x->C, x->H, x->W, relu, gamma, beta, save_mean, save_invstd};
  float* partial = (float*)scratch;
  float* sums = partial + (size_t)bn_max_splits(x->C) * 2 * x->C;
  const double count = (double)x->N * x->H * x->W;
  int st = launch_reduce<1>(p, x, BnFin{1, x->C, count, 0.f, nullptr, nullptr, nullptr, sums, dgamma, dbeta, accumulate_params}, partial, s, planes_vec_ok(x) && planes_vec_ok(dy));
  if (st != AD_OK) return st;
  BnApply a{bview(x), bview(dy), bview(dx), bview(addend ? addend : dx), x->N, x->C, x->H, x->W, dx->sc == 1 && dx->C > 1, relu, addend != nullptr,
            gamma, beta, save_mean, save_invstd, sums, 1, count};
  return launch_apply<1>(a, x, vec_view_ok(x) && vec_view_ok(dy) && vec_view_ok(dx) && (!addend || vec_view_ok(addend)),
                         planes_vec_ok(x) && planes_vec_ok(dy) && planes_vec_ok(dx) && (!addend || planes_vec_ok(addend)), s);
}

extern "C" int ad_bn_bwd(const ad_tensor4* x, const ad_tensor4* dy, const ad_tensor4* dx, const float* gamma,
                         const float* beta, const float* save_mean, const float* save_invstd, float* dgamma,
                         float* dbeta, int32_t relu, int32_t accumulate_dx, void* scratch, size_t scratch_bytes,
                         void* stream) {
  return ad_bn_bwd_add(x, dy, accumulate_dx ? dx : nullptr, dx, gamma, beta, save_mean, save_invstd, dgamma, dbeta, relu, 1, scratch, scratch_bytes,
                       stream);
}

static int pool_params(const ad_tensor4* x, const ad_tensor4* y, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw,
                       PoolP& p) {
  if (!x || !y || !x->base || !y->base || kh == 0 || kw == 0 || sh == 0 || sw == 0) return AD_ERR_BAD_ARG;
  if (x->H < kh || x->W < kw) return AD_ERR_BAD_ARG;
  const uint32_t P = (x->H - kh) / sh + 1, Q = (x->W - kw) / sw + 1;
  if (y->N != x->N || y->C != x->C || y->H != P || y->W != Q || y->dtype != x->dtype) return AD_ERR_BAD_ARG;
  p.x = bview(x);
  p.N = x->N; p.C = x->C; p.H = x->H; p.W = x->W; p.P = P; p.Q = Q;
  p.kh = kh; p.kw = kw; p.sh = sh; p.sw = sw;
  return AD_OK;
}

extern "C" int ad_maxpool2d_fwd(const ad_tensor4* x, const ad_tensor4* y, uint32_t kh, uint32_t kw, uint32_t sh,
                                uint32_t sw, void* stream) {
  PoolP p{};
  int st = pool_params(x, y, kh, kw, sh, sw, p);
  if (st != AD_OK) return st;
  p.y = bview(y);
  p.c_fastest = y->sc == 1 && y->C > 1;
  const size_t total = (size_t)p.N * p.C * p.P * p.Q;
  if (total == 0) return AD_OK;
  cudaStream_t cs = as_stream(stream);
  if (pool_vec_ok(x) && pool_vec_ok(y)) {
    if (kh == 3 && kw == 3) launch(maxpool_fwd_vec<3>, grid_for(total / 8, 256, 16), 256, 0, cs, p);
    else if (kh == 2 && kw == 2) launch(maxpool_fwd_vec<2>, grid_for(total / 8, 256, 16), 256, 0, cs, p);
    else launch(maxpool_fwd_vec<0>, grid_for(total / 8, 256, 16), 256, 0, cs, p);
  } else if (pool_plane_ok(p, x, y, nullptr, false)) {
    const unsigned grid = (unsigned)((size_t)p.N * p.C * ((p.P + 7) / 8) * ((p.Q + 31) / 32));
    AD_DISPATCH_DTYPE(x->dtype, (launch(maxpool_fwd_plane<T>, grid, 256, 0, cs, p)));
  } else AD_DISPATCH_DTYPE(x->dtype, (launch(maxpool_fwd_kernel<T>, grid_for(total, 256, 16), 256, 0, as_stream(stream), p)));
  count_launch();
  return launch_status();
}

extern "C" int ad_maxpool2d_bwd(const ad_tensor4* x, const ad_tensor4* dy, const ad_tensor4* dx, uint32_t kh,
                                uint32_t kw, uint32_t sh, uint32_t sw, int32_t accumulate, void* stream) {
  PoolP p{};
  int st = pool_params(x, dy, kh, kw, sh, sw, p);
  if (st != AD_OK) return st;
  if (!dx || !dx->base || dx->N != x->N || dx->C != x->C || dx->H != x->H || dx->W != x->W || dx->dtype != x->dtype)
    return AD_ERR_BAD_ARG;
  p.dy = bview(dy);
  p.dx = bview(dx);
  p.c_fastest = dx->sc == 1 && dx->C > 1;
  p.accumulate = accumulate;
  const size_t total = (size_t)p.N * p.C * p.H * p.W;
  if (total == 0) return AD_OK;
  cudaStream_t cs = as_stream(stream);
  const bool vec = pool_vec_ok(x) && pool_vec_ok(dy) && pool_vec_ok(dx);
  if (vec && pool_tile_ok(p)) {
    if (kh == 3 && kw == 3 && sh == 2 && sw == 2) {
      const uint32_t gchunks = (p.C / 8 + 7) / 8;
      launch(maxpool_bwd_quads, dim3((p.W + kPoolTile - 1) / kPoolTile * gchunks, (p.H + kPoolTile - 1) / kPoolTile, p.N), 256, 0, cs, p, gchunks);
      count_launch();
      return launch_status();
    }
    if (kh == 3 && kw == 3 && sh == 1 && sw == 1) return launch_pool_bwd_tile<3, 1>(p, cs);
    if (kh == 2 && kw == 2 && sh == 2 && sw == 2) return launch_pool_bwd_tile<2, 2>(p, cs);
    return launch_pool_bwd_tile<0, 0>(p, cs);
  }
  if (vec) launch(maxpool_bwd_vec, grid_for(total / 8, 256, 16), 256, 0, cs, p);
  else if (pool_plane_ok(p, x, dy, dx, true)) {
    const unsigned grid = (unsigned)((size_t)p.N * p.C * ((p.H + kPlaneTile - 1) / kPlaneTile) * ((p.W + kPlaneTile - 1) / kPlaneTile));
    const size_t smem = pool_windows(p, kPlaneTile, kPlaneTile) * sizeof(float2);
    if (kh == 3 && kw == 3 && sh == 2 && sw == 2) AD_DISPATCH_DTYPE(x->dtype, (launch(maxpool_bwd_plane<T, 3, 2>, grid, 256, smem, cs, p)));
    else AD_DISPATCH_DTYPE(x->dtype, (launch(maxpool_bwd_plane<T, 0, 0>, grid, 256, smem, cs, p)));
  }
  else AD_DISPATCH_DTYPE(x->dtype, (launch(maxpool_bwd_kernel<T>, grid_for(total, 256, 16), 256, 0, cs, p)));
  count_launch();
  return launch_status();
}

// ------------------------------------------------------------------ allocation-free variant
// Some callers of this library are not in a position to allocate device memory for the
// statistics scratch: an op body running inside a host framework that has handed the whole
// device to its own memory pool, or a latency-critical loop in which cudaMalloc (which may
// synchronise the device) must not appear.  For them the scratch of the batch-norm forward
// lives in this file-scope device array, sized for at most kBnStaticMaxC channels.  The array
// exists once per GPU that loads the library and is held until the process exits.
constexpr uint32_t kBnStaticMaxC = 2048;
constexpr size_t kBnStaticBytes = (size_t)(adk::kBnMaxSplits + 1) * 2 * kBnStaticMaxC * sizeof(float);
static __device__ __align__(256) unsigned char g_bn_static_scratch[kBnStaticBytes];

// In host code the array's name is only a handle for the runtime, never a device address:
// the address has to be asked for, once per device, with that device current.
// The per-device cache is a table of atomics: host threads that make the first call on one device at the
// same time each look the symbol up and store the same value; none can read a half-written pointer.
static int bn_static_scratch_address(void** out) {
  constexpr int kMaxDevices = 64;
  static std::atomic<void*> addr[kMaxDevices];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) { cudaGetLastError(); return AD_ERR_CUDA; }
  void* p = addr[dev].load(std::memory_order_acquire);
  if (!p) {
    if (cudaGetSymbolAddress(&p, g_bn_static_scratch) != cudaSuccess || !p) { cudaGetLastError(); return AD_ERR_CUDA; }
    addr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return AD_OK;
}

extern "C" int ad_bn_fwd_train_noalloc(const ad_tensor4* x, const ad_tensor4* y, const float* gamma, const float* beta,
                                       float* save_mean, float* save_invstd, float* batch_var, float eps, int32_t relu,
                                       void* stream) {
  if (!x) return AD_ERR_BAD_ARG;
  if (x->C > kBnStaticMaxC) return AD_ERR_LIMIT;  // more channels than the built-in scratch holds
  void* scratch = nullptr;
  int st = bn_static_scratch_address(&scratch);
  if (st != AD_OK) return st;
  // Every word of the scratch that the kernels read is written earlier in the same call, so
  // nothing has to be cleared even though the array keeps the previous call's contents.
  return ad_bn_fwd_train(x, y, gamma, beta, save_mean, save_invstd, batch_var, eps, relu, scratch, kBnStaticBytes, stream);
}
