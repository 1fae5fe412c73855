// Bilinear x`scale` upsample (half-pixel centres, edges clamped) of a strip of a 4-D tensor and its
// gradient, on strided views.  The reference has no such operator; it is the segmentation head of the
// 1024x2048 configuration (logits at 1/8 resolution -> full resolution before the per-pixel loss).
//
// Strip form: the views hold rows [x_row0, x_row0 + x.H) of an input whose full height is in_rows_total
// and rows [y_row0, y_row0 + y.H) of the upsampled output; source rows are computed in global
// coordinates, so a strip with one halo row on each inner edge gives exactly the rows of the
// unpartitioned result.  HBM-bound: the output is scale^2 times the input.
#include <algorithm>

#include "common.cuh"

namespace adk {

struct UpView { char* base; long long sn, sc, sy, sx; };
static UpView upview(const ad_tensor4* t) { return UpView{(char*)t->base, t->sn, t->sc, t->sy, t->sx}; }

struct UpP {
  UpView x, y;            // x: low-resolution side, y: high-resolution side
  uint32_t N, C, XH, XW, YH, YW, scale;
  int32_t x_row0;
  uint32_t in_rows_total, y_row0;
  int c_fastest, accumulate;
};

// source cell pair and weight for output index o (global), as torch's align_corners = false
__device__ __forceinline__ void bilin_src(uint32_t o, float inv_scale, uint32_t in_size, int& i0, int& i1, float& f) {
  float src = ((float)o + 0.5f) * inv_scale - 0.5f;
  if (src < 0.f) src = 0.f;
  int a = (int)floorf(src);
  if (a > (int)in_size - 1) a = (int)in_size - 1;
  i0 = a;
  i1 = a + 1 < (int)in_size ? a + 1 : (int)in_size - 1;
  f = src - (float)a;
}

template <typename T>
__global__ void __launch_bounds__(256) upsample_fwd_kernel(UpP p) {
  grid_dependency();
  const uint32_t total = p.N * p.C * p.YH * p.YW, nt = gridDim.x * blockDim.x;
  const float inv = 1.0f / (float)p.scale;
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {   // past 2^32 on the last step
    uint32_t n, c, oy, ox, r = (uint32_t)i;
    if (p.c_fastest) { c = r % p.C; r /= p.C; ox = r % p.YW; r /= p.YW; oy = r % p.YH; n = r / p.YH; }
    else { ox = r % p.YW; r /= p.YW; oy = r % p.YH; r /= p.YH; c = r % p.C; n = r / p.C; }
    int y0, y1, x0, x1;
    float fy, fx;
    bilin_src(p.y_row0 + oy, inv, p.in_rows_total, y0, y1, fy);
    bilin_src(ox, inv, p.XW, x0, x1, fx);
    y0 -= p.x_row0; y1 -= p.x_row0;
    const T* X = (const T*)p.x.base + n * p.x.sn + c * p.x.sc;
    const float a = ld_f(X + y0 * p.x.sy + x0 * p.x.sx), b = ld_f(X + y0 * p.x.sy + x1 * p.x.sx);
    const float d = ld_f(X + y1 * p.x.sy + x0 * p.x.sx), e = ld_f(X + y1 * p.x.sy + x1 * p.x.sx);
    const float v = (1.f - fy) * ((1.f - fx) * a + fx * b) + fy * ((1.f - fx) * d + fx * e);
    st_f((T*)p.y.base + n * p.y.sn + c * p.y.sc + oy * p.y.sy + ox * p.y.sx, v);
  }
}

// Gather form of the gradient: one thread per low-resolution element sums, in a fixed order, the
// high-resolution gradients whose source pair contains it -- no atomics, reproducible.
template <typename T>
__global__ void __launch_bounds__(256) upsample_bwd_kernel(UpP p) {
  grid_dependency();
  const uint32_t total = p.N * p.C * p.XH * p.XW, nt = gridDim.x * blockDim.x;
  const float inv = 1.0f / (float)p.scale;
  const int s = (int)p.scale;
  for (size_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {   // past 2^32 on the last step
    uint32_t n, c, yl, xl, r = (uint32_t)i;
    if (p.c_fastest) { c = r % p.C; r /= p.C; xl = r % p.XW; r /= p.XW; yl = r % p.XH; n = r / p.XH; }
    else { xl = r % p.XW; r /= p.XW; yl = r % p.XH; r /= p.XH; c = r % p.C; n = r / p.C; }
    const int yg = (int)yl + p.x_row0, xg = (int)xl;
    float acc = 0.f;
    if (yg >= 0 && yg < (int)p.in_rows_total) {
      // candidates: outputs whose source coordinate lies in (g - 1, g + 1); edge cells also take the clamped ones
      int oy_lo = yg == 0 ? 0 : (yg - 1) * s, oy_hi = yg == (int)p.in_rows_total - 1 ? (int)p.in_rows_total * s - 1 : (yg + 2) * s - 1;
      int ox_lo = xg == 0 ? 0 : (xg - 1) * s, ox_hi = xg == (int)p.XW - 1 ? (int)p.XW * s - 1 : (xg + 2) * s - 1;
      if (oy_lo < (int)p.y_row0) oy_lo = (int)p.y_row0;
      if (oy_hi > (int)(p.y_row0 + p.YH) - 1) oy_hi = (int)(p.y_row0 + p.YH) - 1;
      const T* G = (const T*)p.y.base + n * p.y.sn + c * p.y.sc;
      for (int oy = oy_lo; oy <= oy_hi; ++oy) {
        int y0, y1;
        float fy;
        bilin_src((uint32_t)oy, inv, p.in_rows_total, y0, y1, fy);
        const float wy = (y0 == yg ? 1.f - fy : 0.f) + (y1 == yg ? fy : 0.f);
        if (wy == 0.f) continue;
        float row = 0.f;
        for (int ox = ox_lo; ox <= ox_hi; ++ox) {
          int x0, x1;
          float fx;
          bilin_src((uint32_t)ox, inv, p.XW, x0, x1, fx);
          const float wx = (x0 == xg ? 1.f - fx : 0.f) + (x1 == xg ? fx : 0.f);
          if (wx != 0.f) row = fmaf(wx, ld_f(G + (oy - (int)p.y_row0) * p.y.sy + ox * p.y.sx), row);
        }
        acc = fmaf(wy, row, acc);
      }
    }
    T* o = (T*)p.x.base + n * p.x.sn + c * p.x.sc + yl * p.x.sy + xl * p.x.sx;
    st_f(o, p.accumulate ? ld_f(o) + acc : acc);
  }
}

// ------------------------------------------------------------------ row kernels
// Views whose rows are contiguous (x fastest, or channel fastest with packed pixels) are rows of W * Ci elements, Ci = C
// or 1 channels interleaved and the other planes outside.  The bound is HBM: the high-resolution side, once.
//   forward   a block blends the two low-resolution rows behind an output row into shared memory (fp32) and then writes
//             the row in pairs of elements, each a blend of two shared-memory values: two multiply-adds and no global read
//             per element.  (Eight elements per thread would save index arithmetic, but put the lanes' shared-memory reads
//             eight words apart: 172 us instead of 95.)
//   gradient  a thread owns a 16-byte vector of columns and sums it down the 2 * scale output rows that meet the
//             low-resolution row (coalesced reads, weights by row), into shared memory; each low-resolution element then
//             sums its 2 * scale columns there.  Every output row is read by two blocks, the second time from L2.
// Both cut wide rows into chunks of low-resolution columns that fit the shared memory.
// 2 x 19 x 128 x 256 bf16, x 8: forward 434 -> 95 us (by cells, below: 32), gradient 355 -> 57 us (159 MB of logits: 24 us at the copy rate).
struct UpRowP {
  UpP u;
  uint32_t Ci, planes;    // interleaved channels; N * C / Ci outer planes
  uint32_t XC, chunks;    // low-resolution columns per block
  uint32_t rb, tpr;       // forward: output rows per block, threads per row
  uint32_t wtab;          // gradient: where the weight table lies in shared memory (floats)
  uint32_t smem;          // bytes of dynamic shared memory
  uint32_t row_len;       // elements of a high-resolution row
  int vec;                // high-resolution rows start on the boundaries of the vectors
  uint32_t period;        // forward: pairs of outputs per low-resolution column (0: the general form)
  uint32_t cell0, cells;  // forward by cells: the first row of cells (between two source rows) that the strip meets, their number
};
constexpr uint32_t kUpThreads = 256, kUpFloats = 5120;    // 20 KB of rows per block where that holds three columns: 8 blocks per SM
constexpr uint32_t kUpFloatsMax = 12000;

template <typename T> __device__ __forceinline__ void st_pair(T* p, float a, float b);
template <> __device__ __forceinline__ void st_pair<float>(float* p, float a, float b) { *(float2*)p = make_float2(a, b); }
template <> __device__ __forceinline__ void st_pair<__nv_bfloat16>(__nv_bfloat16* p, float a, float b) { *(__nv_bfloat162*)p = __floats2bfloat162_rn(a, b); }
template <typename T> __device__ __forceinline__ void ld_vec(const T* p, float (&v)[16 / sizeof(T)]);
template <> __device__ __forceinline__ void ld_vec<float>(const float* p, float (&v)[4]) {
  const float4 q = *(const float4*)p;
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template <> __device__ __forceinline__ void ld_vec<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 q = *(const uint4*)p;
  const __nv_bfloat162* h = (const __nv_bfloat162*)&q;
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 t = __bfloat1622float2(h[j]); v[2 * j] = t.x; v[2 * j + 1] = t.y; }
}
__device__ __forceinline__ long long plane_off(const UpView& v, uint32_t plane, uint32_t per_n) {
  const uint32_t n = plane / per_n, c = plane - n * per_n;
  return (long long)n * v.sn + (long long)c * v.sc;
}

template <typename T>
__global__ void __launch_bounds__(kUpThreads) upsample_fwd_rows(UpRowP p) {
  grid_dependency();
  extern __shared__ __align__(16) float L[];   // [rb][XC + 2 low-resolution columns, clamped to the image][Ci]
  const UpP& u = p.u;
  const float inv = 1.0f / (float)u.scale;
  const uint32_t chunk = blockIdx.x % p.chunks, xa = chunk * p.XC, xb = xa + p.XC < u.XW ? xa + p.XC : u.XW;
  const uint32_t lo = xa > 0 ? xa - 1 : 0, hi = xb < u.XW ? xb + 1 : u.XW, cols = (hi - lo) * p.Ci, pitch = (p.XC + 2) * p.Ci;
  const uint32_t row0 = blockIdx.x / p.chunks * p.rb, rows_total = p.planes * u.YH;
  const uint32_t nr = rows_total - row0 < p.rb ? rows_total - row0 : p.rb, per_n = u.C / p.Ci;
  for (uint32_t r = 0; r < nr; ++r) {
    const uint32_t oy = (row0 + r) % u.YH, plane = (row0 + r) / u.YH;
    int y0, y1;
    float fy;
    bilin_src(u.y_row0 + oy, inv, u.in_rows_total, y0, y1, fy);
    const T* X = (const T*)u.x.base + plane_off(u.x, plane, per_n) + (long long)lo * p.Ci;
    const T *X0 = X + (y0 - u.x_row0) * u.x.sy, *X1 = X + (y1 - u.x_row0) * u.x.sy;
    // one column of zeros past the last: the right edge blends it with weight 0 (an infinity there, times 0, would be NaN).  Only the
    // chunk that holds the last column has room for it: a chunk that ends one before reads all of its row
    for (uint32_t i = threadIdx.x; i < cols; i += kUpThreads) L[r * pitch + i] = (1.f - fy) * ld_f(X0 + i) + fy * ld_f(X1 + i);
    if (xb == u.XW)
      for (uint32_t i = threadIdx.x; i < p.Ci; i += kUpThreads) L[r * pitch + cols + i] = 0.f;
  }
  int2* tab = (int2*)(L + (((size_t)p.rb * pitch + 1) & ~(size_t)1));   // per output column: where its left source column lies, weight of the right one
  const uint32_t oxa = xa * u.scale, oxb = xb * u.scale;
  for (uint32_t i = threadIdx.x; i < oxb - oxa; i += kUpThreads) {
    int x0, x1;
    float fx;
    bilin_src(oxa + i, inv, u.XW, x0, x1, fx);
    tab[i] = make_int2((int)(((uint32_t)x0 - lo) * p.Ci), __float_as_int(x1 == x0 ? 0.f : fx));
  }
  __syncthreads();
  // pairs of neighbouring elements: a warp writes 64 of them in one run, and its shared-memory reads lie side by side
  const uint32_t e0 = xa * u.scale * p.Ci, e1 = xb * u.scale * p.Ci, v0 = e0 / 2, nv = (e1 + 1) / 2 - v0;
  const uint32_t step_x = 2 * p.tpr / p.Ci, step_c = 2 * p.tpr % p.Ci;
  for (uint32_t r = threadIdx.x / p.tpr; r < nr; r += kUpThreads / p.tpr) {
    const uint32_t oy = (row0 + r) % u.YH, plane = (row0 + r) / u.YH;
    const float* Lr = L + r * pitch;
    T* o = (T*)u.y.base + plane_off(u.y, plane, per_n) + (long long)oy * u.y.sy;
    uint32_t i = threadIdx.x % p.tpr, e = (v0 + i) * 2, ox = e / p.Ci, c = e - ox * p.Ci;
    for (; i < nv; i += p.tpr) {
      // an element outside the chunk (an odd end) is computed from the nearest column and not written
      const uint32_t c1 = c + 1 == p.Ci ? 0 : c + 1, ox1 = c + 1 == p.Ci ? ox + 1 : ox;
      const int2 t0 = tab[ox < oxa ? 0 : ox - oxa], t1 = tab[(ox1 < oxb ? ox1 : oxb - 1) - oxa];
      const float f0 = __int_as_float(t0.y), f1 = __int_as_float(t1.y);
      const float *a0 = Lr + t0.x + c, *a1 = Lr + t1.x + c1;
      const float v = (1.f - f0) * a0[0] + f0 * a0[p.Ci], w = (1.f - f1) * a1[0] + f1 * a1[p.Ci];
      if (p.vec && e >= e0 && e + 2 <= e1) st_pair<T>(o + e, v, w);
      else {
        if (e >= e0 && e < e1) st_f(o + e, v);
        if (e + 1 >= e0 && e + 1 < e1) st_f(o + e + 1, w);
      }
      e += 2 * p.tpr; ox += step_x; c += step_c;
      if (c >= p.Ci) { c -= p.Ci; ++ox; }
    }
  }
}

// Forward, scale a power of two (S, 0: at run time): the output rows between two neighbouring source rows, scale of them, are
// blends of the same two blended rows, and the pairs of one source column's outputs, scale * Ci / 2 of them, recur from column
// to column with the same channels and exactly the same weights.  A block takes such a cell of rows and some columns, a thread
// stays with its pair and steps over columns: 8 reads of shared memory and 8 FMAs for the two blends, then two FMAs, a
// conversion and a store per pair and row.  Bound by instructions before (a table of columns and weights, a row per block: 99
// us and 92 M; pairs with a row per block 55 us and 49 M), by the stores now: 2 x 19 x 128 x 256 x 8 bf16
// 32 us (25 at the copy rate), 2 x 19 x 64 x 128 x 8 fp32, whose planes took the table, 60 -> 16.
template <typename T, int S>
__global__ void __launch_bounds__(kUpThreads) upsample_fwd_cells(UpRowP p) {
  grid_dependency();
  extern __shared__ __align__(16) float L[];   // [2 source rows][XC + 2 columns, clamped to the image][Ci], weights of the cell's rows
  const UpP& u = p.u;
  const int s = S ? S : (int)u.scale;
  const float inv = 1.0f / (float)s;
  const uint32_t chunk = blockIdx.x % p.chunks, at = blockIdx.x / p.chunks, plane = at / p.cells, cell = p.cell0 + at % p.cells;
  const uint32_t xa = chunk * p.XC, xb = xa + p.XC < u.XW ? xa + p.XC : u.XW;
  const uint32_t lo = xa > 0 ? xa - 1 : 0, hi = xb < u.XW ? xb + 1 : u.XW, cols = (hi - lo) * p.Ci, pitch = (p.XC + 2) * p.Ci, Ci = p.Ci;
  // rows ra .. rb - 1 of the cell's s lie in this strip
  const int oy0 = (int)cell * s - s / 2, first = (int)u.y_row0, last_y = (int)(u.y_row0 + u.YH);
  const int ra = oy0 < first ? first - oy0 : 0, rb = oy0 + s > last_y ? last_y - oy0 : s;
  int y0, y1;
  float fy;
  bilin_src((uint32_t)(oy0 + ra), inv, u.in_rows_total, y0, y1, fy);   // the same two rows for the whole cell
  const uint32_t per_n = u.C / Ci;
  const T* X = (const T*)u.x.base + plane_off(u.x, plane, per_n) + (long long)lo * Ci;
  const T *X0 = X + (y0 - u.x_row0) * u.x.sy, *X1 = X + (y1 - u.x_row0) * u.x.sy;
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < cols; i += kUpThreads) { L[i] = ld_f(X0 + i); L[pitch + i] = ld_f(X1 + i); }
  if (xb == u.XW)   // a column of zeros past the last: the right edge blends it with weight 0 (an infinity there, times 0, would be NaN)
    for (uint32_t i = threadIdx.x; i < Ci; i += kUpThreads) L[cols + i] = L[pitch + cols + i] = 0.f;
  float* const W = L + 2 * pitch;
  if ((int)threadIdx.x >= ra && (int)threadIdx.x < rb) {
    bilin_src((uint32_t)(oy0 + (int)threadIdx.x), inv, u.in_rows_total, y0, y1, fy);
    W[threadIdx.x] = fy;
  }
  __syncthreads();
  const uint32_t m = kUpThreads / p.period, k0 = threadIdx.x / p.period, e = threadIdx.x % p.period * 2;
  if (k0 >= m) return;
  const uint32_t ph0 = e / Ci, c0 = e - ph0 * Ci, ph1 = (e + 1) / Ci, c1 = e + 1 - ph1 * Ci;
  const int d0 = 2 * (int)ph0 < s ? -1 : 0, d1 = 2 * (int)ph1 < s ? -1 : 0;
  const float f0 = ((float)ph0 + 0.5f) * inv - 0.5f - (float)d0, f1 = ((float)ph1 + 0.5f) * inv - 0.5f - (float)d1;
  const float g0 = 1.f - f0, g1 = 1.f - f1;
  const uint32_t hop = m * Ci, ohop = hop * (uint32_t)s;
  const long long sy = u.y.sy;
  T* o = (T*)u.y.base + plane_off(u.y, plane, per_n) + (long long)(oy0 - first) * sy + (long long)(xa + k0) * s * Ci + e;
  const float *a0 = L + (int)(xa + k0 - lo + d0) * (int)Ci + (int)c0, *a1 = L + (int)(xa + k0 - lo + d1) * (int)Ci + (int)c1;
  uint32_t x = xa + k0;
  auto edge = [&] {   // left of the first or right of the last column: that column's value, weight 0 on its neighbour
    const int x0 = (int)x + d0, x1 = (int)x + d1, last = (int)u.XW - 1;
    const float h0 = x0 < 0 || x0 >= last ? 0.f : f0, h1 = x1 < 0 || x1 >= last ? 0.f : f1;
    const float *b0 = x0 < 0 ? a0 + Ci : a0, *b1 = x1 < 0 ? a1 + Ci : a1;
    const float t0 = (1.f - h0) * b0[0] + h0 * b0[Ci], t1 = (1.f - h1) * b1[0] + h1 * b1[Ci];
    const float v0 = (1.f - h0) * b0[pitch] + h0 * b0[pitch + Ci], v1 = (1.f - h1) * b1[pitch] + h1 * b1[pitch + Ci];
    for (int r = ra; r < rb; ++r) {
      const float w = W[r];
      st_f(o + r * sy, (1.f - w) * t0 + w * v0);
      st_f(o + r * sy + 1, (1.f - w) * t1 + w * v1);
    }
  };
  auto next = [&] { x += m; a0 += hop; a1 += hop; o += ohop; };
  if (x == 0 && x < xb) { edge(); next(); }
  const uint32_t xe = xb == u.XW ? xb - 1 : xb;
  auto blends = [&](float& t0, float& t1, float& v0, float& v1) {
    t0 = g0 * a0[0] + f0 * a0[Ci]; t1 = g1 * a1[0] + f1 * a1[Ci];
    v0 = g0 * a0[pitch] + f0 * a0[pitch + Ci]; v1 = g1 * a1[pitch] + f1 * a1[pitch + Ci];
  };
  if (S && p.vec && ra == 0 && rb == s) {
    float w[S ? S : 1], q[S ? S : 1];
#pragma unroll
    for (int r = 0; r < S; ++r) { w[r] = W[r]; q[r] = 1.f - w[r]; }
#pragma unroll 2
    for (; x < xe; next()) {
      float t0, t1, v0, v1;
      blends(t0, t1, v0, v1);
      T* or_ = o;
#pragma unroll
      for (int r = 0; r < S; ++r, or_ += sy) st_pair<T>(or_, q[r] * t0 + w[r] * v0, q[r] * t1 + w[r] * v1);
    }
  } else {
    for (; x < xe; next()) {
      float t0, t1, v0, v1;
      blends(t0, t1, v0, v1);
      for (int r = ra; r < rb; ++r) {
        const float w = W[r], a = (1.f - w) * t0 + w * v0, b = (1.f - w) * t1 + w * v1;
        if (p.vec) st_pair<T>(o + r * sy, a, b);
        else { st_f(o + r * sy, a); st_f(o + r * sy + 1, b); }
      }
    }
  }
  if (x < xb) edge();
}

template <typename T>
__global__ void __launch_bounds__(kUpThreads) upsample_bwd_rows(UpRowP p) {
  grid_dependency();
  extern __shared__ __align__(16) float S[];   // column sums of the chunk's output columns (and one low-resolution column either side)
  constexpr uint32_t V = 16 / sizeof(T);
  const UpP& u = p.u;
  const int s = (int)u.scale;
  const float inv = 1.0f / (float)s;
  const uint32_t chunk = blockIdx.x % p.chunks, row = blockIdx.x / p.chunks, yl = row % u.XH, plane = row / u.XH, per_n = u.C / p.Ci;
  const uint32_t xa = chunk * p.XC, xb = xa + p.XC < u.XW ? xa + p.XC : u.XW;
  const uint32_t oxa = xa > 0 ? (xa - 1) * s : 0, oxb = xb < u.XW ? (xb + 1) * s : u.XW * s;
  const int yg = (int)yl + u.x_row0;
  int oy_lo = 0, oy_hi = -1;
  if (yg >= 0 && yg < (int)u.in_rows_total) {
    // outputs whose source coordinate lies in (g - 1, g + 1); edge cells also take the clamped ones.  At an odd scale the
    // outputs at g - 1 and g + 1 have no part in g: an infinite gradient there must not meet a weight of 0.
    oy_lo = yg == 0 ? 0 : (yg - 1) * s + (s + 1) / 2;
    oy_hi = yg == (int)u.in_rows_total - 1 ? (int)u.in_rows_total * s - 1 : (yg + 1) * s + s / 2 - 1;
    if (oy_lo < (int)u.y_row0) oy_lo = (int)u.y_row0;
    if (oy_hi > (int)(u.y_row0 + u.YH) - 1) oy_hi = (int)(u.y_row0 + u.YH) - 1;
  }
  const T* G = (const T*)u.y.base + plane_off(u.y, plane, per_n);
  const uint32_t e0 = oxa * p.Ci, e1 = oxb * p.Ci, v0 = e0 / V, nv = (e1 + V - 1) / V - v0;
  // weights of the output rows, and of the output columns (xg - 1) * s + (s + 1) / 2 + t around a column xg away from the edges
  float* const wyt = S + p.wtab;
  for (int oy = oy_lo + (int)threadIdx.x; oy <= oy_hi; oy += kUpThreads) {
    int y0, y1;
    float fy;
    bilin_src((uint32_t)oy, inv, u.in_rows_total, y0, y1, fy);
    wyt[oy - oy_lo] = (y0 == yg ? 1.f - fy : 0.f) + (y1 == yg ? fy : 0.f);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nv; i += kUpThreads) {
    const uint32_t e = (v0 + i) * V;
    float acc[V];
#pragma unroll
    for (uint32_t j = 0; j < V; ++j) acc[j] = 0.f;
    const bool full = p.vec && e + V <= p.row_len;
    const T* g = G + (long long)(oy_lo - (int)u.y_row0) * u.y.sy + e;
    const int n = oy_hi - oy_lo + 1;
    if (full) {
#pragma unroll 8
      for (int k = 0; k < n; ++k, g += u.y.sy) {
        float v[V];
        ld_vec<T>(g, v);
        const float wy = wyt[k];
#pragma unroll
        for (uint32_t j = 0; j < V; ++j) acc[j] = fmaf(wy, v[j], acc[j]);
      }
    } else {
      for (int k = 0; k < n; ++k, g += u.y.sy)
#pragma unroll
        for (uint32_t j = 0; j < V; ++j)
          if (e + j < p.row_len) acc[j] = fmaf(wyt[k], ld_f(g + j), acc[j]);
    }
#pragma unroll
    for (uint32_t j = 0; j < V; j += 4) *(float4*)&S[i * V + j] = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
  }
  __syncthreads();
  // the column weights take the place of the row weights
  const int nt = 2 * s + s / 2 - (s + 1) / 2;          // outputs that an inner column has a part in
  for (int t = (int)threadIdx.x; t < nt; t += kUpThreads) {
    int x0, x1;
    float fx;
    bilin_src((uint32_t)((s + 1) / 2 + t), inv, 1u << 20, x0, x1, fx);      // around column 1 of a wide row
    wyt[t] = (x0 == 1 ? 1.f - fx : 0.f) + (x1 == 1 ? fx : 0.f);
  }
  __syncthreads();
  T* O = (T*)u.x.base + plane_off(u.x, plane, per_n) + (long long)yl * u.x.sy;
  const float* Sr = S + (e0 - v0 * V);
  for (uint32_t i = threadIdx.x; i < (xb - xa) * p.Ci; i += kUpThreads) {
    const uint32_t xl = xa + i / p.Ci, c = i % p.Ci;
    const int xg = (int)xl;
    const int ox_lo = xg == 0 ? 0 : (xg - 1) * s + (s + 1) / 2, ox_hi = xg == (int)u.XW - 1 ? (int)u.XW * s - 1 : (xg + 1) * s + s / 2 - 1;
    float acc = 0.f;
    const float* sp = Sr + ((uint32_t)ox_lo - oxa) * p.Ci + c;
    if (xg > 0 && xg < (int)u.XW - 1) {
#pragma unroll 4
      for (int t = 0; t < nt; ++t, sp += p.Ci) acc = fmaf(wyt[t], *sp, acc);
    } else {
      for (int ox = ox_lo; ox <= ox_hi; ++ox, sp += p.Ci) {
        int x0, x1;
        float fx;
        bilin_src((uint32_t)ox, inv, u.XW, x0, x1, fx);
        acc = fmaf((x0 == xg ? 1.f - fx : 0.f) + (x1 == xg ? fx : 0.f), *sp, acc);
      }
    }
    T* o = O + (long long)xl * p.Ci + c;
    st_f(o, u.accumulate ? ld_f(o) + acc : acc);
  }
}

// Contiguous rows on both sides?  ci: interleaved channels
static bool up_rows(const ad_tensor4* lo, const ad_tensor4* hi, bool bwd, UpRowP& r) {
  const UpP& u = r.u;
  auto cfast = [](const ad_tensor4* t) { return t->sc == 1 && t->sx == (long long)t->C; };
  if (cfast(lo) && cfast(hi)) r.Ci = u.C;
  else if (lo->sx == 1 && hi->sx == 1) r.Ci = 1;
  else return false;
  r.planes = u.N * (u.C / r.Ci);
  if ((unsigned long long)u.YW * r.Ci >= (1ull << 31)) return false;
  r.row_len = u.YW * r.Ci;
  // a block per row (or a few) has too little to do on short ones: a thread per element (planes of 22 elements: 66 -> 28 us)
  if (r.row_len < 128) return false;
  const int es = hi->dtype == AD_F32 ? 4 : 2;
  const uint32_t V = 16 / es;
  // the gradient reads 16-byte vectors, the forward writes pairs
  const uint32_t A = bwd ? V : 2, mask = bwd ? 15u : (uint32_t)(2 * es - 1);
  r.vec = ((uintptr_t)hi->base & mask) == 0 && hi->sy % A == 0 && hi->sn % A == 0 && (r.Ci > 1 || hi->sc % A == 0);
  // floats of shared memory per low-resolution column: column sums, or the blended row and the column table
  const uint32_t per_col = bwd ? r.Ci * u.scale : r.Ci + 2 * u.scale;
  if ((unsigned long long)per_col * 3 + 2 * V > kUpFloatsMax) return false;
  const uint32_t floats = (unsigned long long)per_col * 10 + 2 * V > kUpFloats ? kUpFloatsMax : kUpFloats;
  r.XC = (floats - 2 * V) / per_col - 2;
  if (r.XC > u.XW) r.XC = u.XW;
  r.chunks = (u.XW + r.XC - 1) / r.XC;
  r.XC = (u.XW + r.chunks - 1) / r.chunks;
  r.chunks = (u.XW + r.XC - 1) / r.XC;
  // short rows: several per block, as many as the shared memory holds and 16 elements per thread need
  r.rb = 1;
  r.tpr = kUpThreads;
  if (!bwd && r.chunks == 1) {
    const uint32_t want = 16 * kUpThreads / r.row_len, fit = (floats - (r.XC + 2) * 2 * u.scale) / ((r.XC + 2) * r.Ci);
    r.rb = want < fit ? want : fit;
    if (r.rb > 64) r.rb = 64;
    if (r.rb < 1) r.rb = 1;
    while (r.tpr > 8 && r.tpr * 2 >= r.row_len && kUpThreads / r.tpr < r.rb) r.tpr >>= 1;
  }
  // an even, power-of-two scale whose pairs fit the block (Ci <= 64 at scale 8, <= 256 at 2), 16 outputs per thread in a cell of
  // one row (shorter rows share a block in the general form)
  r.period = !bwd && u.scale % 2 == 0 && (u.scale & (u.scale - 1)) == 0 && r.Ci * u.scale / 2 <= kUpThreads &&
                     (unsigned long long)r.row_len * u.scale >= 16 * kUpThreads ? r.Ci * u.scale / 2 : 0;
  if (r.period) {
    // two source rows in shared memory; blocks of so few columns that the machine has six per SM
    r.cell0 = (u.y_row0 + u.scale / 2) / u.scale;
    r.cells = (u.y_row0 + u.YH - 1 + u.scale / 2) / u.scale - r.cell0 + 1;
    const uint32_t most = std::max(1u, (kUpFloats / (2 * r.Ci)) - 2), lanes = kUpThreads / r.period;
    const unsigned long long rows = (unsigned long long)r.planes * r.cells;
    const uint32_t want = (uint32_t)std::max<unsigned long long>(1, (unsigned long long)u.XW * rows / (6 * kNumSMs));
    r.XC = std::min(std::min(most, u.XW), std::max(want, std::min(4 * lanes, u.XW)));
    r.chunks = (u.XW + r.XC - 1) / r.XC;
    r.XC = (u.XW + r.chunks - 1) / r.chunks;
    r.chunks = (u.XW + r.XC - 1) / r.XC;
    r.smem = (2 * (r.XC + 2) * r.Ci + u.scale) * 4;
    return u.scale <= kUpThreads && r.smem <= 49152 && rows * r.chunks < (1ull << 31);
  }
  r.wtab = (r.XC + 2) * u.scale * r.Ci + 16;
  r.smem = bwd ? ((r.XC + 2) * u.scale * r.Ci + 16 + 3 * u.scale + 2) * 4 : ((r.rb * (r.XC + 2) * r.Ci + 2) + (r.XC + 2) * 2 * u.scale) * 4;
  return r.smem <= 49152 && (unsigned long long)r.planes * (bwd ? u.XH : u.YH) * r.chunks < (1ull << 31);
}

static int up_params(const ad_tensor4* lo, const ad_tensor4* hi, uint32_t scale, int32_t x_row0, uint32_t in_rows_total,
                     uint32_t y_row0, UpP& p) {
  if (!lo || !hi || !lo->base || !hi->base || scale == 0 || in_rows_total == 0) return AD_ERR_BAD_ARG;
  if (lo->N != hi->N || lo->C != hi->C || lo->dtype != hi->dtype || hi->W != lo->W * scale) return AD_ERR_BAD_ARG;
  if ((size_t)hi->N * hi->C * hi->H * hi->W >= (1ull << 32) || (size_t)in_rows_total * scale >= (1ull << 31)) return AD_ERR_LIMIT;
  if ((size_t)y_row0 + hi->H > (size_t)in_rows_total * scale) return AD_ERR_BAD_ARG;
  // every source row the high-resolution rows refer to must lie inside the low-resolution view
  if (hi->H > 0) {
    auto src_rows = [&](uint32_t o, long long& a, long long& b) {
      double src = ((double)o + 0.5) / (double)scale - 0.5;
      if (src < 0.0) src = 0.0;
      long long i0 = (long long)src;
      if (i0 > (long long)in_rows_total - 1) i0 = (long long)in_rows_total - 1;
      a = i0;
      b = i0 + 1 < (long long)in_rows_total ? i0 + 1 : (long long)in_rows_total - 1;
    };
    long long a0, b0, a1, b1;
    src_rows(y_row0, a0, b0);
    src_rows(y_row0 + hi->H - 1, a1, b1);
    if (a0 < x_row0 || b1 >= (long long)x_row0 + lo->H) return AD_ERR_BAD_ARG;
  }
  p.x = upview(lo); p.y = upview(hi);
  p.N = lo->N; p.C = lo->C; p.XH = lo->H; p.XW = lo->W; p.YH = hi->H; p.YW = hi->W; p.scale = scale;
  p.x_row0 = x_row0; p.in_rows_total = in_rows_total; p.y_row0 = y_row0;
  return AD_OK;
}

}  // namespace adk

using namespace adk;

extern "C" int ad_upsample_bilinear_fwd(const ad_tensor4* x, const ad_tensor4* y, uint32_t scale, int32_t x_row0,
                                        uint32_t in_rows_total, uint32_t y_row0, void* stream) {
  UpP p{};
  int st = up_params(x, y, scale, x_row0, in_rows_total, y_row0, p);
  if (st != AD_OK) return st;
  const size_t total = (size_t)p.N * p.C * p.YH * p.YW;
  if (total == 0) return AD_OK;
  p.c_fastest = y->sc == 1 && y->C > 1;
  UpRowP r{};
  r.u = p;
  if (up_rows(x, y, false, r)) {
    const unsigned grid = r.period ? (unsigned)((size_t)r.planes * r.cells * r.chunks) : (unsigned)((((size_t)r.planes * p.YH + r.rb - 1) / r.rb) * r.chunks);
    const auto go = [&](auto kernel) { launch(kernel, grid, kUpThreads, r.smem, as_stream(stream), r); };
    AD_DISPATCH_DTYPE(x->dtype, (!r.period ? go(upsample_fwd_rows<T>) : scale == 2 ? go(upsample_fwd_cells<T, 2>) : scale == 4 ? go(upsample_fwd_cells<T, 4>)
                                                                      : scale == 8 ? go(upsample_fwd_cells<T, 8>) : go(upsample_fwd_cells<T, 0>)));
  } else
    AD_DISPATCH_DTYPE(x->dtype, (launch(upsample_fwd_kernel<T>, grid_for(total, 256, 16), 256, 0, as_stream(stream), p)));
  count_launch();
  return launch_status();
}

extern "C" int ad_upsample_bilinear_bwd(const ad_tensor4* dy, const ad_tensor4* dx, uint32_t scale, int32_t x_row0,
                                        uint32_t in_rows_total, uint32_t y_row0, int32_t accumulate, void* stream) {
  UpP p{};
  int st = up_params(dx, dy, scale, x_row0, in_rows_total, y_row0, p);
  if (st != AD_OK) return st;
  const size_t total = (size_t)p.N * p.C * p.XH * p.XW;
  if (total == 0) return AD_OK;
  p.c_fastest = dx->sc == 1 && dx->C > 1;
  p.accumulate = accumulate;
  UpRowP r{};
  r.u = p;
  if (up_rows(dx, dy, true, r)) {
    const unsigned grid = (unsigned)((size_t)r.planes * p.XH * r.chunks);
    AD_DISPATCH_DTYPE(dx->dtype, (launch(upsample_bwd_rows<T>, grid, kUpThreads, r.smem, as_stream(stream), r)));
  } else
    AD_DISPATCH_DTYPE(dx->dtype, (launch(upsample_bwd_kernel<T>, grid_for(total, 256, 16), 256, 0, as_stream(stream), p)));
  count_launch();
  return launch_status();
}
