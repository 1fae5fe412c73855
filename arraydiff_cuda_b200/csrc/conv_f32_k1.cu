// fp32 NCHW convolution, 1x1 filters without padding: forward and data gradient, and the products of the two-step
// data gradient into few channels.  A plain GEMM over channels whose right operand, planes of pixels, is contiguous as it
// lies: 16-byte asynchronous copies where planes and images are multiples of four floats apart, per-pixel gathers otherwise.
// The general tiles of conv_f32.cu work an address and a test out for every element.  Packed FMAs, splits over clusters
// and the order of sums are those of conv_f32_k3.cu; running sums of 64 terms.  Long reductions are bound by the issue of
// packed FMAs, short ones by the start of a CTA and its way out through the tile.
// A strided layer gathers every stride-th pixel forward; its data gradient writes them between zeros set in front.
// Measured (one B200; before -> now, the other direction has the sizes exchanged): 2 x 64 x 224 x 224 -> 147: forward 154 -> 82 us,
// data gradient 99 -> 62; 4 x 512 x 14 x 14 -> 2048: 92 -> 59 and 86 -> 62; 4 x 64 x 56 x 56 -> 256: 35 -> 21 and 25 -> 19.  Over 150
// drawn layers: forward 1.63, data gradient 1.45 times as fast in sum, none slower; error against 64 bits as before
// (means 1.17 -> 1.15e-7, 1.34 -> 1.31e-7).  Strides 2 and 3, 150 layers: 1.36 and 2.3 times (4 x 64 x 112 x 112 -> 128, stride 2: 27 -> 17,
// 31 -> 21 us).
#include <algorithm>

#include "conv_f32.cuh"

namespace adk {

// A thread owns 8 output channels (pairs of them in one packed FMA) of 8 pixels, a CTA 32 WM channels of 256 / WM pixels in the
// order of their images.  Shared memory: three stages of 16 channels ([channel][m], [channel][pixel]) beside the main
// accumulators ([pixel][m]).
constexpr int kK1Threads = 128;
template <int WM> struct K1Tile {
  static constexpr int BM = 32 * WM, BN = 256 / WM, NB = BN / 8, CH = 16, STAGES = WM == 2 ? 3 : 2;
  static constexpr int PA = BM + 4, PT = BM + 4, flush = 4;
  static constexpr int w_floats = CH * PA, stage_floats = w_floats + CH * BN;
  static constexpr int smem = (STAGES * stage_floats + BN * PT) * 4;
};

// VX: 16-byte copies of pixels.  VW: output channels are contiguous in the filter (data gradient) and come by 16 bytes.
// SPREAD: the data gradient of a strided layer: a pixel of dy adds to or writes every stride-th pixel of every stride-th row
template <int WM, bool VX, bool VW, bool SPREAD>
__global__ void __launch_bounds__(kK1Threads, 3) conv1_f32(const GemmF32 p) {
  grid_dependency();
  typedef K1Tile<WM> T;
  constexpr int BM = T::BM, BN = T::BN, NB = T::NB, CH = T::CH, PA = T::PA, PT = T::PT, STAGES = T::STAGES;
  extern __shared__ __align__(16) float sm[];
  float* const tile = sm + STAGES * T::stage_floats;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t m_base = blockIdx.y * BM, n_base = blockIdx.x / cs * BN, PW = SPREAD ? p.IW : p.OW, hw = (SPREAD ? p.IH : p.OH) * PW, npx = p.NI * hw;
  const uint32_t per = ((p.CR + cs - 1) / cs + CH - 1) / CH * CH;   // this CTA's share of the input channels
  const uint32_t c_lo = rank * per < p.CR ? rank * per : p.CR, c_hi = c_lo + per < p.CR ? c_lo + per : p.CR;
  const uint32_t steps = (c_hi - c_lo + CH - 1) / CH;

  auto in_at = [&](uint32_t px) {
    const uint32_t n = px / hw, r = px - n * hw, y = r / PW, x = r - y * PW;
    return p.in + (long long)n * p.in_img + (long long)(SPREAD ? y : y * p.sh) * p.in_pitch + (SPREAD ? x : x * p.sw);
  };
  // what this thread copies of the input: 4 pixels of every XS-th channel, or XN pixels of every channel
  constexpr uint32_t XT = BN / 4, XS = kK1Threads / XT, XN = BN / kK1Threads;
  const float* x_src[VX ? 1 : XN];
  bool x_have[VX ? 1 : XN];
#pragma unroll
  for (uint32_t u = 0; u < (VX ? 1u : XN); ++u) {
    const uint32_t px = n_base + (VX ? tid % XT * 4 : tid + u * kK1Threads);
    x_have[u] = px < npx;
    x_src[u] = (x_have[u] ? in_at(px) : p.in) + (long long)(c_lo + (VX ? tid / XT : 0u)) * p.in_plane;
  }
  uint32_t c_next = c_lo;
  auto load = [&](uint32_t slot) {      // the next stage
    const uint32_t base = smem_addr(sm + (size_t)slot * T::stage_floats), x0 = base + T::w_floats * 4;
    if (VX) {
#pragma unroll
      for (uint32_t i = 0; i < CH / XS; ++i) {
        const uint32_t c = tid / XT + i * XS;
        const bool have = x_have[0] && c_next + c < c_hi;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\tcp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(x0 + (c * BN + tid % XT * 4) * 4),
                     "l"(x_src[0] + (long long)(i * XS) * p.in_plane), "r"((uint32_t)have) : "memory");
      }
      x_src[0] += (long long)CH * p.in_plane;
    } else {
#pragma unroll
      for (uint32_t u = 0; u < XN; ++u) {
#pragma unroll 8
        for (uint32_t c = 0; c < CH; ++c) {
          gather4_if(x0 + (c * BN + tid + u * kK1Threads) * 4, x_src[VX ? 0 : u], x_have[VX ? 0 : u] && c_next + c < c_hi);
          x_src[VX ? 0 : u] += p.in_plane;
        }
      }
    }
    if (VW) {
#pragma unroll
      for (uint32_t i = 0; i < CH * BM / 4 / kK1Threads; ++i) {
        const uint32_t at = tid + i * kK1Threads, c = at / (BM / 4), m = at % (BM / 4) * 4;
        const bool have = c_next + c < c_hi && m_base + m < p.M;     // M is a multiple of 4
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\tcp.async.cg.shared.global [%0], [%1], 16, p;\n\t}" ::"r"(base + (c * PA + m) * 4),
                     "l"(p.w + (long long)(c_next + c) * p.w_c + m_base + m), "r"((uint32_t)have) : "memory");
      }
    } else {
      // 8 channels x 4 m per warp: neighbours in memory whichever of the two is contiguous, free of bank conflicts
      const uint32_t c0 = lane & 7, m0 = warp * (BM / 4) + (lane >> 3);
      const float* src = p.w + (long long)(m_base + m0) * p.w_m + (long long)(c_next + c0) * p.w_c;
#pragma unroll
      for (uint32_t g = 0; g < BM / 16; ++g) {
#pragma unroll
        for (uint32_t i = 0; i < CH / 8; ++i)
          gather4_if(base + ((c0 + i * 8) * PA + m0 + g * 4) * 4, src + (long long)(i * 8) * p.w_c, m_base + m0 + g * 4 < p.M && c_next + c0 + i * 8 < c_hi);
        src += 4 * p.w_m;
      }
    }
    c_next += CH;
  };

  // pixels n0 .. n0 + 3 and n0 + 32 .. n0 + 35
  const uint32_t m0 = (warp % WM) * 32 + lane / 8 * 8, wn = warp / WM, n0 = wn * 64 + lane % 8 * 4, blk = wn * 8 + lane % 8;
  u64 acc[8][4];                        // [pixel][pair of channels]
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0ull;
  // tile row of pixel j of a thread: free of bank conflicts here and for neighbouring pixels at the end
  auto tile_row = [&](uint32_t j, uint32_t b) { return j * NB + (b ^ ((j & 3u) << 1)); };
  auto flush = [&](bool first) {        // running sums -> main accumulators (this thread's own elements)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      ulonglong2* t = (ulonglong2*)(tile + tile_row(j, blk) * PT + m0);
      if (!first) {
        const ulonglong2 a = t[0], b = t[1];
        fadd2(acc[j][0], a.x); fadd2(acc[j][1], a.y); fadd2(acc[j][2], b.x); fadd2(acc[j][3], b.y);
      }
      t[0] = make_ulonglong2(acc[j][0], acc[j][1]);
      t[1] = make_ulonglong2(acc[j][2], acc[j][3]);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[j][i] = 0ull;
    }
  };
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if ((uint32_t)st < steps) load(st);
    cp_async_commit();
  }
  bool first = true;
  uint32_t slot = 0, to_flush = T::flush;
#pragma unroll 1
  for (uint32_t st = 0; st < steps; ++st) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < steps) load(slot == 0 ? STAGES - 1 : slot - 1);
    cp_async_commit();
    const float* ws = sm + (size_t)slot * T::stage_floats + m0;
    const float* xs = sm + (size_t)slot * T::stage_floats + T::w_floats + n0;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const ulonglong2 w0 = *(const ulonglong2*)(ws + c * PA), w1 = *(const ulonglong2*)(ws + c * PA + 4);
      const float4 x0 = *(const float4*)(xs + c * BN), x1 = *(const float4*)(xs + c * BN + 32);
      const u64 w[4] = {w0.x, w0.y, w1.x, w1.y};
      const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) ffma2(acc[j][i], w[i], dup2(x[j]));
    }
    if (--to_flush == 0 || st + 1 == steps) { flush(first); first = false; to_flush = T::flush; }
    if (++slot == STAGES) slot = 0;
  }
  if (first) flush(true);
  if (cs > 1) cluster.sync();
  else __syncthreads();
  // each CTA of the cluster finishes BM / cs channels; threads follow the pixels
  const uint32_t rows = BM / cs;
#pragma unroll 1
  for (uint32_t e = tid; e < (uint32_t)BN; e += kK1Threads) {
    const uint32_t px = n_base + e;
    if (px >= npx) continue;
    const uint32_t n = px / hw, r = px - n * hw, y = r / PW, x = r - y * PW;
    float* out = p.out + (long long)n * p.out_img + (long long)(SPREAD ? y * p.sh : y) * p.out_pitch + (SPREAD ? x * p.sw : x);
    const uint32_t row = tile_row((e >> 5 & 1u) * 4 + (e & 3u), (e >> 6) * 8 + (e >> 2 & 7u));
#pragma unroll 1
    for (uint32_t m = rank * rows; m < (rank + 1) * rows; m += 4) {
      const float4 v4 = cluster_total4<kF32Most>(cluster, tile, cs, (size_t)row * PT + m);
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (m_base + m + i >= p.M) break;
        float* o = out + (long long)(m_base + m + i) * p.out_plane;
        float f = v[i];
        if (p.bias) f += p.bias[m_base + m + i];
        if (p.relu) f = fmaxf(f, 0.f);
        if (p.accumulate) f += *o;
        *o = f;
      }
    }
  }
  if (cs > 1) cluster.sync();           // nobody leaves while its tile is still read
}

template <int WM, bool VX, bool VW, bool SPREAD>
static int launch_conv1_f32(const GemmF32& p, cudaStream_t s) {
  typedef K1Tile<WM> T;
  static F32Launch l;
  const uint32_t npx = SPREAD ? p.NI * p.IH * p.IW : p.NI * p.OH * p.OW, tn = (npx + T::BN - 1) / T::BN, tm = (p.M + T::BM - 1) / T::BM;
  auto held = [](uint32_t n) { return f32_held(conv1_f32<WM, VX, VW, SPREAD>, kK1Threads, T::smem, n, l); };
  const uint32_t cs = f32_k3_cluster(held, (unsigned long long)tn * tm, (p.CR + T::CH - 1) / T::CH, std::min(kF32Most, T::BM / 4), kNumSMs);
  return launch_f32(conv1_f32<WM, VX, VW, SPREAD>, dim3(tn * cs, tm), kK1Threads, T::smem, cs, p, l, s);
}
template <bool SPREAD>
static int run_conv1_f32(const GemmF32& p, cudaStream_t s) {
  auto in4 = [](long long v) { return v % 4 == 0; };
  const long long px = SPREAD ? (long long)p.IH * p.IW : (long long)p.OH * p.OW;
  const bool vx = p.in_pitch * p.IH == px && in4(p.in_plane) && in4(p.in_img) && in4(px) && !((uintptr_t)p.in & 15u);
  const bool vw = p.w_m == 1 && in4(p.w_c) && in4(p.M) && !((uintptr_t)p.w & 15u);
  if (p.M <= 32) return vx ? (vw ? launch_conv1_f32<1, true, true, SPREAD>(p, s) : launch_conv1_f32<1, true, false, SPREAD>(p, s))
                           : (vw ? launch_conv1_f32<1, false, true, SPREAD>(p, s) : launch_conv1_f32<1, false, false, SPREAD>(p, s));
  return vx ? (vw ? launch_conv1_f32<2, true, true, SPREAD>(p, s) : launch_conv1_f32<2, true, false, SPREAD>(p, s))
            : (vw ? launch_conv1_f32<2, false, true, SPREAD>(p, s) : launch_conv1_f32<2, false, false, SPREAD>(p, s));
}
template <bool DGRAD>
int f32_k1_gemm(const GemmF32& p, cudaStream_t s) {
  if (!DGRAD || (p.sh == 1 && p.sw == 1)) return run_conv1_f32<false>(p, s);
  // the pixels between: zeroed in front.  Written along by the kernel, one by one, they took most of its time for few tiles
  // (168 -> 33 channels, 27 x 22, stride 3: 39 us)
  if (!p.accumulate && cudaMemsetAsync(p.out, 0, (size_t)p.NI * p.out_img * 4, s) != cudaSuccess) { cudaGetLastError(); return AD_ERR_CUDA; }
  return run_conv1_f32<true>(p, s);
}
template int f32_k1_gemm<false>(const GemmF32&, cudaStream_t);
template int f32_k1_gemm<true>(const GemmF32&, cudaStream_t);

}  // namespace adk
