// fp32 NCHW convolution, 3x3 filters: forward (stride 1 under any dilation, stride 2), data gradient (stride 1, any dilation),
// filter and bias gradient (as the forward pass) from patches of the input in shared memory.  The general tiles of conv_f32.cu gather every input element once per tap and read four
// 16-byte operands from shared memory for 32 packed FMAs; their 12 warps per SM mostly wait.  Here a thread holds the window
// of its pixels in registers and meets all nine taps with it: a third of the gathers, 24 reads for 288 packed FMAs.
// What bounds the kernels is the issue of packed FMAs (63 TFLOP/s in a loop of them and their reads: a scheduler issues one
// in 2.4 clocks, and everything else in between costs a clock) and, for the filter gradient, the main accumulators' way
// through shared memory.  A factor that is the same in both halves of a packed FMA costs nothing as a scalar register
// (mov.b64 {v, v}); kept twice in shared memory instead, the kernels were 15 % slower.
// Measured (one B200, 3.7 GFLOP each; before -> now): 4 x 64 x 112 x 112 -> 64: forward 135 -> 94 us, data gradient 134 -> 92, filter
// and bias gradient 172 -> 127; 4 x 128 x 56 x 56 -> 128: 131 -> 94, 131 -> 90, 261 -> 115; 4 x 512 x 14 x 14 -> 512: 181 -> 127,
// 180 -> 123, 135 -> 125.  Over 630 drawn layers: forward 1.33, data gradient 1.33, filter gradient 1.2 times as fast.  Stride 2, 1.9
// GFLOP: 4 x 64 x 112 x 112 -> 128: forward 75 -> 60, filter gradient 95 -> 76; 4 x 128 x 56 x 56 -> 256: 72 -> 60, 132 -> 70.  Over 250 drawn
// layers of stride 2 or dilations 2 to 4, the ones that stay with the general tiles included: forward 1.20, data gradient 1.10,
// filter gradient 1.23 times as fast.
// A map under dilation d is d x d maps without: blocks and segments take every d-th row and column, neighbouring blocks
// the neighbouring phases, which share the sectors that they read.
// Sums, splits over clusters and slices, and their order of addition are as in conv_f32.cu: fp32 FMAs, running sums of 18 to
// 54 (filter gradient: 32 to 128) terms, partial tiles in rank order; no atomics.
#include <algorithm>

#include "conv_f32.cuh"

namespace adk {

constexpr int kK3Threads = 128;

// ---------------------------------------------------------------- forward / data gradient
// A thread owns 8 output channels (pairs of them in one packed FMA) of a block of 4 rows x 2 columns of pixels; a CTA owns
// 32 WM channels of 16 / WM x 2 blocks, taken from the list of all blocks of all images in order, so that small maps fill
// tiles too.  Per input channel: 6 reads of the block's 6 x 4 input patch (9 x 5 with a stride of 2: 12 reads), 18 of the filter, 288
// packed FMAs.  A packed FMA
// takes more than two of a scheduler's issue slots, so that every other instruction costs: gathers advance their addresses by
// additions and take their conditions from predicates.
// Shared memory: three stages of 2 channels ([channel, tap][m], [channel][block][6][4]; pitches free of bank conflicts)
// beside the tile of main accumulators ([pixel][m]), to which the running sums go.
template <int WM, bool DGRAD, int S> struct K3Tile {
  static constexpr int BM = 32 * WM, NB = 32 / WM, BN = NB * 8;
  static constexpr int XR = 3 * S + 3, XC = S + 3;      // a block's patch of the input
  static constexpr int CH = 2, STAGES = S == 2 && WM == 1 ? 2 : 3, PA = BM + (DGRAD ? 8 : 4), PX = S == 1 ? 28 : 52, PT = BM + 4;
  static constexpr int w_floats = CH * 9 * PA, stage_floats = w_floats + CH * NB * PX;
  static constexpr int smem = (STAGES * stage_floats + BN * PT) * 4;
};

template <int WM, bool DGRAD, int S>
__global__ void __launch_bounds__(kK3Threads, 3) conv3_f32(const GemmF32 p) {
  grid_dependency();
  typedef K3Tile<WM, DGRAD, S> T;
  constexpr int BM = T::BM, NB = T::NB, CH = T::CH, PA = T::PA, PX = T::PX, PT = T::PT, STAGES = T::STAGES;
  // a pass of the threads covers RS rows of all patches (S 1) or RS elements of them (S 2)
  constexpr int RS = (S == 1 ? 32 : kK3Threads) / NB, NG = S == 1 ? 6 / RS : (T::XR * T::XC + RS - 1) / RS;
  // a pass over the filter takes WK (channel, tap) x 24 / WK m per warp: neighbours in memory, free of bank conflicts
  constexpr int WK = DGRAD ? 3 : 6, WR = 24 / WK, MG = BM / (4 * WR);
  extern __shared__ __align__(16) float sm[];
  float* const tile = sm + STAGES * T::stage_floats;
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t m_base = blockIdx.y * BM, blk_base = blockIdx.x / cs * NB;
  const uint32_t BX = ((p.OW + p.dw - 1) / p.dw + 1) / 2, BY = ((p.OH + p.dh - 1) / p.dh + 3) / 4, blocks = p.NI * BY * BX * p.dh * p.dw;
  auto place = [&](uint32_t b, uint32_t& n, uint32_t& y, uint32_t& x) {    // a block's image and first pixel
    uint32_t fx = 0, fy = 0;
    if (S == 1 && p.dw > 1) { fx = b % p.dw; b /= p.dw; }
    x = fx + b % BX * 2 * p.dw; b /= BX;
    y = b % BY * 4 * p.dh; b /= BY;
    if (S == 1 && p.dh > 1) { fy = b % p.dh; b /= p.dh; }
    y += fy;
    n = b;
  };

  const uint32_t per = ((p.CR + cs - 1) / cs + CH - 1) / CH * CH;   // this CTA's share of the input channels
  const uint32_t c_lo = rank * per < p.CR ? rank * per : p.CR, c_hi = c_lo + per < p.CR ? c_lo + per : p.CR;
  const uint32_t steps = (c_hi - c_lo + CH - 1) / CH;

  // what this thread gathers of the input: column gc of rows gr, gr + RS, .. of a block's patch
  const uint32_t gc = S == 1 ? tid & 3 : 0, gb = S == 1 ? (tid >> 2) & (NB - 1) : (lane & 7) | (warp & (NB / 8 - 1)) << 3;
  const uint32_t gr = S == 1 ? tid / (4 * NB) : lane / 8 + warp / (NB / 8) * 4;
  const float* x_src = p.in + (long long)c_lo * p.in_plane;
  bool x_have[NG];
  int x_off[S == 1 ? 1 : NG];
#pragma unroll
  for (int i = 0; i < NG; ++i) x_have[i] = false;
  {
    const uint32_t b = blk_base + gb;
    if (b < blocks) {
      uint32_t n, y, x;
      place(b, n, y, x);
      const int dh = (int)p.dh, dw = (int)p.dw;
      int iy = (int)y * S + (DGRAD ? p.ph - 2 * dh : -p.ph), ix = (int)x * S + (DGRAD ? p.pw - 2 * dw : -p.pw);
      if (S == 1) { iy += (int)gr * dh; ix += (int)gc * dw; }
      x_src += (long long)n * p.in_img + (long long)iy * p.in_pitch + ix;
#pragma unroll
      for (int i = 0; i < NG; ++i) {
        if (S == 1) {
          x_have[i] = (unsigned)ix < p.IW && (unsigned)(iy + i * RS * dh) < p.IH;
        } else {
          const int e = (int)gr + i * RS, r = e / T::XC, c = e - r * T::XC;
          x_have[i] = e < T::XR * T::XC && (unsigned)(ix + c) < p.IW && (unsigned)(iy + r) < p.IH;
        }
      }
    }
#pragma unroll
    for (int i = 0; S > 1 && i < NG; ++i) {
      const int e = (int)gr + i * RS;
      x_off[i] = e / T::XC * (int)p.in_pitch + e % T::XC;
    }
  }
  const long long x_row = (long long)RS * (int)p.dh * p.in_pitch;
  const uint32_t x_dst = (T::w_floats + gb * PX + (S == 1 ? gr * 4 + gc : gr)) * 4;
  const uint32_t lm = lane / WK, lt = lane - lm * WK, wm = warp * (BM / 4) + lm;      // lanes 24 .. 31: none
  const float* w_src[MG];
  bool w_have[MG];
#pragma unroll
  for (int g = 0; g < MG; ++g) {
    w_src[g] = p.w + (long long)(m_base + wm + g * WR) * p.w_m + (long long)c_lo * p.w_c + lt;
    w_have[g] = m_base + wm + g * WR < p.M;
  }
  const uint32_t w_dst = ((DGRAD ? 8 - lt : lt) * PA + wm) * 4;     // the data gradient meets the taps mirrored

  uint32_t c_next = c_lo;
  auto load = [&](uint32_t slot) {    // the next stage
    const uint32_t base = smem_addr(sm + (size_t)slot * T::stage_floats);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const bool in = c_next + c < c_hi;
      if (S == 1) {
        const float* src = x_src;
#pragma unroll
        for (int i = 0; i < NG; ++i) {
          gather4_if(base + x_dst + (c * NB * PX + i * RS * 4) * 4, src, in && x_have[i]);
          src += x_row;
        }
      } else {
#pragma unroll
        for (int i = 0; i < NG; ++i) gather4_if(base + x_dst + (c * NB * PX + i * RS) * 4, x_src + x_off[S == 1 ? 0 : i], in && x_have[i]);
      }
      x_src += p.in_plane;
    }
    if (lane < 24) {
#pragma unroll
      for (int g = 0; g < MG; ++g) {
#pragma unroll
        for (int k = 0; k < CH * 9; k += WK) {
          const int c = k / 9, t = k - c * 9;        // forward: k may run over a channel's last tap, which lt decides
          if (DGRAD)
            gather4_if(base + w_dst + ((c * 9 - t) * PA + g * WR) * 4, w_src[g] + (c ? p.w_c : 0ll) + t, w_have[g] && c_next + c < c_hi);
          else
            gather4_if(base + w_dst + (k * PA + g * WR) * 4, w_src[g] + k, w_have[g] && c_next + (k + lt) / 9 < c_hi);
        }
        w_src[g] += CH * p.w_c;
      }
    }
    c_next += CH;
  };

  const uint32_t m0 = (warp % WM) * 32 + lane / 8 * 8, blk = warp / WM * 8 + lane % 8;
  u64 acc[8][4];                      // [pixel: row * 2 + column][pair of channels]
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[j][i] = 0ull;
  // tile row of a pixel: free of bank conflicts for threads of neighbouring blocks (here) and of neighbouring columns (the end)
  auto tile_row = [&](uint32_t j, uint32_t b) { return j * NB + (b ^ ((j & 1u) << 2)); };
  auto flush = [&](bool first) {      // running sums -> main accumulators (this thread's own elements)
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
  const uint32_t period = steps <= 2 ? 1 : steps <= 8 ? 2 : 3;     // running sums of 18, 36, 54 terms
  uint32_t slot = 0, to_flush = period;
#pragma unroll 1
  for (uint32_t st = 0; st < steps; ++st) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < steps) load(slot == 0 ? STAGES - 1 : slot - 1);
    cp_async_commit();
    const float* ws = sm + (size_t)slot * T::stage_floats + m0;
    const float* xs = sm + (size_t)slot * T::stage_floats + T::w_floats + blk * PX;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      float x[(T::XR * T::XC + 3) / 4 * 4];
#pragma unroll
      for (int r = 0; r < (T::XR * T::XC + 3) / 4; ++r) *(float4*)(x + r * 4) = *(const float4*)(xs + c * NB * PX + r * 4);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          const float* wt = ws + (c * 9 + r * 3 + s) * PA;
          const ulonglong2 w0 = *(const ulonglong2*)wt, w1 = *(const ulonglong2*)(wt + 4);
          const u64 w[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) ffma2(acc[j][i], w[i], dup2(x[((j >> 1) * S + r) * T::XC + (j & 1) * S + s]));
        }
    }
    if (--to_flush == 0 || st + 1 == steps) { flush(first); first = false; to_flush = period; }
    if (++slot == STAGES) slot = 0;
  }
  if (first) flush(true);
  if (cs > 1) cluster.sync();
  else __syncthreads();
  // each CTA of the cluster finishes BM / cs channels; threads follow the pixels along x
  const uint32_t rows = BM / cs;
#pragma unroll 1
  for (uint32_t e = tid; e < (uint32_t)T::BN; e += kK3Threads) {
    const uint32_t px = e & 1, b = (e >> 1) & (NB - 1), py = e / (2 * NB), at = blk_base + b;
    uint32_t n, y, x;
    place(at, n, y, x);
    const uint32_t oy = y + py * p.dh, ox = x + px * p.dw;
    if (at >= blocks || oy >= p.OH || ox >= p.OW) continue;
    float* out = p.out + (long long)n * p.out_img + (long long)oy * p.out_pitch + ox;
#pragma unroll 1
    for (uint32_t m = rank * rows; m < (rank + 1) * rows; m += 4) {
      const float4 v4 = cluster_total4<kF32Most>(cluster, tile, cs, (size_t)tile_row(py * 2 + px, b) * PT + m);
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (m_base + m + i >= p.M) break;
        float* o = out + (long long)(m_base + m + i) * p.out_plane;
        float f = v[i];
        if (!DGRAD) {
          if (p.bias) f += p.bias[m_base + m + i];
          if (p.relu) f = fmaxf(f, 0.f);
        } else if (p.accumulate) {
          f += *o;
        }
        *o = f;
      }
    }
  }
  if (cs > 1) cluster.sync();         // nobody leaves while its tile is still read
}

template <int WM, bool DGRAD, int S>
static int launch_conv3_f32(const GemmF32& p, cudaStream_t s) {
  typedef K3Tile<WM, DGRAD, S> T;
  static F32Launch l;
  const uint32_t blocks = p.NI * (uint32_t)f32_k3_blocks(p.OH, p.OW, p.dh, p.dw), tn = (blocks + T::NB - 1) / T::NB, tm = (p.M + T::BM - 1) / T::BM;
  auto held = [](uint32_t n) { return f32_held(conv3_f32<WM, DGRAD, S>, kK3Threads, T::smem, n, l); };
  const uint32_t cs = f32_k3_cluster(held, (unsigned long long)tn * tm, (p.CR + T::CH - 1) / T::CH, std::min(kF32Most, T::BM / 4), kNumSMs);
  return launch_f32(conv3_f32<WM, DGRAD, S>, dim3(tn * cs, tm), kK3Threads, T::smem, cs, p, l, s);
}

template <bool DGRAD>
int f32_k3_gemm(const GemmF32& p, cudaStream_t s) {
  if constexpr (!DGRAD) {
    if (p.sh == 2) return p.M <= 32 ? launch_conv3_f32<1, false, 2>(p, s) : launch_conv3_f32<2, false, 2>(p, s);
  }
  return p.M <= 32 ? launch_conv3_f32<1, DGRAD, 1>(p, s) : launch_conv3_f32<2, DGRAD, 1>(p, s);
}
template int f32_k3_gemm<false>(const GemmF32&, cudaStream_t);
template int f32_k3_gemm<true>(const GemmF32&, cudaStream_t);

// ---------------------------------------------------------------- filter gradient
// A thread owns the nine taps of one input channel for 8 output channels (pairs of them in one packed FMA); a CTA owns
// 8 KGS output channels x 128 / KGS input channels.  The reduction runs over segments of up to 8 pixels of an output
// row, whose columns of x are three registers that move along with the pixel: per pixel 36 packed FMAs, 2 reads of dy, 9/8 of
// x (9/4 with a stride of 2).  Pixels past the end of a row are skipped, not multiplied by zero.
// Shared memory: two stages of 4 segments, one per warp that gathers it ([pixel][k], [channel][3 rows][12 or 20 columns]), beside
// the tile of main accumulators ([tap][channel][k], 16-byte pieces of k swizzled).
template <int KGS, int S> struct K3Wg {
  static constexpr int BK = 8 * KGS, NCH = kK3Threads / KGS, SEGS = 4, SEG = 8, PK = BK + 4, XC = S == 1 ? 10 : 17, XP = S == 1 ? 12 : 20, PC = 3 * XP;
  static constexpr int dy_floats = SEGS * SEG * PK, stage_floats = dy_floats + SEGS * NCH * PC;
  static constexpr int smem = (2 * stage_floats + 9 * NCH * BK) * 4;
};

template <int KGS, int S>
__global__ void __launch_bounds__(kK3Threads, S == 1 ? 3 : 2) conv3_wgrad_f32(const WgradF32 p) {
  grid_dependency();
  typedef K3Wg<KGS, S> T;
  constexpr int BK = T::BK, NCH = T::NCH, SEGS = T::SEGS, SEG = T::SEG, PK = T::PK, PC = T::PC;
  extern __shared__ __align__(16) float sm[];
  float* const tile = sm + 2 * T::stage_floats;
  __shared__ uint32_t count[2][SEGS];
  __shared__ float sdb[BK];
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t c_base = (blockIdx.x / cs) * NCH, k_base = blockIdx.y * BK, slice = blockIdx.z;
  const uint32_t row_segs = ((p.Q + p.dw_ - 1) / p.dw_ + SEG - 1) / SEG * p.dw_, segs = p.N * p.P * row_segs;
  const uint32_t all = (segs + SEGS - 1) / SEGS, parts = cs * p.slices, per = (all + parts - 1) / parts, me = slice * cs + rank;
  const uint32_t s_lo = me * per < all ? me * per : all, steps = (s_lo + per < all ? s_lo + per : all) - s_lo;
  const long long x_plane = (long long)p.H * p.W;
  const int nk = (int)(p.K - k_base < (uint32_t)BK ? p.K - k_base : BK), nc = (int)(p.C - c_base < (uint32_t)NCH ? p.C - c_base : NCH);
  auto load = [&](uint32_t st) {
    const uint32_t seg = (s_lo + st) * SEGS + warp;
    float* stage = sm + (size_t)(st & 1u) * T::stage_floats;
    const bool in = seg < segs;
    const uint32_t sx = in ? seg % row_segs : 0, r = in ? seg / row_segs : 0, oy = r % p.P, n = r / p.P;
    // every dw-th pixel of a row, from one of the first dw on
    const uint32_t ox = p.dw_ == 1 ? sx * SEG : sx / p.dw_ * SEG * p.dw_ + sx % p.dw_;
    const uint32_t left = !in || ox >= p.Q ? 0u : p.dw_ == 1 ? p.Q - ox : (p.Q - ox + p.dw_ - 1) / p.dw_, cnt = left < (uint32_t)SEG ? left : SEG;
    if (lane == 0) count[st & 1u][warp] = cnt;
    {
      const uint32_t px = lane & 7, k = lane >> 3;
      const float* src = p.dy + ((long long)n * p.K + k_base + k) * p.dy_plane + (long long)oy * p.dy_pitch + ox + px * p.dw_;
      const uint32_t dst = smem_addr(stage + (warp * SEG + px) * PK + k);
      const bool have = px < cnt;
#pragma unroll
      for (int i = 0; i < BK / 4; ++i) {     // rows past the last output channel: zeros
        gather4_if(dst + i * 16, src, have && (int)k + i * 4 < nk);
        src += 4 * p.dy_plane;
      }
    }
#pragma unroll
    for (uint32_t e = lane; e < 3 * T::XC; e += 32) {    // 3 x 10 or 3 x 17 elements of the segment's patch
      const uint32_t lr = e / T::XC, lc = e - lr * T::XC;
      const int iy = (int)(oy * S + lr * p.dh) - p.ph, ix = (int)(ox * S + lc * p.dw_) - p.pw;
      const float* src = p.x + ((long long)n * p.C + c_base) * x_plane + (long long)iy * p.W + ix;
      const uint32_t dst = smem_addr(stage + T::dy_floats + warp * NCH * PC + lr * T::XP + lc);
      const bool have = in && (unsigned)iy < p.H && (unsigned)ix < p.W;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        gather4_if(dst + c * PC * 4, src, have && c < nc);
        src += x_plane;
      }
    }
  };

  const uint32_t kg = lane % KGS, ch = warp * (32 / KGS) + lane / KGS;
  u64 acc[9][4];                      // [tap][pair of output channels: 4 kg .. and 4 (KGS + kg) ..]
#pragma unroll
  for (int t = 0; t < 9; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[t][i] = 0ull;
  float dbs = 0.f, db_main = 0.f;
  const bool with_db = p.db && c_base == 0;
  auto piece = [&](uint32_t t, uint32_t c, uint32_t q) { return (size_t)(t * NCH + c) * BK + ((q ^ ((t + c) & 7u)) << 2); };
  auto flush = [&](bool first) {
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ulonglong2* o = (ulonglong2*)(tile + piece(t, ch, h * KGS + kg));
        if (!first) {
          const ulonglong2 a = *o;
          fadd2(acc[t][2 * h], a.x); fadd2(acc[t][2 * h + 1], a.y);
        }
        *o = make_ulonglong2(acc[t][2 * h], acc[t][2 * h + 1]);
        acc[t][2 * h] = acc[t][2 * h + 1] = 0ull;
      }
  };
  if (steps) load(0);
  cp_async_commit();
  const uint32_t period = steps <= 2 ? 1 : steps <= 24 ? 2 : 4;     // running sums of 32, 64, 128 pixels: a flush costs as much as 8
  uint32_t to_flush = period;
  bool first = true;
  for (uint32_t st = 0; st < steps; ++st) {
    cp_async_wait<0>();
    __syncthreads();
    if (st + 1 < steps) load(st + 1);
    cp_async_commit();
    const float* stage = sm + (size_t)(st & 1u) * T::stage_floats;
#pragma unroll 1
    for (int g = 0; g < SEGS; ++g) {
      const uint32_t cnt = count[st & 1u][g];
      const float* xs = stage + T::dy_floats + (g * NCH + ch) * PC;
      const float* ds = stage + g * SEG * PK + kg * 4;
      // 4 pixels at a time; the next pixel's dy (of the next segment or the patches, past the last) is read underneath this one's products
      ulonglong2 d0 = *(const ulonglong2*)ds, d1 = *(const ulonglong2*)(ds + KGS * 4);
      auto pixel = [&](const float (&x)[3][4 * S + 4], int px, int next) {
        const u64 d[4] = {d0.x, d0.y, d1.x, d1.y};
        { d0 = *(const ulonglong2*)(ds + next * PK); d1 = *(const ulonglong2*)(ds + next * PK + KGS * 4); }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int s = 0; s < 3; ++s) ffma2(acc[r * 3 + s][i], d[i], dup2(x[r][px * S + s]));
      };
#pragma unroll 1
      for (int h = 0; h < SEG; h += 4) {
        if ((uint32_t)h >= cnt) break;
        float x[3][4 * S + 4];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          const float* xr = xs + r * T::XP + h * S;
          *(float4*)x[r] = *(const float4*)xr;
          if (S == 1) *(float2*)(x[r] + 4) = *(const float2*)(xr + 4);
          else { *(float4*)(x[r] + 4) = *(const float4*)(xr + 4); x[r][4 * S] = xr[4 * S]; }
        }
        if (cnt >= (uint32_t)h + 4) {
#pragma unroll
          for (int px = 0; px < 4; ++px) pixel(x, px, h + px + 1);
        } else {
#pragma unroll
          for (int px = 0; px < 3; ++px) {
            if (h + px >= cnt) break;
            pixel(x, px, h + px + 1);
          }
        }
      }
    }
    if (with_db && tid < BK) {        // the bias gradient: column sums of the same dy tile (zeros past the ends)
      float d[SEGS * SEG / 4];
#pragma unroll
      for (int q = 0; q < SEGS * SEG / 4; ++q) {
        const float* v = stage + q * 4 * PK + tid;
        d[q] = (v[0] + v[PK]) + (v[2 * PK] + v[3 * PK]);
      }
      dbs += ((d[0] + d[1]) + (d[2] + d[3])) + ((d[4] + d[5]) + (d[6] + d[7]));
      if ((st & 7u) == 7u) { db_main += dbs; dbs = 0.f; }
    }
    if (--to_flush == 0 || st + 1 == steps) { flush(first); first = false; to_flush = period; }
  }
  if (first) flush(true);
  if (with_db && tid < BK) sdb[tid] = db_main + dbs;
  if (cs > 1) cluster.sync();
  else __syncthreads();
  const uint32_t NC = p.C * 9;
  float* const dw = p.slices > 1 ? p.part + (size_t)slice * ((size_t)p.K * NC + p.K) : p.dw;
  float* const db = p.slices > 1 ? dw + (size_t)p.K * NC : p.db;
  const bool acc_out = p.accumulate && p.slices == 1;
  const uint32_t rows = BK / cs;      // each CTA of the cluster finishes BK / cs output channels
#pragma unroll 1
  for (uint32_t e = tid; e < rows / 4 * (9 * NCH); e += kK3Threads) {
    const uint32_t q = e / (9 * NCH), n = e - q * (9 * NCH), c = n / 9, t = n - c * 9, k = rank * rows + q * 4;
    const float4 v4 = cluster_total4<8>(cluster, tile, cs, piece(t, c, k >> 2));
    const float v[4] = {v4.x, v4.y, v4.z, v4.w};
    if (c_base + c >= p.C) continue;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (k_base + k + i >= p.K) break;
      float* o = dw + (size_t)(k_base + k + i) * NC + c_base * 9 + n;
      *o = acc_out ? *o + v[i] : v[i];
    }
  }
  if (with_db && tid < rows && k_base + rank * rows + tid < p.K) {
    float v = 0.f;
    for (uint32_t q = 0; q < cs; ++q) v += (cs > 1 ? cluster.map_shared_rank(sdb, q) : sdb)[rank * rows + tid];
    float* o = db + k_base + rank * rows + tid;
    *o = acc_out ? *o + v : v;
  }
  if (cs > 1) cluster.sync();
}

F32Split f32_k3_wgrad_split(uint32_t K, uint32_t C, uint32_t N, uint32_t P, uint32_t Q, uint32_t stride, uint32_t dil) {
  const uint32_t bk = K > 32 ? 64 : 32, nch = K > 32 ? 16 : 32;
  const unsigned long long tiles = (unsigned long long)((K + bk - 1) / bk) * ((C + nch - 1) / nch);
  return f32_k3_split(tiles, ((unsigned long long)N * P * f32_k3_segments(Q, dil) + 3) / 4, 9ull * K * C, kNumSMs, stride == 1 ? 3 : 2);
}

template <int KGS, int S>
static int launch_conv3_wgrad(const WgradF32& p, uint32_t most, cudaStream_t s) {
  typedef K3Wg<KGS, S> T;
  static F32Launch l;
  const uint32_t tn = (p.C + T::NCH - 1) / T::NCH, tm = (p.K + T::BK - 1) / T::BK;
  auto held = [](uint32_t n) { return f32_held(conv3_wgrad_f32<KGS, S>, kK3Threads, T::smem, n, l); };
  const uint32_t cs = f32_largest_cluster(held, most);
  return launch_f32(conv3_wgrad_f32<KGS, S>, dim3(tn * cs, tm, p.slices), kK3Threads, T::smem, cs, p, l, s);
}
// p.slices == 1: straight into dw and db, else partial gradients in p.part
int f32_k3_wgrad(const WgradF32& p, uint32_t cs, cudaStream_t s) {
  if (p.sh == 2) return p.K > 32 ? launch_conv3_wgrad<8, 2>(p, cs, s) : launch_conv3_wgrad<4, 2>(p, cs, s);
  return p.K > 32 ? launch_conv3_wgrad<8, 1>(p, cs, s) : launch_conv3_wgrad<4, 1>(p, cs, s);
}

}  // namespace adk
