// fp32 NCHW convolution with fp32 FMA accumulate, as tiled implicit GEMMs: forward, data gradient, filter and bias
// gradient.  Every product and every sum is an fp32 FMA (packed two to an instruction: fma.rn.f32x2 rounds each half as
// fmaf does), and long sums are kept short in two levels: a running sum of 64 terms (filter gradient: 128) is added to the
// main accumulator and restarted.
//
// The bound is the fp32 FMA pipe (148 SMs x 128 FMA per clock: 74 TFLOP/s on paper, 60-68 in a loop of nothing else)
// and, just below it, the 128 bytes per clock a shared-memory read brings into registers: an 8 x 8 outputs-per-thread
// tile needs all of both (58-62 TFLOP/s in a loop of reads and packed FMAs, 8 x 4 outputs 52).  So a thread owns 8 x 8
// outputs, pairs of which sit in one packed FMA, and what is left goes into cheap gathers: operands come by 4-byte
// cp.async into a ring of stages, ~6 instructions per element (table entry, test, address, a predicated copy or a
// predicated store of zero for the implicit padding).
//
// A shape with few output tiles splits its reduction over the CTAs of a cluster (up to 16, filter gradients 8), whose partial tiles meet
// through distributed shared memory in rank order, and a filter gradient further over slices of the caller's scratch:
// no atomics, reproducible.
//
// Measured on a B200 against one thread per output (the kernels of conv_direct.cu, which remain for geometries outside
// f32_gemm_ok and for the smallest calls, direct_wins): figures at the launchers.
#include <algorithm>
#include <cstdlib>

#include "conv_f32.cuh"

namespace adk {

constexpr int kF32Group = 128;           // threads that share one tile; a CTA is one or two such groups
constexpr int kF32MaxK = 15;             // filter rows / columns: one bit each in a 32-bit word (rows 0.., columns 16..)

// A group is 4 warps, WM x WN of them over rows and columns; a warp's lanes are LM x (32 / LM) over rows and columns, a
// thread owns 8 rows x 8 columns.  A CTA of G = 2 groups (filter gradients) halves every stage's pixels between them: 8
// warps where the grid leaves an SM one CTA.
template <int LM, int WM, int WN, int G> struct F32Tile {
  static constexpr int LN = 32 / LM, BM = 8 * LM * WM, BN = 8 * LN * WN, threads = kF32Group * G;
  static_assert(WM * WN == 4, "four warps");
};

// Sum of one element of the tiles of all groups of all CTAs of the cluster, in order; all loads are in flight together
template <int G, int MOST = 8>
__device__ __forceinline__ float cluster_total(cg::cluster_group& cluster, float* sm, uint32_t cs, size_t at, size_t group_stride) {
  float v[MOST * G];
#pragma unroll
  for (uint32_t q = 0; q < MOST; ++q)
#pragma unroll
    for (int g = 0; g < G; ++g) v[q * G + g] = q < cs ? (cs > 1 ? cluster.map_shared_rank(sm, q) : sm)[at + g * group_stride] : 0.f;
  float t = v[0];
#pragma unroll
  for (uint32_t q = 1; q < MOST * G; ++q) if (q < cs * G) t += v[q];
  return t;
}

// ---------------------------------------------------------------- forward / data gradient
// GEMM: rows m = output channels of the pass, columns = output pixels, reduction kd = (channel, tap), tap fastest.
// A data gradient of a strided layer is one such GEMM per residue class of its pixels (blockIdx.z): the pixels
// (y mod sh, x mod sw) = (ry, rx) meet only the taps whose distance is a multiple of the stride, so no tap is multiplied
// that does not contribute.
// Shared memory: a ring of stages ([kd][m], pitch BM + 4, and [kd][pixel]; KB reduction indices each) beside the BM x BN
// tile of main accumulators, to which the running sums of 64 terms go
template <int LM, int WM, int WN> struct GemmTile : F32Tile<LM, WM, WN, 1> {
  typedef F32Tile<LM, WM, WN, 1> B;
  static constexpr int KB = B::BN > 512 ? 8 : 16, flush = 64 / KB;
  static constexpr int PA = B::BM + 4, stage_floats = KB * (PA + B::BN);
  static constexpr int stages = B::BN > 256 ? 2 : 3;
  static constexpr int smem = (stages * stage_floats + B::BM * B::BN) * 4;
};

template <int LM, int WM, int WN, bool DGRAD>
__global__ void __launch_bounds__(kF32Group, 3) conv_gemm_f32(const GemmF32 p) {
  grid_dependency();
  typedef GemmTile<LM, WM, WN> T;
  constexpr int BM = T::BM, BN = T::BN, LN = T::LN, KB = T::KB, PA = T::PA, STAGES = T::stages;
  constexpr int NPX = BN / kF32Group;                                          // pixels a thread gathers for
  extern __shared__ __align__(16) float sm[];
  float* const tile = sm + STAGES * T::stage_floats;
  __shared__ int tap_off[64], tap_bits[64], tap_w[64], row_t[16], col_t[16], s_ntaps;
  __shared__ int4 tab[2][KB];         // per reduction index of a stage: input offset, needed row and column bits, filter offset

  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t m_base = blockIdx.y * BM;

  // the class of pixels and its taps
  uint32_t ry = 0, rx = 0, my = p.sh, mx = p.sw, OHc = p.OH, OWc = p.OW;
  if (DGRAD) {
    ry = blockIdx.z / p.sw; rx = blockIdx.z % p.sw;
    my = mx = 1;
    OHc = p.OH > ry ? (p.OH - ry + p.sh - 1) / p.sh : 0;
    OWc = p.OW > rx ? (p.OW - rx + p.sw - 1) / p.sw : 0;
  }
  if (warp == 0) {
    // row and column offsets of the taps (INT_MIN / 2: the class does not meet that row or column)
    constexpr int kNone = -(1 << 30);
    int vy = kNone, vx = kNone;
    if (lane < p.kh) {
      const int ay = (int)ry + p.ph - (int)(lane * p.dh);
      vy = DGRAD ? (ay % (int)p.sh == 0 ? ay / (int)p.sh : kNone) : (int)(lane * p.dh) - p.ph;
    }
    if (lane < p.kw) {
      const int ax = (int)rx + p.pw - (int)(lane * p.dw);
      vx = DGRAD ? (ax % (int)p.sw == 0 ? ax / (int)p.sw : kNone) : (int)(lane * p.dw) - p.pw;
    }
    if (lane < 16) { row_t[lane] = vy; col_t[lane] = vx; }
    __syncwarp();
    const int taps = (int)(p.kh * p.kw);
    int base = 0;
    for (int t0 = 0; t0 < taps; t0 += 32) {
      const int t = t0 + (int)lane, i = t / (int)p.kw, j = t - i * (int)p.kw;
      const int ty = t < taps ? row_t[i] : kNone, tx = t < taps ? col_t[j] : kNone;
      const bool ok = ty != kNone && tx != kNone;
      const unsigned b = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        const int at = base + __popc(b & ((1u << lane) - 1u));
        tap_off[at] = (int)(ty * p.in_pitch) + tx;
        tap_bits[at] = (int)((1u << i) | (1u << (16 + j)));
        tap_w[at] = t;
      }
      base += __popc(b);
    }
    if (lane == 0) s_ntaps = base;
  }
  __syncthreads();
  const uint32_t ntaps = (uint32_t)s_ntaps;
  const uint32_t npx = p.NI * OHc * OWc, n_base = (blockIdx.x / cs) * BN;
  if (n_base >= npx) return;          // the whole cluster shares the tile

  // this CTA's share of the reduction
  const uint32_t Kd = p.CR * ntaps;
  const uint32_t per = ((Kd + cs - 1) / cs + KB - 1) / KB * KB;
  const uint32_t k_lo = rank * per < Kd ? rank * per : Kd, k_hi = k_lo + per < Kd ? k_lo + per : Kd;
  const uint32_t steps = (k_hi - k_lo + KB - 1) / KB;

  // the pixels this thread gathers for (and writes): where their windows start, which rows and columns lie inside
  const float* in_px[NPX];
  float* out_px[NPX];
  uint32_t bits[NPX];
#pragma unroll
  for (int u = 0; u < NPX; ++u) {
    const uint32_t pxi = n_base + tid + u * kF32Group;
    in_px[u] = p.in; out_px[u] = nullptr; bits[u] = 0;
    if (pxi < npx) {
      const uint32_t ox = pxi % OWc, r = pxi / OWc, oy = r % OHc, n = r / OHc;
      const int iy0 = (int)(oy * my), ix0 = (int)(ox * mx);
      in_px[u] = p.in + (long long)n * p.in_img + (long long)iy0 * p.in_pitch + ix0;
      for (uint32_t i = 0; i < p.kh; ++i) if ((unsigned)(iy0 + row_t[i]) < p.IH) bits[u] |= 1u << i;
      for (uint32_t j = 0; j < p.kw; ++j) if ((unsigned)(ix0 + col_t[j]) < p.IW) bits[u] |= 1u << (16 + j);
      const uint32_t fy = DGRAD ? oy * p.sh + ry : oy, fx = DGRAD ? ox * p.sw + rx : ox;
      out_px[u] = p.out + (long long)n * p.out_img + (long long)fy * p.out_pitch + fx;
    }
  }

  auto make_tab = [&](uint32_t step) {
    if (tid < KB) {
      const uint32_t kd = k_lo + step * KB + tid;
      int4 e = make_int4(0, (int)kF32Never, 0, 0);
      if (kd < k_hi) {
        const uint32_t c = kd / ntaps, t = kd - c * ntaps;
        e = make_int4((int)(c * p.in_plane) + tap_off[t], tap_bits[t], (int)(c * p.w_c) + tap_w[t], 0);
      }
      tab[step & 1u][tid] = e;
    }
  };
  auto load = [&](uint32_t step) {
    const uint32_t a0 = smem_addr(sm + (size_t)(step % STAGES) * T::stage_floats), b0 = a0 + (KB * PA + tid) * 4;
    const int4* tb = tab[step & 1u];
#pragma unroll
    for (int r = 0; r < KB; ++r) {
      const int2 e = *(const int2*)&tb[r];
#pragma unroll
      for (int u = 0; u < NPX; ++u) gather4(b0 + (r * BN + u * kF32Group) * 4, in_px[u] + e.x, bits[u], (uint32_t)e.y);
    }
#pragma unroll
    for (int i = 0; i < (KB * BM + kF32Group - 1) / kF32Group; ++i) {
      const uint32_t idx = tid + i * kF32Group;
      if (KB * BM % kF32Group && idx >= KB * BM) break;
      // filter rows are contiguous along (channel, tap) forward and along m (taps apart) backward
      const uint32_t r = DGRAD ? idx / BM : idx % KB, m = DGRAD ? idx % BM : idx / KB;
      const int4 e = tb[r];
      gather4(a0 + (r * PA + m) * 4, p.w + ((long long)(m_base + m) * p.w_m + e.z), m_base + m < p.M ? 0x7fffffffu : 0u, (uint32_t)e.y);
    }
  };

  const uint32_t m0 = (warp % WM) * 8 * LM + lane / LN * 8, n0 = (warp / WM) * 8 * LN + lane % LN * 4;
  u64 acc[4][8];                      // [pair of rows][column]: columns n0 .. n0 + 3 and n0 + 4 LN .. n0 + 4 LN + 3
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  auto flush = [&](bool first) {      // running sums -> main accumulators in shared memory (this thread's own elements)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 v = unpack2(acc[i][h * 4 + j]);
          lo[j] = v.x; hi[j] = v.y;
          acc[i][h * 4 + j] = 0ull;
        }
        float4* t0 = (float4*)(tile + (size_t)(m0 + 2 * i) * BN + n0 + h * 4 * LN);
        float4* t1 = t0 + BN / 4;
        float4 o0 = make_float4(lo[0], lo[1], lo[2], lo[3]), o1 = make_float4(hi[0], hi[1], hi[2], hi[3]);
        if (!first) {
          const float4 p0 = *t0, p1 = *t1;
          o0.x += p0.x; o0.y += p0.y; o0.z += p0.z; o0.w += p0.w;
          o1.x += p1.x; o1.y += p1.y; o1.z += p1.z; o1.w += p1.w;
        }
        *t0 = o0; *t1 = o1;
      }
  };
  if (steps) {
    for (uint32_t st = 0; st < STAGES - 1; ++st) {
      make_tab(st);
      __syncthreads();
      if (st < steps) load(st);
      cp_async_commit();
    }
    make_tab(STAGES - 1);
  }
  for (uint32_t st = 0; st < steps; ++st) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < steps) load(st + STAGES - 1);
    cp_async_commit();
    make_tab(st + STAGES);
    const float* As = sm + (size_t)(st % STAGES) * T::stage_floats;
    const float* Bs = As + KB * PA + n0;
    As += m0;
    ulonglong2 na0 = *(const ulonglong2*)As, na1 = *(const ulonglong2*)(As + 4);
    float4 nb0 = *(const float4*)Bs, nb1 = *(const float4*)(Bs + 4 * LN);
#pragma unroll
    for (int r = 0; r < KB; ++r) {     // the next row's operands are read underneath this row's products
      const ulonglong2 a0 = na0, a1 = na1;
      const float4 b0 = nb0, b1 = nb1;
      if (r + 1 < KB) {
        na0 = *(const ulonglong2*)(As + (r + 1) * PA); na1 = *(const ulonglong2*)(As + (r + 1) * PA + 4);
        nb0 = *(const float4*)(Bs + (r + 1) * BN); nb1 = *(const float4*)(Bs + (r + 1) * BN + 4 * LN);
      }
      const u64 av[4] = {a0.x, a0.y, a1.x, a1.y};
      const float bf[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const u64 bb = dup2(bf[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) ffma2(acc[i][j], av[i], bb);
      }
    }
    if (st % T::flush == T::flush - 1) flush(st == T::flush - 1);
  }
  if (steps % T::flush || steps == 0) flush(steps < T::flush);
  if (cs > 1) cluster.sync();
  else __syncthreads();
  // each CTA of the cluster finishes BM / cs rows
  const uint32_t rows = BM / cs;
  for (uint32_t i = 0; i < rows; ++i) {
    const uint32_t m = rank * rows + i;
#pragma unroll
    for (int u = 0; u < NPX; ++u) {
      float v = cluster_total<1, kF32Most>(cluster, tile, cs, (size_t)m * BN + tid + u * kF32Group, 0);
      if (out_px[u] && m_base + m < p.M) {
        float* o = out_px[u] + (long long)(m_base + m) * p.out_plane;
        if (!DGRAD) {
          if (p.bias) v += p.bias[m_base + m];
          if (p.relu) v = fmaxf(v, 0.f);
        } else if (p.accumulate) {
          v += *o;
        }
        *o = v;
      }
    }
  }
  if (cs > 1) cluster.sync();         // nobody leaves while its tile is still read
}

template <int LM, int WM, int WN, bool DGRAD>
static int launch_gemm_f32(const GemmF32& p, uint32_t npx, uint32_t classes, uint32_t Kd, cudaStream_t s) {
  typedef GemmTile<LM, WM, WN> T;
  static F32Launch l;
  const uint32_t tn = (npx + T::BN - 1) / T::BN, tm = (p.M + T::BM - 1) / T::BM;
  // every CTA of a cluster finishes at least one of the BM rows.  Clusters of 16 are for few tiles and long reductions:
  // 4 x 512 x 7 x 7 -> 512, 3x3 (16 tiles) 92 -> 67 us against 8.
  auto held = [](uint32_t n) { return f32_held(conv_gemm_f32<LM, WM, WN, DGRAD>, T::threads, T::smem, n, l); };
  const uint32_t cs = f32_cluster_size(held, (unsigned long long)tn * tm * classes, Kd / T::KB, std::min(kF32Most, (int)T::BM), kNumSMs);
  return launch_f32(conv_gemm_f32<LM, WM, WN, DGRAD>, dim3(tn * cs, tm, classes), T::threads, T::smem, cs, p, l, s);
}

// The parity tests: "2" sends every layer that the 3x3 kernels can serve to them (conv_direct.cu has the other values)
static bool f32_k3_forced() {
  const char* t = getenv("ARRAYDIFF_B200_F32_TILES");
  return t && t[0] == '2';
}

// The 3x3 kernels own blocks of 4 x 2 pixels.  Where more than a fifth of them lies past the edges of the map (a third, if the
// reduction is long), for 16 rows and fewer, and for long reductions into few tiles of 32 rows, which go to 8 CTAs at
// most, the general tiles are as fast or faster: 17 x 42 x 13 x 5 -> 346 channels, two thirds used, 25 against 31 us;
// 9 x 440 x 18 x 22 -> 27, 16 tiles, 48 against 65.  The other way: 4 x 512 x 7 x 7 -> 512 data gradient, two thirds used, 94 -> 66.
// A map under dilation is counted as the maps that it falls into.  With a stride of 2 (forward only) a patch is 45 elements
// instead of 24 and three quarters of a tile's rows and pixels have to be used: 137 -> 209, 2 x 14 x 34, 0.71, 33 against 39 us;
// 156 -> 276, 4 x 12 x 21, 0.82, the other way, 47 -> 43.
static bool f32_k3_gemm_wins(const GemmF32& p, bool dgrad) {
  if (p.kh != 3 || p.kw != 3 || p.sh != p.sw || p.sh > (dgrad ? 1u : 2u) || (p.sh == 2 && (p.dh != 1 || p.dw != 1))) return false;
  if (f32_k3_forced()) return true;
  if (p.M <= 16) return false;
  const unsigned long long used = (unsigned long long)p.OH * p.OW, blocks = f32_k3_blocks(p.OH, p.OW, p.dh, p.dw);
  if (p.M <= 32 && p.CR > 128 && p.NI * blocks < (p.sh == 2 ? 48 : 24) * 32) return false;
  if (p.sh == 2 && p.M > 32 && 4 * used * p.M < 3 * 8 * blocks * ((p.M + 63) / 64 * 64)) return false;
  return used * 20 >= blocks * 8 * (p.CR >= 192 ? 13 : 16);
}

// Tiles of 32 rows and more: for 16 and fewer most of one would be zeros.  Faster or equal at every size measured above that
// (300 layers of 17 to 600 channels, strides 1 to 3, maps from 7 x 7) but where single pixels are gathered from far apart for
// few rows (8 x 192 x 235 x 280 -> 21, stride 3: 68 against 60 us).
static bool f32_k1_gemm_wins(const GemmF32& p, bool dgrad) {
  if (!dgrad && p.M <= 32 && p.sh * p.sw > 4) return false;
  return p.kh == 1 && p.kw == 1 && !p.ph && !p.pw && p.M > 16;
}

// Tile height by the row count: a row of the tile costs the same FMAs whether it holds a channel or not, a column is
// gathered once per tile row: 64 x 128 for more than 32 channels, 32 x 256, 16 x 512 and 8 x 1024 below.
template <bool DGRAD>
static int run_gemm_f32(const GemmF32& p, cudaStream_t s) {
  const uint32_t classes = DGRAD ? p.sh * p.sw : 1;
  const uint32_t OHc = DGRAD ? (p.OH + p.sh - 1) / p.sh : p.OH, OWc = DGRAD ? (p.OW + p.sw - 1) / p.sw : p.OW;
  const uint32_t npx = p.NI * OHc * OWc, Kd = p.CR * ((p.kh * p.kw + classes - 1) / classes);
  if (f32_k3_gemm_wins(p, DGRAD)) return f32_k3_gemm<DGRAD>(p, s);
  if (f32_k1_gemm_wins(p, DGRAD)) return f32_k1_gemm<DGRAD>(p, s);
  if (p.M <= 8) return launch_gemm_f32<1, 1, 4, DGRAD>(p, npx, classes, Kd, s);
  if (p.M <= 16) return launch_gemm_f32<2, 1, 4, DGRAD>(p, npx, classes, Kd, s);
  if (p.M <= 32) return launch_gemm_f32<4, 1, 4, DGRAD>(p, npx, classes, Kd, s);
  return launch_gemm_f32<4, 2, 2, DGRAD>(p, npx, classes, Kd, s);
}

// ---------------------------------------------------------------- filter gradient
// GEMM: rows m = output channels, columns n = (input channel, tap), reduction = output pixels, which is the order both
// operands have in memory.  The reduction is split over the CTAs of a cluster and over `slices` of the grid; with more
// than one slice the clusters write partial gradients to scratch and wgrad_f32_finish adds them in order.
// Shared memory: a ring of stages ([row][32 pixels], pitch 36: reads and writes free of bank conflicts) beside the BM x BN
// tile of main accumulators.  One packed FMA multiplies two neighbouring pixels; the halves are added at the end.
constexpr int kWgKB = 32, kWgPitch = 36, kWgStages = 2, kWgFlush = 8;

template <int LM, int WM, int WN, int G> struct WgTile : F32Tile<LM, WM, WN, G> {
  typedef F32Tile<LM, WM, WN, G> B;
  static constexpr int group_floats = (B::BM + B::BN) * kWgPitch, stage_floats = G * group_floats;
  static constexpr int smem = (kWgStages * stage_floats + G * B::BM * B::BN) * 4;
};

template <int LM, int WM, int WN, int G>
__global__ void __launch_bounds__(kF32Group * G, G == 1 ? 2 : 1) conv_wgrad_gemm_f32(const WgradF32 p) {
  grid_dependency();
  typedef WgTile<LM, WM, WN, G> T;
  constexpr int BM = T::BM, BN = T::BN, LN = T::LN, STAGES = kWgStages, PITCH = kWgPitch, KB = kWgKB;
  extern __shared__ __align__(16) float sm[];
  float* const tile = sm + STAGES * T::stage_floats;
  __shared__ int2 col[BN];            // per column: input offset of (channel, tap), row and column bits
  __shared__ int row_t[16], col_t[16];
  __shared__ float sdb[G * BM];
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t group = threadIdx.x / kF32Group, tid = threadIdx.x % kF32Group, warp = tid >> 5, lane = tid & 31;
  const uint32_t taps = p.kh * p.kw, NC = p.C * taps;
  const uint32_t n_base = (blockIdx.x / cs) * BN, m_base = blockIdx.y * BM, slice = blockIdx.z;
  const long long x_img = (long long)p.C * p.H * p.W, dy_img = (long long)p.K * p.dy_plane;
  if (threadIdx.x < 16) { row_t[tid] = (int)(tid * p.dh) - p.ph; col_t[tid] = (int)(tid * p.dw_) - p.pw; }
  for (uint32_t i = threadIdx.x; i < BN; i += T::threads) {
    const uint32_t n = n_base + i;
    int2 e = make_int2(0, (int)kF32Never);
    if (n < NC) {
      const uint32_t c = n / taps, t = n - c * taps, ti = t / p.kw, tj = t - ti * p.kw;
      e = make_int2((int)(c * p.H * p.W) + ((int)(ti * p.dh) - p.ph) * (int)p.W + (int)(tj * p.dw_) - p.pw, (int)((1u << ti) | (1u << (16 + tj))));
    }
    col[i] = e;
  }
  __syncthreads();
  const uint32_t npx = p.N * p.P * p.Q, pq = p.P * p.Q;
  const uint32_t all = (npx + KB * G - 1) / (KB * G), parts = cs * p.slices, per = (all + parts - 1) / parts, me = slice * cs + rank;
  const uint32_t s_lo = me * per < all ? me * per : all, steps = (s_lo + per < all ? s_lo + per : all) - s_lo;

  auto load = [&](uint32_t st) {
    const uint32_t pxi = ((s_lo + st) * G + group) * KB + lane;
    float* As = sm + (size_t)(st % STAGES) * T::stage_floats + group * T::group_floats;
    const bool in = pxi < npx;
    const uint32_t n = in ? pxi / pq : 0, r = in ? pxi - n * pq : 0, oy = r / p.Q, ox = r - oy * p.Q;
    const float* dp = p.dy + (long long)n * dy_img + (long long)oy * p.dy_pitch + ox + (long long)(m_base + warp) * p.dy_plane;
    const uint32_t a0 = smem_addr(As + warp * PITCH + lane), b0 = a0 + BM * PITCH * 4;
#pragma unroll 16
    for (int i = 0; i < BM / 4; ++i) {
      gather4(a0 + i * 4 * PITCH * 4, dp, in && m_base + warp + i * 4 < p.K, 1u);
      dp += 4 * p.dy_plane;
    }
    const int iy0 = (int)(oy * p.sh), ix0 = (int)(ox * p.sw);
    uint32_t bits = 0;
    if (in) {
      for (uint32_t i = 0; i < p.kh; ++i) if ((unsigned)(iy0 + row_t[i]) < p.H) bits |= 1u << i;
      for (uint32_t j = 0; j < p.kw; ++j) if ((unsigned)(ix0 + col_t[j]) < p.W) bits |= 1u << (16 + j);
    }
    const float* xp = p.x + (long long)n * x_img + (long long)iy0 * p.W + ix0;
    // columns past the last (channel, tap) are left as they are: what is summed there is not written (9 columns of 512, one
    // input channel: most of the time went into zeros)
    const int rows = (int)(NC - n_base < BN ? NC - n_base : BN) - (int)warp;
#pragma unroll 16
    for (int i = 0; i < BN / 4; ++i) {
      if (i * 4 >= rows) break;
      const int2 e = col[warp + i * 4];
      gather4(b0 + i * 4 * PITCH * 4, xp + e.x, bits, (uint32_t)e.y);
    }
  };

  const uint32_t m0 = (warp % WM) * 8 * LM + lane / LN, n0 = (warp / WM) * 8 * LN + lane % LN;
  u64 acc[8][8];                      // rows m0 + i LM, columns n0 + j LN
  float dbs = 0.f;
  const bool with_db = p.db && n_base == 0;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  auto flush = [&](bool first) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 v = unpack2(acc[i][j]);
        float* t = tile + ((size_t)group * BM + m0 + i * LM) * BN + n0 + j * LN;
        *t = first ? v.x + v.y : *t + (v.x + v.y);
        acc[i][j] = 0ull;
      }
  };
  for (uint32_t st = 0; st < STAGES - 1; ++st) {
    if (st < steps) load(st);
    cp_async_commit();
  }
  for (uint32_t st = 0; st < steps; ++st) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    if (st + STAGES - 1 < steps) load(st + STAGES - 1);
    cp_async_commit();
    const float* As = sm + (size_t)(st % STAGES) * T::stage_floats + group * T::group_floats;
    const float* a0 = As + m0 * PITCH;
    const float* b0 = As + (BM + n0) * PITCH;
#pragma unroll
    for (int q = 0; q < KB / 4; ++q) {
      ulonglong2 b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = *(const ulonglong2*)(b0 + j * LN * PITCH + q * 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const ulonglong2 a = *(const ulonglong2*)(a0 + i * LM * PITCH + q * 4);
#pragma unroll
        for (int j = 0; j < 8; ++j) { ffma2(acc[i][j], a.x, b[j].x); ffma2(acc[i][j], a.y, b[j].y); }
      }
    }
    if (with_db && tid < BM) {        // the bias gradient: row sums of the same dy tile
      float d = 0.f;
#pragma unroll
      for (int q = 0; q < KB / 4; ++q) {
        const float4 v = *(const float4*)(As + tid * PITCH + q * 4);
        d += (v.x + v.y) + (v.z + v.w);
      }
      dbs += d;
    }
    if (st % kWgFlush == kWgFlush - 1) flush(st == kWgFlush - 1);
  }
  if (steps % kWgFlush || steps == 0) flush(steps < kWgFlush);
  if (with_db && tid < BM) sdb[group * BM + tid] = dbs;
  if (cs > 1) cluster.sync();
  else __syncthreads();
  const uint32_t rows = BM / cs;
  float* const dw = p.slices > 1 ? p.part + (size_t)slice * ((size_t)p.K * NC + p.K) : p.dw;
  float* const db = p.slices > 1 ? dw + (size_t)p.K * NC : p.db;
  const bool acc_out = p.accumulate && p.slices == 1;
  for (uint32_t e = threadIdx.x; e < rows * BN; e += T::threads) {
    const uint32_t m = rank * rows + e / BN, n = e % BN;
    const float v = cluster_total<G>(cluster, tile, cs, (size_t)m * BN + n, (size_t)BM * BN);
    if (m_base + m < p.K && n_base + n < NC) {
      float* o = dw + (size_t)(m_base + m) * NC + n_base + n;
      *o = acc_out ? *o + v : v;
    }
  }
  if (with_db && threadIdx.x < rows && m_base + rank * rows + threadIdx.x < p.K) {
    const uint32_t m = rank * rows + threadIdx.x;
    const float v = cluster_total<G>(cluster, sdb, cs, m, BM);
    float* o = db + m_base + m;
    *o = acc_out ? *o + v : v;
  }
  if (cs > 1) cluster.sync();
}

// dw (+)= sum of the slices, in order; the bias gradient's K values follow the filter's
__global__ void __launch_bounds__(256) wgrad_f32_finish(size_t n, uint32_t K, uint32_t slices, const float* __restrict__ part, float* dw,
                                                        float* db, int accumulate) {
  grid_dependency();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x, stride = n + K;
  if (i >= (db ? stride : n)) return;
  float v[16], t = 0.f;
#pragma unroll
  for (uint32_t s = 0; s < 16; ++s) v[s] = s < slices ? part[s * stride + i] : 0.f;
#pragma unroll
  for (uint32_t s = 0; s < 16; ++s) t += v[s];
  float* o = i < n ? dw + i : db + (i - n);
  *o = accumulate ? *o + t : t;
}

static uint32_t wg_rows(uint32_t K) { return K > 32 ? 64u : (K > 16 ? 32u : 16u); }
static uint32_t wg_cols(uint32_t K) { return 8192u / wg_rows(K); }
// Slices of the pixel range beyond a cluster of 8, each CTA with at least eight stages of pixels: as many clusters as the
// machine holds at a time with two CTAs per SM.  That is the number of the form with 64 rows and one group (88 KB); the forms
// of 32 and 16 rows and the one of two groups (116 to 185 KB) have one CTA per SM and hold about half as many, so that
// their last slices are a second wave.
constexpr unsigned long long kWgHeld = 33;
static uint32_t wg_slices(const ad_conv2d_args* a, uint32_t P, uint32_t Q) {
  const unsigned long long tiles = (unsigned long long)((a->K + wg_rows(a->K) - 1) / wg_rows(a->K)) *
                                   ((a->C * a->kh * a->kw + wg_cols(a->K) - 1) / wg_cols(a->K));
  const unsigned long long steps = ((unsigned long long)a->N * P * Q + kWgKB - 1) / kWgKB;
  const unsigned long long fit = kWgHeld / tiles, most = steps / (8 * 8);
  const unsigned long long n = fit < most ? fit : most;
  return (uint32_t)(n > 16 ? 16 : (n < 1 ? 1 : n));
}

static int finish_wgrad_f32(const WgradF32& p, cudaStream_t s) {
  const size_t n = (size_t)p.K * p.C * p.kh * p.kw;
  launch(wgrad_f32_finish, (unsigned)((n + p.K + 255) / 256), 256, 0, s, n, p.K, p.slices, p.part, p.dw, p.db, p.accumulate);
  count_launch();
  return launch_status();
}

template <int LM, int WM, int WN, int G>
static int launch_wgrad_f32(WgradF32& p, cudaStream_t s) {
  typedef WgTile<LM, WM, WN, G> T;
  static F32Launch l;
  const uint32_t tn = (p.C * p.kh * p.kw + T::BN - 1) / T::BN, tm = (p.K + T::BM - 1) / T::BM;
  const uint32_t steps = p.N * p.P * p.Q / (kWgKB * G) / p.slices;
  auto held = [](uint32_t n) { return f32_held(conv_wgrad_gemm_f32<LM, WM, WN, G>, T::threads, T::smem, n, l); };
  const uint32_t cs = p.slices > 1 ? f32_largest_cluster(held, 8) : f32_cluster_size(held, (unsigned long long)tn * tm, steps, 8, kNumSMs);
  int st = launch_f32(conv_wgrad_gemm_f32<LM, WM, WN, G>, dim3(tn * cs, tm, p.slices), T::threads, T::smem, cs, p, l, s);
  return st != AD_OK || p.slices == 1 ? st : finish_wgrad_f32(p, s);
}

// ---------------------------------------------------------------- entry points (called by conv_direct.cu)
static bool fits31(long long v) { return v >= 0 && v < (1ll << 31); }

// Limits of the tiled kernels: 32-bit offsets inside one image and one filter, 31-bit pixel counts, a bit per filter row
// and column.
bool f32_gemm_ok(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane) {
  if (a->kh > kF32MaxK || a->kw > kF32MaxK || a->kh * a->kw > 64) return false;
  if ((unsigned long long)a->stride_h * a->stride_w > 65535) return false;
  const long long reach = ((long long)a->dil_h * (a->kh - 1) + a->pad_h + 1) * ((long long)a->W + y_pitch) + (long long)a->dil_w * (a->kw - 1) + a->pad_w;
  return fits31(reach) && fits31((long long)a->C * a->H * a->W + reach) && fits31((long long)a->K * y_plane + reach) &&
         fits31((long long)a->N * P * Q) && fits31((long long)a->N * a->H * a->W) && fits31((long long)a->K * a->C * a->kh * a->kw) &&
         a->K <= 65535u * 8 && a->C <= 65535u * 8 && y_pitch >= 0 && y_plane >= 0;
}

// The 3x3 kernel's tiles are 64 x 16 channels (32 x 32 for up to 32 output channels), the general one's 64 x 128 (channel, tap)
// columns: it wins from 16 channels on where more than half of its tiles is used (11 channels: 35 against 47 us, 14: 36
// against 63, 17: 109 against 137, 33 output channels: 79 against 103; the other way 25: 430 -> 367, 32: 54 -> 52).  One tile
// alone is split into 128 CTAs at most: with more than four stages for each, the general kernel, which has more of them, is
// faster (8 x 24 x 60 x 60 -> 32: 47 against 56 us).
static bool f32_k3_wgrad_wins(const ad_conv2d_args* a, uint32_t P, uint32_t Q) {
  if (a->kh != 3 || a->kw != 3 || a->stride_h != a->stride_w || a->stride_h > 2) return false;
  if (a->stride_h == 2 && (a->dil_h != 1 || a->dil_w != 1)) return false;
  if (f32_k3_forced()) return true;
  if (a->K <= 16 || a->C < 16) return false;
  if (a->K <= 64 && a->C <= (a->K <= 32 ? 32u : 16u) && (unsigned long long)a->N * P * f32_k3_segments(Q, a->dil_w) > 4 * 4 * 128) return false;
  // under dilation a segment's pixels are dil apart: seven tenths of segments and tiles together (27 x 41 x 14 x 33 -> 57, dilation 4,
  // 0.37: 39 against 54 us; 29 x 26 x 16 x 58 -> 177, 0.68: 118 against 131)
  const unsigned bk = a->K <= 32 ? 32 : 64, bc = a->K <= 32 ? 32 : 16;
  const unsigned long long k = (a->K + bk - 1) / bk * bk, c = (a->C + bc - 1) / bc * bc;
  if (a->dil_w > 1 && (a->dil_w > Q || 10ull * a->K * a->C * Q < 7ull * k * c * f32_k3_segments(Q, a->dil_w) * 8)) return false;
  if (a->K <= 32) return true;
  return 25ull * a->K * a->C >= 14ull * k * c;
}
size_t f32_wgrad_scratch(const ad_conv2d_args* a, uint32_t P, uint32_t Q) {
  const uint32_t s = f32_k3_wgrad_wins(a, P, Q) ? f32_k3_wgrad_split(a->K, a->C, a->N, P, Q, a->stride_w, a->dil_w).slices : wg_slices(a, P, Q);
  return s > 1 ? (size_t)s * ((size_t)a->K * a->C * a->kh * a->kw + a->K) * 4 : 0;
}

// Measured (one B200; per call, thread per output -> these tiles): 64 -> 64 channels, 3x3, 64 x 64 pixels, one image: forward
// 188 -> 21 us, data gradient 158 -> 25, filter and bias gradient 286 -> 31.  4 x 64 x 112 x 112, 64 -> 64 3x3: 1440 -> 135, 1500 ->
// 134, 2330 -> 172 us (27 / 28 / 21 TFLOP/s); conv_f32_k3.cu, which serves these two now, takes 17, 21, 23 and 94, 92, 127.
// What is left above the FMA pipe: 12 warps per SM do not hide the latency of the shared-memory reads (issue slots 42 % busy);
// 4 x 8 outputs per thread or packed pairs along the reduction were slower.
int f32_gemm_fprop(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s) {
  GemmF32 p = {};
  p.in = (const float*)a->x; p.w = (const float*)a->w; p.bias = a->bias; p.out = (float*)a->y;
  p.M = a->K; p.CR = a->C; p.NI = a->N; p.IH = a->H; p.IW = a->W;
  p.in_pitch = a->W; p.in_plane = (long long)a->H * a->W; p.in_img = p.in_plane * a->C;
  p.OH = P; p.OW = Q; p.out_pitch = y_pitch; p.out_plane = y_plane; p.out_img = y_plane * a->K;
  p.w_m = (long long)a->C * a->kh * a->kw; p.w_c = (long long)a->kh * a->kw;
  p.kh = a->kh; p.kw = a->kw; p.sh = a->stride_h; p.sw = a->stride_w; p.dh = a->dil_h; p.dw = a->dil_w;
  p.ph = (int)a->pad_h; p.pw = (int)a->pad_w; p.relu = a->relu;
  return run_gemm_f32<false>(p, s);
}

// Data gradient into few channels (an image's three), with scratch: per pixel of dy the products of all (channel, tap) rows
// with the filter as one GEMM -- Z[n][channel, tap][pixel], a 1x1 convolution of dy -- and then the sum over the taps of
// each input pixel, in tap order.  As the GEMM above, 3 of 8 rows of a tile are used and every element of dy is gathered
// once per tap: bound by the gathers.  4 x 64 x 224 x 224 -> 3, 7x7: 730 -> 250 us.
// Images are taken as many at a time as fit kFewZ bytes (f32_few_images); larger ones go the other way.
constexpr size_t kFewZ = 64u << 20;
static size_t few_z_bytes(const ad_conv2d_args* a, uint32_t P, uint32_t Q) { return (size_t)P * Q * a->C * a->kh * a->kw * 4; }   // one image
static uint32_t few_images(const ad_conv2d_args* a, uint32_t P, uint32_t Q) {
  return f32_few_images(a->N, (unsigned long long)a->C * a->H * a->W, few_z_bytes(a, P, Q), kFewZ);
}
size_t f32_dgrad_scratch(const ad_conv2d_args* a, uint32_t P, uint32_t Q) {
  if (a->C > 8 || a->kh * a->kw < 4 || a->K < 16) return 0;
  return few_z_bytes(a, P, Q) * few_images(a, P, Q);
}
__global__ void __launch_bounds__(256) dgrad_few_sum(const float* __restrict__ z, float* dx, uint32_t N, uint32_t C, uint32_t H, uint32_t W,
                                                     uint32_t P, uint32_t Q, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw,
                                                     uint32_t dh, uint32_t dw, int ph, int pw, int accumulate) {
  grid_dependency();
  const uint32_t total = N * C * H * W, pq = P * Q;   // below 2^31: f32_few_images
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < total; i += gridDim.x * 256) {
    const uint32_t x = i % W, r = i / W, y = r % H, nc = r / H;
    const float* zc = z + (size_t)nc * kh * kw * pq;
    float v = 0.f;
    for (uint32_t ti = 0; ti < kh; ++ti) {
      const int ay = (int)y + ph - (int)(ti * dh);
      if (ay < 0 || ay % (int)sh || (uint32_t)ay / sh >= P) continue;
      const float* zr = zc + (size_t)ti * kw * pq + (size_t)((uint32_t)ay / sh) * Q;
#pragma unroll 7
      for (uint32_t tj = 0; tj < kw; ++tj) {
        const int ax = (int)x + pw - (int)(tj * dw);
        const uint32_t ox = (uint32_t)ax / sw;
        v += ax >= 0 && ox * sw == (uint32_t)ax && ox < Q ? zr[(size_t)tj * pq + ox] : 0.f;
      }
    }
    dx[i] = accumulate ? dx[i] + v : v;
  }
}
static int f32_dgrad_few(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s) {
  const uint32_t M = a->C * a->kh * a->kw, step = few_images(a, P, Q);
  for (uint32_t n0 = 0; n0 < a->N; n0 += step) {
    const uint32_t n = std::min(step, a->N - n0);
    GemmF32 p = {};
    p.in_pitch = y_pitch; p.in_plane = y_plane; p.in_img = y_plane * a->K;
    p.in = (const float*)a->y + (long long)n0 * p.in_img; p.w = (const float*)a->w; p.out = (float*)a->scratch;
    p.M = M; p.CR = a->K; p.NI = n; p.IH = P; p.IW = Q;
    p.OH = P; p.OW = Q; p.out_pitch = Q; p.out_plane = (long long)P * Q; p.out_img = p.out_plane * M;
    p.w_m = 1; p.w_c = M;
    p.kh = p.kw = p.sh = p.sw = p.dh = p.dw = 1;
    const int rc = run_gemm_f32<false>(p, s);
    if (rc != AD_OK) return rc;
    launch(dgrad_few_sum, grid_for((size_t)n * a->C * a->H * a->W, 256, 16), 256, 0, s, (const float*)a->scratch,
           (float*)a->dx + (size_t)n0 * a->C * a->H * a->W, n, a->C, a->H, a->W, P, Q, a->kh, a->kw, a->stride_h, a->stride_w, a->dil_h,
           a->dil_w, (int)a->pad_h, (int)a->pad_w, a->accumulate);
    count_launch();
  }
  return launch_status();
}

int f32_gemm_dgrad(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s) {
  const size_t need = f32_dgrad_scratch(a, P, Q);
  if (need && a->scratch && a->scratch_bytes >= need) return f32_dgrad_few(a, P, Q, y_pitch, y_plane, s);
  GemmF32 p = {};
  p.in = (const float*)a->y; p.w = (const float*)a->w; p.out = (float*)a->dx;
  p.M = a->C; p.CR = a->K; p.NI = a->N; p.IH = P; p.IW = Q;
  p.in_pitch = y_pitch; p.in_plane = y_plane; p.in_img = y_plane * a->K;
  p.OH = a->H; p.OW = a->W; p.out_pitch = a->W; p.out_plane = (long long)a->H * a->W; p.out_img = p.out_plane * a->C;
  p.w_m = (long long)a->kh * a->kw; p.w_c = (long long)a->C * a->kh * a->kw;
  p.kh = a->kh; p.kw = a->kw; p.sh = a->stride_h; p.sw = a->stride_w; p.dh = a->dil_h; p.dw = a->dil_w;
  p.ph = (int)a->pad_h; p.pw = (int)a->pad_w; p.accumulate = a->accumulate;
  return run_gemm_f32<true>(p, s);
}

int f32_gemm_wgrad(const ad_conv2d_args* a, uint32_t P, uint32_t Q, long long y_pitch, long long y_plane, cudaStream_t s) {
  WgradF32 p = {};
  p.x = (const float*)a->x; p.dy = (const float*)a->y; p.dw = (float*)a->dw; p.db = a->db;
  p.K = a->K; p.C = a->C; p.N = a->N; p.P = P; p.Q = Q; p.H = a->H; p.W = a->W;
  p.kh = a->kh; p.kw = a->kw; p.sh = a->stride_h; p.sw = a->stride_w; p.dh = a->dil_h; p.dw_ = a->dil_w;
  p.ph = (int)a->pad_h; p.pw = (int)a->pad_w;
  p.dy_pitch = y_pitch; p.dy_plane = y_plane; p.accumulate = a->accumulate;
  p.slices = 1;
  const size_t need = f32_wgrad_scratch(a, P, Q);
  const bool k3 = f32_k3_wgrad_wins(a, P, Q), parts = need && a->scratch && a->scratch_bytes >= need;
  const F32Split split = k3 ? f32_k3_wgrad_split(a->K, a->C, a->N, P, Q, a->stride_w, a->dil_w) : F32Split{8, wg_slices(a, P, Q)};
  if (parts) { p.slices = split.slices; p.part = (float*)a->scratch; }
  if (k3) {
    const int rc = f32_k3_wgrad(p, parts || split.slices == 1 ? split.cs : 8, s);
    return rc != AD_OK || p.slices == 1 ? rc : finish_wgrad_f32(p, s);
  }
  // clusters of 8 fill at most one CTA per SM: two groups per CTA (9 tiles of 4096 pixels: 31 -> 27 us)
  const unsigned long long tiles = (unsigned long long)((a->K + 63) / 64) * ((a->C * a->kh * a->kw + 127) / 128) * p.slices;
  switch (wg_rows(a->K)) {
    case 64: return tiles * 8 <= kNumSMs ? launch_wgrad_f32<4, 2, 2, 2>(p, s) : launch_wgrad_f32<4, 2, 2, 1>(p, s);
    case 32: return launch_wgrad_f32<4, 1, 4, 1>(p, s);
    default: return launch_wgrad_f32<2, 1, 4, 1>(p, s);
  }
}

}  // namespace adk
