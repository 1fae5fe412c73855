// Implicit-GEMM convolution on the 5th-generation tensor cores (tcgen05.mma, accumulators in
// tensor memory), operands staged by TMA tile loads into 128-byte-swizzled shared memory.
// NHWC bf16 activations, KRSC bf16 filters, fp32 accumulate.
//
//   forward / data gradient   conv_tc_fwd_kernel
//       GEMM  M = 128 output pixels (a TH x TW patch of one image), N = BN output channels,
//       K = taps x channels walked in 64-channel slabs.  For every (tap, slab) ONE 4-D TMA box
//       load fetches the shifted (dilated, strided) activation patch [128 pixels][64 ch], which
//       lands exactly in the K-major SWIZZLE_128B operand layout, so no im2col is materialised.
//       The data gradient of a stride-1 convolution is the same kernel run over dy with the
//       taps mirrored and the filter transposed to C,R,S,K.
//       Persistent CTAs (one per SM) loop over tiles; warp 0 = TMA producer, warp 1 = MMA
//       issuer (one elected thread), warps 2-9 = two epilogue groups of four.  Two accumulators in
//       tensor memory let the epilogue of tile i overlap the MMAs of tile i+1.
//   filter gradient           conv_tc_wgrad_kernel
//       GEMM  M = 128 output channels of dy, N = BN input channels of x, K = pixels.  Both
//       operands are the NHWC tiles as TMA delivers them ([pixel][64 ch] rows), consumed as
//       MN-major operands; warps 2-5 are the epilogue.  The pixel range is split across CTAs; each split writes an fp32
//       partial to caller scratch and a second kernel sums the partials in a fixed order
//       (reproducible, no atomics).
//
// Every mbarrier wait is bounded; on expiry the kernel raises an abort flag, all roles leave
// their loops, tensor memory is freed and AD_ERR_TIMEOUT is written to a status word.
// No TMA load here uses cluster multicast.
#include "common.cuh"
#include <algorithm>

#include "bias_grad.cuh"
#include "conv_tc_plan.h"
#include "overlap.h"
#include "tc_common.cuh"

#include <cstdlib>
#include <mutex>
#include <vector>

namespace adk {
namespace tc {

EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
    else
      cudaGetLastError();
  });
  return fn;
}

int make_tmap_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box, const uint32_t* elem_strides) {
  EncodeTiledFn enc = get_encode_tiled();
  if (!enc) return AD_ERR_CUDA;
  if (((uintptr_t)base & 15u) != 0) return AD_ERR_ALIGN;
  cuuint64_t gdim[5], gstr[5];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = elem_strides[i];
    if (box[i] == 0 || box[i] > 256) return AD_ERR_UNSUPPORTED;
  }
  for (int i = 1; i < rank; ++i) {
    gstr[i - 1] = strides_bytes[i];
    if (strides_bytes[i] % 16) return AD_ERR_ALIGN;
  }
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bx, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? AD_OK : AD_ERR_CUDA;
}

constexpr int kTileM = 128;         // pixels (fwd) / dy channels (wgrad) per tile = TMEM lanes
constexpr int kSlabBytes = 16384;   // one [128 rows][64 bf16] swizzled operand slab
constexpr int kThreads = 192;       // filter-gradient kernel: warp 0 TMA, warp 1 MMA, warps 2..5 epilogue
constexpr int kFwdThreads = 320;    // forward kernel: warp 0 TMA, warp 1 MMA, two groups of 4 epilogue warps

// The forward kernel is persistent, one CTA per SM, with two accumulators.  What bounds it where the contraction is long is the
// rate at which an SM gets operand tiles from the L2 (64 bytes per clock): a [128 pixels][256 channels] tile takes 48 KB per 64 of
// depth.  PAIR: two CTAs make [256][256] together (cta_group::2), each loading its own pixels and half of the filter
// rows, 32 KB.  512 -> 512 channels, 3x3, 65,536 pixels: 198 -> 180 us, 1024 -> 2048
// 1x1 261 -> 179.
// The outputs that a launch computes fall into classes of one tap list each: one class, except for the data gradient of a
// strided layer (conv_tc_dgrad), where a pixel's taps depend on its row and column modulo the stride.
struct FwdClass {
  uint32_t tile0;           // first pixel tile
  uint32_t OP, OQ, tiles_y, tiles_x;
  uint32_t nr, ns;          // taps: rows x columns (nr * ns = 0: the outputs are zero)
  int32_t offy, offx;
  uint32_t tap0, tap_r, tap_s;   // place in the filter of tap (r, s): tap0 + r * tap_r + s * tap_s
  long long out_off;        // element offset of its first output
};
constexpr int kFwdClasses = 4;
struct FwdParams {
  uint32_t NI, OP, OQ, OC;  // output: images, rows, cols, channels
  uint32_t CK;              // reduction channels per tap (multiple of 64)
  uint32_t kh, kw, sh, sw, dh, dw;
  int32_t offy, offx;       // input row = oy*sh + r*dh + offy
  uint32_t TH, TW, tiles_y, tiles_x, tiles_n;
  uint32_t TN, tiles_b;     // a tile spans TN images of TH x TW pixels (small maps); tiles_b = ceil(NI / TN)
  long long out_pitch, out_plane;  // elements between output rows / images
  __nv_bfloat16* out;
  const float* bias;
  int32_t relu, accumulate;
  int32_t* status;
  int32_t tma_store;   // epilogue: stage 64-channel chunks in shared memory, one TMA tile store each
  long long out_px;    // elements between output pixels of a row
  const __nv_bfloat16* add;   // tma_store, one class: added to the rounded outputs (a residual sum); pixels OC apart
  long long add_pitch, add_plane;
};
struct FwdClasses { FwdClass c[kFwdClasses]; uint32_t n; };
template <int NC> struct FwdOut { CUtensorMap map[NC]; };
// Where tile number `tile` of the launch lies: channel tile tn, pixel tile (n, ty, tx) of class cls (n >= NI: none, a CTA
// pair has an odd tile too many).  The channel tiles of one pixel tile (of the two of a pair) follow one another, so that
// they read it together: with all pixel tiles of one channel tile first, wide inputs came from DRAM once per channel tile
// (1024 -> 2048, 1x1, 65,536 pixels: 291 -> 231 us without pairs).
struct FwdTile { uint32_t tn, tx, ty, n, cls; };
template <int NC, bool PAIR>
__device__ __forceinline__ FwdTile fwd_tile(const FwdParams& p, const FwdClasses& k, uint32_t rank, uint32_t tile) {
  FwdTile t;
  t.tn = tile % p.tiles_n;
  uint32_t tm = tile / p.tiles_n * (PAIR ? 2 : 1) + rank;
  uint32_t tx = p.tiles_x, ty = p.tiles_y;
  t.cls = 0;
  if (NC > 1) {
    while (t.cls + 1 < k.n && tm >= k.c[t.cls + 1].tile0) ++t.cls;
    tm -= k.c[t.cls].tile0;
    tx = k.c[t.cls].tiles_x; ty = k.c[t.cls].tiles_y;
  }
  t.tx = tm % tx; t.ty = (tm / tx) % ty; t.n = tm / (tx * ty) * p.TN;
  return t;
}

constexpr int kStagingBytes = 4 * 16384;   // two 64-channel chunks for each of the two epilogue groups

struct SmemCtl {
  unsigned long long full[8], empty[8], tfull[2], tempty[2], stg_full[4], stg_free[4];
  uint32_t tmem_base;
  volatile int abort_flag;
};

// End of a CTA pair's producer: every stage has been given back.  The arrivals come from the other CTA, so a CTA must not
// leave (and its shared memory must not go to another one) before they are there.
template <int STAGES>
__device__ __forceinline__ void await_stages(SmemCtl* ctl, uint32_t stage, uint32_t phase, volatile int* abortf) {
  for (int i = 0; i < STAGES; ++i) {
    if (!mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1u, abortf)) return;
    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
  }
}

__device__ __forceinline__ uint32_t pow2_cols(uint32_t c) {
  uint32_t p = 32;
  while (p < c) p <<= 1;
  return p;
}

template <int BN, int STAGES, int NC, bool PAIR>
__global__ void __launch_bounds__(kFwdThreads, 1)
conv_tc_fwd_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ FwdOut<NC> out, const FwdParams p, const __grid_constant__ FwdClasses cl) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kCtas = PAIR ? 2 : 1;
  constexpr uint32_t kStageBytes = kSlabBytes + BN / kCtas * 128;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* osm = smem + (size_t)STAGES * kStageBytes;
  SmemCtl* ctl = (SmemCtl*)(osm + kStagingBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles_m = NC > 1 ? p.tiles_x : p.tiles_b * p.tiles_y * p.tiles_x;   // classes: the host has summed them up
  const uint32_t total_tiles = (tiles_m + kCtas - 1) / kCtas * p.tiles_n;
  const uint32_t rank = PAIR ? cluster_rank() : 0u, first = blockIdx.x / kCtas, step = gridDim.x / kCtas;
  const uint32_t slabs = p.CK / 64;
  constexpr uint32_t kTmemCols = 2 * BN < 32 ? 32 : 2 * BN;  // BN in {32,64,128,256} -> power of two

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ctl->full[s]), 1);
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ctl->tfull[a]), 1);
      // an accumulator is drained by both epilogue groups when a tile has several 64-channel chunks
      mbar_init(smem_u32(&ctl->tempty[a]), ((p.tma_store && BN >= 128) ? 8 : 4) * kCtas);
    }
    for (int b = 0; b < 4; ++b) {
      mbar_init(smem_u32(&ctl->stg_full[b]), 4);
      mbar_init(smem_u32(&ctl->stg_free[b]), 1);
    }
    ctl->abort_flag = 0;
    mbar_init_fence();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    if (p.tma_store)
      for (uint32_t c = 0; c < (NC > 1 ? cl.n : 1u); ++c) tma_prefetch_desc(&out.map[c]);
  }
  if (PAIR) cluster_sync();   // the other CTA runs and its barriers are initialised
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(smem_u32(&ctl->tmem_base), kTmemCols); tmem_relinquish_pair(); }
    else { tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();   // both have their tensor memory
  tc_fence_after();
  grid_dependency();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abortf = &ctl->abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      for (uint32_t tile = first; tile < total_tiles && !*abortf; tile += step) {
        const FwdTile t = fwd_tile<NC, PAIR>(p, cl, rank, tile);
        const FwdClass& k = cl.c[NC > 1 ? t.cls : 0];
        const int x0 = (int)(t.tx * p.TW * p.sw) + (NC > 1 ? k.offx : p.offx), y0 = (int)(t.ty * p.TH * p.sh) + (NC > 1 ? k.offy : p.offy);
        const uint32_t nr = NC > 1 ? k.nr : p.kh, ns = NC > 1 ? k.ns : p.kw;
        bool ok = true;
        for (uint32_t r = 0; r < nr && ok; ++r)
          for (uint32_t s = 0; s < ns && ok; ++s)
            for (uint32_t cb = 0; cb < slabs; ++cb) {
              if (!mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1u, abortf)) { ok = false; break; }
              const uint32_t full = smem_u32(&ctl->full[stage]);
              uint8_t* st = smem + (size_t)stage * kStageBytes;
              if (rank == 0) mbar_expect_tx(full, kStageBytes * kCtas);
              const uint32_t tap = NC > 1 ? k.tap0 + r * k.tap_r + s * k.tap_s : r * p.kw + s;
              const int ac = (int)(cb * 64), ax = x0 + (int)(s * p.dw), ay = y0 + (int)(r * p.dh);
              const int bk = (int)(tap * p.CK + cb * 64), bn = (int)(t.tn * BN + rank * (BN / kCtas));
              if (PAIR) {
                const uint32_t bar = cluster_first(full);
                tma_load_4d_pair(smem_u32(st), &map_a, bar, ac, ax, ay, (int)t.n);
                tma_load_2d_pair(smem_u32(st + kSlabBytes), &map_b, bar, bk, bn);
              } else {
                tma_load_4d(smem_u32(st), &map_a, full, ac, ax, ay, (int)t.n);
                tma_load_2d(smem_u32(st + kSlabBytes), &map_b, full, bk, bn);
              }
              if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            }
        if (!ok) break;
      }
      if (PAIR) await_stages<STAGES>(ctl, stage, phase, abortf);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_bf16(BN, 0, 0, 128 * kCtas);
      uint32_t stage = 0, phase = 0, it = 0;
      for (uint32_t tile = first; tile < total_tiles && !*abortf; tile += step, ++it) {
        const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
        if (!mbar_wait(smem_u32(&ctl->tempty[acc]), acc_phase ^ 1u, abortf)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * BN;
        const FwdClass& c = cl.c[NC > 1 ? fwd_tile<NC, PAIR>(p, cl, rank, tile).cls : 0];
        const uint32_t kiters = (NC > 1 ? c.nr * c.ns : p.kh * p.kw) * slabs;
        bool ok = true;
        for (uint32_t k = 0; k < kiters; ++k) {
          if (!mbar_wait(smem_u32(&ctl->full[stage]), phase, abortf)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + (size_t)stage * kStageBytes);
          const uint64_t da = smem_desc_sw128(sa, 16, 1024), db = smem_desc_sw128(sa + kSlabBytes, 16, 1024);
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk) {  // 4 x (K = 16 bf16 = 32 bytes) inside the 128-byte row
            if (PAIR) umma_bf16_pair(d, da + 2 * kk, db + 2 * kk, idesc, (k | kk) != 0u);
            else umma_bf16(d, da + 2 * kk, db + 2 * kk, idesc, (k | kk) != 0u);
          }
          if (PAIR) umma_commit_pair(smem_u32(&ctl->empty[stage]));
          else umma_commit(smem_u32(&ctl->empty[stage]));
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if (PAIR) umma_commit_pair(smem_u32(&ctl->tfull[acc]));
        else umma_commit(smem_u32(&ctl->tfull[acc]));
      }
    }
  } else {
    const uint32_t q = (uint32_t)warp & 3u;  // TMEM lane quarter this warp may read
    const uint32_t grp = ((uint32_t)warp - 2u) >> 2;   // epilogue warps 2..5 = group 0, 6..9 = group 1
    const bool leader = (((uint32_t)warp - 2u) & 3u) == 0u;
    auto drained = [&](uint32_t acc) {   // this warp has read its part of the accumulator
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(cluster_first(smem_u32(&ctl->tempty[acc])));
        else mbar_arrive(smem_u32(&ctl->tempty[acc]));
      }
    };
    uint32_t it = 0, gk = 0;   // gk: chunks this group has staged so far
    for (uint32_t tile = first; tile < total_tiles && !*abortf; tile += step, ++it) {
      const uint32_t acc = it & 1u, acc_phase = (it >> 1) & 1u;
      const FwdTile t = fwd_tile<NC, PAIR>(p, cl, rank, tile);
      const uint32_t tn = t.tn, tx = t.tx, ty = t.ty, n = t.n;
      const FwdClass& kc = cl.c[NC > 1 ? t.cls : 0];
      const bool none = NC > 1 && kc.nr * kc.ns == 0;   // no taps: nothing was accumulated
      const uint32_t m = q * 32 + lane;
      if (BN >= 64 && p.tma_store) {
        // 64-channel chunks of the tile go through a swizzled [128 px][64 ch] staging buffer and one TMA
        // tile store each: coalesced, clipped to the tensor, no per-thread scattered 16-byte stores.  The
        // two warp groups take alternate chunks (alternate tiles when a tile is one chunk), each with two
        // staging buffers of its own: a group converts a chunk while its last one is still being read
        // (64 -> 256 channels, 262,144 pixels, bound by these stores: 44 -> 35 us).
        constexpr uint32_t kChunks = BN / 64;
        if (kChunks == 1 && (it & 1u) != grp) continue;
        // the addend's 128 bytes per pixel and chunk are on their way while the accumulator is awaited
        uint4 ad[8];
        const __nv_bfloat16* arow = nullptr;
        if (NC == 1 && p.add) {
          const uint32_t mi = m / (p.TW * p.TH), mr = m - mi * (p.TW * p.TH);
          const uint32_t oy = ty * p.TH + mr / p.TW, ox = tx * p.TW + mr % p.TW, on = n + mi;
          if (oy < p.OP && ox < p.OQ && on < p.NI) arow = p.add + (long long)on * p.add_plane + (long long)oy * p.add_pitch + (long long)ox * p.OC;
        }
        auto load_add = [&](uint32_t cb) {
#pragma unroll
          for (uint32_t g8 = 0; g8 < 8; ++g8) ad[g8] = arow && cb + g8 * 8 < p.OC ? *(const uint4*)(arow + cb + g8 * 8) : make_uint4(0u, 0u, 0u, 0u);
        };
        if (NC == 1 && p.add) load_add(tn * BN + (kChunks == 1 ? 0u : grp) * 64);
        if (!mbar_wait(smem_u32(&ctl->tfull[acc]), acc_phase, abortf)) break;
        tc_fence_after();
        const uint32_t m7 = m & 7u;
        bool live = true;
#pragma unroll 1
        for (uint32_t c64 = (kChunks == 1 ? 0u : grp); c64 < kChunks && live; c64 += 2, ++gk) {
          uint32_t v[64];
          const uint32_t taddr = tmem_base + ((q * 32u) << 16) + acc * BN + c64 * 64;
          tmem_ld32(taddr, *(uint32_t(*)[32])&v[0]);
          tmem_ld32(taddr + 32, *(uint32_t(*)[32])&v[32]);
          tmem_ld_wait();
          if (none) {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] = 0u;
          }
          if (c64 + 2 >= kChunks) drained(acc);
          const uint32_t sb = grp * 2 + (gk & 1u);
          uint8_t *stg = osm + (size_t)sb * 16384, *srow = stg + m * 128u;
          bool ok = true;
          if (gk >= 2) ok = mbar_wait(smem_u32(&ctl->stg_free[sb]), ((gk >> 1) - 1u) & 1u, abortf);
          if (!__all_sync(0xffffffffu, ok)) { live = false; break; }
          const uint32_t cbase = tn * BN + c64 * 64;
          if (p.bias && cbase + 64 <= p.OC && !((uintptr_t)p.bias & 15u)) {
#pragma unroll
            for (int j = 0; j < 64; j += 4) {
              const float4 b = *(const float4*)(p.bias + cbase + j);
              v[j] = __float_as_uint(__uint_as_float(v[j]) + b.x); v[j + 1] = __float_as_uint(__uint_as_float(v[j + 1]) + b.y);
              v[j + 2] = __float_as_uint(__uint_as_float(v[j + 2]) + b.z); v[j + 3] = __float_as_uint(__uint_as_float(v[j + 3]) + b.w);
            }
          } else if (p.bias) {
#pragma unroll
            for (int j = 0; j < 64; ++j)
              if (cbase + j < p.OC) v[j] = __float_as_uint(__uint_as_float(v[j]) + p.bias[cbase + j]);
          }
          if (p.relu) {
#pragma unroll
            for (int j = 0; j < 64; ++j) v[j] = __float_as_uint(fmaxf(__uint_as_float(v[j]), 0.f));
          }
#pragma unroll
          for (uint32_t g8 = 0; g8 < 8; ++g8) {
            uint4 pk;
            __nv_bfloat162* p2 = (__nv_bfloat162*)&pk;
#pragma unroll
            for (int j = 0; j < 4; ++j)
              p2[j] = __floats2bfloat162_rn(__uint_as_float(v[g8 * 8 + 2 * j]), __uint_as_float(v[g8 * 8 + 2 * j + 1]));
            if (NC == 1 && p.add) {
              const __nv_bfloat162* a2 = (const __nv_bfloat162*)&ad[g8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 r = __bfloat1622float2(p2[j]), e = __bfloat1622float2(a2[j]);
                p2[j] = __floats2bfloat162_rn(r.x + e.x, r.y + e.y);
              }
            }
            *(uint4*)(srow + ((g8 ^ m7) * 16u)) = pk;
          }
          if (NC == 1 && p.add && c64 + 2 < kChunks) load_add(cbase + 128);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl->stg_full[sb]));
          if (leader && lane == 0) {
            if (mbar_wait(smem_u32(&ctl->stg_full[sb]), (gk >> 1) & 1u, abortf)) {
              if (cbase < p.OC && n < p.NI)
                asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(&out.map[NC > 1 ? t.cls : 0]),
                             "r"(smem_u32(stg)), "r"((int)cbase), "r"((int)(tx * p.TW)), "r"((int)(ty * p.TH)), "r"((int)n)
                             : "memory");
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
              if (gk >= 1) mbar_arrive(smem_u32(&ctl->stg_free[sb ^ 1u]));   // the chunk before has been read
            }
          }
          __syncwarp();
        }
        if (!live) break;
        continue;
      }
      if (grp != 0) continue;   // the scattered-store form is served by the first group alone
      if (!mbar_wait(smem_u32(&ctl->tfull[acc]), acc_phase, abortf)) break;
      tc_fence_after();
      const uint32_t mi = m / (p.TW * p.TH), mr = m - mi * (p.TW * p.TH);   // image inside the tile, pixel inside the image
      const uint32_t oy = ty * p.TH + mr / p.TW, ox = tx * p.TW + mr % p.TW, on = n + mi;
      const bool valid = oy < (NC > 1 ? kc.OP : p.OP) && ox < (NC > 1 ? kc.OQ : p.OQ) && on < p.NI;
      __nv_bfloat16* orow = p.out + (NC > 1 ? kc.out_off : 0) + (long long)on * p.out_plane + (long long)oy * p.out_pitch + (long long)ox * p.out_px;
#pragma unroll 1
      for (uint32_t ch = 0; ch < BN / 32; ++ch) {
        uint32_t v[32];
        tmem_ld32(tmem_base + ((q * 32u) << 16) + acc * BN + ch * 32, v);
        tmem_ld_wait();
        if (none) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        const uint32_t c0 = tn * BN + ch * 32;
        if (valid && c0 < p.OC) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const uint32_t cg = c0 + g * 8;
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              f[j] = __uint_as_float(v[g * 8 + j]);
              if (p.bias && cg + j < p.OC) f[j] += p.bias[cg + j];
            }
            if (cg + 8 <= p.OC && (p.OC & 7u) == 0) {
              if (p.accumulate) {
                uint4 old = *(const uint4*)(orow + cg);
                const __nv_bfloat162* o2 = (const __nv_bfloat162*)&old;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  float2 t = __bfloat1622float2(o2[j]);
                  f[2 * j] += t.x; f[2 * j + 1] += t.y;
                }
              }
              if (p.relu) {
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = fmaxf(f[j], 0.f);
              }
              uint4 pk;
              __nv_bfloat162* p2 = (__nv_bfloat162*)&pk;
#pragma unroll
              for (int j = 0; j < 4; ++j) p2[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
              *(uint4*)(orow + cg) = pk;
            } else {
              for (int j = 0; j < 8; ++j)
                if (cg + j < p.OC) {
                  float t = f[j];
                  if (p.accumulate) t += __bfloat162float(orow[cg + j]);
                  if (p.relu) t = fmaxf(t, 0.f);
                  orow[cg + j] = __float2bfloat16_rn(t);
                }
            }
          }
        }
      }
      drained(acc);
    }
    if (p.tma_store && leader && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (*abortf) {
    // Let any tile copy that is still in flight land before shared memory is released.
    for (int i = 0; i < 2000; ++i) __nanosleep(500);
    if (threadIdx.x == 0 && p.status) *p.status = AD_ERR_TIMEOUT;
  }
  __syncthreads();
  if (PAIR) cluster_sync();   // neither CTA leaves while the other's copies, arrivals or MMAs may reach it
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
  if (PAIR) cluster_sync();   // the release concerns both CTAs
}

// ---------------------------------------------------------------- filter gradient
struct WgParams {
  uint32_t NI, OP, OQ;  // dy: images, rows, cols
  uint32_t KO, CI;      // dy channels (GEMM M), x channels (GEMM N)
  uint32_t kh, kw, sh, sw, dh, dw;
  int32_t offy, offx;
  uint32_t TH, TW, tiles_y, tiles_x;
  uint32_t TN, tiles_b;  // a tile spans TN images (small maps); tiles_b = ceil(NI / TN)
  uint32_t ktiles, ctiles, splits;
  float* partial;       // [splits][KO][kh*kw][CI]
  int32_t* status;
};

// A work item is one [128 dy channels][BN x channels] block of one tap, summed over the pixel tiles of one split.  The kernel
// is persistent, one CTA per SM: the copies of the next item start while the last one is still multiplied, and two
// accumulators let the epilogue drain one item under the next.  With a CTA per item, layers of a few pixel tiles per item
// (small feature maps) spent most of the time in set-up, pipeline fill and drain.
// PAIR: two CTAs work on one item of 256 dy channels and load half of the x tile each: 48 KB instead of 64 per 128 pixels
// and SM; the operand tiles come out of the L2, whose rate (~16 TB/s) is the bound of the plain form: 512 -> 512 channels,
// 3x3, 65,536 pixels 306 -> 269 us, 1024 -> 256, 1x1 93 -> 67.
// Items of one split come one after another, so that the blocks at work at any time read the same pixels.
template <int BN, int STAGES, bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
conv_tc_wgrad_kernel(const __grid_constant__ CUtensorMap map_dy, const __grid_constant__ CUtensorMap map_x,
                     const WgParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kCtas = PAIR ? 2 : 1;
  constexpr uint32_t kABytes = 2 * kSlabBytes, kBSlabs = BN / 64 / kCtas, kStageBytes = kABytes + kBSlabs * kSlabBytes;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  SmemCtl* ctl = (SmemCtl*)(smem + (size_t)STAGES * kStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kTmemCols = 2 * BN;   // 128 or 256
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  const uint32_t sp_tiles = p.tiles_b * p.tiles_y * p.tiles_x;
  const uint32_t outer = p.kh * p.kw * (p.ktiles / kCtas) * p.ctiles, items = outer * p.splits;
  const uint32_t first = blockIdx.x / kCtas, step = gridDim.x / kCtas;

  struct Item { uint32_t split, tap, kt, ct, tiles; };
  auto item_at = [&](uint32_t i) {
    Item t;
    t.split = i / outer;
    uint32_t rem = i - t.split * outer;
    t.ct = rem % p.ctiles; rem /= p.ctiles;
    t.kt = rem % (p.ktiles / kCtas) * kCtas + rank;
    t.tap = rem / (p.ktiles / kCtas);
    t.tiles = t.split < sp_tiles ? (sp_tiles - t.split + p.splits - 1) / p.splits : 0;
    return t;
  };

  if (threadIdx.x == 0) {
    for (int st = 0; st < STAGES; ++st) {
      mbar_init(smem_u32(&ctl->full[st]), 1);
      mbar_init(smem_u32(&ctl->empty[st]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ctl->tfull[a]), 1);
      mbar_init(smem_u32(&ctl->tempty[a]), 4 * kCtas);
    }
    ctl->abort_flag = 0;
    mbar_init_fence();
    tma_prefetch_desc(&map_dy);
    tma_prefetch_desc(&map_x);
  }
  if (PAIR) cluster_sync();   // the other CTA runs and its barriers are initialised
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(smem_u32(&ctl->tmem_base), kTmemCols); tmem_relinquish_pair(); }
    else { tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();   // both have their tensor memory
  tc_fence_after();
  grid_dependency();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile int* abortf = &ctl->abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (uint32_t i = first; i < items && ok; i += step) {
        const Item t = item_at(i);
        const uint32_t r = t.tap / p.kw, s = t.tap % p.kw;
        for (uint32_t j = 0; j < t.tiles; ++j) {
          const uint32_t tm = t.split + j * p.splits;
          const uint32_t tx = tm % p.tiles_x, ty = (tm / p.tiles_x) % p.tiles_y, n = tm / (p.tiles_x * p.tiles_y) * p.TN;
          if (!mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1u, abortf)) { ok = false; break; }
          uint32_t full = smem_u32(&ctl->full[stage]);
          uint8_t* st = smem + (size_t)stage * kStageBytes;
          if (rank == 0) mbar_expect_tx(full, kStageBytes * kCtas);
          if (PAIR) full = cluster_first(full);
          const int qx = (int)(tx * p.TW), qy = (int)(ty * p.TH), c0 = (int)(t.ct * BN + rank * (BN / kCtas));
          const int ix = qx * (int)p.sw + (int)(s * p.dw) + p.offx, iy = qy * (int)p.sh + (int)(r * p.dh) + p.offy;
          auto load = [&](uint32_t dst, const CUtensorMap* map, int c, int x, int y) {
            if (PAIR) tma_load_4d_pair(dst, map, full, c, x, y, (int)n);
            else tma_load_4d(dst, map, full, c, x, y, (int)n);
          };
          load(smem_u32(st), &map_dy, (int)(t.kt * 128), qx, qy);
          load(smem_u32(st + kSlabBytes), &map_dy, (int)(t.kt * 128 + 64), qx, qy);
#pragma unroll
          for (uint32_t b = 0; b < kBSlabs; ++b) load(smem_u32(st + kABytes + b * kSlabBytes), &map_x, c0 + (int)b * 64, ix, iy);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (PAIR) await_stages<STAGES>(ctl, stage, phase, abortf);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_bf16(BN, 1, 1, 128 * kCtas);
      uint32_t stage = 0, phase = 0, it = 0;
      bool ok = true;
      for (uint32_t i = first; i < items && ok; i += step, ++it) {
        const uint32_t tiles = item_at(i).tiles, acc = it & 1u;
        if (!mbar_wait(smem_u32(&ctl->tempty[acc]), ((it >> 1) & 1u) ^ 1u, abortf)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * BN;
        for (uint32_t j = 0; j < tiles; ++j) {
          if (!mbar_wait(smem_u32(&ctl->full[stage]), phase, abortf)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + (size_t)stage * kStageBytes);
#pragma unroll
          for (uint32_t ks = 0; ks < 8; ++ks) {  // 8 x (K = 16 pixels = 16 rows of 128 B)
            const uint64_t da = smem_desc_sw128(sa + ks * 2048, kSlabBytes, 1024);
            const uint64_t db = smem_desc_sw128(sa + kABytes + ks * 2048, kSlabBytes, 1024);
            if (PAIR) umma_bf16_pair(d, da, db, idesc, (j | ks) != 0u);
            else umma_bf16(d, da, db, idesc, (j | ks) != 0u);
          }
          if (PAIR) umma_commit_pair(smem_u32(&ctl->empty[stage]));
          else umma_commit(smem_u32(&ctl->empty[stage]));
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if (PAIR) umma_commit_pair(smem_u32(&ctl->tfull[acc]));
        else umma_commit(smem_u32(&ctl->tfull[acc]));
      }
    }
  } else {
    const uint32_t q = (uint32_t)warp & 3u;
    const uint32_t taps = p.kh * p.kw;
    uint32_t it = 0;
    for (uint32_t i = first; i < items; i += step, ++it) {
      const Item t = item_at(i);
      const uint32_t acc = it & 1u, k = t.kt * 128 + q * 32 + lane;
      float* orow = p.partial + (((size_t)t.split * p.KO + k) * taps + t.tap) * p.CI + (size_t)t.ct * BN;
      if (!mbar_wait(smem_u32(&ctl->tfull[acc]), (it >> 1) & 1u, abortf)) break;
      tc_fence_after();
#pragma unroll 1
      for (uint32_t ch = 0; ch < BN / 32; ++ch) {
        uint32_t v[32];
        tmem_ld32(tmem_base + ((q * 32u) << 16) + acc * BN + ch * 32, v);
        tmem_ld_wait();
        if (t.tiles == 0) {   // more splits than pixel tiles: nothing was accumulated
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        if (k < p.KO) {
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const uint32_t c = t.ct * BN + ch * 32 + g * 4;
            if (c + 4 <= p.CI)
              *(float4*)(orow + ch * 32 + g * 4) = make_float4(__uint_as_float(v[g * 4]), __uint_as_float(v[g * 4 + 1]),
                                                               __uint_as_float(v[g * 4 + 2]), __uint_as_float(v[g * 4 + 3]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(cluster_first(smem_u32(&ctl->tempty[acc])));
        else mbar_arrive(smem_u32(&ctl->tempty[acc]));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abortf) {
    for (int i = 0; i < 2000; ++i) __nanosleep(500);
    if (threadIdx.x == 0 && p.status) *p.status = AD_ERR_TIMEOUT;
  }
  __syncthreads();
  if (PAIR) cluster_sync();   // neither CTA leaves while the other's copies, arrivals or MMAs may reach it
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
  if (PAIR) cluster_sync();   // the release concerns both CTAs
}

// dw (+)= sum over splits of partial[s][k][tap][c], fixed order: lane l of four sums splits l, l+4, ... (8 loads of 16 bytes in
// flight), the lanes are combined in order.  The partials were written by the kernel before, so this is bound by L2 latency.
__device__ __forceinline__ float4 wgrad_lane_sum(const float* src, size_t part_stride, uint32_t splits, uint32_t lane) {
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t s0 = lane; s0 < splits; s0 += 32) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t si = s0 + 4 * u;
      v[u] = si < splits ? *(const float4*)(src + (size_t)si * part_stride) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) { t.x += v[u].x; t.y += v[u].y; t.z += v[u].z; t.w += v[u].w; }
  }
  return t;
}
// KRSC filters, and 1x1 ones in either order (kcrs): 64 x 4 outputs x 4 lanes per block.  C is a multiple of 64.
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(size_t n, size_t part_stride, uint32_t splits,
                                                           const float* __restrict__ partial, float* dw, int accumulate,
                                                           uint32_t taps, uint32_t C, int kcrs, BiasParts bias) {
  grid_dependency();
  if (bias_finish_blocks(bias, accumulate)) return;
  const uint32_t tx = threadIdx.x & 63, pl = threadIdx.x >> 6, block = blockIdx.x - bias.blocks;
  const size_t i = ((size_t)block * 64 + tx) * 4;
  __shared__ float4 sh[4][64];
  if (i < n) sh[pl][tx] = wgrad_lane_sum(partial + i, part_stride, splits, pl);
  __syncthreads();
  // thread t finishes output t of the block's 256
  const size_t j = (size_t)block * 256 + threadIdx.x;
  if (j >= n) return;
  const float* f = (const float*)sh + threadIdx.x;
  const float t = ((f[0] + f[256]) + f[512]) + f[768];
  size_t o = j;
  if (kcrs) {
    const uint32_t c = (uint32_t)(j % C);
    const size_t r = j / C;
    const uint32_t tap = (uint32_t)(r % taps);
    o = ((r / taps) * C + c) * taps + tap;
  }
  dw[o] = accumulate ? dw[o] + t : t;
}
// KCRS filters of several taps: a block owns 32 channels x all taps of one filter, a contiguous run of dw, and turns them
// round in shared memory; element by element, each 4-byte store met its own 32-byte sector (the reductions of the
// segmentation net's 50 filter gradients: 1.77 -> 1.06 ms).
constexpr uint32_t kWgRedPitch = 36;
__global__ void wgrad_reduce_kcrs_kernel(size_t part_stride, uint32_t splits, const float* __restrict__ partial, float* dw,
                                         int accumulate, uint32_t taps, uint32_t C, BiasParts bias) {
  grid_dependency();
  if (bias_finish_blocks(bias, accumulate)) return;
  extern __shared__ float wr[];   // [4][taps][kWgRedPitch]
  const uint32_t block = blockIdx.x - bias.blocks, ctiles = C / 32, k = block / ctiles, c0 = block % ctiles * 32, items = taps * 8;
  for (uint32_t w = threadIdx.x; w < items * 4; w += blockDim.x) {
    const uint32_t pl = w / items, e = w - pl * items, tap = e >> 3, c4 = e & 7;
    *(float4*)(wr + (pl * taps + tap) * kWgRedPitch + c4 * 4) =
        wgrad_lane_sum(partial + ((size_t)k * taps + tap) * C + c0 + c4 * 4, part_stride, splits, pl);
  }
  __syncthreads();
  float* out = dw + ((size_t)k * C + c0) * taps;
  const uint32_t plane = taps * kWgRedPitch;
  for (uint32_t i = threadIdx.x; i < taps * 32; i += blockDim.x) {
    const uint32_t c = i / taps, tap = i - c * taps;
    const float* f = wr + tap * kWgRedPitch + c;
    const float t = ((f[0] + f[plane]) + f[2 * plane]) + f[3 * plane];
    out[i] = accumulate ? out[i] + t : t;
  }
}
// Filter for the data gradient: wt[c][kh-1-r][kw-1-s][k] = w[k][r][s][c]  (bf16); rows of Kp >= K
// entries, zero past K.
__global__ void __launch_bounds__(256) filter_transpose_flip_kernel(uint32_t K, uint32_t Kp, uint32_t kh, uint32_t kw,
                                                                    uint32_t C, const __nv_bfloat16* __restrict__ w,
                                                                    __nv_bfloat16* wt) {
  grid_dependency();
  const size_t total = (size_t)Kp * kh * kw * C, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    uint32_t k = (uint32_t)(i % Kp);
    size_t rr = i / Kp;
    uint32_t s = (uint32_t)(rr % kw); rr /= kw;
    uint32_t r = (uint32_t)(rr % kh);
    uint32_t c = (uint32_t)(rr / kh);
    wt[i] = k < K ? w[(((size_t)k * kh + (kh - 1 - r)) * kw + (kw - 1 - s)) * C + c] : __float2bfloat16_rn(0.f);
  }
}
// Both tensor-core forms of many fp32 KCRS filters in one launch: KRSC bf16 (rows of `row` elements) and, for the data
// gradient, C,R,S,K bf16 with mirrored taps (Kp entries per row, zero past K).  A block turns KT filters x CT channels x all
// taps round in shared memory: fp32 rows are read and runs of bf16 pairs written.  The shapes that nearly all filters have
// (1x1 and 3x3, whole channel tiles) are compiled with constant extents: with divisions by variable ones the kernel was
// bound by integer arithmetic.  As two launches per layer (one of them in front of every forward and data-gradient
// kernel) the 23.5 M weights of a 53-layer net took 640 us, in one launch of variable extents 200, so 89.
constexpr uint32_t kPrepItems = 32, kPrepFloats = 9216;
struct PrepItem {
  const float* src;
  __nv_bfloat16 *krsc, *crsk;
  uint32_t K, C, taps, Kp, KT, CT, tile0;   // tile0: first tile of this item
  long long row;
};
struct PrepBatch { PrepItem it[kPrepItems]; uint32_t count, tiles; };
template <uint32_t T, uint32_t CT, uint32_t KT>   // constant taps and tile, even KT; T = 0: those of the item
__device__ __forceinline__ void filter_prepare_tile(const PrepItem& p, uint32_t k0, uint32_t c0, float* sm) {
  const uint32_t taps = T ? T : p.taps, ct = T ? CT : p.CT, kt = T ? KT : p.KT;
  const uint32_t nc = T ? CT : (p.C - c0 < ct ? p.C - c0 : ct), run = nc * taps, pitch = ct * taps + 1;   // odd pitch where ct * taps is even
  const uint32_t nk = k0 < p.K ? (p.K - k0 < kt ? p.K - k0 : kt) : 0;
  const float* src = p.src + ((size_t)k0 * p.C + c0) * taps;
  const size_t krow = (size_t)p.C * taps;
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < nk * run; i += 256) {
    const uint32_t k = i / run, e = i - k * run;
    sm[k * pitch + e] = src[k * krow + e];
  }
  __syncthreads();
  if (T) {
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < nk * (run / 2); i += 256) {
      const uint32_t c = i % (nc / 2) * 2, r = i / (nc / 2), tap = r % taps, k = r / taps;
      const float* f = sm + k * pitch + c * taps + tap;
      *(__nv_bfloat162*)(p.krsc + (size_t)(k0 + k) * p.row + (size_t)tap * p.C + c0 + c) = __floats2bfloat162_rn(f[0], f[taps]);
    }
  } else {
    for (uint32_t i = threadIdx.x; i < nk * run; i += 256) {
      const uint32_t c = i % nc, r = i / nc, tap = r % taps, k = r / taps;
      p.krsc[(size_t)(k0 + k) * p.row + (size_t)tap * p.C + c0 + c] = __float2bfloat16_rn(sm[k * pitch + c * taps + tap]);
    }
  }
  if (p.crsk) {
    const uint32_t kk = p.Kp - k0 < kt ? p.Kp - k0 : kt, pairs = kt / 2;   // Kp is even
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < pairs * run; i += 256) {
      const uint32_t k = i % pairs * 2, r = i / pairs, tap = r % taps, c = r / taps;
      const float* f = sm + k * pitch + c * taps + tap;
      if (k < kk)
        *(__nv_bfloat162*)(p.crsk + ((size_t)(c0 + c) * taps + (taps - 1 - tap)) * p.Kp + k0 + k) =
            __floats2bfloat162_rn(k < nk ? f[0] : 0.f, k + 1 < nk ? f[pitch] : 0.f);
    }
  }
}
__global__ void __launch_bounds__(256) filter_prepare_kernel(const __grid_constant__ PrepBatch b) {
  grid_dependency();
  __shared__ float sm[kPrepFloats + 128];
  for (uint32_t tile = blockIdx.x; tile < b.tiles; tile += gridDim.x) {
    uint32_t lo = 0, hi = b.count;   // the last item whose tile0 <= tile: one without tiles shares its tile0 with the next
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (b.it[mid].tile0 <= tile) lo = mid; else hi = mid;
    }
    const PrepItem& p = b.it[lo];
    const uint32_t ctiles = (p.C + p.CT - 1) / p.CT, t = tile - p.tile0, k0 = t / ctiles * p.KT, c0 = t % ctiles * p.CT;
    __syncthreads();
    if (p.taps == 1 && p.KT == 128) filter_prepare_tile<1, 64, 128>(p, k0, c0, sm);
    else if (p.taps == 9 && p.C % 32 == 0 && !(p.row & 1) && !((uintptr_t)p.krsc & 3u)) filter_prepare_tile<9, 32, 32>(p, k0, c0, sm);
    else filter_prepare_tile<0, 0, 0>(p, k0, c0, sm);
  }
}
// dst[pixel][0..Kp) = src[pixel][0..K), zero past K
__global__ void __launch_bounds__(256) pad_channels_kernel(size_t pixels, uint32_t K, uint32_t Kp,
                                                           const __nv_bfloat16* __restrict__ src, __nv_bfloat16* dst) {
  grid_dependency();
  const size_t total = pixels * Kp, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += nt) {
    const uint32_t k = (uint32_t)(i % Kp);
    const size_t px = i / Kp;
    dst[i] = k < K ? src[px * K + k] : __float2bfloat16_rn(0.f);
  }
}

// db[k] (+)= sum over pixels of dy[pixel][k] (dense NHWC bf16), in two fixed-order stages: a block sums its share of the
// pixels into part[block][k], bias_finish_blocks adds the blocks in order.  HBM-bound: dy is read once.
// K a multiple of 8: a thread owns 8 adjacent channels (16-byte loads, eight pixels in flight), 256 / (K / 8) pixel lanes
// per block (K above 2048: channel groups over blockIdx.y).  32 x 512 x 512 pixels of 64 channels: 205 us
// with four pixels in registers, 178 with the ring.
__device__ __forceinline__ void bias_add8(float (&acc)[8], const uint4& v) {
  const uint32_t* w = &v.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[2 * j] += __uint_as_float(w[j] << 16);
    acc[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
  }
}
__global__ void __launch_bounds__(256) bias_grad_vec_kernel(size_t pixels, uint32_t K, uint32_t gb, const __nv_bfloat16* __restrict__ dy, float* part) {
  grid_dependency();
  typedef LoadRing<1, 8> Ring;
  __shared__ __align__(128) uint4 ring_smem[Ring::kBytes / 16];
  Ring ring(ring_smem);
  const uint32_t G = K / 8, gl = threadIdx.x % gb, pl = threadIdx.x / gb, PL = 256 / gb, g = blockIdx.y * gb + gl;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  const size_t stride = (size_t)gridDim.x * PL;
  size_t i = g < G && pl < PL ? (size_t)blockIdx.x * PL + pl : pixels;
  const uint4* src = (const uint4*)dy + g;
  if (pixels > 16 * stride) {
    auto issue = [&](size_t at) {
      if (at < pixels) ring.copy(0, src + at * G);
      ring.commit();
    };
#pragma unroll
    for (int u = 0; u < 7; ++u) issue(i + u * stride);
    for (; i < pixels; i += stride) {
      ring.wait();
      const uint4 v = ring.get(0);
      ring.next();
      issue(i + 7 * stride);
      bias_add8(acc, v);
    }
  } else {   // few pixels per thread: the ring's start costs more than it brings (1 us)
    for (; i + 3 * stride < pixels; i += 4 * stride) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = src[(i + u * stride) * G];
#pragma unroll
      for (int u = 0; u < 4; ++u) bias_add8(acc, v[u]);
    }
    for (; i < pixels; i += stride) bias_add8(acc, src[i * G]);
  }
  float (*red)[9] = (float (*)[9])ring_smem;   // free once every thread has read its last element
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) red[threadIdx.x][j] = acc[j];
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < gb * 8; t += 256) {
    const uint32_t tg = t >> 3, j = t & 7;
    if (blockIdx.y * gb + tg >= G) continue;
    float v = 0.f;
    for (uint32_t q = 0; q < PL; ++q) v += red[q * gb + tg][j];
    part[(size_t)blockIdx.x * K + (blockIdx.y * gb + tg) * 8 + j] = v;
  }
}
// other channel counts (a 19-class head): a thread per channel and pixel lane
__global__ void __launch_bounds__(256) bias_grad_nhwc_kernel(size_t pixels, uint32_t K, const __nv_bfloat16* __restrict__ dy,
                                                             float* part) {
  grid_dependency();
  const uint32_t k = blockIdx.y * 32 + threadIdx.x, split = blockIdx.x, nsplit = gridDim.x;
  const size_t chunk = (pixels + nsplit - 1) / nsplit, lo = (size_t)split * chunk, hi = lo + chunk < pixels ? lo + chunk : pixels;
  float acc = 0.f;
  if (k < K) {
#pragma unroll 4
    for (size_t i = lo + threadIdx.y; i < hi; i += 8) acc += __bfloat162float(dy[i * K + k]);
  }
  __shared__ float red[8][33];
  red[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && k < K) {
    float t = 0.f;
    for (int w = 0; w < 8; ++w) t += red[w][threadIdx.x];
    part[(size_t)split * K + k] = t;
  }
}
// Blocks (= partial rows of K floats) of the first stage: four per SM, each thread with at least two batches of pixels.
// Their sum is part of the reduction of the filter gradient's partials (BiasParts), which lie in front of them in scratch.
static uint32_t bias_grad_blocks(size_t pixels, uint32_t K) {
  const bool vec = K % 8 == 0;
  const uint32_t gb = vec ? std::min(K / 8, 256u) : 32u, lanes = vec ? 256 / gb : 8, groups = vec ? (K / 8 + gb - 1) / gb : (K + 31) / 32;
  const size_t most = pixels / ((size_t)lanes * 8), want = std::max(1u, 4u * kNumSMs / groups);
  return (uint32_t)std::max<size_t>(1, std::min(most, want));
}
size_t bias_grad_bytes(size_t pixels, uint32_t K) { return (size_t)bias_grad_blocks(pixels, K) * K * 4; }
// The first stage, if there is a db; part: at least bias_grad_bytes (less: one block does with what there is)
BiasParts bias_grad_parts(size_t pixels, uint32_t K, const void* dy, float* db, float* part, size_t part_bytes, cudaStream_t s) {
  if (!db) return BiasParts{};
  const uint32_t nsplit = (uint32_t)std::min<size_t>(bias_grad_blocks(pixels, K), part_bytes / ((size_t)K * 4));
  if (K % 8 == 0 && ((uintptr_t)dy & 15u) == 0) {
    const uint32_t gb = K / 8 < 256 ? K / 8 : 256;
    launch(bias_grad_vec_kernel, dim3(nsplit, (K / 8 + gb - 1) / gb), 256, 0, s, pixels, K, gb, (const __nv_bfloat16*)dy, part);
  } else {
    launch(bias_grad_nhwc_kernel, dim3(nsplit, (K + 31) / 32), dim3(32, 8), 0, s, pixels, K, (const __nv_bfloat16*)dy, part);
  }
  count_launch();
  return BiasParts{part, nsplit, K, K, db, (K + 31) / 32};
}

struct BiasGrad { size_t pixels; const void* dy; float *db, *part; size_t part_bytes; };
// The reduction over the splits, with that of the bias gradient's partials in blocks of its own
static void launch_wgrad_reduce(uint32_t K, uint32_t taps, uint32_t C, size_t part_stride, uint32_t splits, const float* partial,
                                float* dw, int accumulate, int kcrs, const BiasGrad& b, cudaStream_t s) {
  const size_t n = (size_t)K * taps * C, smem = (size_t)4 * taps * kWgRedPitch * 4;
  const BiasParts bias = bias_grad_parts(b.pixels, K, b.dy, b.db, b.part, b.part_bytes, s);
  if (kcrs && taps > 1 && smem <= 48 * 1024) {   // more taps than shared memory holds (over 85) take the form below
    const uint32_t threads = std::min((taps * 32 + 31) / 32 * 32, 512u);
    launch(wgrad_reduce_kcrs_kernel, bias.blocks + K * (C / 32), threads, smem, s, part_stride, splits, partial, dw, accumulate, taps, C, bias);
  } else {
    launch(wgrad_reduce_kernel, bias.blocks + (uint32_t)((n + 255) / 256), 256, 0, s, n, part_stride, splits, partial, dw, accumulate, taps, C, kcrs && taps > 1, bias);
  }
  count_launch();
}

// ---------------------------------------------------------------- host side
struct Geo {
  uint32_t P, Q;
};
static int conv_geo(const ad_conv2d_args* a, Geo& g) {
  if (!a) return AD_ERR_BAD_ARG;
  if (a->N == 0 || a->C == 0 || a->H == 0 || a->W == 0 || a->K == 0 || a->kh == 0 || a->kw == 0) return AD_ERR_BAD_ARG;
  if (a->stride_h == 0 || a->stride_w == 0 || a->dil_h == 0 || a->dil_w == 0) return AD_ERR_BAD_ARG;
  const long long eh = (long long)a->H + 2ll * a->pad_h - (long long)a->dil_h * (a->kh - 1) - 1;
  const long long ew = (long long)a->W + 2ll * a->pad_w - (long long)a->dil_w * (a->kw - 1) - 1;
  if (eh < 0 || ew < 0) return AD_ERR_BAD_ARG;
  g.P = (uint32_t)(eh / a->stride_h + 1);
  g.Q = (uint32_t)(ew / a->stride_w + 1);
  return AD_OK;
}

// Patch of 128 output pixels (TN images x TH rows x TW columns) wasting the fewest lanes on partial tiles: large
// maps get one image per tile, small feature maps (7 x 7, 14 x 14) several, which otherwise leave most of a
// 128-pixel tile empty.
static void pick_tile3(uint32_t NI, uint32_t OP, uint32_t OQ, uint32_t sh, uint32_t sw, uint32_t& TN, uint32_t& TH, uint32_t& TW) {
  unsigned long long best = ~0ull;
  TN = 1; TH = 1; TW = 128;
  for (uint32_t tn = 1; tn <= 16; tn <<= 1)
    for (uint32_t tw = 128 / tn; tw >= 8; tw >>= 1) {
      const uint32_t th = 128 / tn / tw;
      if (th == 0 || tw * sw > 256 || th * sh > 256) continue;
      const unsigned long long cost = (unsigned long long)((OQ + tw - 1) / tw * tw) * ((OP + th - 1) / th * th) * ((NI + tn - 1) / tn * tn);
      if (cost < best) { best = cost; TN = tn; TH = th; TW = tw; }
    }
}

// A persistent kernel over `items` tiles: one CTA per SM, or a pair of CTAs per two SMs.  attr_done: the caller's record of
// the devices (a bit each) on which the kernel's shared-memory limit is raised.
template <typename... KArgs, typename... Args>
static int launch_tc(void (*kern)(KArgs...), uint32_t ctas, uint32_t items, int threads, int smem, unsigned& attr_done, cudaStream_t s,
                     const Args&... args) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(attr_done & (1u << (dev & 31)))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      cudaGetLastError();
      return AD_ERR_CUDA;
    }
    attr_done |= 1u << (dev & 31);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(std::min(items, (uint32_t)kNumSMs / ctas) * ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.numAttrs = ctas > 1 ? 1 : 0;
  launch_attr(cfg, at);
  if (cudaLaunchKernelEx(&cfg, kern, KArgs(args)...) != cudaSuccess) {
    cudaGetLastError();
    return AD_ERR_CUDA;
  }
  count_launch();
  return launch_status();
}
template <int BN, int NC, bool PAIR>
static int launch_fwd(const CUtensorMap& ma, const CUtensorMap& mb, const FwdOut<NC>& mo, const FwdParams& p, const FwdClasses& cl, cudaStream_t s) {
  constexpr int kCtas = PAIR ? 2 : 1;
  constexpr int kStageBytes = kSlabBytes + BN / kCtas * 128;
  constexpr int STAGES = (160 * 1024) / kStageBytes > 8 ? 8 : (160 * 1024) / kStageBytes;
  constexpr int smem = STAGES * kStageBytes + kStagingBytes + 1024 + (int)sizeof(SmemCtl);
  const uint32_t tiles_m = NC > 1 ? p.tiles_x : p.tiles_b * p.tiles_y * p.tiles_x;
  static unsigned attr_done = 0;
  return launch_tc(conv_tc_fwd_kernel<BN, STAGES, NC, PAIR>, kCtas, (tiles_m + kCtas - 1) / kCtas * p.tiles_n, kFwdThreads, smem, attr_done, s,
                   ma, mb, mo, p, cl);
}

int conv_tc_row_fwd(const void* act, uint32_t NI, uint32_t IH, uint32_t IW, uint32_t CK, const void* filt, uint32_t OC,
                    uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw, int offy, int offx,
                    uint32_t OP, uint32_t OQ, void* out, long long out_pitch, long long out_plane, const float* bias,
                    int relu, int accumulate, int32_t* status, cudaStream_t s);

size_t conv_tc_row_wgrad_scratch(uint32_t NI, uint32_t CI, uint32_t KO, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw,
                                 uint32_t dh, uint32_t dw, uint32_t OP, uint32_t OQ);
int conv_tc_row_wgrad(const void* x, uint32_t NI, uint32_t IH, uint32_t IW, uint32_t CI, const void* dy, uint32_t KO,
                      uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw, int offy, int offx,
                      uint32_t OP, uint32_t OQ, float* dwt, float* db, int accumulate, int kcrs, void* partial, size_t partial_bytes,
                      int32_t* status, cudaStream_t s);

// The launch of the general kernel: everything but the tensor maps and the channel tiles is in p (and cl, NC > 1).
// all_taps: taps of the filter.
template <int NC>
static int run_fwd_tiles(const void* act, uint32_t IH, uint32_t IW, const void* filt, uint32_t all_taps, FwdParams p, const FwdClasses& cl,
                         cudaStream_t s) {
  g_last_conv_kernel = kConvTcGeneral;
  const uint32_t tiles_m = NC > 1 ? p.tiles_x : p.tiles_b * p.tiles_y * p.tiles_x;
  int BN = p.OC > 128 ? 256 : (p.OC > 64 ? 128 : (p.OC > 32 ? 64 : 32));
  // Short contractions: narrower channel tiles where they still make one round, which takes as long at any width (0.3 us per 64
  // terms) while more SMs share the stores.  2 x 64 x 79 x 21 -> 512, 3x3 9.3 -> 6.5 us, 5 x 256 x 29 x 16 -> 256, 1x1 5.8 -> 4.5; in two rounds
  // 9.7 -> 10.0.  A long contraction occupies twice the SMs for almost as long: 8 - 23 % faster alone, but kernels of other
  // streams wait (two strips of a 50-layer net side by side: 10.93 -> 11.21 ms).
  if (all_taps * (p.CK / 64) <= 9)
    while (BN > 64 && tiles_m * ((p.OC + BN / 2 - 1) / (BN / 2)) <= (uint32_t)kNumSMs) BN /= 2;
  p.tiles_n = (p.OC + BN - 1) / BN;
  const bool aligned = !((uintptr_t)p.out & 15u) && p.out_pitch % 8 == 0 && p.out_plane % 8 == 0;
  if (!aligned && (p.OC & 7u) == 0) return AD_ERR_ALIGN;

  // Pairs save operand traffic where there is a second pixel tile to share the filter rows with and the contraction is long
  // enough to be bound by it; short ones are bound by their stores, which single CTAs spread better in time (65,536
  // pixels, in a net: 256 -> 1024 channels 50 us against 54 as pairs, 512 -> 2048 118 against 144 the other way round).
  const bool pair = BN == 256 && tiles_m > 1 && all_taps * (p.CK / 64) >= 8;
  CUtensorMap ma, mb;
  {
    uint64_t dims[4] = {p.CK, IW, IH, p.NI};
    uint64_t str[4] = {0, (uint64_t)p.CK * 2, (uint64_t)IW * p.CK * 2, (uint64_t)IH * IW * p.CK * 2};
    uint32_t box[4] = {64, p.TW * p.sw, p.TH * p.sh, p.TN};
    uint32_t es[4] = {1, p.sw, p.sh, 1};
    int st = make_tmap_bf16(&ma, act, 4, dims, str, box, es);
    if (st != AD_OK) return st;
  }
  {
    uint64_t dims[2] = {(uint64_t)all_taps * p.CK, p.OC};
    uint64_t str[2] = {0, (uint64_t)all_taps * p.CK * 2};
    uint32_t box[2] = {64, (uint32_t)BN / (pair ? 2 : 1)};
    uint32_t es[2] = {1, 1};
    int st = make_tmap_bf16(&mb, filt, 2, dims, str, box, es);
    if (st != AD_OK) return st;
  }
  FwdOut<NC> mo;
  for (int c = 0; c < NC; ++c) mo.map[c] = ma;
  p.tma_store = (!p.accumulate && BN >= 64 && (p.OC & 7u) == 0 && aligned) ? 1 : 0;
  if (p.tma_store)
    for (uint32_t c = 0; c < (NC > 1 ? cl.n : 1u); ++c) {
      uint64_t dims[4] = {p.OC, NC > 1 ? cl.c[c].OQ : p.OQ, NC > 1 ? cl.c[c].OP : p.OP, p.NI};
      uint64_t str[4] = {0, (uint64_t)p.out_px * 2, (uint64_t)p.out_pitch * 2, (uint64_t)p.out_plane * 2};
      uint32_t box[4] = {64, p.TW, p.TH, p.TN};
      uint32_t es[4] = {1, 1, 1, 1};
      int st = make_tmap_bf16(&mo.map[c], p.out + (NC > 1 ? cl.c[c].out_off : 0), 4, dims, str, box, es);
      if (st != AD_OK) return st;
    }
  switch (BN) {
    case 256: return pair ? launch_fwd<256, NC, true>(ma, mb, mo, p, cl, s) : launch_fwd<256, NC, false>(ma, mb, mo, p, cl, s);
    case 128: return launch_fwd<128, NC, false>(ma, mb, mo, p, cl, s);
    case 64: return launch_fwd<64, NC, false>(ma, mb, mo, p, cl, s);
    default: return launch_fwd<32, NC, false>(ma, mb, mo, p, cl, s);
  }
}

// out += add, dims of add: for the forms whose epilogue does not
static int add_to_output(const ad_tensor4* add, void* out, long long pitch, long long plane, cudaStream_t s) {
  ad_tensor4 y = *add;
  y.base = out;
  y.sc = 1; y.sx = add->C; y.sy = pitch; y.sn = plane;
  return ad_add(&y, add, &y, s);
}

// Generic forward-style implicit GEMM launch (fprop, or dgrad expressed as fprop).
static int run_fwd_gemm(const void* act, uint32_t NI, uint32_t IH, uint32_t IW, uint32_t CK, const void* filt,
                        uint32_t OC, uint32_t kh, uint32_t kw, uint32_t sh, uint32_t sw, uint32_t dh, uint32_t dw,
                        int offy, int offx, uint32_t OP, uint32_t OQ, void* out, long long out_pitch,
                        long long out_plane, const float* bias, int relu, int accumulate, int32_t* status,
                        cudaStream_t s, const ad_tensor4* add = nullptr) {
  if (CK % 64 != 0) return AD_ERR_UNSUPPORTED;
  if (!getenv("ARRAYDIFF_B200_NO_ROW_KERNEL") && !(add && OQ < 96)) {
    // 64-channel layers: the row kernels fetch each activation patch once (conv_tc_row.cu); narrow maps with an addend stay with the
    // general kernel, whose epilogue adds it
    int st = conv_tc_row_fwd(act, NI, IH, IW, CK, filt, OC, kh, kw, sh, sw, dh, dw, offy, offx, OP, OQ, out, out_pitch,
                             out_plane, bias, relu, accumulate, status, s);
    if (st != AD_ERR_UNSUPPORTED) {
      g_last_conv_kernel = kConvTcRow;
      return st == AD_OK && add ? add_to_output(add, out, out_pitch, out_plane, s) : st;
    }
  }
  FwdParams p{};
  p.NI = NI; p.OP = OP; p.OQ = OQ; p.OC = OC; p.CK = CK;
  p.kh = kh; p.kw = kw; p.sh = sh; p.sw = sw; p.dh = dh; p.dw = dw; p.offy = offy; p.offx = offx;
  pick_tile3(NI, OP, OQ, sh, sw, p.TN, p.TH, p.TW);
  p.tiles_y = (OP + p.TH - 1) / p.TH;
  p.tiles_x = (OQ + p.TW - 1) / p.TW;
  p.tiles_b = (NI + p.TN - 1) / p.TN;
  p.out_px = OC;
  p.out_pitch = out_pitch ? out_pitch : (long long)OQ * OC;
  p.out_plane = out_plane ? out_plane : (long long)OP * OQ * OC;
  p.out = (__nv_bfloat16*)out;
  p.bias = bias; p.relu = relu; p.accumulate = accumulate; p.status = status;
  // In the epilogue where it stores by TMA and the addend's pixels are as dense as the output's
  const bool in_epilogue = add && OC > 32 && OC % 8 == 0 && add->sc == 1 && add->sx == (int64_t)OC && !(add->sy & 7) && !(add->sn & 7) &&
                           !((uintptr_t)add->base & 15u) && !((uintptr_t)out & 15u) && p.out_pitch % 8 == 0 && p.out_plane % 8 == 0;
  if (in_epilogue) { p.add = (const __nv_bfloat16*)add->base; p.add_pitch = add->sy; p.add_plane = add->sn; }
  const int st = run_fwd_tiles<1>(act, IH, IW, filt, kh * kw, p, FwdClasses{}, s);
  return st == AD_OK && add && !in_epilogue ? add_to_output(add, out, p.out_pitch, p.out_plane, s) : st;
}

template <int BN, bool PAIR>
static int launch_wgrad(const CUtensorMap& mdy, const CUtensorMap& mx, const WgParams& p, cudaStream_t s) {
  constexpr int kCtas = PAIR ? 2 : 1;
  constexpr int kStageBytes = 2 * kSlabBytes + (BN / 64 / kCtas) * kSlabBytes;
  // three stages as a pair: 146 KB leave room for a block of a batch norm pass on the main stream (LoadRing::kSmem), which
  // waits for memory while this waits for the tensor cores (segmentation net's step 20.1 -> 19.9 ms against four)
  constexpr int STAGES = PAIR ? 3 : (200 * 1024) / kStageBytes;
  constexpr int smem = STAGES * kStageBytes + 1024 + (int)sizeof(SmemCtl);
  static unsigned attr_done = 0;
  return launch_tc(conv_tc_wgrad_kernel<BN, STAGES, PAIR>, kCtas, p.splits * p.kh * p.kw * (p.ktiles / kCtas) * p.ctiles, kThreads, smem,
                   attr_done, s, mdy, mx, p);
}

static size_t round_1k(size_t b) { return (b + 1023) / 1024 * 1024; }
// Gradient channel counts the tensor-core kernels take as they are: the data gradient reduces over K in
// 64-channel slabs, the filter gradient needs 16-byte pixel pitches of dy.  Other counts (a 19-class head)
// run on a zero-padded copy of dy kept in scratch.
static uint32_t dgrad_kp(uint32_t K) { return (K + 63) / 64 * 64; }
static uint32_t wgrad_kp(uint32_t K) { return (K + 7) / 8 * 8; }

// Scratch layouts:
//   pass 1 (data gradient):   [status 16 B | transposed filter C,R,S,Kp bf16] [dy padded to Kp channels, if Kp != K]
//   pass 2 (filter gradient): [status 16 B] [dy padded, if Kp != K] [fp32 partials]
size_t conv_tc_scratch_bytes(const ad_conv2d_args* a, int pass) {
  Geo g;
  if (conv_geo(a, g) != AD_OK) return 0;
  const size_t pixels = (size_t)a->N * g.P * g.Q;
  if (pass == 1) {
    const uint32_t Kp = dgrad_kp(a->K);
    size_t b = round_1k((size_t)Kp * a->kh * a->kw * a->C * 2 + 16);
    if (Kp != a->K) b += round_1k(pixels * Kp * 2);
    return b;
  }
  if (pass == 2) {
    const uint32_t Kp = wgrad_kp(a->K);
    const size_t wcount = (size_t)Kp * a->kh * a->kw * a->C;
    uint32_t TN, TH, TW;
    pick_tile3(a->N, g.P, g.Q, a->stride_h, a->stride_w, TN, TH, TW);
    const uint32_t sp = ((a->N + TN - 1) / TN) * ((g.P + TH - 1) / TH) * ((g.Q + TW - 1) / TW);
    size_t general = (size_t)wgrad_splits(sp, Kp, a->C, a->kh * a->kw, kNumSMs) * wcount * 4;
    size_t row = conv_tc_row_wgrad_scratch(a->N, a->C, a->K, a->kh, a->kw, a->stride_h, a->stride_w, a->dil_h, a->dil_w, g.P, g.Q);
    const size_t part = std::max(general + bias_grad_bytes(pixels, a->K), row);
    size_t b = 1024 + part;
    if (Kp != a->K) b += round_1k(pixels * Kp * 2);
    return b;
  }
  return 16;
}

int conv_tc_fprop(const ad_conv2d_args* a, const ad_tensor4* addend, cudaStream_t s) {
  Geo g;
  int st = conv_geo(a, g);
  if (st != AD_OK) return st;
  if (!a->x || !a->w || !a->y) return AD_ERR_BAD_ARG;
  if (a->pad_h || a->pad_w) {
    // Implicit padding is served by TMA's out-of-bounds zero fill (negative start coordinates).
  }
  int32_t* status = (a->scratch && a->scratch_bytes >= 16) ? (int32_t*)a->scratch : nullptr;
  // A row range is the same problem with fewer output rows: shift the input row offset and the
  // output pointer, keep the pitches of the full tensor.
  uint32_t q0 = 0, nq = g.P;
  if (a->out_row_count) {
    if ((unsigned long long)a->out_row_begin + a->out_row_count > g.P) return AD_ERR_BAD_ARG;
    q0 = a->out_row_begin; nq = a->out_row_count;
  }
  const long long pitch = a->y_pitch ? a->y_pitch : (long long)g.Q * a->K;
  const long long plane = a->y_plane ? a->y_plane : (long long)g.P * g.Q * a->K;
  __nv_bfloat16* out = (__nv_bfloat16*)a->y + (long long)q0 * pitch;
  ad_tensor4 add;
  if (addend) {
    if (!addend->base || addend->dtype != AD_BF16 || addend->N != a->N || addend->C != a->K || addend->H != g.P || addend->W != g.Q) return AD_ERR_BAD_ARG;
    add = *addend;
    add.H = nq;
    add.base = (__nv_bfloat16*)addend->base + (long long)q0 * addend->sy;
    // the forms without the sum in their epilogue write y first: an addend in its place would be the new y in those and
    // the old one in the others
    const long long ax = (long long)(g.Q - 1) * add.sx, ac = (long long)(a->K - 1) * add.sc;
    const ByteRows to{(intptr_t)out, a->N, nq, plane * 2, pitch * 2, 0, (long long)g.Q * a->K * 2};
    const ByteRows from{(intptr_t)add.base, a->N, nq, add.sn * 2, add.sy * 2, 2 * (std::min(0ll, ax) + std::min(0ll, ac)),
                        2 * (std::max(0ll, ax) + std::max(0ll, ac) + 1)};
    if (rows_meet(to, from)) return AD_ERR_BAD_ARG;
  }
  return run_fwd_gemm(a->x, a->N, a->H, a->W, a->C, a->w, a->K, a->kh, a->kw, a->stride_h, a->stride_w, a->dil_h,
                      a->dil_w, -(int)a->pad_h + (int)(q0 * a->stride_h), -(int)a->pad_w, nq, g.Q, out, pitch, plane, a->bias,
                      a->relu, 0, status, s, addend ? &add : nullptr);
}

// Data gradient of a strided layer.  Output row y takes the taps r with (y + pad - r * dil) divisible by the stride, a list
// that depends on y modulo the stride only, and reads row (y + pad - r * dil) / stride of dy: so the rows and columns of
// one class are a stride-1 problem over dy with part of the taps, and all classes together do each multiplication once.
// (dy with zeros inserted, the plain problem on it, does stride^2 times as many, and writes and reads the copy:
// 16 x 128 x 75 x 57 <- 256, 3x3 stride 2, 62 + 14 us against 25.)  The taps keep their order, so the sums are the same to the bit.
struct TapList { uint32_t first, count, step; int off, dil; };   // r' = first + t * step reads dy at i + off + t * dil
static TapList class_taps(uint32_t y0, uint32_t pad, uint32_t k, uint32_t dil, uint32_t stride) {
  uint32_t g = stride, h = dil;
  while (h) { const uint32_t t = g % h; g = h; h = t; }   // gcd
  TapList l{0, 0, stride / g, 0, (int)(dil / g)};
  for (uint32_t r = 0; r < k; ++r) {
    const long long v = (long long)y0 + pad - (long long)r * dil;
    if (v % (long long)stride) continue;
    ++l.count;
    l.first = k - 1 - r;   // the last r comes first: taps are mirrored
    l.off = (int)(v / (long long)stride);
  }
  return l;
}
static int conv_tc_dgrad_strided(const ad_conv2d_args* a, const Geo& g, const void* dy, uint32_t Kp, const void* wt, uint32_t c0, uint32_t nc,
                                 int32_t* status, cudaStream_t s) {
  std::vector<FwdClass> all;
  FwdParams p{};
  for (uint32_t cy = 0; cy < a->stride_h && cy < a->H; ++cy)
    for (uint32_t cx = 0; cx < a->stride_w && cx < nc; ++cx) {
      const TapList ly = class_taps(cy, a->pad_h, a->kh, a->dil_h, a->stride_h), lx = class_taps(c0 + cx, a->pad_w, a->kw, a->dil_w, a->stride_w);
      FwdClass k{};
      k.OP = (a->H - cy + a->stride_h - 1) / a->stride_h; k.OQ = (nc - cx + a->stride_w - 1) / a->stride_w;
      k.nr = ly.count; k.ns = lx.count;
      k.offy = ly.off; k.offx = lx.off;
      k.tap0 = ly.first * a->kw + lx.first; k.tap_r = ly.step * a->kw; k.tap_s = lx.step;
      k.out_off = ((long long)cy * a->W + cx) * a->C;
      p.dh = (uint32_t)ly.dil; p.dw = (uint32_t)lx.dil;
      if (k.nr * k.ns || !a->accumulate) all.push_back(k);
    }
  std::stable_sort(all.begin(), all.end(), [](const FwdClass& x, const FwdClass& y) { return x.nr * x.ns > y.nr * y.ns; });   // long tiles first
  p.NI = a->N; p.OC = a->C; p.CK = Kp;
  p.sh = p.sw = 1;
  p.out_px = (long long)a->stride_w * a->C; p.out_pitch = (long long)a->stride_h * a->W * a->C; p.out_plane = (long long)a->H * a->W * a->C;
  p.out = (__nv_bfloat16*)a->dx + (size_t)c0 * a->C;
  p.accumulate = a->accumulate; p.status = status;
  pick_tile3(a->N, (a->H + a->stride_h - 1) / a->stride_h, (nc + a->stride_w - 1) / a->stride_w, 1, 1, p.TN, p.TH, p.TW);
  for (size_t i = 0; i < all.size(); i += kFwdClasses) {
    FwdClasses cl{};
    cl.n = (uint32_t)std::min(all.size() - i, (size_t)kFwdClasses);
    p.tiles_x = 0;
    for (uint32_t c = 0; c < cl.n; ++c) {
      FwdClass& k = cl.c[c] = all[i + c];
      k.tiles_y = (k.OP + p.TH - 1) / p.TH; k.tiles_x = (k.OQ + p.TW - 1) / p.TW;
      k.tile0 = p.tiles_x;
      p.tiles_x += ((a->N + p.TN - 1) / p.TN * k.tiles_y * k.tiles_x + 1) & ~1u;   // both tiles of a pair are of one class
    }
    const int st = run_fwd_tiles<kFwdClasses>(dy, g.P, g.Q, wt, a->kh * a->kw, p, cl, s);
    if (st != AD_OK) return st;
  }
  return AD_OK;
}

// wt: the filter as C,R,S,K with mirrored taps (NULL: made in scratch); status: where waits that run out report (NULL: the
// first word of scratch)
int conv_tc_dgrad(const ad_conv2d_args* a, const void* prepared, int32_t* status, cudaStream_t s) {
  Geo g;
  int st = conv_geo(a, g);
  if (st != AD_OK) return st;
  if (!a->y || !a->w || !a->dx || !a->scratch) return AD_ERR_BAD_ARG;
  if (a->y_pitch || a->y_plane) return AD_ERR_UNSUPPORTED;  // dy must be dense for the TMA view
  if (a->scratch_bytes < conv_tc_scratch_bytes(a, 1)) return AD_ERR_SCRATCH;
  const uint32_t Kp = dgrad_kp(a->K);
  if (!status) status = (int32_t*)a->scratch;
  const void* wt = prepared;
  char* next = (char*)a->scratch + round_1k((size_t)Kp * a->kh * a->kw * a->C * 2 + 16);
  const size_t wcount = (size_t)Kp * a->kh * a->kw * a->C;
  if (!wt) {
    __nv_bfloat16* made = (__nv_bfloat16*)((char*)a->scratch + 16);
    launch(filter_transpose_flip_kernel, grid_for(wcount, 256), 256, 0, s, a->K, Kp, a->kh, a->kw, a->C, (const __nv_bfloat16*)a->w, made);
    count_launch();
    wt = made;
  }
  const void* dy = a->y;
  if (Kp != a->K) {
    const size_t pixels = (size_t)a->N * g.P * g.Q;
    launch(pad_channels_kernel, grid_for(pixels * Kp, 256, 16), 256, 0, s, pixels, a->K, Kp, (const __nv_bfloat16*)a->y,
                                                                        (__nv_bfloat16*)next);
    count_launch();
    dy = next;
    next += round_1k(pixels * Kp * 2);
  }
  // A column range is the same problem with fewer output columns: shift the input column offset and the
  // output pointer, keep the pitches of the full tensor.
  uint32_t c0 = 0, nc = a->W;
  if (a->dx_col_count) {
    if ((unsigned long long)a->dx_col_begin + a->dx_col_count > a->W) return AD_ERR_BAD_ARG;
    c0 = a->dx_col_begin; nc = a->dx_col_count;
  }
  if (a->stride_h != 1 || a->stride_w != 1) return conv_tc_dgrad_strided(a, g, dy, Kp, wt, c0, nc, status, s);
  // dx[n,yy,xx,c] = sum_{r',s',k} dy[n, yy + ph - (kh-1)*dh + r'*dh, xx + ..., k] * wt[c][r'][s'][k]
  const int offy = (int)a->pad_h - (int)((a->kh - 1) * a->dil_h), offx = (int)a->pad_w - (int)((a->kw - 1) * a->dil_w);
  return run_fwd_gemm(dy, a->N, g.P, g.Q, Kp, wt, a->C, a->kh, a->kw, 1, 1, a->dil_h, a->dil_w, offy, offx + (int)c0, a->H,
                      nc, (__nv_bfloat16*)a->dx + (size_t)c0 * a->C, (long long)a->W * a->C, (long long)a->H * a->W * a->C,
                      nullptr, 0, a->accumulate, status, s);
}

int conv_tc_wgrad(const ad_conv2d_args* a, int32_t* status, cudaStream_t s) {
  Geo g;
  int st = conv_geo(a, g);
  if (st != AD_OK) return st;
  if (!a->x || !a->y || !a->dw || !a->scratch) return AD_ERR_BAD_ARG;
  if (a->y_pitch || a->y_plane) return AD_ERR_UNSUPPORTED;
  if (a->C % 64 != 0) return AD_ERR_UNSUPPORTED;
  if (a->scratch_bytes < conv_tc_scratch_bytes(a, 2)) return AD_ERR_SCRATCH;
  if (!status) status = (int32_t*)a->scratch;
  const uint32_t Kp = wgrad_kp(a->K);
  const void* dy = a->y;
  char* part_base = (char*)a->scratch + 1024;
  if (Kp != a->K) {
    const size_t pixels = (size_t)a->N * g.P * g.Q;
    launch(pad_channels_kernel, grid_for(pixels * Kp, 256, 16), 256, 0, s, pixels, a->K, Kp, (const __nv_bfloat16*)a->y,
                                                                        (__nv_bfloat16*)part_base);
    count_launch();
    dy = part_base;
    part_base += round_1k(pixels * Kp * 2);
  }
  const size_t part_bytes = a->scratch_bytes - (size_t)(part_base - (char*)a->scratch);
  if (Kp == a->K && !getenv("ARRAYDIFF_B200_NO_ROW_KERNEL")) {
    // 64-channel layers: one CTA serves all taps from one fetch of x and dy (conv_tc_row.cu)
    st = conv_tc_row_wgrad(a->x, a->N, a->H, a->W, a->C, a->y, a->K, a->kh, a->kw, a->stride_h, a->stride_w, a->dil_h,
                           a->dil_w, -(int)a->pad_h, -(int)a->pad_w, g.P, g.Q, (float*)a->dw, a->db, a->accumulate, a->dw_kcrs,
                           part_base, part_bytes, status, s);
    if (st != AD_ERR_UNSUPPORTED) {
      g_last_conv_kernel = kConvTcRow;
      return st;
    }
  }
  g_last_conv_kernel = kConvTcGeneral;
  WgParams p{};
  p.NI = a->N; p.OP = g.P; p.OQ = g.Q; p.KO = Kp; p.CI = a->C;
  p.kh = a->kh; p.kw = a->kw; p.sh = a->stride_h; p.sw = a->stride_w; p.dh = a->dil_h; p.dw = a->dil_w;
  p.offy = -(int)a->pad_h; p.offx = -(int)a->pad_w;
  // The tile is chosen for the dy grid; the x box is the same patch scaled by the stride.
  pick_tile3(a->N, g.P, g.Q, a->stride_h, a->stride_w, p.TN, p.TH, p.TW);
  p.tiles_y = (g.P + p.TH - 1) / p.TH;
  p.tiles_x = (g.Q + p.TW - 1) / p.TW;
  p.tiles_b = (a->N + p.TN - 1) / p.TN;
  const int BN = wgrad_bn(a->C);
  p.ktiles = (Kp + 127) / 128;
  p.ctiles = (a->C + BN - 1) / BN;
  const uint32_t sp_tiles = p.tiles_b * p.tiles_y * p.tiles_x;
  p.splits = wgrad_splits(sp_tiles, Kp, a->C, p.kh * p.kw, kNumSMs);
  p.status = status;
  p.partial = (float*)part_base;
  const size_t wcount_p = (size_t)Kp * a->kh * a->kw * a->C;
  if (part_bytes < (size_t)p.splits * wcount_p * 4) return AD_ERR_SCRATCH;

  CUtensorMap mdy, mx;
  {
    uint64_t dims[4] = {Kp, g.Q, g.P, a->N};
    uint64_t str[4] = {0, (uint64_t)Kp * 2, (uint64_t)g.Q * Kp * 2, (uint64_t)g.P * g.Q * Kp * 2};
    uint32_t box[4] = {64, p.TW, p.TH, p.TN};
    uint32_t es[4] = {1, 1, 1, 1};
    st = make_tmap_bf16(&mdy, dy, 4, dims, str, box, es);
    if (st != AD_OK) return st;
  }
  {
    uint64_t dims[4] = {a->C, a->W, a->H, a->N};
    uint64_t str[4] = {0, (uint64_t)a->C * 2, (uint64_t)a->W * a->C * 2, (uint64_t)a->H * a->W * a->C * 2};
    uint32_t box[4] = {64, p.TW * a->stride_w, p.TH * a->stride_h, p.TN};
    uint32_t es[4] = {1, a->stride_w, a->stride_h, 1};
    st = make_tmap_bf16(&mx, a->x, 4, dims, str, box, es);
    if (st != AD_OK) return st;
  }
  // pairs need an even number of 128-channel tiles of dy, and 64 channels of x per CTA
  st = BN == 128 ? (p.ktiles % 2 == 0 ? launch_wgrad<128, true>(mdy, mx, p, s) : launch_wgrad<128, false>(mdy, mx, p, s))
                 : launch_wgrad<64, false>(mdy, mx, p, s);
  if (st != AD_OK) return st;
  const size_t filter_bytes = (size_t)p.splits * wcount_p * 4;
  launch_wgrad_reduce(a->K, a->kh * a->kw, a->C, wcount_p, p.splits, p.partial, (float*)a->dw, a->accumulate, a->dw_kcrs,
                      BiasGrad{(size_t)a->N * g.P * g.Q, a->y, a->db, (float*)(part_base + filter_bytes), part_bytes - filter_bytes}, s);
  return launch_status();
}

}  // namespace tc

// fp32 direct path (conv_direct.cu)
int conv_direct_fprop(const ad_conv2d_args* a, cudaStream_t s);
int conv_direct_dgrad(const ad_conv2d_args* a, cudaStream_t s);
int conv_direct_wgrad(const ad_conv2d_args* a, cudaStream_t s);
size_t conv_direct_scratch_bytes(const ad_conv2d_args* a, int pass);

}  // namespace adk

using namespace adk;

static int path_of(const ad_conv2d_args* a) {
  if (!a) return -1;
  if (a->dtype == AD_F32 && a->layout == AD_NCHW) return 0;
  if (a->dtype == AD_BF16 && a->layout == AD_NHWC) return 1;
  return -1;
}

extern "C" size_t ad_conv2d_scratch_bytes(const ad_conv2d_args* a, int32_t pass) {
  switch (path_of(a)) {
    case 0: return conv_direct_scratch_bytes(a, pass);
    case 1: return tc::conv_tc_scratch_bytes(a, pass);
    default: return 0;
  }
}

// ---------------------------------------------------------------- per-call timing (ad_conv2d_profile)
namespace {
struct ProfRec {
  ad_conv2d_profile_entry e;
  cudaEvent_t e0, e1;
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::vector<ProfRec> g_prof;

template <typename F>
int profiled(int pass, const ad_conv2d_args* a, void* stream, F&& call) {
  if (!g_prof_on || !a) return call();
  ProfRec r{};
  if (cudaEventCreate(&r.e0) != cudaSuccess || cudaEventCreate(&r.e1) != cudaSuccess) {
    cudaGetLastError();
    return call();
  }
  cudaEventRecord(r.e0, as_stream(stream));
  const int st = call();
  cudaEventRecord(r.e1, as_stream(stream));
  r.e.pass = pass; r.e.kernel = g_last_conv_kernel; r.e.status = st;
  r.e.N = a->N; r.e.C = a->C; r.e.H = a->H; r.e.W = a->W; r.e.K = a->K; r.e.kh = a->kh; r.e.kw = a->kw;
  r.e.stride = a->stride_h; r.e.dil = a->dil_h; r.e.pad = a->pad_h;
  r.e.out_rows = pass == 0 ? a->out_row_count : 0;
  std::lock_guard<std::mutex> lk(g_prof_mu);
  g_prof.push_back(r);
  return st;
}
}  // namespace

extern "C" int ad_conv2d_profile(int32_t enable) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  for (auto& r : g_prof) { cudaEventDestroy(r.e0); cudaEventDestroy(r.e1); }
  g_prof.clear();
  g_prof_on = enable != 0;
  return AD_OK;
}
extern "C" size_t ad_conv2d_profile_read(ad_conv2d_profile_entry* out, size_t max_entries) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  if (!out) return g_prof.size();
  size_t n = 0;
  for (auto& r : g_prof) {
    if (n == max_entries) break;
    cudaEventSynchronize(r.e1);
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, r.e0, r.e1) != cudaSuccess) { cudaGetLastError(); ms = -1.f; }
    r.e.ms = ms;
    out[n++] = r.e;
  }
  return n;
}

static int fprop_call(const ad_conv2d_args* a, const ad_tensor4* addend, void* stream) {
  return profiled(0, a, stream, [&] {
    switch (path_of(a)) {
      case 0: g_last_conv_kernel = kConvDirectF32; return addend ? (int)AD_ERR_UNSUPPORTED : conv_direct_fprop(a, as_stream(stream));
      case 1: return tc::conv_tc_fprop(a, addend, as_stream(stream));
      default: return (int)(a ? AD_ERR_UNSUPPORTED : AD_ERR_BAD_ARG);
    }
  });
}
extern "C" int ad_conv2d_fprop(const ad_conv2d_args* a, void* stream) { return fprop_call(a, nullptr, stream); }
extern "C" int ad_conv2d_fprop_add(const ad_conv2d_args* a, const ad_tensor4* addend, void* stream) { return fprop_call(a, addend, stream); }
static int dgrad_call(const ad_conv2d_args* a, const void* w_crsk, int32_t* status, void* stream) {
  return profiled(1, a, stream, [&] {
    switch (path_of(a)) {
      case 0: g_last_conv_kernel = kConvDirectF32; return conv_direct_dgrad(a, as_stream(stream));
      case 1: return tc::conv_tc_dgrad(a, w_crsk, status, as_stream(stream));
      default: return (int)(a ? AD_ERR_UNSUPPORTED : AD_ERR_BAD_ARG);
    }
  });
}
extern "C" int ad_conv2d_dgrad(const ad_conv2d_args* a, void* stream) { return dgrad_call(a, nullptr, nullptr, stream); }
extern "C" int ad_conv2d_dgrad_ex(const ad_conv2d_args* a, const void* w_crsk, int32_t* status, void* stream) {
  return dgrad_call(a, w_crsk, status, stream);
}
static int wgrad_call(const ad_conv2d_args* a, int32_t* status, void* stream) {
  return profiled(2, a, stream, [&] {
    switch (path_of(a)) {
      case 0: g_last_conv_kernel = kConvDirectF32; return conv_direct_wgrad(a, as_stream(stream));
      case 1: return tc::conv_tc_wgrad(a, status, as_stream(stream));
      default: return (int)(a ? AD_ERR_UNSUPPORTED : AD_ERR_BAD_ARG);
    }
  });
}
extern "C" int ad_conv2d_wgrad(const ad_conv2d_args* a, void* stream) { return wgrad_call(a, nullptr, stream); }
extern "C" int ad_conv2d_wgrad_ex(const ad_conv2d_args* a, int32_t* status, void* stream) {
  LateLaunch late;
  return wgrad_call(a, status, stream);
}

extern "C" int ad_filter_prepare(uint32_t count, const ad_filter_item* items, void* stream) {
  if (count && !items) return AD_ERR_BAD_ARG;
  for (uint32_t i = 0; i < count; ++i) {
    const ad_filter_item& f = items[i];
    if (!f.src || !f.krsc || !f.K || !f.C || !f.kh || !f.kw || (f.crsk && (f.crsk_k < f.K || (f.crsk_k & 1) || ((uintptr_t)f.crsk & 3u)))) return AD_ERR_BAD_ARG;
    if (f.krsc_row < (int64_t)f.kh * f.kw * f.C || (f.crsk && f.krsc_row != (int64_t)f.kh * f.kw * f.C)) return AD_ERR_UNSUPPORTED;
  }
  const cudaStream_t s = as_stream(stream);
  for (uint32_t i0 = 0; i0 < count; i0 += tc::kPrepItems) {
    tc::PrepBatch b{};
    b.count = std::min(count - i0, tc::kPrepItems);
    for (uint32_t i = 0; i < b.count; ++i) {
      const ad_filter_item& f = items[i0 + i];
      tc::PrepItem& p = b.it[i];
      if ((uint64_t)f.kh * f.kw * 32 > tc::kPrepFloats) {   // more taps than the tile holds (over 288): element by element
        const int64_t taps = (int64_t)f.kh * f.kw;
        ad_tensor4 src = {(void*)f.src, AD_F32, f.K, f.C, f.kh, f.kw, f.C * taps, taps, f.kw, 1};
        ad_tensor4 dst = {f.krsc, AD_BF16, f.K, f.C, f.kh, f.kw, f.krsc_row, 1, (int64_t)f.kw * f.C, f.C};
        if (int rc = ad_convert(&src, &dst, 0, stream)) return rc;
        if (f.crsk) {
          launch(tc::filter_transpose_flip_kernel, grid_for((size_t)f.C * taps * f.crsk_k, 256), 256, 0, s, f.K, f.crsk_k, f.kh, f.kw, f.C, (const __nv_bfloat16*)f.krsc, (__nv_bfloat16*)f.crsk);
          count_launch();
        }
        p.tile0 = b.tiles;
        p.K = p.C = p.taps = p.Kp = p.KT = p.CT = 1;
        continue;
      }
      p.src = f.src; p.krsc = (__nv_bfloat16*)f.krsc; p.crsk = (__nv_bfloat16*)f.crsk;
      p.K = f.K; p.C = f.C; p.taps = f.kh * f.kw; p.Kp = f.crsk ? f.crsk_k : f.K; p.row = f.krsc_row;
      const bool pairs = !(p.row & 1) && !((uintptr_t)f.krsc & 3u);
      p.KT = p.taps == 1 && p.C % 64 == 0 && pairs ? 128 : 32;
      p.CT = p.KT == 128 ? 64 : std::min(32u, tc::kPrepFloats / (32 * p.taps));
      p.tile0 = b.tiles;
      b.tiles += (p.Kp + p.KT - 1) / p.KT * ((p.C + p.CT - 1) / p.CT);
    }
    if (!b.tiles) continue;
    launch(tc::filter_prepare_kernel, std::min(b.tiles, (uint32_t)kNumSMs * 6), 256, 0, s, b);
    count_launch();
  }
  return launch_status();
}
