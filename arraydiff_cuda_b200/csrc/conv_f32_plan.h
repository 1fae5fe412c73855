// Host-side choices of the fp32 convolutions (conv_f32.cu) in plain C++: what they decide can be checked without a GPU.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace adk {

// CTAs that share one tile's reduction of `steps` stages: the size with the shortest time by a count of waves.  held(cs):
// clusters of cs CTAs that the machine holds at a time; a size of which it holds none cannot be launched and is passed over.
// A CTA costs its stages and about six more to start and finish; one CTA on an SM takes 2.2 per stage, two 2.5, three 3 (12
// warps hide most of what they wait for).  Of the sizes 1 .. 16 this picks the fastest or one within a tenth of it for 18 of
// 20 layers measured.  Before, the size went by CTAs per SM alone: 35 clusters of 8 where the machine holds 33
// took two waves (filter gradient 64 -> 64, 4 x 112 x 112: 228 us against 168 for 30).
template <typename Held>
uint32_t f32_cluster_size(Held held, unsigned long long tiles, uint32_t steps, uint32_t most, uint32_t sms) {
  static const double per_stage[4] = {0, 2.2, 2.5, 3.0};
  uint32_t best = 0;
  double best_cost = 0;
  for (uint32_t cs = 1; cs <= most && (cs == 1 || steps >= 4 * cs); cs *= 2) {
    const unsigned long long h = held(cs);
    if (!h) continue;
    auto wave = [&](unsigned long long clusters) { return per_stage[std::min<unsigned long long>((clusters * cs + sms - 1) / sms, 3)]; };
    const double cta = (steps + cs - 1) / cs + 6, cost = cta * (tiles / h * wave(h) + (tiles % h ? wave(tiles % h) : 0));
    if (!best || cost < best_cost) { best = cs; best_cost = cost; }
  }
  return best ? best : 1;
}

// The 3x3 and 1x1 kernels (conv_f32_k3.cu, conv_f32_k1.cu: stages of 18 and 16 terms) keep the FMA pipe busy with one CTA per SM, so that CTAs on one SM take turns (a stage
// measured 1.1 us alone, 1.9 beside one other, 2.7 beside two), and the SM with the most of them counts.  A cluster stays
// within one group of SMs, so that larger ones are spread less evenly: 36 clusters of 4 leave some SMs two CTAs (filter gradient
// 64 -> 64, 4 x 112 x 112: 184 us, 32 clusters of 4 133), and so do 16 of 8 already (half of the SMs were idle).
inline double f32_k3_share(unsigned long long ctas, uint32_t cs, uint32_t sms, double one, double two) {
  const double per_stage[4] = {0, one, two, 3.0};
  const double even = (double)ctas * (cs >= 8 ? 1.15 : cs >= 4 ? 1.1 : cs == 2 ? 1.02 : 1.0) / sms;
  return per_stage[even > 2 ? 3 : even > 1 || (cs >= 8 && even > 0.5) ? 2 : ctas ? 1 : 0];
}
template <typename Held>
uint32_t f32_k3_cluster(Held held, unsigned long long tiles, uint32_t steps, uint32_t most, uint32_t sms) {
  uint32_t best = 0;
  double best_cost = 0;
  for (uint32_t cs = 1; cs <= most && (cs == 1 || steps >= 2 * cs); cs *= 2) {
    const unsigned long long h = held(cs);
    if (!h) continue;
    const double cost = (steps + cs - 1) / cs * (tiles / h * f32_k3_share(h * cs, cs, sms, 1.2, 2.1) + f32_k3_share(tiles % h * cs, cs, sms, 1.2, 2.1)) + 0.75 * cs;
    // a CTA sums over 128 stages (256 channels) at most where that can be: the sum of its running sums loses precision with
    // their number (371 channels in one CTA: 2.0e-7 against 1.7e-7 in two)
    if (!best || cost < best_cost || (steps > 128 * best)) { best = cs; best_cost = cost; }
  }
  return best ? best : 1;
}

// Blocks of 4 x 2 pixels of the 3x3 kernels in an image: a map under dilation falls into dh x dw maps without
inline unsigned long long f32_k3_blocks(uint32_t OH, uint32_t OW, uint32_t dh, uint32_t dw) {
  return (unsigned long long)(((OH + dh - 1) / dh + 3) / 4) * (((OW + dw - 1) / dw + 1) / 2) * dh * dw;
}
// Segments of up to 8 pixels of a row
inline uint32_t f32_k3_segments(uint32_t Q, uint32_t dw) { return ((Q + dw - 1) / dw + 7) / 8 * dw; }

// Filter gradient of the 3x3 kernels: CTAs of a cluster x slices of the grid that share a tile's `all` stages of pixels
struct F32Split { uint32_t cs, slices; };
// A stage takes 3.0 us alone, 4.8 beside one other, 7.0 beside two: the most CTAs that are resident together win, up to what
// their start, and writing and adding the slices' `words` (the gradient's size), cost.  The constants are not these times (which
// are 1.3 and 2.1 where the longest counts 3) but a fit to 1000 times of whole calls of 40 layers: the choice is on average 1.6 %
// above the fastest (7.6 % with the forward kernels' ones: 256 -> 256, 4 x 14 x 14 52 -> 44 us, 191 -> 75, 3 x 71 x 10 68 -> 54).
// The slices' scratch stays within 32 MB.  The clusters that are held at a time are those of a whole GPU, not asked of the device:
// the size of the scratch, which follows from the split, can be asked for where there is none.
inline F32Split f32_k3_split(unsigned long long tiles, unsigned long long all, unsigned long long words, uint32_t sms, uint32_t per_sm) {
  // clusters of 1, 2, 4, 8 CTAs at a time, two or three CTAs per SM
  static const unsigned held2[4] = {296, 148, 70, 33}, held3[4] = {444, 222, 104, 48};
  const unsigned* const held = per_sm == 2 ? held2 : held3;
  F32Split best = {1, 1};
  double best_cost = 0;
  for (uint32_t i = 0; i < 4; ++i)
    for (uint32_t sl = 1; sl <= 16; ++sl) {
      const uint32_t cs = 1u << i, parts = cs * sl;
      if ((parts > 1 && all < 2ull * parts) || (sl > 1 && sl * words > (8ull << 20))) break;
      const unsigned long long h = held[i], n = tiles * sl;
      const double cta = (double)((all + parts - 1) / parts) + 1.75 + 0.5 * cs;
      const double cost = cta * (n / h * f32_k3_share(h * cs, cs, sms, 1.8, 2.35) + f32_k3_share(n % h * cs, cs, sms, 1.8, 2.35)) +
                          (sl > 1 ? 2.1 + (0.1 + 0.63e-6 * words) * sl : 0);
      if (best_cost == 0 || cost < best_cost) { best = {cs, sl}; best_cost = cost; }
    }
  return best;
}

// `most` CTAs, or the largest smaller power of two of which the machine holds a cluster
template <typename Held>
uint32_t f32_largest_cluster(Held held, uint32_t most) {
  uint32_t cs = most;
  while (cs > 1 && !held(cs)) cs /= 2;
  return cs;
}

// Images that the two-step data gradient into few channels takes at a time: as many as fit `limit` bytes of scratch, z bytes
// each, and whose input elements a 32-bit index counts with room for a step of the grid (an image has fewer than 2^31; with a
// stride of 32 and more, small maps of dy belong to a gradient of more than 2^32 elements).  0: one image does not fit.
inline uint32_t f32_few_images(uint32_t N, unsigned long long image, unsigned long long z, unsigned long long limit) {
  return (uint32_t)std::min<unsigned long long>(N, std::min(limit / z, ((1ull << 31) - 1) / image));
}

}  // namespace adk
