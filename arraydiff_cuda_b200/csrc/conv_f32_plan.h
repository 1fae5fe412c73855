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
