// Choices of the tensor-core convolutions that need no GPU.
#pragma once

#include <algorithm>
#include <cstdint>

namespace adk {
namespace tc {

// Input channels per CTA of the general filter-gradient kernel.  (A 256-wide tile halves the L2 fetches of the dy
// tile but leaves room for two pipeline stages only: measured 15 % slower on the 512 -> 512 layers.)
inline int wgrad_bn(uint32_t C) { return C > 64 ? 128 : 64; }
// Splits of the pixel range of which an accumulator in tensor memory sums one: twice as many items as SMs, at most 64.  Fewer make
// longer runs of sums in the accumulator, which cuts the last bit off at every step, always towards zero: the error grows with
// the length of a run.  Half as many (what the rule below would take by time alone) gave 4.0e-6 against 64 bits on average
// over 95 layers where these give 2.1e-6, at worst 7.3e-5 against 2.4e-5 (512 -> 512, 3x3 on 65,536 pixels).
inline uint32_t wgrad_least_splits(uint32_t sp_tiles, uint32_t KO, uint32_t C, uint32_t taps, uint32_t sms) {
  const uint32_t BN = (uint32_t)wgrad_bn(C), outer = taps * ((KO + 127) / 128) * ((C + BN - 1) / BN);
  return std::max(1u, std::min(std::min((2 * sms + outer - 1) / outer, sp_tiles), 64u));
}
// From there on the count with the shortest time by rounds of the machine's CTAs (pairs) and by what the partial gradients cost on
// their way out and back (a pixel tile of an item takes about 0.5 us, 2.5 MB): a count that leaves the last round nearly
// empty costs most.  95 layers, us in sum: the least count 5060 (with the bias gradient in launches of its own), this
// 4500, by time alone 4180; error 1.7e-6.
inline uint32_t wgrad_splits(uint32_t sp_tiles, uint32_t KO, uint32_t C, uint32_t taps, uint32_t sms) {
  const uint32_t BN = (uint32_t)wgrad_bn(C), ktiles = (KO + 127) / 128, least = wgrad_least_splits(sp_tiles, KO, C, taps, sms);
  const bool pair = BN == 128 && ktiles % 2 == 0;
  const unsigned long long outer = (unsigned long long)taps * (pair ? ktiles / 2 : ktiles) * ((C + BN - 1) / BN), units = pair ? sms / 2 : sms;
  const double part = (double)KO * taps * C * 8 / 2.5e6;
  uint32_t best = least;
  double best_cost = 0;
  for (uint32_t n = least; n <= sp_tiles && n <= 64; ++n) {   // above 64 the reduction takes a third trip to the L2 (64 -> 256: 36 us, 74 splits 39)
    const double cost = (double)((outer * n + units - 1) / units) * ((sp_tiles + n - 1) / n) + n * part;
    if (n == least || cost < best_cost) { best = n; best_cost = cost; }
    if (outer * n > 8 * units) break;
  }
  return best;
}

}  // namespace tc
}  // namespace adk
