// Do two strided views share memory?  Plain C++: what it decides can be checked without a GPU.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

namespace adk {

// N x H rows of [lo, hi) bytes from base + n * sn + y * sy (strides in bytes, of either sign)
struct ByteRows {
  intptr_t base;
  uint32_t N, H;
  long long sn, sy, lo, hi;
};

// A view inside the gaps of another (the other half of a padded row, every other image) shares nothing with it.  Rows are
// looked at one by one only where the extents meet, which those of two allocations never do.
inline bool rows_meet(const ByteRows& a, const ByteRows& b) {
  struct Span { intptr_t lo, hi; int of; };
  auto extent = [](const ByteRows& r) {
    const long long n = (long long)(r.N - 1) * r.sn, y = (long long)(r.H - 1) * r.sy;
    return Span{(intptr_t)(r.base + std::min(0ll, n) + std::min(0ll, y) + r.lo), (intptr_t)(r.base + std::max(0ll, n) + std::max(0ll, y) + r.hi), 0};
  };
  if (!a.N || !a.H || !b.N || !b.H) return false;
  const Span ea = extent(a), eb = extent(b);
  if (ea.hi <= eb.lo || eb.hi <= ea.lo) return false;
  std::vector<Span> spans;
  spans.reserve((size_t)a.N * a.H + (size_t)b.N * b.H);
  for (const ByteRows* r : {&a, &b})
    for (uint32_t n = 0; n < r->N; ++n)
      for (uint32_t y = 0; y < r->H; ++y) {
        const intptr_t at = (intptr_t)(r->base + (long long)n * r->sn + (long long)y * r->sy);
        spans.push_back({(intptr_t)(at + r->lo), (intptr_t)(at + r->hi), r == &b});
      }
  std::sort(spans.begin(), spans.end(), [](const Span& x, const Span& y) { return x.lo < y.lo; });
  intptr_t end[2] = {INTPTR_MIN, INTPTR_MIN};   // how far the rows so far reach
  for (const Span& s : spans) {
    if (s.lo < end[1 - s.of]) return true;
    end[s.of] = std::max(end[s.of], s.hi);
  }
  return false;
}

}  // namespace adk
