// svo_route.h -- host-side rules of the casts: plain functions of sizes, addresses and flags, which need no device.
#pragma once

#include <cstdint>
#include <utility>
#include <vector>

#include "svo_internal.h"

namespace svo {

// Whether a cast can work on host arrays in place, without the staged copies (which take any address).
// The kernels load and store whole elements: an array of 4-byte elements off a 4-byte boundary would fault.
inline bool arrays_aligned(const svo_rays& rays, const svo_hits& hits) {
  const float* const in[6] = {rays.ox, rays.oy, rays.oz, rays.dx, rays.dy, rays.dz};
  void* const* out = reinterpret_cast<void* const*>(&hits);
  uintptr_t bits = 0;
  for (const float* p : in) bits |= reinterpret_cast<uintptr_t>(p) & 3u;
  for (int f = 0; f < kHitFields; ++f) bits |= reinterpret_cast<uintptr_t>(out[f]) & (kHitFieldBytes[f] - 1u);
  return bits == 0;
}

// Whether hits written in place may change rays that are still to be read: a hit field over a ray array, other than element
// for element (a ray is read before its own hit is written).  Copies of a batch are complete before its cast.
inline bool hits_over_rays(const svo_rays& rays, const svo_hits& hits, uint64_t n) {
  const float* const in[6] = {rays.ox, rays.oy, rays.oz, rays.dx, rays.dy, rays.dz};
  void* const* out = reinterpret_cast<void* const*>(&hits);
  uintptr_t low = UINTPTR_MAX, high = 0;  // all rays lie between these
  for (const float* p : in) {
    const uintptr_t r = reinterpret_cast<uintptr_t>(p);
    low = r < low ? r : low;
    high = r > high ? r : high;
  }
  high += sizeof(float) * n;
  for (int f = 0; f < kHitFields; ++f) {
    const uintptr_t h = reinterpret_cast<uintptr_t>(out[f]);
    if (!h || h >= high || h + kHitFieldBytes[f] * n <= low) continue;
    for (const float* p : in) {
      const uintptr_t r = reinterpret_cast<uintptr_t>(p);
      if (h == r && kHitFieldBytes[f] == sizeof(float)) continue;
      if (h < r + sizeof(float) * n && r < h + kHitFieldBytes[f] * n) return true;
    }
  }
  return false;
}

// Spans [a, b) of elements, added in order; those fewer than `gap` apart become one.
using Spans = std::vector<std::pair<uint64_t, uint64_t>>;
inline void add_span(Spans& spans, uint64_t a, uint64_t b, uint64_t gap) {
  if (spans.empty() || a - spans.back().second >= gap)
    spans.push_back({a, b});
  else
    spans.back().second = b;
}

}  // namespace svo
