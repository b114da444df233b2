// svo_route.h -- host-side rules of the casts: plain functions of sizes, addresses and flags, which need no device.
#pragma once

#include <cstdint>

#include "svo_internal.h"

namespace svo {

// Whether a cast can work on host arrays in place, without the staged copies (which take any address).
// The kernels load and store whole elements: an array of 4-byte elements off a 4-byte boundary would fault.
inline bool arrays_aligned(const svo_rays& rays, const svo_hits& hits) {
  const float* const in[6] = {rays.ox, rays.oy, rays.oz, rays.dx, rays.dy, rays.dz};
  void* const* out = reinterpret_cast<void* const*>(&hits);
  for (const float* p : in)
    if (reinterpret_cast<uintptr_t>(p) % sizeof(float)) return false;
  for (int f = 0; f < kHitFields; ++f)
    if (reinterpret_cast<uintptr_t>(out[f]) % kHitFieldBytes[f]) return false;
  return true;
}

}  // namespace svo
