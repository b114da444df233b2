// svo_unit.cuh -- node heads: a node as rays of one direction octant see it.
#pragma once

#include "svo_cast.cuh"

namespace svo {

#define SVO_UHD __host__ __device__ __forceinline__

// ------------------------------------------------------------------ node heads
// One node as rays of one direction octant see it (uint4: x, y, z, w).
//   x, y  bit m of the 64: a cell of the node's 4x4x4 occupancy lies in the box between mirrored cell m
//         (mx | my << 2 | mz << 4) and the far corner; 0 for a UniformLeaf, which is always left after its probe
//   z     [7:0] mirrored octants that stop an ADVANCE (an Internal node's occupied octants with a child,
//         a Leaf's bricks that are not Empty; all or none for a UniformLeaf), [15:8] mirrored octants whose
//         brick is Solid, [17:16] content kind, [19:18] MIP brick kind
//   w     the MIP brick's value
constexpr uint32_t kHeadPlanes = 8;

// The head of node record n for rays whose positive axes are `dir` (octant bit layout).
SVO_UHD uint4 node_head(const DevNode& n, uint32_t dir) {
  const uint32_t kind = n.meta & 3u, flip = dir ^ 7u;
  uint64_t occ = n.ocbits;
  // mirrored occupancy: reverse the cells along each axis the ray travels towards -
  if (flip & 1u) {
    occ = ((occ & 0x5555555555555555ull) << 1) | ((occ >> 1) & 0x5555555555555555ull);
    occ = ((occ & 0x3333333333333333ull) << 2) | ((occ >> 2) & 0x3333333333333333ull);
  }
  if (flip & 4u) {
    occ = ((occ & 0x0F0F0F0F0F0F0F0Full) << 4) | ((occ >> 4) & 0x0F0F0F0F0F0F0F0Full);
    occ = ((occ & 0x00FF00FF00FF00FFull) << 8) | ((occ >> 8) & 0x00FF00FF00FF00FFull);
  }
  if (flip & 2u) {
    occ = ((occ & 0x0000FFFF0000FFFFull) << 16) | ((occ >> 16) & 0x0000FFFF0000FFFFull);
    occ = (occ << 32) | (occ >> 32);
  }
  uint32_t live = 0, solid = 0;
  for (uint32_t m = 0; m < 8; ++m) {
    const uint32_t o = m ^ flip, bk = (n.meta >> (8 + 2 * (kind == kKindLeaf ? o : 0u))) & 3u;
    bool on;
    if (kind == kKindInternal)
      on = n.slot[o] != kInvalidChild && (n.ocbits & octant_mask(o)) != 0;
    else
      on = (kind == kKindLeaf || kind == kKindUniform) && bk != kBkEmpty;
    live |= (on ? 1u : 0u) << m;
    solid |= ((kind == kKindLeaf || kind == kKindUniform) && bk == kBkSolid ? 1u : 0u) << m;
  }
  // the union over all cells at or beyond each cell, axis by axis (+1, then +2, within 4 cells)
  uint64_t r = occ;
  r |= (r >> 1) & 0x7777777777777777ull;
  r |= (r >> 2) & 0x3333333333333333ull;
  r |= (r >> 4) & 0x0FFF0FFF0FFF0FFFull;
  r |= (r >> 8) & 0x00FF00FF00FF00FFull;
  r |= r >> 16;
  r |= r >> 32;
  if (kind == kKindUniform) r = 0;
  uint4 hd;
  hd.x = (uint32_t)r;
  hd.y = (uint32_t)(r >> 32);
  hd.z = live | (solid << 8) | (kind << 16) | (((n.meta >> 24) & 3u) << 18);
  hd.w = n.mip;
  return hd;
}

}  // namespace svo
