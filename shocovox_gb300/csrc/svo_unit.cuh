// svo_unit.cuh -- node heads, and the arithmetic of the cast's form for rays of unit direction (svo_flow.cuh).
//
// That form visits the same nodes and voxels as cast_ray_fast_from (svo_cast.cuh) and moves the point by the
// same f32 operations, so its hits are the same bit for bit.  What differs is the bookkeeping:
//
//  * Everything is mirrored into the ray's own direction octant: in mirrored octants and cells, "far"
//    (bit set) is the side the ray leaves by.  A step can only turn near into far, so it leaves the
//    parent exactly when a moved axis is far already.
//  * The node is kept as its centre c and half size h, the target cell (a child, of size h) as the
//    planes X that the ray leaves it by.  The reference's distance to leave, for a direction towards
//    +, is fl(size - fl(p - min)).  fl(p - min) is exact when p >= min / 2, and then the distance is
//    fl((min + size) - p) = fl(X - p).  p < min / 2 cannot happen: an axis' cell changes only when the
//    step ends on that cell's plane, up to the rounding of p and to the error of |d|, both below
//    min / 2 by far for a unit direction (min is a multiple of the cell left, or 0, where p - 0 is
//    exact).  For a direction towards - both forms are |p - min|.
//  * A cell index is one fused multiply-add rounded down: floor((p - min) * q) + 2^23.  The
//    reference takes floor(fl(p - min) * q) clamped at 0: fl(p - min) is exact for p >= min / 2 and
//    negative otherwise.  Its octant test fl(p - min) >= half is p >= min + half for the same reason.
//  * Steps are not counted one by one.  A visit, its probe and its ADVANCE make at most
//    work_per_visit(D) steps, so the cap of 2^22 steps cannot have been passed before kWorkCap /
//    work_per_visit(D) visits.
//
// A ray that is not eligible (unit_eligible), or that makes too many visits or a restart run whose end is
// not certain to lie below the cap, is cast by the general forms instead, from its start.
#pragma once

#include "svo_cast.cuh"

#ifdef __CUDA_ARCH__
#define SVO_LD(p) __ldg(p)
#else
#include <cfenv>
#include <cmath>
#define SVO_LD(p) (*(p))
#endif

namespace svo {

#define SVO_UHD __host__ __device__ __forceinline__

// fma(a, b, c) rounded down
SVO_UHD float fma_down(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rd(a, b, c);
#else
  std::fesetround(FE_DOWNWARD);
  volatile float va = a, vb = b, vc = c;
  volatile float r = std::fmaf(va, vb, vc);
  std::fesetround(FE_TONEAREST);
  return r;
#endif
}
// fma(a, b, c) where a * b is exact (b a power of two or 0, +-1): one rounding either way
SVO_UHD float fma_near(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fmaf(a, b, c);
#endif
}
// max(min(a, b), 0)
SVO_UHD int min_relu(int a, int b) {
#ifdef __CUDA_ARCH__
  return __vimin_s32_relu(a, b);
#else
  const int m = a < b ? a : b;
  return m > 0 ? m : 0;
#endif
}

// hash_region (src/spatial/math/mod.rs:11-19) and the bitmap position's clamp
SVO_UHD uint32_t octant_of(float x, float y, float z, float half) {
  return (x >= half ? 1u : 0u) + (z >= half ? 2u : 0u) + (y >= half ? 4u : 0u);
}
SVO_UHD float clamp_bitmap(float x) { return fminf(fmaxf(x, kTol), 4.0f - kTol); }

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

// ------------------------------------------------------------------ eligibility
// Steps of one visit at most: the visit, an ADVANCE of 4 and a brick's 3 D + 2, and as much again to spare.
SVO_UHD uint32_t work_per_visit(uint32_t dim) { return 16u * (dim + 4u); }

// Rays of unit direction that start within 1024 octree sizes, whose direction octant in the reference's
// table (1 + d >= 1) is that of their signs (a component in (-2^-25, -0] breaks this).
SVO_UHD bool unit_eligible(const SceneView& s, float ox, float oy, float oz, float dx, float dy, float dz) {
  const float len2 = (dx * dx + dy * dy) + dz * dz;
  const float far = s.size * 1024.0f;
  auto same = [](float d) { return (1.0f + d >= 1.0f) == !signbit(d); };
  return !s.literal && s.visit_limit != 0u && fabsf(len2 - 1.0f) <= 0x1p-12f && fabsf(ox) <= far && fabsf(oy) <= far && fabsf(oz) <= far &&
         same(dx) && same(dy) && same(dz);
}

// ------------------------------------------------------------------ the traversal
struct UnitRay {
  float dx, dy, dz;  // direction
  float fx, fy, fz;  // dda scale factors
  float gx, gy, gz;  // signs of the direction, +-1
  float px, py, pz;  // current point
};

// dda_step_to_next_sibling (raytracing_on_cpu.rs:124-152) to the planes (Xx, Xy, Xz)
SVO_UHD void unit_step(UnitRay& r, float Xx, float Xy, float Xz, bool& mx, bool& my, bool& mz) {
  const float ax = fabsf((Xx - r.px) * r.fx), ay = fabsf((Xy - r.py) * r.fy), az = fabsf((Xz - r.pz) * r.fz);
  const float m = fminf(fminf(ax, ay), az);
  r.px = r.px + r.dx * m;
  r.py = r.py + r.dy * m;
  r.pz = r.pz + r.dz * m;
  mx = m == ax;
  my = m == ay;
  mz = m == az;
}

// cube_impact_normal (src/spatial/raytracing/mod.rs:106-134) of the cube with centre (cx, cy, cz).  One
// largest component v gives v / sqrt(v * v) = +-1 exactly (v * v neither over- nor underflows in the
// range tested); ties (an edge) take the reference's operations.
SVO_UHD void unit_normal(const UnitRay& r, float cx, float cy, float cz, HitRecord& h) {
  const float mx = cx - r.px, my = cy - r.py, mz = cz - r.pz;
  const float m = fmaxf(fmaxf(fabsf(mx), fabsf(my)), fabsf(mz));
  const bool ex = fabsf(mx) == m, ey = fabsf(my) == m, ez = fabsf(mz) == m;
  h.nx = ex ? copysignf(1.0f, -mx) : 0.0f;
  h.ny = ey ? copysignf(1.0f, -my) : 0.0f;
  h.nz = ez ? copysignf(1.0f, -mz) : 0.0f;
  if ((ex && ey) || (ex && ez) || (ey && ez) || !(m > 0x1p-40f && m < 0x1p40f)) {
    const float vx = ex ? -mx : 0.0f, vy = ey ? -my : 0.0f, vz = ez ? -mz : 0.0f;
    const float len = sqrtf((vx * vx + vy * vy) + vz * vz);
    h.nx = vx / len;
    h.ny = vy / len;
    h.nz = vz / len;
  }
}

SVO_UHD int unit_bits(float v) {  // the integer part of a float in [2^23, 2^24)
#ifdef __CUDA_ARCH__
  return __float_as_int(v) - 0x4B000000;
#else
  return (int)f32_bits(v) - 0x4B000000;
#endif
}

#ifdef __CUDACC__
// ------------------------------------------------------------------ any ray
// How a ray is cast: in the unit-direction form, the fast form (no NaN in the direction), or literally.
enum : uint32_t { kFormLiteral = 0, kFormFast = 1, kFormUnit = 2 };

__device__ __forceinline__ uint32_t ray_form(const SceneView& s, float ox, float oy, float oz, float dx, float dy,
                                             float dz) {
  if (unit_eligible(s, ox, oy, oz, dx, dy, dz)) return kFormUnit;
  return (!s.literal && !isnan(dx) && !isnan(dy) && !isnan(dz)) ? kFormFast : kFormLiteral;
}
#endif  // __CUDACC__

}  // namespace svo
