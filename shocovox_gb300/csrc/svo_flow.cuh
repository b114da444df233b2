// svo_flow.cuh -- many rays per warp through the unit-direction form, one step of each at a time.
//
// Rays in no order walk paths of very different lengths and are never at the same kind of step: a warp that
// casts 32 of them to their ends, each kind of step in a loop of its own, runs 4 of 32 lanes (2^22 random rays on
// 512^3: 905 M warp instructions, 1,015 us, bound by instruction issue).  Here a lane's ray is a small state
// (Flow) that advances by a visit, a step or both per turn of one loop, and lanes whose rays have ended take new
// ones: 10 of 32 lanes, 526 M warp instructions, 635 us.  The state is what bounds the form: little of it may
// spill, so what is read rarely lives in shared memory, and what is a function of the rest (the node's
// 1 / size, the direction's signs as masks) is formed again.  It fits 72 registers (7 blocks per SM) in a
// kernel of its own, 80 (6) beside queue_cast or with its scenes in a table.
#pragma once

#include "svo_unit.cuh"

namespace svo {

// What a lane's ray does next.
enum : uint32_t {
  kIdle = 0,     // the lane has no ray
  kHit = 1,      // ended on a voxel or a Solid brick: X holds its centre, slot its brick or value
  kEnded = 2,    // the node stack is empty: a restart, or a miss
  kPanic = 3,    // the reference panics
  kGeneral = 4,  // the general forms have to cast it
  kVisit = 8,    // running: a node visit ...
  kVisited = 9,  // ... whose brick has been probed
  kStep = 10,    // ... an ADVANCE step
  kPop = 11,     // ... a POP
  kBrick = 12,   // ... a voxel of a brick
};

// Cells and voxels are packed x | z << 10 | y << 20, mirrored, so that a step adds 1 to the moved fields
// and has left its parent once a field reaches the parent's extent (2 cells, or D voxels).
constexpr uint32_t kX = 1u, kZ = 1u << 10, kY = 1u << 20, kXYZ = kX | kY | kZ;

struct Flow {
  UnitRay r;
  float cx, cy, cz, hs;  // the node: centre, half size
  float Xx, Xy, Xz, cs;  // the cell, a target cell of the node or a voxel: the planes it is left by, size
  uint32_t mode, at;     // what comes next; the cell's place in the node or brick
  uint32_t cur, fm;      // node; all bits of the fields whose axes are mirrored
  uint32_t misc;         // [2:0] mirrored axes as an octant, [4:3] depth mod 4, [7:5] entries of the node stack, [31:8] visits
  uint32_t info, slot;   // the head's info; child key, brick slot or Solid value under the target
  uint32_t w0, w1, w2;   // node: reach bits, ADVANCE's first target; brick: voxel, the target cell, occupancy word
};
struct FlowShared {      // one entry per thread and array: no bank conflicts
  uint2 ring[4][128];    // the node stack: keys of the ancestors and the target cells in them
  float from[3][128];    // where an ADVANCE began
};
SVO_UHD uint32_t trunc_u32(float v) { return v > 0.0f ? (uint32_t)v : 0u; }  // `as usize` of a value below 2^32
constexpr uint32_t kDepthOne = 1u << 3, kDepthMask = 3u << 3, kCountOne = 1u << 5, kCountMask = 7u << 5, kVisitOne = 1u << 8;

SVO_UHD uint32_t pack_octant(uint32_t o) { return (o & 1u) | ((o & 2u) << 9) | ((o & 4u) << 18); }
SVO_UHD uint32_t octant_at(uint32_t at) { return ((at | (at >> 9)) | (at >> 18)) & 7u; }
// 4 / size of the node: a power of two, by its exponent
SVO_UHD float flow_q4(const Flow& f) { return f32_from(0x7F800000u - f32_bits(f.hs)); }

SVO_UHD void flow_head(Flow& f, const SceneView& s) {
  const uint4 hd = SVO_LD(s.heads + (((f.misc & 7u) ^ 7u) * s.head_stride + f.cur));
  f.w0 = hd.x;
  f.w1 = hd.y;
  f.info = hd.z;
}
SVO_UHD void flow_slot(Flow& f, const SceneView& s) {
  f.slot = SVO_LD(s.nodes[f.cur].slot + (octant_at(f.at) ^ (f.misc & 7u)));
}
// the planes the target cell is left by
SVO_UHD void flow_planes(Flow& f) {
  f.Xx = (f.at & kX) ? fma_near(f.r.gx, f.hs, f.cx) : f.cx;
  f.Xy = (f.at & kY) ? fma_near(f.r.gy, f.hs, f.cy) : f.cy;
  f.Xz = (f.at & kZ) ? fma_near(f.r.gz, f.hs, f.cz) : f.cz;
  f.cs = f.hs;
}
SVO_UHD void flow_root(Flow& f, const SceneView& s, uint32_t octant) {
  f.at = pack_octant(octant ^ (f.misc & 7u));
  f.cur = 0;
  f.misc = (f.misc & ~(kCountMask | kDepthMask)) | kCountOne;
  f.hs = s.size * 0.5f;
  f.cx = f.cy = f.cz = f.hs;
  flow_planes(f);
  f.mode = kVisit;
}

SVO_UHD void flow_start(Flow& f, const SceneView& s, float dx, float dy, float dz, float px, float py,
                                           float pz, uint32_t target) {
  UnitRay& r = f.r;
  r.dx = dx;
  r.dy = dy;
  r.dz = dz;
  r.gx = copysignf(1.0f, dx);
  r.gy = copysignf(1.0f, dy);
  r.gz = copysignf(1.0f, dz);
  r.px = px;
  r.py = py;
  r.pz = pz;
  const float a = dz / dx, b = dy / dx, c = dx / dy, d = dz / dy, e = dx / dz, g = dy / dz;
  r.fx = sqrtf((1.0f + a * a) + b * b);
  r.fy = sqrtf((c * c + 1.0f) + d * d);
  r.fz = sqrtf((e * e + 1.0f) + g * g);
  f.misc = (signbit(dx) ? 1u : 0u) | (signbit(dz) ? 2u : 0u) | (signbit(dy) ? 4u : 0u);
  f.fm = (signbit(dx) ? 1023u * kX : 0u) | (signbit(dz) ? 1023u * kZ : 0u) | (signbit(dy) ? 1023u * kY : 0u);
  flow_root(f, s, target);
  flow_head(f, s);
  flow_slot(f, s);
}

// The reach bit of the packed mirrored cell c: bit x + 4 y + 16 z of the 64.
SVO_UHD bool flow_reach(uint32_t c, uint32_t lo, uint32_t hi) {
  const uint32_t k = (c & 3u) | ((c >> 18) & 12u);
  return (((c & (2u * kZ)) ? hi : lo) >> (k + ((c & kZ) ? 16u : 0u))) & 1u;
}

// A ray whose node stack is empty: the 0.1 nudge, then a restart (kVisit) or the end (kEnded stays: a miss).
SVO_UHD void flow_restart(Flow& f, const SceneView& s) {
  UnitRay& r = f.r;
  const float nx = r.dx * 0.1f, ny = r.dy * 0.1f, nz = r.dz * 0.1f;
  const float S = s.size;
  r.px = r.px + nx;
  r.py = r.py + ny;
  r.pz = r.pz + nz;
  if (!(r.px < S && r.py < S && r.pz < S && r.px > 0.0f && r.py > 0.0f && r.pz > 0.0f)) return;
  f.cur = 0;
  flow_head(f, s);
  const uint32_t rk = (f.info >> 16) & 3u;
  if (rk == kKindInternal || rk == kKindNothing) {
    const float q4 = s.inv_size * 4.0f;
    const int ix = min_relu(unit_bits(fma_down(r.px, q4, 0x1p23f)), 3);
    const int iy = min_relu(unit_bits(fma_down(r.py, q4, 0x1p23f)), 3);
    const int iz = min_relu(unit_bits(fma_down(r.pz, q4, 0x1p23f)), 3);
    if (!flow_reach((uint32_t)(ix + (iz << 10) + (iy << 20)) ^ (f.fm & (3u * kXYZ)), f.w0, f.w1)) {
      const float cmax = fmaxf(fmaxf(fabsf(nx), fabsf(ny)), fabsf(nz));
      const float done = (float)(f.misc / kVisitOne + 1u) * (float)work_per_visit(s.dim);
      if (!(cmax >= S * 0x1p-22f && done + S / (0.5f * cmax) + 2.0f < (float)kWorkCap)) f.mode = kGeneral;
      return;
    }
  }
  flow_root(f, s, octant_of(r.px, r.py, r.pz, S * 0.5f));
  flow_slot(f, s);
}

// The visit of a running lane's node.
SVO_UHD void flow_visit(Flow& f, const SceneView& s, FlowShared& sh, uint32_t tid) {
  UnitRay& r = f.r;
  const uint32_t o = octant_at(f.at);
  const bool leafy = (f.info >> 17) & 1u;  // a Leaf or UniformLeaf
  const bool live = (f.info >> o) & 1u;
  const float q4 = flow_q4(f);
  f.misc += kVisitOne;
  if (live && leafy && f.mode == kVisit) {
    // the brick over the UniformLeaf's cube, or over the Leaf's target cell
    const bool uni = (f.info >> 16) & 1u, solid = (f.info >> (8u + o)) & 1u;
    if (uni) f.slot = SVO_LD(s.nodes[f.cur].slot);
    f.w1 = f.at;
    f.mode = kBrick;
    const float q = uni ? f.hs : f.hs * 0.5f, k = (uni ? q4 * 0.25f : q4 * 0.5f) * (float)s.dim;
    const float bx = (uni ? f.cx : fma_near(-r.gx, q, f.Xx)) - q;
    const float by = (uni ? f.cy : fma_near(-r.gy, q, f.Xy)) - q;
    const float bz = (uni ? f.cz : fma_near(-r.gz, q, f.Xz)) - q;
    const float half = q * s.inv_dim, unit = half * 2.0f;
    const float top = 0x1p23f + (float)(s.dim - 1u);
    const float wx = fminf(fmaxf(fma_down(r.px, k, fma_near(-bx, k, 0x1p23f)), 0x1p23f), top);
    const float wy = fminf(fmaxf(fma_down(r.py, k, fma_near(-by, k, 0x1p23f)), 0x1p23f), top);
    const float wz = fminf(fmaxf(fma_down(r.pz, k, fma_near(-bz, k, 0x1p23f)), 0x1p23f), top);
    const uint32_t ix = (uint32_t)unit_bits(wx), iy = (uint32_t)unit_bits(wy), iz = (uint32_t)unit_bits(wz);
    const uint32_t L = s.dim_log;
    f.w0 = ix + (iy << L) + (iz << (2u * L));
    f.w2 = 0xFFFFFFFFu;
    if (solid)
      f.w0 = 0xFFFFFFFFu;  // a hit at once
    else
      f.w2 = SVO_LD(s.vbits + ((size_t)f.slot * s.vwords + (f.w0 >> 5)));
    f.at = (ix | (iz << 10) | (iy << 20)) ^ (f.fm & ((s.dim - 1u) * kXYZ));
    f.Xx = fma_near(r.gx, half, fma_near(wx - 0x1p23f, unit, bx + half));
    f.Xy = fma_near(r.gy, half, fma_near(wy - 0x1p23f, unit, by + half));
    f.Xz = fma_near(r.gz, half, fma_near(wz - 0x1p23f, unit, bz + half));
    f.cs = unit;
  } else {
    const int ix = min_relu(unit_bits(fma_down(r.px, q4, fma_near(-f.cx, q4, 0x1p23f + 2.0f))), 3);
    const int iy = min_relu(unit_bits(fma_down(r.py, q4, fma_near(-f.cy, q4, 0x1p23f + 2.0f))), 3);
    const int iz = min_relu(unit_bits(fma_down(r.pz, q4, fma_near(-f.cz, q4, 0x1p23f + 2.0f))), 3);
    const uint32_t cell = (uint32_t)(ix + (iz << 10) + (iy << 20)) ^ (f.fm & (3u * kXYZ));
    if (!flow_reach(cell, f.w0, f.w1)) {
      f.mode = kPop;
    } else if (live && !leafy) {
      // PUSH
      sh.ring[(f.misc >> 3) & 3u][tid] = make_uint2(f.cur, f.at);
      const float q = f.hs * 0.5f;
      f.cx = fma_near(-r.gx, q, f.Xx);
      f.cy = fma_near(-r.gy, q, f.Xy);
      f.cz = fma_near(-r.gz, q, f.Xz);
      const uint32_t upper = cell >> 1;
      f.at = (((upper ^ f.at) & upper) | (~(upper ^ f.at) & cell)) & kXYZ;
      f.Xx = (f.at & kX) ? f.Xx : f.cx;
      f.Xy = (f.at & kY) ? f.Xy : f.cy;
      f.Xz = (f.at & kZ) ? f.Xz : f.cz;
      const uint32_t deeper = (f.misc + kDepthOne) & kDepthMask;
      f.misc = ((f.misc & ~kDepthMask) | deeper) + ((f.misc & (4u * kCountOne)) ? 0u : kCountOne);
      f.cur = f.slot;
      f.hs = f.cs = q;
      flow_head(f, s);
      flow_slot(f, s);
      f.mode = kVisit;
    } else {
      // ADVANCE: where the point stands, for the reference's bitmap position
      f.mode = kStep;
      sh.from[0][tid] = r.px;
      sh.from[1][tid] = r.py;
      sh.from[2][tid] = r.pz;
      f.w2 = f.at | (((f.hs <= 1.0f ? ~0u : cell >> 1) & ~f.at & kXYZ) ? 0x80000000u : 0u);
    }
  }
}

// One step of a running lane's ray to the planes of its cell.
SVO_UHD void flow_step(Flow& f, const SceneView& s, FlowShared& sh, uint32_t tid) {
  UnitRay& r = f.r;
  if (f.mode == kPop) {
    f.misc -= kCountOne;
    if (!(f.misc & kCountMask)) {
      f.mode = kEnded;
      return;
    }
    f.misc = (f.misc & ~kDepthMask) | ((f.misc - kDepthOne) & kDepthMask);
    const uint2 up = sh.ring[(f.misc >> 3) & 3u][tid];
    f.cur = up.x;
    f.at = up.y;
    f.Xx = fma_near(r.gx, f.hs, f.cx);
    f.Xy = fma_near(r.gy, f.hs, f.cy);
    f.Xz = fma_near(r.gz, f.hs, f.cz);
    f.cx = (f.at & kX) ? fma_near(-r.gx, f.hs, f.cx) : f.Xx;
    f.cy = (f.at & kY) ? fma_near(-r.gy, f.hs, f.cy) : f.Xy;
    f.cz = (f.at & kZ) ? fma_near(-r.gz, f.hs, f.cz) : f.Xz;
    f.hs = f.cs = f.hs * 2.0f;
  }
  bool mx, my, mz;
  unit_step(r, f.Xx, f.Xy, f.Xz, mx, my, mz);
  if (mx) {
    f.Xx = fma_near(r.gx, f.cs, f.Xx);
    f.at += kX;
  }
  if (my) {
    f.Xy = fma_near(r.gy, f.cs, f.Xy);
    f.at += kY;
  }
  if (mz) {
    f.Xz = fma_near(r.gz, f.cs, f.Xz);
    f.at += kZ;
  }
  const bool out = f.at & ((f.mode == kBrick ? s.dim : 2u) * kXYZ);
  if (f.mode == kBrick) {
    if (out) {
      f.at = f.w1;
      flow_planes(f);
      flow_head(f, s);
      f.mode = kVisited;
    } else {
      const uint32_t v = f.at ^ (f.fm & ((s.dim - 1u) * kXYZ)), L = s.dim_log;
      f.w0 = (v & 1023u) + ((v >> 20) << L) + (((v >> 10) & 1023u) << (2u * L));
      f.w2 = SVO_LD(s.vbits + ((size_t)f.slot * s.vwords + (f.w0 >> 5)));
    }
  } else if (out) {
    f.misc += kVisitOne;
    f.mode = kPop;
  } else {
    bool visit = true;
    if (f.mode == kPop) {
      flow_head(f, s);
    } else {
      const bool live = (f.info >> octant_at(f.at)) & 1u, leafy = (f.info >> 17) & 1u, check = f.w2 >> 31;
      visit = live;
      if (check || (live && !leafy)) {
        const uint32_t m = f.at ^ f.w2;
        const float q4 = flow_q4(f);
        float ux = clamp_bitmap((sh.from[0][tid] - (f.cx - f.hs)) * q4),
              uy = clamp_bitmap((sh.from[1][tid] - (f.cy - f.hs)) * q4),
              uz = clamp_bitmap((sh.from[2][tid] - (f.cz - f.hs)) * q4);
        if (m & kX) ux = fma_near(r.gx, q4, ux);
        if (m & kY) uy = fma_near(r.gy, q4, uy);
        if (m & kZ) uz = fma_near(r.gz, q4, uz);
        if (!leafy)
          visit = live && flow_reach((trunc_u32(ux) + (trunc_u32(uz) << 10) + (trunc_u32(uy) << 20)) ^
                                         (f.fm & (3u * kXYZ)), f.w0, f.w1);
        if (ux >= 4.0f || uy >= 4.0f || uz >= 4.0f) {
          f.mode = kPanic;
          visit = false;
        }
      }
    }
    if (visit) {
      flow_slot(f, s);
      f.mode = kVisit;
    }
  }
}

// The record of a lane whose ray has ended.
SVO_UHD void flow_record(Flow& f, const SceneView& s, HitRecord& h) {
  miss_record(h);
  if (f.mode == kPanic) h.status = 3;
  if (f.mode != kHit) return;
  const UnitRay& r = f.r;
  const bool uni = (f.info >> 16) & 1u, solid = f.w0 == 0xFFFFFFFFu;
  h.status = 1;
  h.node = f.cur;
  h.octant = uni ? 0u : octant_at(f.w1) ^ (f.misc & 7u);
  h.voxel = f.w0;
  h.pix = solid ? f.slot : SVO_LD(s.voxels + (((size_t)f.slot << (3u * s.dim_log)) + f.w0));
  h.px = r.px;
  h.py = r.py;
  h.pz = r.pz;
  // the cube's centre: the node's, the target cell's or the voxel's
  if (solid) {
    f.at = f.w1;
    flow_planes(f);
  }
  const float half = f.cs * 0.5f;
  const bool node = solid && uni;
  unit_normal(r, node ? f.cx : fma_near(-r.gx, half, f.Xx), node ? f.cy : fma_near(-r.gy, half, f.Xy),
              node ? f.cz : fma_near(-r.gz, half, f.Xz), h);
}

// One warp's lists: unit-direction rays that have entered their root, with the point where they enter,
// and rays for the general forms.
template <class Id>
struct FlowLists {
  float p[3][64];
  Id id[64];
  Id other[96];  // fewer than 32 wait before a claim; it adds 32 at most, and so do the rays in flight
  Id lane[32];   // the lanes' rays
  uint8_t target[64];
};

// A batch's rays, by one warp among gridDim.x * 4.  Src names the rays:
//   bool claimed(c, lane, id)  the ray of `lane` in claim c
//   ray(id, o, d)              its origin and direction
//   scene(id)                  its scene
//   put(id, h)                 writes its record
// c is the warp's next claim, from the counter *queue like queue_cast's: whichever of the two a block runs, each
// claim is cast once; `count` and `others` rays wait in the lists, none of them at first.
// Returns once a warp of rays waits for the general forms, or nothing but some of those is left, with no ray in flight
// (so their registers are free): flow_batch casts them and calls again.
//
// Rays that miss the root box get their miss at once, the others wait in the warp's list.  Once
// kFlowRefill lanes (or `refill`) have no running ray, their records are written and the next listed rays
// taken: the long sequences at a ray's two ends run with many lanes, and rays of very different lengths
// keep the lanes busy.  Between two such points every running lane makes one visit, one step or both
// per turn of the loop, whatever its ray is at -- a POP, an ADVANCE and a voxel of a brick take the same
// step code -- so rays that have nothing in common still run most instructions together.
constexpr uint32_t kFlowRefill = 12;  // 8 to 16 measured alike

__device__ __forceinline__ unsigned long long flow_claim(unsigned long long* __restrict__ queue) {
  unsigned long long c = 0;
  if ((threadIdx.x & 31u) == 0u) c = atomicAdd(queue, 1ull);
  return __shfl_sync(0xFFFFFFFFu, c, 0);
}

template <class Src, class Id>
__device__ __forceinline__ void flow_cast(const Src& src, uint64_t claims, uint32_t refill,
                                              unsigned long long* __restrict__ queue, unsigned long long& c,
                                              uint32_t& count, uint32_t& others, FlowShared& sh, FlowLists<Id>& w) {
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  uint32_t tid = threadIdx.x;
  asm volatile("" : "+r"(tid));  // kept in a register: each use read the special register again (680 -> 665 us)
  w.lane[lane] = Id{};
  __syncwarp();
  Flow f{};  // every field set: nothing of a ray lives on from the last call
  for (;;) {
    // ---- hand out: restarts, records of ended rays, new rays for idle lanes
    if (f.mode != kIdle) {
      const SceneView& s = src.scene(w.lane[lane]);
      if (f.mode < kVisit && f.misc / kVisitOne > s.visit_limit) f.mode = kGeneral;
      if (f.mode == kEnded) flow_restart(f, s);
      if (f.mode < kVisit && f.mode != kGeneral) {
        HitRecord h;
        flow_record(f, s, h);
        src.put(w.lane[lane], h);
        f.mode = kIdle;
      }
    }
    __syncwarp();
    const unsigned g = __ballot_sync(0xFFFFFFFFu, f.mode == kGeneral);
    if (f.mode == kGeneral) {
      w.other[others + __popc(g & below)] = w.lane[lane];
      f.mode = kIdle;
    }
    others += __popc(g);
    const unsigned idle = __ballot_sync(0xFFFFFFFFu, f.mode == kIdle);
    const uint32_t need = __popc(idle);
    // claims until every idle lane can have a ray, or a warp of rays waits for the general forms: those are cast
    // when the rays in flight have ended
    while (c < claims && count < need && others < 32u) {
      bool unit = false, other = false;
      float p[3] = {};
      uint32_t target = 0;
      Id id{};
      if (src.claimed(c, lane, id)) {
        float o[3], d[3];
        src.ray(id, o, d);
        const SceneView& s = src.scene(id);
        const uint32_t form = ray_form(s, o[0], o[1], o[2], d[0], d[1], d[2]);
        if (form == kFormLiteral || fast_entry(s, o[0], o[1], o[2], d[0], d[1], d[2], p[0], p[1], p[2], target)) {
          unit = form == kFormUnit;
          other = !unit;
        } else {
          HitRecord h;
          miss_record(h);
          src.put(id, h);
        }
      }
      const unsigned mu = __ballot_sync(0xFFFFFFFFu, unit), mo = __ballot_sync(0xFFFFFFFFu, other);
      if (unit) {
        const uint32_t k = count + __popc(mu & below);
        w.p[0][k] = p[0];
        w.p[1][k] = p[1];
        w.p[2][k] = p[2];
        w.target[k] = (uint8_t)target;
        w.id[k] = id;
      }
      if (other) w.other[others + __popc(mo & below)] = id;
      count += __popc(mu);
      others += __popc(mo);
      c = flow_claim(queue);
    }
    __syncwarp();
    const uint32_t take = others >= 32u ? 0u : count < need ? count : need;
    if (f.mode == kIdle) {
      const uint32_t k = __popc(idle & below);
      if (k < take) {
        const uint32_t at = count - take + k;
        const Id id = w.id[at];
        w.lane[lane] = id;
        float o[3], d[3];
        src.ray(id, o, d);
        flow_start(f, src.scene(id), d[0], d[1], d[2], w.p[0][at], w.p[1][at], w.p[2][at], w.target[at]);
      }
    }
    count -= take;
    __syncwarp();
    const bool left = others < 32u && (count > 0 || c < claims);
    if (!left && !__any_sync(0xFFFFFFFFu, f.mode != kIdle)) return;
    // ---- run until `refill` lanes have no running ray (all lanes, once nothing is left to hand out)
    const uint32_t stop = left ? 32u - refill : 0u;
    while (__popc(__ballot_sync(0xFFFFFFFFu, f.mode >= kVisit)) > stop) {
      const SceneView& s = src.scene(w.lane[lane]);
      if ((f.mode & ~1u) == kVisit) flow_visit(f, s, sh, tid);
      __syncwarp();
      if (f.mode == kBrick && ((f.w2 >> (f.w0 & 31u)) & 1u)) f.mode = kHit;
      if (f.mode >= kStep) flow_step(f, s, sh, tid);
      __syncwarp();
    }
  }
}

// A batch's rays, all of them.  Rays for the general forms are cast a warp of them at a time (cast a claim's few at a time,
// as they came, 2^22 random rays on 512^3 of which a tenth are not of unit length took 1,626 us, all of them 1,598).
template <class Src, class Id>
__device__ __forceinline__ void flow_batch(const Src& src, uint64_t claims, uint32_t refill,
                                           unsigned long long* __restrict__ queue, FlowShared& sh, FlowLists<Id>& w) {
  const uint32_t lane = threadIdx.x & 31u;
  unsigned long long c = flow_claim(queue);
  uint32_t count = 0, others = 0;
  for (;;) {
    flow_cast(src, claims, refill, queue, c, count, others, sh, w);
    if (others == 0u) return;
    const uint32_t take = others < 32u ? others : 32u;
    others -= take;
    if (lane < take) {
      const Id id = w.other[others + lane];
      float o[3], d[3];
      src.ray(id, o, d);
      HitRecord h;
      cast_one<false>(src.scene(id), kLuts, o[0], o[1], o[2], d[0], d[1], d[2], h);
      src.put(id, h);
    }
    __syncwarp();
  }
}

// One scene's rays in arrays.
struct RayId {
  unsigned long long i;
};
struct ArraySource {
  SceneView s;
  RaysView rays;
  HitsView out;
  uint64_t n;
  ClaimOrder order;
  __device__ __forceinline__ bool claimed(uint64_t c, uint32_t lane, RayId& id) const {
    id.i = claimed_ray(order, c, lane, n);
    return id.i < n;
  }
  __device__ __forceinline__ void ray(const RayId& id, float (&o)[3], float (&d)[3]) const {
    o[0] = __ldg(rays.ox + id.i);
    o[1] = __ldg(rays.oy + id.i);
    o[2] = __ldg(rays.oz + id.i);
    d[0] = __ldg(rays.dx + id.i);
    d[1] = __ldg(rays.dy + id.i);
    d[2] = __ldg(rays.dz + id.i);
  }
  __device__ __forceinline__ const SceneView& scene(const RayId&) const { return s; }
  __device__ __forceinline__ void put(const RayId& id, HitRecord& h) const { write_hit(s, out, id.i, h); }
};

svo_status launch_plain(const SceneView& v, const RaysView& rays, const HitsView& hits, uint64_t n, uint32_t refill,
                        uint32_t blocks_per_sm, unsigned long long* queue, cudaStream_t st);

// The first rays of the 32 pairs that rays_mixed looks at, one in each 32nd of the batch.  Where in it is scattered: at
// equal distances the pairs of an image of 1920 x 1080 x 4 rays lay at 32 neighbouring columns, those at the row's end
// with one ray on the next row, and its cast took 3.49 ms instead of 3.13.  Pairs are 8 apart, so that
// few of them straddle a row's end from 64 columns on.
constexpr uint32_t kPairApart = 8;
SVO_UHD uint64_t pair_at(uint64_t n, uint32_t k) {
  uint32_t h = (k + 1u) * 0x9E3779B1u;
  h = (h ^ (h >> 15)) * 0x2C1B3C6Du;
  h ^= h >> 13;
  const uint64_t step = n <= kPairApart + 32u ? 0u : (n - kPairApart) / 32u;
  return step * k + ((step * (h >> 8)) >> 24);
}

// Whether neighbouring rays of a batch go their own ways: of 32 pairs of rays, spread over the batch,
// fewer than 24 head into one octant, within 25 degrees, from origins within an eighth of the octree; and half of them or
// more are of the unit form (2^22 random rays on 512^3, a quarter of them not of unit length: 885 us in flow_cast, 979 in
// queue_cast; 30%: 951, 975; 40%: 1,003, 961).  Every warp of a launch reads the same 12 x 32 values and comes to the same answer.
__device__ __forceinline__ bool rays_mixed(const RaysView& r, uint64_t n, const SceneView& s) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t a = pair_at(n, lane), b = n <= kPairApart ? n - 1u : a + kPairApart;
  const float ax = __ldg(r.dx + a), ay = __ldg(r.dy + a), az = __ldg(r.dz + a);
  const float bx = __ldg(r.dx + b), by = __ldg(r.dy + b), bz = __ldg(r.dz + b);
  const float ux = __ldg(r.ox + a), uy = __ldg(r.oy + a), uz = __ldg(r.oz + a);
  const float vx = __ldg(r.ox + b), vy = __ldg(r.oy + b), vz = __ldg(r.oz + b);
  const float near = s.size * 0.125f;
  const bool along = signbit(ax) == signbit(bx) && signbit(ay) == signbit(by) && signbit(az) == signbit(bz) &&
                     ax * bx + ay * by + az * bz > 0.9f && fabsf(ux - vx) < near && fabsf(uy - vy) < near &&
                     fabsf(uz - vz) < near;
  const bool unit = unit_eligible(s, ux, uy, uz, ax, ay, az) && unit_eligible(s, vx, vy, vz, bx, by, bz);
  return __popc(__ballot_sync(0xFFFFFFFFu, along)) < 24 && __popc(__ballot_sync(0xFFFFFFFFu, unit)) >= 16;
}

}  // namespace svo
