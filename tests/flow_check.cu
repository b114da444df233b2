// The unit-direction form (svo_flow.cuh) on the host: the functions that the kernels run, one ray at a time,
// over a scene's node records.  Built by test_flow_host.py into a shared library of its own.
#include "../shocovox_gb300/csrc/svo_device.cu"

namespace {
float nan_min(float a, float b) { return std::isnan(a) ? b : (std::isnan(b) ? a : (b < a ? b : a)); }
float nan_max(float a, float b) { return std::isnan(a) ? b : (std::isnan(b) ? a : (b > a ? b : a)); }

// Cube::intersect_ray on the root (src/spatial/raytracing/mod.rs:32-61)
bool enters(const SceneView& s, const float* o, const float* d, float* p, uint32_t& target) {
  float lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    const float a = (0.0f - o[k]) / d[k], b = ((0.0f + s.size) - o[k]) / d[k];
    lo[k] = nan_min(a, b);
    hi[k] = nan_max(a, b);
  }
  const float t0 = nan_max(nan_max(lo[0], lo[1]), lo[2]), t1 = nan_min(nan_min(hi[0], hi[1]), hi[2]);
  if (t1 < 0.0f || t0 > t1) return false;
  const float t = t0 < 0.0f ? 0.0f : t0;
  for (int k = 0; k < 3; ++k) p[k] = o[k] + d[k] * t;
  target = octant_of(p[0], p[1], p[2], s.size * 0.5f);
  return true;
}
}  // namespace

// n rays (origins o, directions d, 3 floats each).  form: 0 not eligible, 1 cast, 2 left to the general forms.
// rec: 12 words a ray: status, brick octant, node, voxel, pix, point, normal.
extern "C" void flow_check(svo_scene* sc, const float* o, const float* d, uint64_t n, uint8_t* form, uint32_t* rec) {
  HostOctree& t = sc->tree;
  const uint64_t nodes = t.nodes(), words = vwords_of(t);
  std::vector<DevNode> records(nodes);
  std::vector<uint32_t> bits(t.arena.slots() * words + 1);
  for (uint64_t k = 0; k < nodes; ++k) build_node(t, k, records[k]);
  for (uint32_t k = 0; k < t.arena.slots(); ++k) build_vbits(t, k, &bits[k * words]);
  std::vector<uint4> heads(nodes * kHeadPlanes);
  for (uint32_t p = 0; p < kHeadPlanes; ++p)
    for (uint64_t k = 0; k < nodes; ++k) heads[p * nodes + k] = node_head(records[k], p);
  sc->dev.node_cap = nodes;
  SceneView v = scene_view(sc);
  v.nodes = records.data();
  v.heads = heads.data();
  v.vbits = bits.data();
  v.voxels = t.arena.raw().data();
  static FlowShared sh;
  for (uint64_t i = 0; i < n; ++i, o += 3, d += 3, rec += 12) {
    for (int k = 0; k < 12; ++k) rec[k] = 0;
    form[i] = unit_eligible(v, o[0], o[1], o[2], d[0], d[1], d[2]) ? 1 : 0;
    float p[3];
    uint32_t target;
    if (!form[i] || !enters(v, o, d, p, target)) continue;
    Flow f{};
    flow_start(f, v, d[0], d[1], d[2], p[0], p[1], p[2], target);
    while (f.mode >= kVisit) {
      if ((f.mode & ~1u) == kVisit) flow_visit(f, v, sh, 0);
      if (f.mode == kBrick && ((f.w2 >> (f.w0 & 31u)) & 1u)) f.mode = kHit;
      if (f.mode >= kStep) flow_step(f, v, sh, 0);
      if (f.mode < kVisit && f.misc / kVisitOne > v.visit_limit) f.mode = kGeneral;
      if (f.mode == kEnded) flow_restart(f, v);
    }
    if (f.mode == kGeneral) {
      form[i] = 2;
      continue;
    }
    HitRecord h;
    flow_record(f, v, h);
    rec[0] = h.status;
    if (h.status != 1) continue;
    const uint32_t ids[4] = {h.octant, h.node, h.voxel, h.pix};
    const float fl[6] = {h.px, h.py, h.pz, h.nx, h.ny, h.nz};
    std::memcpy(rec + 1, ids, sizeof(ids));
    std::memcpy(rec + 5, fl, sizeof(fl));
  }
}

// The rays that tell a batch's order (rays_mixed): the first of pair k of n rays.
extern "C" uint64_t flow_pair(uint64_t n, uint32_t k) { return pair_at(n, k); }
extern "C" uint32_t flow_pair_apart() { return kPairApart; }
