// svo_batch.cu -- batched multi-scene cast: one persistent launch over many
// (scene, ray batch) items.
//
// Work distribution: the claims of all items form one global index space
// (item prefix sums; an item spans 32 indices per claim of its ClaimOrder, so
// an item of camera rays with a row length is cast in 8 x 4 ray blocks).  Each
// warp repeatedly claims `rays_per_chunk` consecutive indices from a device
// work counter with one atomicAdd, maps every lane's index to its item by
// binary search over the prefix sums held in shared memory, and casts with the
// shared per-ray restatement of Octree::get_by_ray (svo_cast.cuh).  Items of
// different octree sizes and brick dimensions mix freely; a ray's result does
// not depend on which warp or launch casts it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "svo_cast.cuh"
#include "svo_flow.cuh"
#include "svo_queue.h"
#include "svo_trace.h"

namespace svo {

struct BatchItemDev {
  SceneView scene;
  RaysView rays;
  HitsView hits;
  ClaimOrder order;  // the item's rays by claim and lane
  uint64_t begin;    // first global index of the item (a multiple of 32)
  uint64_t n;
  const DevNode* stage_src;  // the first item of each staged scene: its top table, which blocks copy
  uint32_t stage_off;        // the scene's staged records in the block's copy: [stage_off, + stage_n)
  uint32_t stage_n;          // 0: the scene's nodes are read from L1/L2
};

constexpr uint32_t kBatchStageRecords = 768;  // 48 KB of staged records per block at most

// Shares the staged records out among the scenes of a call's items in claim order (the others' kernel stages nothing),
// in order of first appearance, at staging depth `depth` while they fit kBatchStageRecords; returns the
// records a block copies.
inline uint32_t assign_staging(BatchItemDev* table, const svo_batch_item* items, uint32_t n_items, uint32_t depth) {
  uint32_t total = 0;
  for (uint32_t i = 0; i < n_items; ++i) {
    table[i].stage_src = nullptr;
    table[i].stage_off = 0;
    table[i].stage_n = 0;
  }
  if (depth == 0) return 0;
  for (uint32_t i = 0; i < n_items; ++i) {
    if (table[i].n == 0) continue;
    uint32_t first = i;
    for (uint32_t j = 0; j < i; ++j)
      if (table[j].n != 0 && items[j].scene == items[i].scene) {
        first = j;
        break;
      }
    if (first < i) {  // a later item of a scene seen before: the same staged records
      table[i].stage_off = table[first].stage_off;
      table[i].stage_n = table[first].stage_n;
      continue;
    }
    const uint32_t n = table[i].scene.literal ? 0u : staged_records(items[i].scene, depth);
    if (n == 0 || total + n > kBatchStageRecords) continue;
    table[i].stage_src = table[i].scene.top;
    table[i].stage_off = total;
    table[i].stage_n = n;
    total += n;
  }
  return total;
}

// The staged records of every scene of the table into the block's shared-memory copy.
__device__ __forceinline__ void stage_items(DevNode* stg, const BatchItemDev* items, uint32_t n_items) {
  for (uint32_t i = 0; i < n_items; ++i) {
    const DevNode* src = items[i].stage_src;
    if (src) stage_records(stg + items[i].stage_off, src, items[i].stage_n);
  }
}

// fills the device form of one item at global index `begin`; returns the indices it spans
// (none when the item's rays are cast by batch_flow_kernel instead: `claimed` false)
uint64_t item_dev(const svo_batch_item& it, uint64_t begin, uint32_t shape, BatchItemDev& d, bool claimed = true) {
  d.scene = scene_view(it.scene);
  d.rays = RaysView{it.rays.ox, it.rays.oy, it.rays.oz, it.rays.dx, it.rays.dy, it.rays.dz};
  d.hits = hits_view_of(it.hits);
  d.n = claimed ? it.n : 0;
  d.order = claim_order(d.n, it.row_length, shape);
  d.begin = begin;
  return 32 * d.order.claims;
}

constexpr uint32_t kMaxSharedItems = 256;  // prefix sums staged in shared memory (the rest read from the table)

// At most kBatchMaxBlock threads per block with 7 resident blocks per SM (72 registers, a few
// spilled bytes); the launch configuration is checked against the block limit.
constexpr uint32_t kBatchMaxBlock = 128;

// Rays that miss their octree's root box get their miss written at once; the entering rays of a
// partly entering round of 32 indices wait in the warp's slice of shared memory (their index, item,
// the point where they enter and its octant) until `pack` of them (pack_target) are there; their origin and
// direction are read again when they are cast (less shared memory per block leaves more L1).
struct WaitingBatchRays {
  float p[3][64];
  uint32_t target[64];  // octant of the entry point; bit 31: fast form
  uint32_t item[64];
  unsigned long long i[64];
};

template <bool kCount, bool kStage = false>
__global__ void __launch_bounds__(kBatchMaxBlock, 7)
    batched_kernel(const BatchItemDev* __restrict__ items, uint32_t n_items, uint64_t total,
                   unsigned long long* __restrict__ counter, uint32_t chunk, uint32_t pack) {
  __shared__ uint64_t s_begin[kMaxSharedItems];
  __shared__ WaitingBatchRays waiting[kBatchMaxBlock / 32];
  extern __shared__ uint4 staged_smem[];
  DevNode* stg = reinterpret_cast<DevNode*>(staged_smem);
  const uint32_t staged = n_items < kMaxSharedItems ? n_items : kMaxSharedItems;
  for (uint32_t i = threadIdx.x; i < staged; i += blockDim.x) s_begin[i] = items[i].begin;
  const SharedLuts* luts = &kLuts;  // read by the literal form and, staged, by the fast form
  if constexpr (kStage) {
    __shared__ SharedLuts L;
    fill_shared_luts(L);
    stage_items(stg, items, n_items);
    luts = &L;
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31u;
  WaitingBatchRays& w = waiting[threadIdx.x >> 5];
  uint32_t count = 0;                 // rays waiting (the same in every lane)
  bool more = true;                   // chunks left
  unsigned long long base = 0;        // the warp's chunk
  uint32_t next = chunk;              // offset of the next round of 32 indices in it
  for (;;) {
    bool have = false, fast = false, waited = false;
    uint64_t i = 0;
    uint32_t item = 0, target = 0;
    float ox = 0.0f, oy = 0.0f, oz = 0.0f, dx = 0.0f, dy = 0.0f, dz = 0.0f, px = 0.0f, py = 0.0f, pz = 0.0f;
    while (count < pack) {
      if (next >= chunk) {
        if (!more) break;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)chunk);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= total) {
          more = false;
          break;
        }
        next = 0;
      }
      const uint64_t g = base + next + lane;
      const bool in_chunk = next + lane < chunk;
      next += 32;
      bool enters = false;
      if (in_chunk && g < total) {
        // largest item with begin <= g (items are sorted by begin)
        uint32_t lo = 0, hi = n_items - 1;
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          const uint64_t b = mid < kMaxSharedItems ? s_begin[mid] : items[mid].begin;
          if (b <= g)
            lo = mid;
          else
            hi = mid - 1;
        }
        const BatchItemDev& it = items[lo];
        const uint64_t x = g - it.begin;  // an empty item shares its begin with the next one
        const uint64_t j =
            x < 32 * it.order.claims ? claimed_ray(it.order, x >> 5, (uint32_t)(x & 31u), it.n) : it.n;
        if (j < it.n) {
          const RaysView& r = it.rays;
          ox = __ldg(r.ox + j);
          oy = __ldg(r.oy + j);
          oz = __ldg(r.oz + j);
          dx = __ldg(r.dx + j);
          dy = __ldg(r.dy + j);
          dz = __ldg(r.dz + j);
          fast = !it.scene.literal && !isnan(dx) && !isnan(dy) && !isnan(dz);
          enters = !fast || fast_entry(it.scene, ox, oy, oz, dx, dy, dz, px, py, pz, target);
          if (!enters) {
            HitRecord h;
            miss_record(h);
            write_hit(it.scene, it.hits, j, h);
            if (kCount) write_counters(it.hits, j, h);
          }
          i = j;
          item = lo;
        }
      }
      const unsigned m = __ballot_sync(0xFFFFFFFFu, enters);
      if (m == 0xFFFFFFFFu && count == 0) {  // a full round: cast in place
        have = true;
        break;
      }
      if (enters) {
        const uint32_t k = count + __popc(m & ((1u << lane) - 1u));
        w.p[0][k] = px;
        w.p[1][k] = py;
        w.p[2][k] = pz;
        w.target[k] = target | (fast ? 0x80000000u : 0u);
        w.item[k] = item;
        w.i[k] = i;
      }
      count += __popc(m);
      __syncwarp();
    }
    if (!have) {
      if (count == 0) break;  // no chunks left and nothing waiting
      const uint32_t take = count < 32 ? count : 32;
      if (lane < take) {
        const uint32_t k = count - take + lane;
        px = w.p[0][k];
        py = w.p[1][k];
        pz = w.p[2][k];
        target = w.target[k] & 0x7FFFFFFFu;
        fast = (w.target[k] >> 31) != 0u;
        item = w.item[k];
        i = w.i[k];
        have = true;
        waited = true;
      }
      count -= take;
      __syncwarp();
    }
    if (!have) continue;
    const BatchItemDev& it = items[item];
    if (waited) {  // origin and direction again from the item's arrays
      const RaysView& r = it.rays;
      ox = __ldg(r.ox + i);
      oy = __ldg(r.oy + i);
      oz = __ldg(r.oz + i);
      dx = __ldg(r.dx + i);
      dy = __ldg(r.dy + i);
      dz = __ldg(r.dz + i);
    }
    HitRecord h;
    cast_entered<kCount, false, kStage>(it.scene, *luts, ox, oy, oz, dx, dy, dz, fast, px, py, pz, target, h, 0.0f,
                                        stg + it.stage_off, it.stage_n);
    write_hit(it.scene, it.hits, i, h);
    if (kCount) write_counters(it.hits, i, h);
  }
}

// ---- rays in no order (svo_launch_config.sort_key = 1) ------------------------------------------
//
// The items without a row length are cast by flow_cast (svo_flow.cuh), 32 consecutive rays of an item per
// claim.  It keeps a warp's lanes busy with rays that have nothing in common, so putting like rays into one
// warp first does not pay: binning, scanning and scattering 2^20 rays took 60 us, and the cast of the sorted
// rays 300; in index order flow_cast takes 260 in all (GB300, 512^3, 17% entering; 20,000 rays 90 us, 198 sorted).
struct LooseItemDev {
  uint64_t begin;  // the item's first claim
  uint64_t n;      // its rays (0: the item is cast in claim order)
};

struct BatchRayId {
  unsigned long long i;
  uint32_t item;
};
struct BatchSource {
  const BatchItemDev* items;
  const LooseItemDev* loose;
  uint32_t n_items;
  __device__ __forceinline__ bool claimed(uint64_t c, uint32_t lane, BatchRayId& id) const {
    uint32_t lo = 0, hi = n_items - 1;  // the item: largest with begin <= c; an empty one shares its begin with the next
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (loose[mid].begin <= c)
        lo = mid;
      else
        hi = mid - 1;
    }
    id.item = lo;
    id.i = (c - loose[lo].begin) * 32u + lane;
    return id.i < loose[lo].n;
  }
  __device__ __forceinline__ void ray(const BatchRayId& id, float (&o)[3], float (&d)[3]) const {
    const RaysView& r = items[id.item].rays;
    o[0] = __ldg(r.ox + id.i);
    o[1] = __ldg(r.oy + id.i);
    o[2] = __ldg(r.oz + id.i);
    d[0] = __ldg(r.dx + id.i);
    d[1] = __ldg(r.dy + id.i);
    d[2] = __ldg(r.dz + id.i);
  }
  __device__ __forceinline__ const SceneView& scene(const BatchRayId& id) const { return items[id.item].scene; }
  __device__ __forceinline__ void put(const BatchRayId& id, HitRecord& h) const {
    const BatchItemDev& it = items[id.item];
    write_hit(it.scene, it.hits, id.i, h);
  }
};

__global__ void __launch_bounds__(128, 6)
    batch_flow_kernel(const __grid_constant__ BatchSource src, uint64_t claims, uint32_t refill,
                      unsigned long long* __restrict__ queue) {
  __shared__ FlowShared sh;
  __shared__ FlowLists<BatchRayId> lists[4];
  queue_begin(queue);
  flow_batch(src, claims, refill, queue, sh, lists[threadIdx.x >> 5]);
}

}  // namespace svo

namespace svo {
// Rays per claim where the caller gives none: 64, which halves the claims, but 32 while a warp of a full GPU (28 per SM)
// would get fewer than 8 claims of 64.  The launch ends when its last claim does, and a claim of 64 is two casts
// one after the other: 24 items of 861 K rays take 354 us at 32, 443 at 64 and 620 at 128.
inline uint32_t default_chunk(uint64_t total, int sm_count) { return total < (uint64_t)sm_count * 28u * 8u * 64u ? 32u : 64u; }

// The claim-order persistent launch of a prepared item table (device copy at d_items), with
// staged_n records of the call's top tables staged by every block.
svo_status launch_claimed(const BatchItemDev* d_items, uint32_t n_items, uint64_t total,
                          unsigned long long* d_counter, uint32_t chunk, uint32_t block, const svo_launch_config* cfg,
                          bool count, uint32_t staged_n, int sm_count, cudaStream_t st) {
  const size_t smem = (size_t)staged_n * sizeof(DevNode);
  auto kern = staged_n ? (count ? batched_kernel<true, true> : batched_kernel<false, true>)
                       : (count ? batched_kernel<true> : batched_kernel<false>);
  SVO_CUDA_TRY(allow_dynamic_smem(kern, smem));
  int per_sm = (cfg && cfg->blocks_per_sm) ? (int)cfg->blocks_per_sm : 0;
  if (per_sm == 0) {
    SVO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, block, smem));
    per_sm = std::max(per_sm, 1);
  }
  const uint64_t warps_needed = (total + chunk - 1) / chunk;
  uint64_t grid = (uint64_t)sm_count * (uint64_t)per_sm;
  grid = std::min<uint64_t>(grid, (warps_needed * 32 + block - 1) / block);
  grid = std::max<uint64_t>(grid, 1);
  SVO_CUDA_TRY(cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st));
  kern<<<(unsigned)grid, block, smem, st>>>(d_items, n_items, total, d_counter, chunk,
                                            pack_target(total / 32, (uint64_t)sm_count * per_sm * (block / 32)));
  SVO_CUDA_TRY(cudaGetLastError());
  return SVO_OK;
}
}  // namespace svo

// Workspace of the batched cast: device item table + work counter, and a
// pinned host staging copy of the table.  Grows only when the item count grows.
struct svo_batch_workspace {
  svo::BatchItemDev* d_items = nullptr;
  unsigned long long* d_counter = nullptr;  // [0] claim-order work counter, from [2] on the words of the loose items' launches
  svo::QueueTurn turn;
  bool zeroed = false;  // the words have been zeroed, by the first launch that took one of the pair
  svo::BatchItemDev* h_items = nullptr;     // pinned
  svo::LooseItemDev* d_loose = nullptr;     // the items of batch_flow_kernel
  svo::LooseItemDev* h_loose = nullptr;     // pinned
  cudaEvent_t copied = nullptr;             // the last table upload has left h_items and h_loose
  uint32_t cap = 0;
  int sm_count = 0;
};

using namespace svo;

extern "C" {

svo_status svo_batch_workspace_create(svo_batch_workspace** out) {
  if (!out) return fail(SVO_ERR_ARGUMENT, "NULL argument");
  svo_batch_workspace* ws = new svo_batch_workspace();
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ws->sm_count, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaMalloc(&ws->d_counter, (2 + kQueueWords) * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ws->copied, cudaEventDisableTiming);
  if (e != cudaSuccess) {
    cudaFree(ws->d_counter);
    if (ws->copied) cudaEventDestroy(ws->copied);
    delete ws;
    return fail(SVO_ERR_CUDA, std::string("svo_batch_workspace_create: ") + cudaGetErrorString(e));
  }
  *out = ws;
  return SVO_OK;
}

void svo_batch_workspace_destroy(svo_batch_workspace* ws) {
  if (!ws) return;
  cudaFree(ws->d_items);
  cudaFree(ws->d_counter);
  cudaFreeHost(ws->h_items);
  cudaFree(ws->d_loose);
  cudaFreeHost(ws->h_loose);
  if (ws->copied) cudaEventDestroy(ws->copied);
  delete ws;
}

svo_status svo_cast_batched(svo_batch_workspace* ws, const svo_batch_item* items, uint32_t n_items,
                            const svo_launch_config* cfg, void* stream) {
  TraceRange range("svo_cast_batched");
  if (!ws || (!items && n_items)) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: NULL argument");
  if (n_items == 0) return SVO_OK;
  cudaStream_t st = (cudaStream_t)stream;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  SVO_CUDA_TRY(cudaStreamIsCapturing(st, &capturing));
  const bool in_capture = capturing != cudaStreamCaptureStatusNone;
  if (n_items > ws->cap) {
    if (in_capture) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: workspace must be sized before stream capture");
    // the previous table may still be read by an in-flight launch on this stream
    SVO_CUDA_TRY(cudaStreamSynchronize(st));
    cudaFree(ws->d_items);
    cudaFreeHost(ws->h_items);
    cudaFree(ws->d_loose);
    cudaFreeHost(ws->h_loose);
    ws->d_items = nullptr;
    ws->h_items = nullptr;
    ws->d_loose = nullptr;
    ws->h_loose = nullptr;
    ws->cap = 0;
    const uint32_t cap = std::max<uint32_t>(n_items, 16);
    SVO_CUDA_TRY(cudaMalloc(&ws->d_items, cap * sizeof(BatchItemDev)));
    SVO_CUDA_TRY(cudaMallocHost(&ws->h_items, cap * sizeof(BatchItemDev)));
    SVO_CUDA_TRY(cudaMalloc(&ws->d_loose, cap * sizeof(LooseItemDev)));
    SVO_CUDA_TRY(cudaMallocHost(&ws->h_loose, cap * sizeof(LooseItemDev)));
    ws->cap = cap;
  } else if (!in_capture) {
    // the pinned staging tables are reused: wait until their previous upload has left them
    SVO_CUDA_TRY(cudaEventSynchronize(ws->copied));
  }
  const uint32_t shape = (cfg && cfg->block_shape) ? cfg->block_shape : 3;
  if (shape < 3 || shape > 5) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: block_shape must be 0, 3, 4 or 5");
  const uint32_t sort_key = cfg ? cfg->sort_key : 0;
  if (sort_key > 1) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: sort_key must be 0 or 1");
  const uint32_t depth = cfg ? cfg->staging_depth : 0;
  if (depth > kMaxStageDepth)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: staging_depth must be 0.." + std::to_string(kMaxStageDepth));
  const uint32_t refill = cfg ? cfg->refill_below : 0;
  if (refill > 32) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: refill_below must be 0..32");
  uint64_t total = 0, loose_rays = 0, loose_claims = 0;
  uint32_t n_loose = 0, one = 0;
  bool count = false;
  for (uint32_t i = 0; i < n_items; ++i) {
    const svo_batch_item& it = items[i];
    if (!it.scene) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: NULL scene");
    if (!it.scene->dev.valid) return fail(SVO_ERR_NOT_UPLOADED, "svo_cast_batched: scene not uploaded");
    if (it.n && (!it.rays.ox || !it.rays.oy || !it.rays.oz || !it.rays.dx || !it.rays.dy || !it.rays.dz))
      return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: NULL ray array");
    count |= counts_requested(it.hits);
  }
  // the instrumented cast counts in claim order, whatever the key
  for (uint32_t i = 0; i < n_items; ++i) {
    const svo_batch_item& it = items[i];
    const bool unordered = sort_key == 1 && it.row_length == 0 && it.n > 0;
    if (unordered) loose_rays += it.n;
    const bool loose = unordered && !count;
    total += item_dev(it, total, shape, ws->h_items[i], !loose);
    ws->h_loose[i].begin = loose_claims;
    ws->h_loose[i].n = loose ? it.n : 0;
    if (loose) {
      loose_claims += (it.n + 31) / 32;
      ++n_loose;
      one = i;
    }
  }
  if (total == 0 && n_loose == 0) return SVO_OK;
  if (loose_rays >= (1ull << 32))
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: sort_key 1 takes fewer than 2^32 rays per call");
  const uint32_t staged_n = assign_staging(ws->h_items, items, n_items, depth);
  const uint32_t block = (cfg && cfg->block) ? cfg->block : 128;
  const uint32_t chunk = (cfg && cfg->rays_per_chunk) ? cfg->rays_per_chunk : default_chunk(total, ws->sm_count);
  if (block % 32 != 0 || block > kBatchMaxBlock || chunk == 0)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched: block must be a multiple of 32 and at most 128");
  // the tables are read by the claim-order kernel and by batch_flow_kernel; a lone loose item needs neither
  if (total > 0 || n_loose > 1)
    SVO_CUDA_TRY(cudaMemcpyAsync(ws->d_items, ws->h_items, n_items * sizeof(BatchItemDev), cudaMemcpyHostToDevice, st));
  if (n_loose > 1)
    SVO_CUDA_TRY(cudaMemcpyAsync(ws->d_loose, ws->h_loose, n_items * sizeof(LooseItemDev), cudaMemcpyHostToDevice, st));
  if (!in_capture) SVO_CUDA_TRY(cudaEventRecord(ws->copied, st));
  if (n_loose) {
    const uint32_t below = refill ? 33u - refill : kFlowRefill;
    QueueLaunch take;
    SVO_CUDA_TRY(queue_take({ws->d_counter + 2, &ws->turn}, st, take));
    if (!take.captured && !ws->zeroed) {
      SVO_CUDA_TRY(cudaMemsetAsync(ws->d_counter + 2, 0, 2 * sizeof(unsigned long long), st));
      ws->zeroed = true;
    }
    const uint32_t per_sm = cfg ? cfg->blocks_per_sm : 0;
    if (n_loose == 1) {
      const BatchItemDev& d = ws->h_items[one];
      const svo_status rc = launch_plain(d.scene, d.rays, d.hits, items[one].n, below, per_sm, take.word, st);
      if (rc != SVO_OK) return rc;
    } else {
      int per = (int)per_sm;
      if (per == 0) {
        SVO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, batch_flow_kernel, 128, 0));
        per = std::max(per, 1);
      }
      const uint64_t grid = std::min<uint64_t>((uint64_t)ws->sm_count * (uint64_t)per, (loose_claims + 3) / 4);
      batch_flow_kernel<<<(unsigned)grid, 128, 0, st>>>(BatchSource{ws->d_items, ws->d_loose, n_items}, loose_claims, below,
                                                        take.word);
      SVO_CUDA_TRY(cudaGetLastError());
    }
    take.launched();
  }
  if (total == 0) return SVO_OK;
  return launch_claimed(ws->d_items, n_items, total, ws->d_counter, chunk, block, cfg, count, staged_n, ws->sm_count, st);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free batched cast.
//
// Some callers of this library cannot allocate device memory at the moment they
// cast: an engine that hands the library a fixed memory budget and forbids
// allocation after start-up, or code running inside a frame loop or a graph of
// its own where a cudaMalloc would synchronise the device.  For them the item
// table and the work counter of the batched cast live in the fixed scratch
// array below instead of an svo_batch_workspace.  The array is reserved on
// every GPU that loads the library, for as long as the process lives.
constexpr uint32_t kNoAllocMaxItems = 128;  // items per call
constexpr size_t kNoAllocTableBytes = kNoAllocMaxItems * sizeof(svo::BatchItemDev);
constexpr size_t kNoAllocCounterOffset = (kNoAllocTableBytes + 255) / 256 * 256;
constexpr size_t kNoAllocBytes = kNoAllocCounterOffset + 256;
static_assert(kNoAllocBytes == 50432, "include/svo.h documents the scratch array's size");
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace {
constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};
int g_noalloc_sms[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device, looked up once per device.
svo_status noalloc_scratch(void** out, int* sms) {
  int dev = 0;
  SVO_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: device ordinal too large");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* ptr = nullptr;
    SVO_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
    int n = 0;
    SVO_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    g_noalloc_ptr[dev] = ptr;
    g_noalloc_sms[dev] = n;
  }
  *out = g_noalloc_ptr[dev];
  *sms = g_noalloc_sms[dev];
  return SVO_OK;
}
}  // namespace

extern "C" {

svo_status svo_cast_batched_noalloc(const svo_batch_item* items, uint32_t n_items, const svo_launch_config* cfg,
                                    void* stream) {
  TraceRange range("svo_cast_batched_noalloc");
  if (!items && n_items) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: NULL items");
  if (n_items > kNoAllocMaxItems)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: " + std::to_string(n_items) + " items exceed the maximum of " +
                                      std::to_string(kNoAllocMaxItems) + " per call");
  if (n_items == 0) return SVO_OK;
  cudaStream_t st = (cudaStream_t)stream;
  // The item table below is copied from this call's stack frame.  Inside a stream capture the copy
  // would become a graph node that reads that frame again at every replay, long after it is gone, so
  // a capturing stream is refused before anything is enqueued.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  SVO_CUDA_TRY(cudaStreamIsCapturing(st, &capture));
  if (capture != cudaStreamCaptureStatusNone)
    return fail(SVO_ERR_ARGUMENT,
                "svo_cast_batched_noalloc: the stream is capturing; its item table is copied from the caller's "
                "stack and cannot be replayed (capture svo_cast_batched with a workspace instead)");
  void* scratch = nullptr;
  int sms = 0;
  svo_status rc = noalloc_scratch(&scratch, &sms);
  if (rc != SVO_OK) return rc;
  BatchItemDev table[kNoAllocMaxItems];
  const uint32_t shape = (cfg && cfg->block_shape) ? cfg->block_shape : 3;
  if (shape < 3 || shape > 5)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: block_shape must be 0, 3, 4 or 5");
  if (cfg && cfg->sort_key)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: sort_key 1 needs a batch workspace");
  uint64_t total = 0;
  bool count = false;
  for (uint32_t i = 0; i < n_items; ++i) {
    const svo_batch_item& it = items[i];
    if (!it.scene) return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: NULL scene");
    if (!it.scene->dev.valid) return fail(SVO_ERR_NOT_UPLOADED, "svo_cast_batched_noalloc: scene not uploaded");
    if (it.n && (!it.rays.ox || !it.rays.oy || !it.rays.oz || !it.rays.dx || !it.rays.dy || !it.rays.dz))
      return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: NULL ray array");
    total += item_dev(it, total, shape, table[i]);
    count |= counts_requested(it.hits);
  }
  if (total == 0) return SVO_OK;
  const uint32_t block = (cfg && cfg->block) ? cfg->block : 128;
  const uint32_t chunk = (cfg && cfg->rays_per_chunk) ? cfg->rays_per_chunk : default_chunk(total, sms);
  if (block % 32 != 0 || block > kBatchMaxBlock || chunk == 0)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: block must be a multiple of 32 and at most 128");
  const uint32_t depth = cfg ? cfg->staging_depth : 0;
  if (depth > kMaxStageDepth)
    return fail(SVO_ERR_ARGUMENT, "svo_cast_batched_noalloc: staging_depth must be 0.." + std::to_string(kMaxStageDepth));
  const uint32_t staged_n = assign_staging(table, items, n_items, depth);
  BatchItemDev* d_items = static_cast<BatchItemDev*>(scratch);
  unsigned long long* d_counter =
      reinterpret_cast<unsigned long long*>(static_cast<unsigned char*>(scratch) + kNoAllocCounterOffset);
  // the table is copied from this stack frame: a pageable source is staged before cudaMemcpyAsync returns;
  // the counter keeps the previous call's final value and is reset for this launch by launch_claimed
  SVO_CUDA_TRY(cudaMemcpyAsync(d_items, table, n_items * sizeof(BatchItemDev), cudaMemcpyHostToDevice, st));
  return launch_claimed(d_items, n_items, total, d_counter, chunk, block, cfg, count, staged_n, sms, st);
}

}  // extern "C"
