// assign_staging (shocovox_gb300/csrc/svo_batch.cu) on the host, for tests/test_staging_host.py.
#include "../shocovox_gb300/csrc/svo_batch.cu"

// Items i of scene scene[i] with n[i] rays in claim order; each scene's staged records at any depth: records[scene].
// out: per item the offset, the records and whether a block copies them for it.  Returns the records a block copies.
extern "C" uint32_t stage_check(uint32_t n_items, const uint32_t* scene, const uint64_t* n, uint32_t n_scenes,
                                const uint32_t* records, uint32_t* out) {
  static DevNode top;
  std::vector<svo_scene*> scenes;
  for (uint32_t k = 0; k < n_scenes; ++k) {
    svo_scene* sc = nullptr;
    if (svo_scene_create(64, 4, &sc) != SVO_OK) return ~0u;
    sc->dev.top = &top;
    for (auto& c : sc->dev.top_count) c = records[k];
    scenes.push_back(sc);
  }
  std::vector<svo_batch_item> items(n_items);
  std::vector<BatchItemDev> table(n_items);
  for (uint32_t i = 0; i < n_items; ++i) {
    items[i] = svo_batch_item{};
    items[i].scene = scenes[scene[i]];
    table[i] = BatchItemDev{};
    table[i].n = n[i];
    table[i].scene.top = &top;
  }
  const uint32_t total = assign_staging(table.data(), items.data(), n_items, 2);
  for (uint32_t i = 0; i < n_items; ++i) {
    out[3 * i] = table[i].stage_off;
    out[3 * i + 1] = table[i].stage_n;
    out[3 * i + 2] = table[i].stage_src != nullptr;
  }
  for (svo_scene* sc : scenes) sc->dev.top = nullptr;  // not device memory; the scenes stay
  return total;
}
