// svo_route.h and svo_queue.h (shocovox_gb300/csrc) for tests/test_routes_host.py, through plain C functions.
#include "../shocovox_gb300/csrc/svo_queue.h"
#include "../shocovox_gb300/csrc/svo_route.h"

extern "C" {

int route_aligned(const svo_rays* rays, const svo_hits* hits) { return svo::arrays_aligned(*rays, *hits) ? 1 : 0; }

int route_overlap(const svo_rays* rays, const svo_hits* hits, uint64_t n) { return svo::hits_over_rays(*rays, *hits, n) ? 1 : 0; }

uint32_t route_spans(const uint64_t* runs, uint64_t n, uint64_t gap, uint64_t* out) {
  svo::Spans s;
  for (uint64_t k = 0; k < n; ++k) svo::add_span(s, runs[2 * k], runs[2 * k + 1], gap);
  for (size_t k = 0; k < s.size(); ++k) {
    out[2 * k] = s[k].first;
    out[2 * k + 1] = s[k].second;
  }
  return (uint32_t)s.size();
}

// a stream's claim words: the one its next launch takes, the one that launch zeroes, and the launch
uint32_t route_words() { return svo::kQueueWords; }
uint32_t route_word(uint32_t turn, int captured) { return svo::QueueTurn{turn}.word(captured != 0); }
uint32_t route_launched(uint32_t turn, int captured) {
  svo::QueueTurn t{turn};
  t.launched(captured != 0);
  return t.turn;
}
uint32_t route_zeroes(uint32_t word) {
  alignas(16) static unsigned long long words[svo::kQueueWords];
  return (uint32_t)(svo::queue_next(words + word) - words);
}

}  // extern "C"
