// svo_queue.h -- the per-stream work counters of a scene, shared by the queued cast
// (svo_device.cu) and the fused render (svo_render.cu).
//
// A queued kernel's warps claim work from a counter word that starts at 0.  Launches on one stream run one after
// another, so a stream takes two words in turn, and a launch zeroes the next one's (queue_begin): a
// launch needs nothing before it, and whatever a launch finds in its word, the one after the next
// starts at 0 again.  A captured launch may be replayed any number of times, beside casts on its stream too: it
// takes a third word, which a memset node before it zeroes.  Launches on different streams may overlap, so every
// stream that uses the scene gets words of its own.  Two more say which of two launches is to cast a batch.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

#include "svo_internal.h"

namespace svo {

constexpr uint32_t kQueueSlots = 64;
// Words of a stream: two that its launches take in turn, the captured launches' and one that those "zero" for nobody,
// and what order_kernel found, captured launches apart from others.
constexpr uint32_t kQueueWords = 6;

// Which of a stream's words its next launch claims from.
struct QueueTurn {
  uint32_t turn = 0;
  uint32_t word(bool captured) const { return captured ? 2u : turn; }
  void launched(bool captured) {  // it is in the stream, and will zero the other word
    if (!captured) turn ^= 1u;
  }
};

// The claim word of the next launch on the stream of the launch whose word `queue` is: the other of the pair.
#ifdef __CUDACC__
__host__ __device__
#endif
inline unsigned long long* queue_next(unsigned long long* queue) {
  return reinterpret_cast<unsigned long long*>(reinterpret_cast<uintptr_t>(queue) ^ sizeof(unsigned long long));
}
#ifdef __CUDACC__
// Zeroes it; no other launch of the stream runs meanwhile.
__device__ __forceinline__ void queue_begin(unsigned long long* queue) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *queue_next(queue) = 0;
}
#endif

struct CastQueues {
  std::mutex m;
  cudaStream_t streams[kQueueSlots] = {};
  QueueTurn turns[kQueueSlots];
  uint32_t used = 0;
  unsigned long long* counters = nullptr;  // kQueueSlots * kQueueWords
  int sm_count = 0, blocks_per_sm = 0, blocks_per_sm_count = 0, blocks_per_sm_plain = 0, blocks_per_sm_flow = 0;
};

// The words of one stream, or of a batch workspace.
struct QueueWords {
  unsigned long long* words = nullptr;  // nullptr: none
  QueueTurn* turn = nullptr;
};

// The words of stream `st` (claimed on first use), or none where the scene has none for it:
// all slots taken, or the per-thread default stream, which names a different stream in every
// host thread.  Call with q->m held until the launch is in the stream.
inline QueueWords queue_words(CastQueues* q, cudaStream_t st) {
  if (!q || st == cudaStreamPerThread) return {};
  uint32_t slot = 0;
  while (slot < q->used && q->streams[slot] != st) ++slot;
  if (slot == q->used) {
    if (q->used == kQueueSlots) return {};
    q->streams[q->used++] = st;
  }
  return {q->counters + kQueueWords * slot, q->turns + slot};
}

// One launch's word: `word` goes to the kernel, `launched` follows its launch.
struct QueueLaunch {
  unsigned long long* word = nullptr;
  unsigned long long* mixed = nullptr;
  QueueTurn* turn = nullptr;
  bool captured = false;
  void launched() { turn->launched(captured); }
};

inline cudaError_t queue_take(const QueueWords& q, cudaStream_t st, QueueLaunch& out) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(st, &capturing);
  out.captured = capturing != cudaStreamCaptureStatusNone;
  out.turn = q.turn;
  out.word = q.words + q.turn->word(out.captured);
  out.mixed = q.words + (out.captured ? 5 : 4);
  if (e == cudaSuccess && out.captured) e = cudaMemsetAsync(out.word, 0, sizeof(unsigned long long), st);
  return e;
}

}  // namespace svo
