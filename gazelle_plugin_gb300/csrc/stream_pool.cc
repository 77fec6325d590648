#include "stream_pool.h"

#include <algorithm>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

namespace gz {

namespace {

// An executor's task slots, all devices together.  Streams that live on cost something: with 57 sets kept
// a first small call on fresh buffers took 50 us instead of 28, with 16 of them 28.
constexpr size_t kPooledSets = 16;
constexpr size_t kPooledEvents = 2048;

struct Pool {
  std::mutex mu;
  std::vector<StreamSet> sets;
  std::map<int, std::vector<cudaEvent_t>> events;
  size_t n_events = 0;
};
// never destroyed: splitters may give sets back during exit
Pool& g_pool = *new Pool;

}  // namespace

void DestroyStreams(StreamSet* set) {
  for (cudaStream_t st : {set->c, set->p, set->s, set->h, set->o})
    if (st) cudaStreamDestroy(st);
  for (cudaEvent_t e : set->ev)
    if (e) cudaEventDestroy(e);
  *set = StreamSet();
}

cudaError_t AcquireStreams(int device, StreamSet* out) {
  StreamSet s;
  {
    std::lock_guard<std::mutex> lk(g_pool.mu);
    for (size_t i = g_pool.sets.size(); i-- > 0;) {
      if (g_pool.sets[i].device != device) continue;
      s = g_pool.sets[i];
      g_pool.sets.erase(g_pool.sets.begin() + (long)i);
      break;
    }
  }
  // host reads, then the plan kernels, get the higher priorities: their few CTAs are
  // scheduled ahead of the remaining CTAs of a running k_scatter; k_hash_count gets the lowest,
  // so it takes the SMs k_scatter leaves idle instead of delaying it
  int least = 0, greatest = 0;
  cudaError_t e = cudaDeviceGetStreamPriorityRange(&least, &greatest);
  if (s.device < 0) {
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&s.c, cudaStreamNonBlocking, greatest);
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&s.p, cudaStreamNonBlocking, std::min(greatest + 1, least));
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&s.h, cudaStreamNonBlocking, least);
    for (int i = 0; i < StreamSet::kEvents && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&s.ev[i], cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&s.s, cudaStreamNonBlocking, std::min(greatest + 2, least));
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s.o, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    DestroyStreams(&s);
    return e;
  }
  s.device = device;
  *out = s;
  return cudaSuccess;
}

void ReleaseStreams(StreamSet* set) {
  if (set->device < 0) return;
  if (set->s) cudaStreamDestroy(set->s);
  if (set->o) cudaStreamDestroy(set->o);
  set->s = set->o = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_pool.mu);
    if (g_pool.sets.size() < kPooledSets) {
      g_pool.sets.push_back(*set);
      *set = StreamSet();
      return;
    }
  }
  DestroyStreams(set);
}

cudaError_t WaitForWord(const uint32_t* word, uint32_t seq, cudaStream_t st) {
  for (uint32_t polls = 1; __atomic_load_n(word, __ATOMIC_ACQUIRE) != seq; polls++) {
    if (polls % 4096) continue;
    // taking long: a failed launch never writes the word
    const cudaError_t e = cudaStreamQuery(st);
    if (e != cudaErrorNotReady) return e;
    cudaGetLastError();
    std::this_thread::yield();
  }
  return cudaSuccess;
}

cudaError_t AcquireEvent(int device, cudaEvent_t* out) {
  {
    std::lock_guard<std::mutex> lk(g_pool.mu);
    auto& v = g_pool.events[device];
    if (!v.empty()) {
      *out = v.back();
      v.pop_back();
      g_pool.n_events--;
      return cudaSuccess;
    }
  }
  return cudaEventCreate(out);
}

void ReleaseEvent(int device, cudaEvent_t ev) {
  if (!ev) return;
  {
    std::lock_guard<std::mutex> lk(g_pool.mu);
    if (g_pool.n_events < kPooledEvents) {
      g_pool.events[device].push_back(ev);
      g_pool.n_events++;
      return;
    }
  }
  cudaEventDestroy(ev);
}

}  // namespace gz
