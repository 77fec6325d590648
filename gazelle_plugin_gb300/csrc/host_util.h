// Host-side helpers of the splitter: a process-wide pool of pinned host blocks (flush outputs
// copied out of HBM) and a small thread pool that spreads large memcpys over several cores
// (staging a caller's host batch before Split returns).
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <functional>
#include <vector>

namespace gz {

struct PinnedBlock {
  uint8_t* ptr = nullptr;
  size_t cap = 0;
};

// Pinned (page-locked) host blocks, reused across splitters.  Acquire returns a block of at
// least `bytes` (cap = its size); ptr == nullptr when cudaHostAlloc failed.  Release takes back
// exactly a block Acquire returned.
PinnedBlock PinnedAcquire(size_t bytes);
void PinnedRelease(PinnedBlock b);
// Adds about `bytes` of pinned slabs of `block` bytes to the pool up front (cudaHostAlloc is
// slow, so a server takes that cost at start instead of inside calls); returns the bytes added.
int64_t PinnedReserve(int64_t bytes, size_t block);
constexpr size_t kPinnedSlab = size_t(1) << 30;

struct CopyJob {
  uint8_t* dst;
  const uint8_t* src;
  size_t n;
};

// Copies every job; large totals are split over worker threads and the caller.  Returns when
// all bytes are copied.
void ParallelCopy(const std::vector<CopyJob>& jobs, size_t total_bytes);

// Runs fn(i) for every i in [0, n) on the calling thread and up to `max_helpers` threads of a
// process-wide pool (shared by all splitters: concurrent calls share its workers); returns when
// every fn(i) has returned.  Items are claimed one at a time (a few at a time when there are hundreds),
// so long and short items balance.
void ParallelFor(size_t n, const std::function<void(size_t)>& fn, int max_helpers = 15);

// A caller about to use the pool's threads a number of times (a task's Stop): while several do, each
// gets its share of them (16 tasks that stop at once, 283 MB, wake and contend for 15 workers otherwise:
// 9.7 to 11.2 ms, 8.9 to 9.1 with shares).
struct ParallelUser {
  ParallelUser();
  ~ParallelUser();
  ParallelUser(const ParallelUser&) = delete;
  ParallelUser& operator=(const ParallelUser&) = delete;
};
// The share, at most `most`.
int ParallelHelpers(int most);

// Starts fn on up to `threads` threads of that pool and returns at once; fn runs at most that often
// (not at all while the pool is busy), possibly after the caller is done: it owns what it uses.
void Background(int threads, const std::function<void()>& fn);

}  // namespace gz
