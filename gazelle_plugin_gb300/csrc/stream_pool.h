// Streams and events kept from one splitter to the next: a splitter uses five streams and a score of
// events, and making and destroying them took 60 and 30 us of a one-batch map task's 480.  The two on which
// it allocates and frees memory are made anew: memory freed on a stream that lives on stays that
// stream's, and to others the pool hands it out slowly, with new mappings (after 16 tasks at once, a task
// of three batches took 1.75 ms instead of 0.8, a reader of 36 short streams 2.2 instead of 1.05).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gz {

struct StreamSet {
  static constexpr int kEvents = 15;
  int device = -1;  // -1: empty
  cudaStream_t c = nullptr, p = nullptr, h = nullptr;  // kept: Splitter's cstream_, pstream_, hstream_
  cudaStream_t s = nullptr, o = nullptr;               // not kept: its stream_, ostream_
  cudaEvent_t ev[kEvents] = {};                        // kept, without timing
};

// A set on the current device `device`, whose streams are idle.
cudaError_t AcquireStreams(int device, StreamSet* out);
// Takes an idle set back (at most kPooledSets are kept, the others destroyed); clears *set.
void ReleaseStreams(StreamSet* set);
void DestroyStreams(StreamSet* set);

// Waits until a launch on `st` has written seq to *word (k_gather_args), or `st` is done without.
cudaError_t WaitForWord(const uint32_t* word, uint32_t seq, cudaStream_t st);

// Timing events of the current device `device`, likewise.
cudaError_t AcquireEvent(int device, cudaEvent_t* out);
void ReleaseEvent(int device, cudaEvent_t ev);

}  // namespace gz
