// Streams and events kept from one splitter to the next: a splitter uses five streams and a score of
// events, and making and destroying them took 60 and 30 us of a one-batch map task's 480.
#pragma once
#include <cuda_runtime.h>

namespace gz {

struct StreamSet {
  static constexpr int kEvents = 15;
  int device = -1;  // -1: empty
  cudaStream_t c = nullptr, p = nullptr, s = nullptr, h = nullptr, o = nullptr;  // Splitter's cstream_ ..
  cudaEvent_t ev[kEvents] = {};                                                  // without timing
};

// A set on the current device `device`, whose streams are idle.
cudaError_t AcquireStreams(int device, StreamSet* out);
// Takes an idle set back (at most kPooledSets are kept, the others destroyed); clears *set.
void ReleaseStreams(StreamSet* set);
void DestroyStreams(StreamSet* set);

// Timing events of the current device `device`, likewise.
cudaError_t AcquireEvent(int device, cudaEvent_t* out);
void ReleaseEvent(int device, cudaEvent_t ev);

}  // namespace gz
