// k_emit: the data file's bytes put together by the device.
//
// Stop used to copy every pass's column regions to pinned host memory and had the CPU gather each
// record batch's buffers out of them into the file, page faults included: 3.7 ms and 12.3 ms of an
// 18.5 ms Stop that writes 720 MB (47 MB through pwritev: 5.5 ms, the file's lock admits one writer).
// Here the pieces of every record batch (headers and padding too, uploaded in one block) go to
// their place in an image of a stretch of the file, in HBM, and the image goes to the file's mapped pages
// in one copy at the link's rate.  The kernel itself is bound by HBM: sources and destinations meet at
// any byte offset, so a warp takes a piece and writes aligned 16-byte words, each shifted together
// from two aligned source words.
#include <cuda_runtime.h>
#include <stdint.h>

#include "copy.cuh"
#include "emit_kernels.h"

namespace gz {

namespace {

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) k_emit(const EmitJob* __restrict__ jobs, uint32_t n_jobs, uint8_t* image,
                                                    uint64_t base) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (kThreads / 32);
  for (uint32_t j = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); j < n_jobs; j += warps) {
    const EmitJob job = jobs[j];
    copy_bytes<32>(image + (job.dst - base), job.src, (uint32_t)job.len, lane);
  }
}

}  // namespace

cudaError_t launch_emit(const EmitJob* jobs, uint32_t n_jobs, uint8_t* image, uint64_t base, cudaStream_t st) {
  if (n_jobs == 0) return cudaSuccess;
  const uint32_t per = kThreads / 32, need = (n_jobs + per - 1) / per;
  k_emit<<<need < 1216u ? need : 1216u, kThreads, 0, st>>>(jobs, n_jobs, image, base);  // eight blocks per SM
  return cudaGetLastError();
}

}  // namespace gz
