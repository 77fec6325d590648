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

#include "emit_kernels.h"

namespace gz {

namespace {

constexpr int kThreads = 256;

// Bytes 4 * Q + sh / 8 .. + 16 of the 32 bytes a, b.
template <int Q>
__device__ __forceinline__ uint4 shift16(const uint4& a, const uint4& b, uint32_t sh) {
  const uint32_t w[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, 0u};
  return make_uint4(__funnelshift_r(w[Q], w[Q + 1], sh), __funnelshift_r(w[Q + 1], w[Q + 2], sh),
                    __funnelshift_r(w[Q + 2], w[Q + 3], sh), __funnelshift_r(w[Q + 3], w[Q + 4], sh));
}

// n 16-byte words of dst from the source bytes at phase s = 4 * Q + sh / 8 of the aligned word a.  Every
// word read holds bytes of the source (with s = 0 the second one of a pair is not read).
template <int Q>
__device__ __forceinline__ void copy_words(uint4* dst, const uint4* a, uint32_t n, uint32_t s) {
  const uint32_t lane = threadIdx.x & 31, sh = (s & 3) * 8, up = s ? 1u : 0u;
#pragma unroll 4
  for (uint32_t i = lane; i < n; i += 32) {
    const uint4 x = a[i], y = a[i + up];
    dst[i] = shift16<Q>(x, y, sh);
  }
}

__global__ void __launch_bounds__(kThreads) k_emit(const EmitJob* __restrict__ jobs, uint32_t n_jobs, uint8_t* image,
                                                    uint64_t base) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (kThreads / 32);
  for (uint32_t j = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); j < n_jobs; j += warps) {
    const EmitJob job = jobs[j];
    uint8_t* dst = image + (job.dst - base);
    const uint8_t* src = job.src;
    uint32_t n = (uint32_t)job.len;
    const uint32_t head = min(n, (16u - ((uint32_t)job.dst & 15)) & 15);
    if (lane < head) dst[lane] = src[lane];
    dst += head;
    src += head;
    n -= head;
    const uint32_t s = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15), nw = n >> 4;
    const uint4* a = reinterpret_cast<const uint4*>(src - s);
    uint4* d = reinterpret_cast<uint4*>(dst);
    switch (s >> 2) {  // the same in the whole warp
      case 0: copy_words<0>(d, a, nw, s); break;
      case 1: copy_words<1>(d, a, nw, s); break;
      case 2: copy_words<2>(d, a, nw, s); break;
      default: copy_words<3>(d, a, nw, s); break;
    }
    if (lane < (n & 15)) dst[(nw << 4) + lane] = src[(nw << 4) + lane];
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
