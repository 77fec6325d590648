// sm_103a kernels of the reduce-side read (PartitionReader): the record batches of a partition's
// IPC streams, already in HBM, concatenated into one set of Arrow columns.  Three job lists, each
// job small enough that one CTA per job keeps every SM busy:
//   byte jobs   (64 KB) values of fixed-width columns and characters of binary columns, copied
//   offset jobs binary offsets (int32, or int64 of the large types) rebased:
//               out[i] = in[i] - in[0] + (the batch's first character)
//   bit jobs    validity / bool bits moved to their row in the output (OR into zeroed words;
//               a batch without a validity buffer contributes ones)
#include <cuda_runtime.h>
#include <stdint.h>

#include "copy.cuh"
#include "device_info.h"
#include "read_kernels.h"

#include <algorithm>

namespace gz {

namespace {

constexpr int kThreads = 256;

// Bits [start, start + len) of `src` (len <= 32) as the low bits of a word.  Reads only the 4-byte
// words that hold those bits.
__device__ __forceinline__ uint32_t extract_bits(const uint32_t* src, uint64_t start, uint32_t len) {
  const uint64_t w = start >> 5;
  const uint32_t sh = (uint32_t)(start & 31);
  uint32_t v = src[w] >> sh;
  if (sh + len > 32) v |= src[w + 1] << (32 - sh);
  return len == 32 ? v : v & ((1u << len) - 1);
}

// The three lists in one launch: blocks take the byte jobs first, then the offset jobs, then the bit jobs.
// Bound by HBM (every byte read and written once).  A record batch's buffers meet the column at any
// byte offset (characters) or element (values): the characters moved byte by byte before, in a launch of
// their own.  The columns of 32 record batches, 141 MB: 207 us as three launches with the lists uploaded
// before each, 54 now, the clearing of the validity words included (5.2 TB/s of loads and stores).
__global__ void __launch_bounds__(kThreads) k_read(const ReadJobs jobs) {
  const uint32_t n = jobs.n_bytes + jobs.n_offs + jobs.n_bits;
  for (uint32_t b = blockIdx.x; b < n; b += gridDim.x) {
    if (b < jobs.n_bytes) {
      const ByteJob job = jobs.bytes[b];
      copy_bytes<kThreads>(job.dst, job.src, (uint32_t)job.bytes, threadIdx.x);
    } else if (b < jobs.n_bytes + jobs.n_offs) {
      const OffsetJob job = jobs.offs[b - jobs.n_bytes];
      if (job.wide) {
        const int64_t* src = static_cast<const int64_t*>(job.src);
        int64_t* dst = static_cast<int64_t*>(job.dst);
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < job.n; i += kThreads) dst[i] = src[i] + job.add;
      } else {
        const int32_t* src = static_cast<const int32_t*>(job.src);
        int32_t* dst = static_cast<int32_t*>(job.dst);
        const int32_t add = (int32_t)job.add;
#pragma unroll 8
        for (uint32_t i = threadIdx.x; i < job.n; i += kThreads) dst[i] = src[i] + add;
      }
    } else {
      const BitJob job = jobs.bits[b - jobs.n_bytes - jobs.n_offs];
      if (job.nbits == 0) continue;
      const uint64_t d0 = job.dst_bit, d1 = job.dst_bit + job.nbits;
      const uint64_t w0 = d0 >> 5, w1 = (d1 - 1) >> 5;
      for (uint64_t w = w0 + threadIdx.x; w <= w1; w += kThreads) {
        const uint64_t lo = w * 32 > d0 ? w * 32 : d0;
        const uint64_t hi = w * 32 + 32 < d1 ? w * 32 + 32 : d1;
        const uint32_t len = (uint32_t)(hi - lo);
        const uint32_t bits = job.src ? extract_bits(job.src, job.src_bit + (lo - d0), len)
                                      : (len == 32 ? 0xffffffffu : (1u << len) - 1);
        if (bits) atomicOr(job.dst + w, bits << (uint32_t)(lo - w * 32));
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_read_words(const int32_t* const* __restrict__ src, int32_t* out, size_t n) {
  cudaGridDependencySynchronize();
  for (size_t i = (size_t)blockIdx.x * kThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kThreads) out[i] = *src[i];
}

unsigned grid_for(uint32_t n_jobs) {
  const uint32_t cap = 8u * (uint32_t)SmCount();
  return n_jobs < cap ? n_jobs : cap;
}

}  // namespace

cudaError_t launch_read_words(const int32_t* const* src, int32_t* out, size_t n, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const size_t blocks = (n + kThreads - 1) / kThreads;
  cudaLaunchAttribute at;  // it comes up while the kernel before it runs
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = (unsigned)std::min<size_t>(blocks, 1024);
  cfg.blockDim = kThreads;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_read_words, src, out, n);
}

cudaError_t launch_read_jobs(const ReadJobs& jobs, cudaStream_t st) {
  const uint32_t n = jobs.n_bytes + jobs.n_offs + jobs.n_bits;
  if (n == 0) return cudaSuccess;
  k_read<<<grid_for(n), kThreads, 0, st>>>(jobs);
  return cudaGetLastError();
}

}  // namespace gz
