// k_emit (emit_kernels.cu): pieces of emitted record batches gathered into an image of the data file.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gz {

constexpr uint32_t kEmitPiece = 16u << 10;  // bytes of a job, at most

struct EmitJob {  // len bytes of src (device memory, or pinned host memory) to byte dst of the file
  const uint8_t* src;
  uint64_t dst;
  uint64_t len;
};

// Runs the jobs (in device memory); `image` (16-byte aligned) holds the file's bytes from `base` (a
// multiple of 16) on.
cudaError_t launch_emit(const EmitJob* jobs, uint32_t n_jobs, uint8_t* image, uint64_t base, cudaStream_t st);

}  // namespace gz
