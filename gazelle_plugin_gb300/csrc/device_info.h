// What the launchers set or ask once a device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace gz {

// Lets launches of `kernel` on the current device use `bytes` of dynamic shared memory.  The limit belongs to
// the device that is current when it is set, and is never lowered: another thread may be about to launch
// the kernel with what it asked for.
cudaError_t AllowSharedMemory(const void* kernel, size_t bytes);

// The current device's SMs.
int SmCount();

}  // namespace gz
