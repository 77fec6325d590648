#include "device_info.h"

#include <map>
#include <mutex>
#include <utility>

namespace gz {

namespace {

struct Known {
  std::mutex mu;
  std::map<std::pair<int, const void*>, size_t> shared;  // (device, kernel): its limit
  std::map<int, int> sms;
};
// never destroyed: launches may come during exit
Known& g_known = *new Known;

}  // namespace

cudaError_t AllowSharedMemory(const void* kernel, size_t bytes) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_known.mu);
  size_t& have = g_known.shared[{dev, kernel}];
  if (have >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) have = bytes;
  return e;
}

int SmCount() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 152;
  std::lock_guard<std::mutex> lk(g_known.mu);
  int& have = g_known.sms[dev];
  if (have == 0 && (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)) return 152;
  if (have == 0) have = sms;
  return have;
}

}  // namespace gz
