"""The host side of the kernel launches against a stand-in for the CUDA runtime with two devices (no GPU is
used): what a device has to be told before a launch is told to every device."""
import os
import subprocess

import pytest

from gazelle_plugin_gb300 import build as B

# Knows of each (device, kernel) the dynamic shared memory allowed, and refuses a launch that asks for more, as
# the runtime does; 48 KB need no leave.
RUNTIME = r"""
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <map>
#include <string>
#include <utility>
#include <vector>
static char g_primary[2], g_other;            // contexts: the devices' primary ones, one of the driver API's own
static char* g_ctx = &g_primary[0];
static int g_dev = 0, g_lowered = 0, g_launched[2] = {0, 0};
static cudaError_t g_last = cudaSuccess;
static std::map<std::pair<int, const void*>, int> g_limit;
static struct { dim3 g, b; size_t sm; cudaStream_t st; } g_cfg;
struct Owned { int dev; };  // a stream or an event
static cudaError_t fail() { return g_last = cudaErrorInvalidResourceHandle; }
static cudaError_t launch(const void* f, size_t sm, cudaStream_t st) {
  if ((st && ((Owned*)st)->dev != g_dev) || g_ctx != &g_primary[g_dev]) return fail();
  auto it = g_limit.find({g_dev, f});
  if (sm > (size_t)(it == g_limit.end() ? 48 * 1024 : it->second)) return g_last = cudaErrorInvalidValue;
  g_launched[g_dev]++;
  return cudaSuccess;
}
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sm, cudaStream_t st) { g_cfg = {g, b, sm, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sm, void* st) {
  *g = g_cfg.g; *b = g_cfg.b; *sm = g_cfg.sm; *(cudaStream_t*)st = g_cfg.st;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t sm, cudaStream_t st) {
  return launch((const void*)k, sm, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaGetLastError() { cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
const char* cudaGetErrorString(cudaError_t) { return "an error"; }
cudaError_t cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_dev = d; g_ctx = &g_primary[d]; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { *v = d == 0 ? 152 : 100; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes*, const void*) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char mem[256]; *p = mem; return g_ctx == &g_primary[g_dev] ? cudaSuccess : fail(); }
static int current(void** c) { *c = g_ctx; return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *f = (void*)current;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    int& have = g_limit[{g_dev, f}];
    if (v < have) g_lowered++;
    have = v;
  }
  return cudaSuccess;
}
// memory is the heap's, copies happen at once, kernels do nothing
static cudaError_t make(void* out) { *(Owned**)out = new Owned{g_dev}; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return make(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return make(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return make(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return ((Owned*)e)->dev == ((Owned*)s)->dev ? cudaSuccess : fail(); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
}
"""


def _object(src, where):
    """The built object of a source file, or one made here when it is missing or older than a source."""
    obj = os.path.join(B.BUILD_DIR, os.path.splitext(src)[0] + ".o")
    newest = max(os.path.getmtime(os.path.join(B.CSRC, f)) for f in os.listdir(B.CSRC))
    if os.path.exists(obj) and os.path.getmtime(obj) >= newest:
        return obj
    obj = os.path.join(where, os.path.basename(obj))
    subprocess.run([B.nvcc(), *B.GENCODE, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", os.path.join(B.ROOT, "include"),
                    "-c", os.path.join(B.CSRC, src), "-o", obj], check=True)
    return obj


def _run(where, objects, main):
    """Builds and runs `main` (C++ statements; check(x, what) notes what does not hold) over the objects."""
    try:
        cuda = os.path.join(os.path.dirname(os.path.dirname(B.nvcc())), "include")
    except RuntimeError:
        pytest.skip("no CUDA toolkit")
    src, exe = os.path.join(where, "m.cc"), os.path.join(where, "m")
    with open(src, "w") as f:
        f.write(RUNTIME + """
#include "gz_kernels.h"
#include "hash_static.h"
#include "lz4_kernels.h"
#include "read_kernels.h"
static int bad = 0;
static void check(bool ok, const char* what) { if (!ok) { bad++; printf("%s\\n", what); } }
int main() {
""" + main + "\n  return bad != 0;\n}\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", cuda, "-I", B.CSRC, "-I", os.path.join(B.ROOT, "include"), src,
                    *[_object(o, where) for o in objects], "-o", exe, "-pthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_every_device_allows_the_shared_memory_of_its_launches(tmp_path):
    _run(str(tmp_path), ["kernels.cu", "lz4_kernels.cu", "read_kernels.cu", "device_info.cc"], r"""
  using namespace gz;
  static SchemaDesc sd;
  static FlushDesc fd;
  fd.n_segs = fd.n_tiles = 1;
  fd.hist_in_smem = 1;
  uint32_t warps[2];
  for (int round = 0; round < 2; round++)
    for (int dev = 0; dev < 2; dev++) {
      cudaSetDevice(dev);
      check(launch_lz4_decode(nullptr, nullptr, 3, nullptr, nullptr, 0) == cudaSuccess, "LZ4 decode");
      check(launch_lz4_compress(nullptr, 3, nullptr, nullptr, nullptr, nullptr, 0, nullptr, false, nullptr, 0) == cudaSuccess, "LZ4 compress");
      for (int lists = 0; lists < 2; lists++) {
        sd.list_mask = lists;
        check(launch_scatter(sd, fd, 0) == cudaSuccess, "k_scatter");
        for (int P : {40000, 20000, 40000}) {
          sd.P = P;
          check(launch_hash_count(sd, fd, 0) == cudaSuccess, "k_hash_count");
        }
      }
      warps[dev] = lz4_compress_warps();
    }
  check(g_launched[0] == g_launched[1], "a launch on one device only");
  check(g_lowered == 0, "a limit lowered, which another thread's launch may rely on");
  check(warps[0] * 100 == warps[1] * 152, "the grid of the other device");
""")


def test_partition_ids_make_the_device_s_primary_context_current(tmp_path):
    """Also when the device is current already: a context of the driver API's own may be, in which neither the
    scratch array nor the kernels are at hand."""
    _run(str(tmp_path), ["hash_static.cu"], r"""
  int64_t counts[8];
  uint16_t ids[8];
  int32_t values[8] = {};
  GzKeyColumn key{};
  key.type = GZ_TYPE_INT32;
  key.values = reinterpret_cast<const uint8_t*>(values);
  std::string msg;
  int launches = 0;
  for (int call = 0; call < 2; call++)
    for (int dev = 0; dev < 2; dev++)
      for (int own = 0; own < 2; own++) {
        cudaSetDevice(0);
        if (own) g_ctx = &g_other;
        check(gz::HashPartitionStatic(dev, 8, &key, 1, 8, ids, counts, 0, &msg) == GZ_OK, "the call");
        check(g_launched[0] + g_launched[1] == (launches += 2), "its launches");
        check(g_dev == 0, "the caller's device is current again");
      }
""")


def test_calls_of_a_thread_on_another_device_use_the_task_s(tmp_path):
    """A memory manager's thread asks a task of device 1 to spill with device 0 current; so does a thread that
    reads the task's ids and times.  Streams, events and launches are the task's device's, and so is what later
    tasks take over from it."""
    _run(str(tmp_path), [s for s in B.SOURCES], r"""
  GzField field{};
  field.type = GZ_TYPE_INT64;
  field.name = "k";
  GzSplitOptions o;
  gz_split_default_options(&o);
  o.device = 1;
  o.prefer_spill = 0;
  const int32_t key = 0;
  int64_t values[10] = {};
  const int64_t addrs[2] = {0, (int64_t)values}, sizes[2] = {0, (int64_t)sizeof(values)};
  for (int what = 0; what < 6; what++) {
    int64_t h = 0, n = 0;
    uint16_t ids[10];
    double times[4];
    check(gz_split_make_fields("hash", 4, &field, 1, &key, 1, &o, &h) == GZ_OK, "make");
    check(gz_split_split(h, 10, addrs, sizes, 2, 0, &n) == GZ_OK, "split");
    cudaSetDevice(0);
    GzStatus st = GZ_OK;
    if (what % 3 == 0) st = gz_split_spill(h, 1 << 20, &n);
    if (what % 3 == 1) st = gz_split_last_pids(h, ids, 10);
    if (what % 3 == 2) st = gz_split_kernel_times(h, times);
    if (st != GZ_OK) printf("call %d: %d\n", what % 3, (int)st);
    check(st == GZ_OK, "a call of a thread with another device current");
    check(gz_split_sync(h) == GZ_OK, "sync");
    check(gz_split_close(h) == GZ_OK, "close");
  }
  check(cudaGetLastError() == cudaSuccess, "an error left behind");
""")
