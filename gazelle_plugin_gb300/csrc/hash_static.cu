// Partition ids of one device-resident batch, computed without allocating device memory
// (C entry point gz_hash_partition_static).
//
// The hash chain and pmod are the splitter's (k_hash_count, restating
// HashSplitter::ComputeAndCountPartitionId, native-sql-engine/cpp/src/shuffle/splitter.cc:1440-1470).
// k_hash_count counts rows per (segment, partition) in memory the splitter allocates for each
// device pass; here the blocks' counts live in one file-scope device array of fixed size, so
// that callers which may not allocate device memory can run the kernel.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "gz_engine.cuh"
#include "gz_hash.cuh"
#include "hash_static.h"

namespace gz {
namespace {

using namespace hash;

constexpr uint32_t kTile = 1024;             // rows behind each row of counters in the limit on a call
constexpr uint32_t kGroup = 4;               // consecutive rows of a thread
constexpr uint32_t kSmemHistMaxP = 57344;    // a block's histogram stays in shared memory (224 KB)
constexpr int kAny = -1, kMixed = -2;         // see k_hash_count_static
constexpr uint32_t kWideHistP = 2048;        // larger histograms: blocks of 1024 threads share one

// Row counts of each block, [block][partition], of the most recent call on this device.  Every call
// shares it and it keeps the last call's contents: each block writes the row it owns.  Host code
// reaches it only through the address cudaGetSymbolAddress returns.
static __device__ __align__(256) uint32_t g_tile_counts[kStaticScratchWords];

struct KeySet {
  const uint8_t* validity[kMaxKeys];
  const uint8_t* values[kMaxKeys];
  int32_t kind[kMaxKeys];
  int32_t n;
};

// Rows r0 .. r0 + 3 (r0 a multiple of 4) of a key as they lie in memory, and their validity bits.
struct Group {
  uint4 lo, hi;    // int64: two rows each; narrower values packed from lo.x on; bool: bits of lo.x
  uint32_t valid;
};

// Bits r0 .. r0 + 3 of a bitmap: one byte holds them.
__device__ __forceinline__ uint32_t load_nibble(const uint8_t* bits, uint32_t r0) {
  return (uint32_t)(__ldg(bits + (r0 >> 3)) >> (r0 & 4)) & 15u;
}

// kBytes per row: one or two wide loads where the buffer's alignment allows them (a batch sliced out of
// a larger one may start anywhere) and no row is past the end, else row by row.
template <int kBytes>
__device__ __forceinline__ void load_values(const uint8_t* values, uint32_t r0, uint32_t m, uint4* lo, uint4* hi) {
  const uint8_t* p = values + (size_t)r0 * kBytes;
  constexpr uint32_t kWide = kBytes * 4 < 16 ? kBytes * 4 : 16;
  if (m == kGroup && (reinterpret_cast<uintptr_t>(p) & (kWide - 1)) == 0) {
    if constexpr (kBytes == 8) *hi = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    if constexpr (kBytes >= 4) {
      *lo = __ldg(reinterpret_cast<const uint4*>(p));
    } else if constexpr (kBytes == 2) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      lo->x = v.x;
      lo->y = v.y;
    } else {
      lo->x = __ldg(reinterpret_cast<const uint32_t*>(p));
    }
    return;
  }
  uint64_t v[kGroup];
#pragma unroll
  for (uint32_t u = 0; u < kGroup; u++) {
    v[u] = 0;
    if (u >= m) continue;
    if constexpr (kBytes == 8) v[u] = reinterpret_cast<const uint64_t*>(p)[u];
    else if constexpr (kBytes == 4) v[u] = reinterpret_cast<const uint32_t*>(p)[u];
    else if constexpr (kBytes == 2) v[u] = reinterpret_cast<const uint16_t*>(p)[u];
    else v[u] = p[u];
  }
  if constexpr (kBytes == 8) {
    *lo = make_uint4((uint32_t)v[0], (uint32_t)(v[0] >> 32), (uint32_t)v[1], (uint32_t)(v[1] >> 32));
    *hi = make_uint4((uint32_t)v[2], (uint32_t)(v[2] >> 32), (uint32_t)v[3], (uint32_t)(v[3] >> 32));
  } else if constexpr (kBytes == 4) {
    *lo = make_uint4((uint32_t)v[0], (uint32_t)v[1], (uint32_t)v[2], (uint32_t)v[3]);
  } else if constexpr (kBytes == 2) {
    lo->x = (uint32_t)(v[0] | v[1] << 16);
    lo->y = (uint32_t)(v[2] | v[3] << 16);
  } else {
    lo->x = (uint32_t)(v[0] | v[1] << 8 | v[2] << 16 | v[3] << 24);
  }
}

__device__ __forceinline__ void load_key(const KeySet& keys, int k, uint32_t r0, uint32_t m, Group* g) {
  const uint8_t* values = keys.values[k];
  switch (keys.kind[k]) {
    case KEY_I64: load_values<8>(values, r0, m, &g->lo, &g->hi); break;
    case KEY_I32: load_values<4>(values, r0, m, &g->lo, &g->hi); break;
    case KEY_I16: load_values<2>(values, r0, m, &g->lo, &g->hi); break;
    case KEY_I8: load_values<1>(values, r0, m, &g->lo, &g->hi); break;
    default: g->lo.x = load_nibble(values, r0); break;
  }
  g->valid = keys.validity[k] != nullptr ? load_nibble(keys.validity[k], r0) : 15u;
}

// The key's hashes chained onto h; a null passes the seed through.
__device__ __forceinline__ void hash_key(int kind, const Group& g, int32_t* h) {
  int32_t x[kGroup];
  if (kind == KEY_I64) {
    x[0] = hash_long((int64_t)((uint64_t)g.lo.y << 32 | g.lo.x), h[0]);
    x[1] = hash_long((int64_t)((uint64_t)g.lo.w << 32 | g.lo.z), h[1]);
    x[2] = hash_long((int64_t)((uint64_t)g.hi.y << 32 | g.hi.x), h[2]);
    x[3] = hash_long((int64_t)((uint64_t)g.hi.w << 32 | g.hi.z), h[3]);
  } else {
    int32_t v[kGroup];
    if (kind == KEY_I32) {
      v[0] = (int32_t)g.lo.x;
      v[1] = (int32_t)g.lo.y;
      v[2] = (int32_t)g.lo.z;
      v[3] = (int32_t)g.lo.w;
    } else if (kind == KEY_I16) {
      v[0] = (int16_t)g.lo.x;
      v[1] = (int16_t)(g.lo.x >> 16);
      v[2] = (int16_t)g.lo.y;
      v[3] = (int16_t)(g.lo.y >> 16);
    } else if (kind == KEY_I8) {
#pragma unroll
      for (uint32_t u = 0; u < kGroup; u++) v[u] = (int8_t)(g.lo.x >> (8 * u));
    } else {
#pragma unroll
      for (uint32_t u = 0; u < kGroup; u++) v[u] = (int32_t)((g.lo.x >> u) & 1u);
    }
#pragma unroll
    for (uint32_t u = 0; u < kGroup; u++) x[u] = hash_int(v[u], h[u]);
  }
#pragma unroll
  for (uint32_t u = 0; u < kGroup; u++)
    if ((g.valid >> u) & 1u) h[u] = x[u];
}

// Every block takes a contiguous range of rows: partition id of every row, and the block's row count
// per partition into row blockIdx.x of `count_rows`.  Bound by the hash's integer instructions.  A
// thread takes four consecutive rows, loaded 16 bytes at a time one key ahead of
// the hashing, and a block keeps one histogram for all its rows, so only a row of counters per
// resident block is left to be added up.  16M rows of two nullable int64 keys and 200 partitions (290
// MB): 156 us with scalar loads and a row of counters per 1024 rows, 84 us with wide loads and few
// counters (59% of the issue slots, 55% of the 64-bit multiply pipe), 70 us with the next key's loads
// ahead and the 32-bit pmod (117 instructions a row, 75% of the issue slots), 55 us (5.2 TB/s) with counters known to be in shared
// memory (a pointer to either memory costs an address test and a branch per row), the last, partial
// groups apart and the alignment and the kind of the keys settled by the host; one int32 key: 47 and 32 us.
// (A ring of four keys' values on their way into shared memory by cp.async: 46 us for one int32 key
// against 47, 90 for the two int64 against 70: not the loads but the instructions bound it.)
// kSmem: the counters are in shared memory.  kKind: all keys are of that kind, their values on the
// boundaries of a group's wide loads and the ids on 8-byte ones; kMixed: any kinds, so aligned; kAny.
template <int kThreads, int kMinBlocks, bool kSmem, int kKind>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
k_hash_count_static(const KeySet keys, uint32_t nrows, uint32_t rows_per_block, PmodDiv pmod,
                    uint16_t* __restrict__ pids, uint32_t* __restrict__ count_rows) {
  extern __shared__ uint32_t smem[];
  cudaTriggerProgrammaticLaunchCompletion();  // k_sum_tile_counts may come up, and wait
  cudaGridDependencySynchronize();            // (this kernel came up early as well)
  const uint32_t P = pmod.P;
  uint32_t* const row = count_rows + (size_t)blockIdx.x * P;
  uint32_t* const H = kSmem ? smem : row;
  const uint32_t lo = blockIdx.x * rows_per_block;  // a multiple of 4
  const uint32_t hi = min(nrows, lo + rows_per_block);
  uint32_t r0 = lo + kGroup * threadIdx.x;
  auto load = [&](int k, uint32_t r, uint32_t m, Group* g) {
    if (kKind == kMixed && m == kGroup) {
      const uint8_t* v = keys.values[k];
      switch (keys.kind[k]) {
        case KEY_I64:
          g->lo = __ldg(reinterpret_cast<const uint4*>(v) + (r >> 1));
          g->hi = __ldg(reinterpret_cast<const uint4*>(v) + (r >> 1) + 1);
          break;
        case KEY_I32: g->lo = __ldg(reinterpret_cast<const uint4*>(v) + (r >> 2)); break;
        case KEY_I16: {
          const uint2 x = __ldg(reinterpret_cast<const uint2*>(v) + (r >> 2));
          g->lo.x = x.x;
          g->lo.y = x.y;
          break;
        }
        case KEY_I8: g->lo.x = __ldg(reinterpret_cast<const uint32_t*>(v) + (r >> 2)); break;
        default: g->lo.x = load_nibble(v, r); break;
      }
      g->valid = keys.validity[k] != nullptr ? load_nibble(keys.validity[k], r) : 15u;
    } else if (kKind >= 0 && m == kGroup) {
      const uint4* v = reinterpret_cast<const uint4*>(keys.values[k]) + (r >> 2) * (kKind == KEY_I64 ? 2 : 1);
      g->lo = __ldg(v);
      if (kKind == KEY_I64) g->hi = __ldg(v + 1);
      g->valid = keys.validity[k] != nullptr ? load_nibble(keys.validity[k], r) : 15u;
    } else {
      load_key(keys, k, r, m, g);
    }
  };
  auto hash = [&](int k, const Group& g, int32_t* h) { hash_key(kKind >= 0 ? kKind : keys.kind[k], g, h); };
  // the ids of m rows from r on
  auto put = [&](const int32_t* h, uint32_t r, uint32_t m) {
    uint32_t p[kGroup];
#pragma unroll
    for (uint32_t u = 0; u < kGroup; u++) p[u] = pmod_div(h[u], pmod);
    if (m == kGroup && (kKind != kAny || (reinterpret_cast<uintptr_t>(pids) & 7) == 0)) {
      *reinterpret_cast<uint2*>(pids + r) = make_uint2(p[0] | p[1] << 16, p[2] | p[3] << 16);
    } else {
#pragma unroll
      for (uint32_t u = 0; u < kGroup; u++)
        if (u < m) pids[r + u] = (uint16_t)p[u];
    }
#pragma unroll
    for (uint32_t u = 0; u < kGroup; u++)
      if (u < m) atomicAdd(&H[p[u]], 1u);
  };
  Group cur, nxt;
  cur.lo = cur.hi = nxt.lo = nxt.hi = make_uint4(0, 0, 0, 0);
  cur.valid = 0;
  if (r0 + kGroup <= hi && keys.n > 0) load(0, r0, kGroup, &cur);
  for (uint32_t i = threadIdx.x; i < P; i += kThreads) H[i] = 0;
  __syncthreads();
  for (; r0 + kGroup <= hi; r0 += kGroup * kThreads) {
    const uint32_t r1 = r0 + kGroup * kThreads;
    int32_t h[kGroup] = {42, 42, 42, 42};
    for (int k = 0; k < keys.n; k++) {
      // the next key, or the next group's first, is on its way while this one is hashed
      if (k + 1 < keys.n) load(k + 1, r0, kGroup, &nxt);
      else if (r1 + kGroup <= hi) load(0, r1, kGroup, &nxt);
      hash(k, cur, h);
      cur = nxt;
    }
    put(h, r0, kGroup);
  }
  if (r0 < hi) {  // the call's last rows, fewer than a group
    int32_t h[kGroup] = {42, 42, 42, 42};
    for (int k = 0; k < keys.n; k++) {
      load(k, r0, hi - r0, &cur);
      hash(k, cur, h);
    }
    put(h, r0, hi - r0);
  }
  if (kSmem) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < P; i += kThreads) row[i] = H[i];
  }
}

// counts[p] = sum over blocks of count_rows[b][p].  Block (32, 32): x picks the partition,
// y strides over the rows; the 32 partial sums of a partition are added in shared memory.
__global__ void __launch_bounds__(1024)
k_sum_tile_counts(const uint32_t* __restrict__ count_rows, uint32_t n_rows, uint32_t P,
                  int64_t* __restrict__ counts) {
  __shared__ unsigned long long part[32][33];
  const uint32_t p = blockIdx.x * 32 + threadIdx.x;
  cudaTriggerProgrammaticLaunchCompletion();  // so may the next call's counting kernel
  cudaGridDependencySynchronize();            // the counting kernel's rows
  unsigned long long s = 0;
  if (p < P) {
#pragma unroll 8
    for (uint32_t t = threadIdx.y; t < n_rows; t += 32) s += count_rows[(size_t)t * P + p];
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && p < P) {
    unsigned long long tot = 0;
    for (int y = 0; y < 32; y++) tot += part[y][threadIdx.x];
    counts[p] = (int64_t)tot;
  }
}

using CountFn = void (*)(const KeySet, uint32_t, uint32_t, PmodDiv, uint16_t*, uint32_t*);
// wide: blocks of 1024 threads share a histogram (always in shared memory)
CountFn CountKernel(bool wide, bool smem, int kind) {
  if (!smem) return k_hash_count_static<512, 3, false, kAny>;
  switch (kind) {
    case KEY_I32: return wide ? k_hash_count_static<1024, 1, true, KEY_I32> : k_hash_count_static<512, 3, true, KEY_I32>;
    case KEY_I64: return wide ? k_hash_count_static<1024, 1, true, KEY_I64> : k_hash_count_static<512, 3, true, KEY_I64>;
    case kMixed: return wide ? k_hash_count_static<1024, 1, true, kMixed> : k_hash_count_static<512, 3, true, kMixed>;
    default: return wide ? k_hash_count_static<1024, 1, true, kAny> : k_hash_count_static<512, 3, true, kAny>;
  }
}

std::mutex g_mu;
// device address of g_tile_counts, per device ordinal, in that device's primary context (the
// one the runtime API uses; other contexts are not supported)
std::vector<uint32_t*> g_addr;
std::vector<int> g_sms;  // SMs per device ordinal
std::vector<CUcontext> g_primary;  // that context
CUresult (*g_ctx_current)(CUcontext*) = nullptr;

// Whether the thread's context is the one that g_addr[device] is of.  cudaSetDevice makes it so, also where a
// context of the driver API's own is current on that device, but on every call it cost 0.13 of 4.4 us; a look costs
// nothing that shows.
bool PrimaryIsCurrent(int device) {
  std::lock_guard<std::mutex> lk(g_mu);
  CUcontext c = nullptr;
  return device >= 0 && device < (int)g_primary.size() && g_primary[device] != nullptr &&
         g_ctx_current(&c) == CUDA_SUCCESS && c == g_primary[device];
}

// Looks up (once per device, with `device` current) the device address of g_tile_counts, and loads
// the kernels, so that no later call adds device code.
cudaError_t ScratchAddress(int device, uint32_t** out, uint32_t* sms) {
  std::lock_guard<std::mutex> lk(g_mu);
  if ((int)g_addr.size() <= device) g_addr.resize(device + 1, nullptr);
  if (g_addr[device] == nullptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_tile_counts);
    cudaFuncAttributes fa;
    for (const bool wide : {false, true})
      for (const bool smem : {false, true})
        for (const int kind : {kAny, kMixed, (int)KEY_I32, (int)KEY_I64}) {
          if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, CountKernel(wide, smem, kind));
          if (e == cudaSuccess && wide && smem)
            e = cudaFuncSetAttribute(CountKernel(wide, smem, kind), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(kSmemHistMaxP * sizeof(uint32_t)));
        }
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k_sum_tile_counts);
    if (e == cudaSuccess && (int)g_sms.size() <= device) g_sms.resize(device + 1, 0);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sms[device], cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    g_addr[device] = static_cast<uint32_t*>(p);
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (g_ctx_current == nullptr) {
      if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &found) != cudaSuccess)
        cudaGetLastError();  // (then cudaSetDevice on every call)
      else if (found == cudaDriverEntryPointSuccess)
        g_ctx_current = reinterpret_cast<CUresult (*)(CUcontext*)>(f);
    }
    if ((int)g_primary.size() <= device) g_primary.resize(device + 1, nullptr);
    if (g_ctx_current != nullptr && g_ctx_current(&g_primary[device]) != CUDA_SUCCESS) g_primary[device] = nullptr;
  }
  *out = g_addr[device];
  *sms = (uint32_t)g_sms[device];
  return cudaSuccess;
}

}  // namespace

GzStatus HashPartitionStatic(int32_t device, int32_t P, const GzKeyColumn* keys, int32_t n_keys,
                             int32_t num_rows, uint16_t* pids, int64_t* counts, cudaStream_t stream,
                             std::string* msg) {
  if (P < 1 || P > 65536) {
    *msg = "num_partitions must be in [1, 65536], got " + std::to_string(P);
    return GZ_INVALID;
  }
  if (keys == nullptr || n_keys < 1 || n_keys > kMaxKeys) {
    *msg = "need 1 to " + std::to_string(kMaxKeys) + " key columns";
    return GZ_INVALID;
  }
  if (num_rows < 0 || counts == nullptr || (num_rows > 0 && pids == nullptr)) {
    *msg = "num_rows must be >= 0 and the output pointers non-null";
    return GZ_INVALID;
  }
  // A null-type key has no hash function and leaves the chain unchanged (the NullType case of
  // HashSplitter::CreateProjector, splitter.cc:1407-1408): it takes no slot of the key list.
  KeySet ks{};
  ks.n = 0;
  for (int k = 0; k < n_keys; k++) {
    if (keys[k].type == GZ_TYPE_NULL) continue;
    int kind;
    switch (keys[k].type) {
      case GZ_TYPE_BOOL: kind = KEY_BOOL; break;
      case GZ_TYPE_INT8: kind = KEY_I8; break;
      case GZ_TYPE_INT16: kind = KEY_I16; break;
      case GZ_TYPE_INT32: case GZ_TYPE_FLOAT32: case GZ_TYPE_DATE32: kind = KEY_I32; break;
      case GZ_TYPE_INT64: case GZ_TYPE_FLOAT64: kind = KEY_I64; break;
      default:
        *msg = "key " + std::to_string(k) + ": type " + std::to_string(keys[k].type) +
               " has no Spark-compatible hash here";
        return GZ_NOT_IMPLEMENTED;
    }
    if (num_rows > 0 && keys[k].values == nullptr) {
      *msg = "key " + std::to_string(k) + ": null values pointer";
      return GZ_INVALID;
    }
    ks.kind[ks.n] = kind;
    ks.validity[ks.n] = keys[k].validity;
    ks.values[ks.n] = keys[k].values;
    ks.n++;
  }
  const uint64_t n_tiles = ((uint64_t)num_rows + kTile - 1) / kTile;
  if (n_tiles * (uint64_t)P > kStaticScratchWords) {
    *msg = std::to_string(num_rows) + " rows x " + std::to_string(P) + " partitions need " +
           std::to_string(n_tiles * (uint64_t)P) + " per-tile counters; the static scratch holds " +
           std::to_string(kStaticScratchWords) + " (16 MiB): split the batch into smaller calls";
    return GZ_INVALID;
  }

  // An error already pending on this thread came from the caller's earlier work, not from this
  // call: report it as such (and leave it pending) instead of taking it for a launch failure.
  {
    const cudaError_t before = cudaPeekAtLastError();
    if (before != cudaSuccess) {
      *msg = std::string("a CUDA error from earlier work on this thread is pending (nothing was "
                         "launched): ") + cudaGetErrorString(before);
      return GZ_CUDA;
    }
  }
  int prev = device;
  cudaError_t e = cudaSuccess;
  if (!PrimaryIsCurrent(device)) {
    e = cudaGetDevice(&prev);
    if (e == cudaSuccess) e = cudaSetDevice(device);
  }
  uint32_t* scratch = nullptr;
  uint32_t sms = 0;
  if (e == cudaSuccess) {
    e = ScratchAddress(device, &scratch, &sms);
    if (e == cudaErrorMemoryAllocation) {
      // with lazy module loading the array is reserved here, on the first call on a device
      cudaGetLastError();
      if (prev >= 0 && prev != device) cudaSetDevice(prev);
      *msg = "out of device memory reserving the library's 16 MiB static scratch array on device " +
             std::to_string(device) + ": make the first call on each device before reserving its free memory";
      return GZ_OOM;
    }
  }
  if (e == cudaSuccess) {
    // Blocks that fill the SMs, each with at least a full sweep of rows.  A histogram of up to 2048
    // partitions is a block of 512 threads' own (three blocks per SM); a larger one is shared by 1024
    // threads, one block per SM, so that fewer rows of counters are written and added up (500k rows,
    // 8000 partitions, three keys: 18.5 us with a row per 1024 rows, 9.0 us); one that exceeds shared
    // memory is counted in its row of the scratch.  (One cluster adding its histograms through distributed shared memory in a
    // single launch was no faster for small batches: 6.2 us a call.)
    const uint32_t n = (uint32_t)num_rows, parts = (uint32_t)P;
    const bool smem_hist = parts <= kSmemHistMaxP, wide = smem_hist && parts > kWideHistP;
    const uint32_t threads = wide ? 1024 : 512;
    const uint64_t sweep = smem_hist ? threads * kGroup : kTile;
    uint64_t blocks = std::min<uint64_t>((n + sweep - 1) / sweep, smem_hist ? (uint64_t)sms * (wide ? 1 : 3) : n_tiles);
    // Both kernels may come up while the one before them on the stream still runs, and wait for it
    // there: calls of 4096 rows in a row take 4.4 us each instead of 9.2 (6.1 with the second kernel only).
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (blocks > 0) {
      const uint32_t per = (uint32_t)((n + blocks - 1) / blocks + 3) & ~3u;
      blocks = (n + per - 1) / per;
      const PmodDiv pmod = make_pmod(parts);
      cfg.gridDim = (unsigned)blocks;
      cfg.blockDim = threads;
      cfg.dynamicSmemBytes = smem_hist ? sizeof(uint32_t) * parts : 0;
      // columns on their boundaries (not slices): no look at that per group, nor at the kind when there is one
      int kind = ks.n > 0 && (ks.kind[0] == KEY_I32 || ks.kind[0] == KEY_I64) ? ks.kind[0] : kMixed;
      if ((reinterpret_cast<uintptr_t>(pids) & 7) != 0) kind = kAny;
      for (int k = 0; k < ks.n && kind != kAny; k++) {
        const uint32_t wide_load = ks.kind[k] == KEY_I8 ? 4 : ks.kind[k] == KEY_I16 ? 8 : ks.kind[k] == KEY_BOOL ? 1 : 16;
        if ((reinterpret_cast<uintptr_t>(ks.values[k]) & (wide_load - 1)) != 0) kind = kAny;
        else if (ks.kind[k] != kind) kind = kMixed;
      }
      e = cudaLaunchKernelEx(&cfg, CountKernel(wide, smem_hist, kind), ks, n, per, pmod, pids, scratch);
    }
    if (e == cudaSuccess) {
      cfg.gridDim = (parts + 31) / 32;
      cfg.blockDim = dim3(32, 32);
      cfg.dynamicSmemBytes = 0;
      e = cudaLaunchKernelEx(&cfg, k_sum_tile_counts, (const uint32_t*)scratch, (uint32_t)blocks, parts, counts);
    }
  }
  if (prev >= 0 && prev != device) {
    cudaError_t e2 = cudaSetDevice(prev);
    if (e == cudaSuccess) e = e2;
  }
  if (e != cudaSuccess) {
    *msg = std::string("CUDA error: ") + cudaGetErrorString(e);
    return GZ_CUDA;
  }
  return GZ_OK;
}

}  // namespace gz
