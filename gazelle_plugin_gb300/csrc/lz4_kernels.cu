// sm_103a kernels of the LZ4_FRAME shuffle codec: block compression (the map side, emitted
// record-batch buffers) and frame decoding (the reduce side).
//
// The reference compresses each body buffer of an emitted record batch with Arrow's
// Lz4FrameCodec (splitter.cc:311-327, 586-600) through the LZ4 library on one CPU core; the
// buffer is written as an int64 uncompressed length followed by one LZ4 frame.  Here the
// buffers are cut into chunks of at most 8 KiB, each staged in shared memory and compressed by
// one warp into one LZ4 block (greedy single-candidate matching, hash table in shared memory:
// every read of the match search is a shared-memory read; 12 KiB of shared memory per warp, 18
// warps per SM), and the host strings the blocks of a buffer into a frame (independent blocks,
// 64 KiB maximum block size in the descriptor, no checksums).  The search is bound by the
// instructions of its dependent chains, so its speed follows the warps per SM and the instructions per
// sequence: against 64 KiB blocks searched in global memory, the Stop compression of the wide
// fact-table bodies runs 2.1x faster, for 1.9% more output (an 8 KiB history); 16 KiB blocks (8
// warps per SM) were 1.0x, 8 KiB blocks with a 4096-entry table (12 warps) 1.5x.  117 thousand
// instructions per block of the wide table's worded columns (94 MB: 2.6 ms, 51% of the issue slots)
// fell to 1.55 ms with short sequences written by one store, positions of the last window looked up
// again instead of read and hashed again, and chunks staged in 16-byte words from any phase.  The output is
// a valid frame for any LZ4 frame decoder; it is not the same byte string the LZ4 library would
// produce (the codec's output is not unique).
//
// Formats (published LZ4 block / frame descriptions):
//   block    sequences of [token: literal length << 4 | match length - 4][literal length
//            bytes when >= 15][literals][offset, 2 bytes LE][match length bytes when >= 15];
//            the last sequence has literals only; a match starts at least 12 bytes before the
//            end of the block and the last 5 bytes are literals
//   frame    magic 0x184D2204, FLG, BD, header checksum, blocks [size (bit 31: stored)]
//            [payload], end mark 0
#include <cuda_runtime.h>
#include <stdint.h>

#include "copy.cuh"
#include "device_info.h"
#include "lz4_kernels.h"

namespace gz {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 4;  // warps per CTA
constexpr int kHashLog = 11;
constexpr int kCWarps = 2;                       // warps per CTA of the compressor
constexpr int kCBlocks = 9;                      // resident CTAs per SM (shared memory)
constexpr uint32_t kStage = kLz4MaxBlock + 32;   // a warp's staged chunk, at its source's 16-byte phase
constexpr size_t kCompressSmem = (size_t)kCWarps * (kStage + (2u << kHashLog));
constexpr uint32_t kAgain = 24;  // window positions from which a new window is read instead (12, 20, 28, 32: 3, 0, 0, 10% slower)
constexpr uint16_t kEmpty = 0xffff;  // no position (position 65535 never starts a match)

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }

__device__ __forceinline__ uint32_t hash4(uint32_t v) { return (v * 2654435761u) >> (32 - kHashLog); }

// Length bytes of a literal or match length field >= 15: (x - 15) as 255s and a last byte < 255.
__device__ __forceinline__ uint32_t ext_bytes(uint32_t x) { return x >= 15 ? (x - 15) / 255 + 1 : 0; }
__device__ __forceinline__ void put_ext(uint8_t* p, uint32_t x, uint32_t nb) {
  for (uint32_t i = lane_id(); i < nb; i += 32) p[i] = i + 1 < nb ? 255 : (uint8_t)((x - 15) - 255 * (nb - 1));
}

// One sequence at dst + o: literals src[anchor, anchor + lit) then (when off != 0) a match of
// mlen bytes at distance off.  Returns the new output position (the same in every lane).
__device__ uint32_t emit(uint8_t* dst, uint32_t o, const uint8_t* src, uint32_t anchor, uint32_t lit,
                         uint32_t off, uint32_t mlen) {
  const uint32_t ml = off ? mlen - 4 : 0;
  if (lane_id() == 0) dst[o] = (uint8_t)(((lit < 15 ? lit : 15) << 4) | (ml < 15 ? ml : 15));
  const uint32_t nl = ext_bytes(lit);
  put_ext(dst + o + 1, lit, nl);
  o += 1 + nl;
  for (uint32_t i = lane_id(); i < lit; i += 32) dst[o + i] = src[anchor + i];
  o += lit;
  if (off) {
    if (lane_id() == 0) {
      dst[o] = (uint8_t)(off & 255);
      dst[o + 1] = (uint8_t)(off >> 8);
    }
    const uint32_t nm = ext_bytes(ml);
    put_ext(dst + o + 2, ml, nm);
    o += 2 + nm;
  }
  return o;
}

// A sequence like emit's whose lengths fit its token: lane j writes byte j, with one store.
__device__ __forceinline__ uint32_t emit_short(uint8_t* dst, uint32_t o, const uint8_t* src, uint32_t anchor, uint32_t lit,
                                               uint32_t off, uint32_t ml) {
  const uint32_t j = lane_id();
  uint32_t b = lit << 4 | ml;
  if (j > lit) b = j == lit + 1 ? off : off >> 8;
  if (j - 1 < lit) b = src[anchor + j - 1];
  if (j < lit + 3) dst[o + j] = (uint8_t)b;
  return o + lit + 3;
}

// Compresses the staged src[0, n) (n <= kLz4MaxBlock) into dst (room for n + n / 255 + 16 bytes); returns the
// block's size.  Positions are scanned 32 at a time: every lane hashes its position's 4 bytes and
// looks up the last earlier position with that hash; the first lane whose candidate matches
// starts the match, which the warp then extends 32 bytes at a time.  Table entries come only from
// earlier windows (inserted after the lookups), so a candidate always precedes its position.
__device__ uint32_t compress_block(const uint8_t* src, uint32_t n, uint16_t* table, uint8_t* dst) {
  const uint32_t lane = lane_id();
  const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3);
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(src - ph);
  // little-endian 4 bytes at position q (q + 8 <= n)
  auto read4 = [&](uint32_t q) {
    const uint32_t i = ph + q;
    return __funnelshift_r(sw[i >> 2], sw[(i >> 2) + 1], (i & 3) * 8);
  };
  uint32_t o = 0, anchor = 0, p = 0;
  uint32_t misses = 0;  // windows in a row without a match
  if (n >= 13) {
    for (uint32_t i = lane; i < (1u << kHashLog) / 8; i += 32)
      reinterpret_cast<uint4*>(table)[i] = make_uint4(~0u, ~0u, ~0u, ~0u);  // kEmpty: past every position
    __syncwarp();
    while (p + 12 <= n) {
      const uint32_t q = p + lane;
      const bool valid = q + 12 <= n;
      uint32_t v = 0, h = 0, cand = kEmpty;
      if (valid) {
        v = read4(q);
        h = hash4(v);
        cand = table[h];
      }
      bool ok = cand < q && read4(cand) == v;
      unsigned m = __ballot_sync(kFull, ok);
      __syncwarp();
      if (m == 0) {
        if (valid) table[h] = (uint16_t)q;
        __syncwarp();
        // acceleration (as LZ4's fast mode): the longer no match turns up, the further the next
        // window jumps, the positions in between staying literals; incompressible data costs a
        // fraction of a full scan
        misses++;
        p += 32u << min(misses >> 3, 4u);
        continue;
      }
      misses = 0;
      const uint32_t base = p;
      for (uint32_t first = 0;;) {
        // the match of lane f, the first with one from position base + first on
        const uint32_t f = __ffs(m) - 1;
        if (valid && lane >= first && lane <= f) table[h] = (uint16_t)q;  // positions up to the match start only
        const uint32_t mq = base + f;
        const uint32_t mc = __shfl_sync(kFull, cand, f);
        __syncwarp();
        uint32_t len = 4;
        for (;;) {  // the match may end at n - 5 at the latest
          const uint32_t a = mq + len + lane;
          const bool eq = a + 5 < n && src[a] == src[mc + len + lane];
          const unsigned ne = __ballot_sync(kFull, !eq);
          if (ne == 0) {
            len += 32;
            continue;
          }
          len += __ffs(ne) - 1;
          break;
        }
        const uint32_t lit = mq - anchor;
        o = lit < 15 && len < 19 ? emit_short(dst, o, src, anchor, lit, mq - mc, len - 4)
                                 : emit(dst, o, src, anchor, lit, mq - mc, len);
        p = mq + len;
        anchor = p;
        // The next window starts at p; a match of a position both windows hold is its first match as well,
        // found by looking those positions up again (their bytes and hashes are at hand)
        first = p - base;
        if (first >= kAgain) break;
        cand = valid && lane >= first ? table[h] : kEmpty;
        ok = cand < q && read4(cand) == v;
        m = __ballot_sync(kFull, ok);
        __syncwarp();
        if (m == 0) break;
      }
    }
  }
  o = emit(dst, o, src, anchor, n - anchor, 0, 0);
  return o;
}

__global__ void __launch_bounds__(kCWarps * 32, kCBlocks)
k_lz4_compress(const Lz4Chunk* __restrict__ chunks, uint32_t n_chunks, uint32_t* next, uint8_t* scratch,
               uint8_t* out, unsigned long long* out_used, unsigned long long out_cap, Lz4Block* res,
               bool skip_stored, int32_t* err) {
  extern __shared__ __align__(16) uint8_t csm[];
  const uint32_t warp = threadIdx.x >> 5;
  uint8_t* sbuf = csm + (size_t)warp * (kStage + (2u << kHashLog));
  uint16_t* table = reinterpret_cast<uint16_t*>(sbuf + kStage);
  uint8_t* slot = scratch + (size_t)(blockIdx.x * kCWarps + warp) * kLz4Slot;
  for (;;) {
    uint32_t c = 0;
    if (lane_id() == 0) c = atomicAdd(next, 1u);
    c = __shfl_sync(kFull, c, 0);
    if (c >= n_chunks) return;
    const Lz4Chunk ch = chunks[c];
    const uint32_t n = ch.raw || ch.len <= kLz4MaxBlock ? ch.len : 0;  // the host cuts blocks to 64 KiB
    uint32_t size = n;
    if (!ch.raw) {
      // the chunk into this warp's shared buffer: the aligned 16-byte words that hold it (each holds a
      // byte of the chunk, so none is outside its allocation)
      const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(ch.src) & 15);
      const uint4* a = reinterpret_cast<const uint4*>(ch.src - phase);
#pragma unroll 4
      for (uint32_t i = lane_id(); i < (phase + n + 15) >> 4; i += 32) reinterpret_cast<uint4*>(sbuf)[i] = __ldg(a + i);
      __syncwarp();
      size = compress_block(sbuf + phase, n, table, slot);
      __syncwarp();
    }
    const bool stored = size >= n;  // a plain copy, or no gain: the block is stored as it is
    if (stored) size = n;
    if (stored && skip_stored) {
      if (lane_id() == 0) res[c] = Lz4Block{0, n, 1u};
      __syncwarp();
      continue;
    }
    unsigned long long pos = 0;
    if (lane_id() == 0) pos = atomicAdd(out_used, (unsigned long long)((size + 15) & ~15u));
    pos = __shfl_sync(kFull, pos, 0);
    if (pos + size > out_cap) {
      if (lane_id() == 0) {
        atomicOr(err, 1);
        res[c] = Lz4Block{0, 0, 0};
      }
      continue;
    }
    uint8_t* d = out + pos;  // 16-byte aligned, like the slot
    if (stored) {
      const uintptr_t a = reinterpret_cast<uintptr_t>(ch.src);
      if ((a & 15) == 0) {
        const uint32_t nv = n >> 4;
        for (uint32_t i = lane_id(); i < nv; i += 32)
          reinterpret_cast<uint4*>(d)[i] = __ldg(reinterpret_cast<const uint4*>(ch.src) + i);
        for (uint32_t i = (nv << 4) + lane_id(); i < n; i += 32) d[i] = __ldg(ch.src + i);
      } else if ((a & 3) == 0) {
        const uint32_t nv = n >> 2;
        for (uint32_t i = lane_id(); i < nv; i += 32)
          reinterpret_cast<uint32_t*>(d)[i] = __ldg(reinterpret_cast<const uint32_t*>(ch.src) + i);
        for (uint32_t i = (nv << 2) + lane_id(); i < n; i += 32) d[i] = __ldg(ch.src + i);
      } else {
        // unaligned source: aligned destination words, each a funnel shift of two aligned source
        // words (both hold bytes of the chunk), then the last bytes one by one
        const uint32_t* base = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
        const uint32_t sh = (uint32_t)(a & 3) * 8;
        const uint32_t nv = n >> 2;
        for (uint32_t i = lane_id(); i < nv; i += 32)
          reinterpret_cast<uint32_t*>(d)[i] = __funnelshift_r(__ldg(base + i), __ldg(base + i + 1), sh);
        for (uint32_t i = (nv << 2) + lane_id(); i < n; i += 32) d[i] = __ldg(ch.src + i);
      }
    } else {
      const uint32_t nv = size >> 4;
      for (uint32_t i = lane_id(); i < nv; i += 32)
        reinterpret_cast<uint4*>(d)[i] = reinterpret_cast<const uint4*>(slot)[i];
      for (uint32_t i = (nv << 4) + lane_id(); i < size; i += 32) d[i] = slot[i];
    }
    if (lane_id() == 0) res[c] = Lz4Block{pos, size, stored ? 1u : 0u};
    __syncwarp();
  }
}

// ---- decoding ---------------------------------------------------------------------------

// xxHash32 of a few bytes (the frame descriptor), seed 0: the published algorithm's path for
// inputs shorter than 16 bytes.
__host__ __device__ uint32_t xxh32_short(const uint8_t* p, uint32_t n) {
  constexpr uint32_t P1 = 2654435761u, P2 = 2246822519u, P3 = 3266489917u, P4 = 668265263u, P5 = 374761393u;
  uint32_t h = P5 + n;
  uint32_t i = 0;
  for (; i + 4 <= n; i += 4) {
    const uint32_t w = (uint32_t)p[i] | (uint32_t)p[i + 1] << 8 | (uint32_t)p[i + 2] << 16 | (uint32_t)p[i + 3] << 24;
    h += w * P3;
    h = ((h << 17) | (h >> 15)) * P4;
  }
  for (; i < n; i++) {
    h += p[i] * P5;
    h = ((h << 11) | (h >> 21)) * P1;
  }
  h ^= h >> 15;
  h *= P2;
  h ^= h >> 13;
  h *= P3;
  h ^= h >> 16;
  return h;
}

__host__ __device__ __forceinline__ uint32_t le32(const uint8_t* p) {
  return (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24;
}

// Decodes one LZ4 block src[0, n) into dst at *op (capacity cap); matches may reach back into the
// frame's earlier blocks.  Every read and write is checked; false on malformed input.
__device__ bool decode_block(const uint8_t* src, uint32_t n, uint8_t* dst, uint64_t cap, uint64_t* op) {
  uint64_t o = *op;
  uint32_t ip = 0;
  while (ip < n) {
    const uint32_t token = src[ip++];
    uint32_t lit = token >> 4;
    if (lit == 15) {
      uint32_t b;
      do {
        if (ip >= n) return false;
        b = src[ip++];
        lit += b;
      } while (b == 255);
    }
    if (lit > n - ip || lit > cap - o) return false;
    for (uint32_t i = lane_id(); i < lit; i += 32) dst[o + i] = src[ip + i];
    ip += lit;
    o += lit;
    if (ip == n) break;
    if (n - ip < 2) return false;
    const uint32_t off = (uint32_t)src[ip] | (uint32_t)src[ip + 1] << 8;
    ip += 2;
    if (off == 0 || off > o) return false;
    uint32_t ml = token & 15;
    if (ml == 15) {
      uint32_t b;
      do {
        if (ip >= n) return false;
        b = src[ip++];
        ml += b;
      } while (b == 255);
    }
    ml += 4;
    if (ml > cap - o) return false;
    __syncwarp();  // the bytes a match copies are written
    // byte i of a match repeats byte i mod off of its source run, so overlapping copies read
    // only bytes written before the match
    for (uint32_t i = lane_id(); i < ml; i += 32) dst[o + i] = dst[o - off + (i % off)];
    __syncwarp();
    o += ml;
  }
  *op = o;
  return true;
}

// ---- frames decoded block by block ---------------------------------------------------------
// A block is a serial chain (each token says where the next one is, each match may copy what the
// last one wrote).  One warp per frame followed it from global memory: 5.3 ms for a map output of
// three wide record batches (100 frames, 1.4 MB decoded), most SMs idle; one warp per block, staged
// in shared memory: 261 us, still the chain (about 1000 sequences of 500 cycles).  The frames the
// splitter writes hold independent blocks of at most kLz4MaxBlock bytes, so here
//   lz4_index     finds the blocks from the frames' headers, on the host while the device reads the stream
//   k_lz4_blocks  gives every block a CTA that follows no long chain: where the next token would be is
//                 computed for every byte position at once; a warp's shuffles find where the chain from each
//                 of 32 positions leaves them, one pass more where it leaves a warp's 512; so one thread
//                 crosses the block in at most 16 steps and one a warp its part in 16 more; the threads
//                 whose positions are entered list their tokens, the sequences' sizes are scanned, and
//                 every output byte's source is followed to a literal by pointer jumping, 16 bytes in a
//                 thread's registers.  Bound by instruction issue (parsing every position and the sources
//                 take a fifth each; 16 warps, two CTAs per SM: three spilled or, with 40 registers,
//                 took longer for the last ones to finish).  Both kernels for a map output of 242
//                 compressed blocks: 80 us with the tokens found by ten rounds of pointer doubling, 55
//                 with a thread per 32 positions and 256 steps, 35 now.
//                 Where a block's bytes go depends on the sizes of the blocks before it, so they
//                 go to a slot of their own
//   k_lz4_place   adds up the sizes and moves slots (and stored blocks) to their place, 128 threads each (a
//                 warp each took 12 us)
// A frame that is anything else (blocks that reach back into earlier ones, larger blocks, more
// blocks than slots, malformed) is decoded as a whole by one warp of k_lz4_place.
constexpr uint32_t kNoSlot = kLz4NoSlot;
constexpr int kDT = 512;                       // threads per block
constexpr int kSegs = kLz4MaxBlock / 32;       // segments of 32 positions, a warp's lanes each
constexpr int kGroups = kDT / 32;              // groups of segments, a warp each
constexpr int kOut = kLz4MaxBlock / kDT;       // output bytes of a thread
constexpr uint32_t kInStage = kLz4MaxBlock + 64;   // + the phase of its first byte
constexpr uint32_t kMaxSeq = kLz4MaxBlock / 4 + 1; // every match yields four bytes or more
constexpr uint32_t kPosRoom = kLz4MaxBlock + 2 * kSegs;
constexpr uint32_t kPtrRoom = kLz4MaxBlock + 2 * kDT;
constexpr uint32_t kChainEnd = kPosRoom - 2;   // entries that no position has: the block's end reached,
constexpr uint32_t kChainBad = kPosRoom - 1;   // or a sequence that cannot be
struct __align__(8) Seq {
  uint16_t start, mst;  // its first output byte, its first match byte
  uint16_t lpos, offs;  // its literals in the input, its match offset
};
constexpr size_t kDecodeSmem = kInStage + 2 * (kPtrRoom + 2 * kPosRoom);
static_assert(kOut == 16 && kSegs % kGroups == 0, "a thread's bytes go out in one store");
static_assert(kPtrRoom >= kPosRoom && sizeof(Seq) * (kMaxSeq + 1) <= 2 * kPosRoom, "what lies over what");
static_assert(kDecodeSmem <= 61 * 1024, "three CTAs per SM");
// index of position o (swz: a segment's 32 entries start in a bank of their own) and of output byte o
// (a thread's 16)
__device__ __forceinline__ uint32_t swz(uint32_t o) { return o + 2 * (o >> 5); }
__device__ __forceinline__ uint32_t swz_out(uint32_t o) { return o + 2 * (o >> 4); }

// Reads and checks a frame's header; false when malformed.  *pos: its first block.
__host__ __device__ bool frame_header(const uint8_t* s, uint64_t n, uint64_t* pos, bool* block_sum, bool* content_sum) {
  if (n < 7 || le32(s) != 0x184D2204u) return false;
  const uint8_t flg = s[4], bd = s[5];
  *block_sum = flg & 0x10;
  *content_sum = flg & 0x04;
  const uint64_t p = 6 + ((flg & 0x08) ? 8 : 0) + ((flg & 0x01) ? 4 : 0);
  if (!((flg >> 6) == 1 && (bd & 0x8F) == 0 && n > p && s[p] == (uint8_t)((xxh32_short(s + 4, (uint32_t)(p - 4)) >> 8) & 0xFF)))
    return false;
  *pos = p + 1;
  return true;
}

// The sequence at position `at` of the staged block in[0, n): its literals, and its match (ml 0:
// the block ends with the literals).  Returns the position after it, or kNoSlot when it is cut off or
// longer than `cap`.
__device__ __forceinline__ uint32_t parse_seq(const uint8_t* in, uint32_t n, uint32_t cap, uint32_t at, uint32_t* lit,
                                              uint32_t* lpos, uint32_t* ml) {
  const uint32_t token = in[at];
  uint32_t p = at + 1, l = token >> 4, b;
  if (l == 15) {
    do {
      if (p >= n) return kNoSlot;
      b = in[p++];
      l += b;
    } while (b == 255 && l <= cap);
  }
  if (l > n - p || l > cap) return kNoSlot;
  *lit = l;
  *lpos = p;
  *ml = 0;
  p += l;
  if (p == n) return p;
  if (n - p < 2) return kNoSlot;
  p += 2;
  uint32_t m = token & 15;
  if (m == 15) {
    do {
      if (p >= n) return kNoSlot;
      b = in[p++];
      m += b;
    } while (b == 255 && m <= cap);
  }
  if (m + 4 > cap) return kNoSlot;
  *ml = m + 4;
  return p;
}

// Where the sequence at position `at` of the staged block ends, or kNoSlot when it is cut off; its lengths
// are checked where they are needed.  (A length byte is read before it is known to be inside the block:
// one byte past it at most, inside the stage.)
__device__ __forceinline__ uint32_t next_seq(const uint8_t* in, uint32_t n, uint32_t at) {
  const uint32_t token = in[at];
  uint32_t p = at + 1, b;
  if (token >= 0xf0) {
    b = in[p++];
    uint32_t l = b;
    while (b == 255 && p < n) {
      b = in[p++];
      l += b;
    }
    p += l;
  }
  p += token >> 4;
  if (p == n) return n;
  p += 2;
  if (p > n) return kNoSlot;
  if ((token & 15) == 15) {
    do {
      b = in[p++];
    } while (b == 255 && p < n);
    // (cut off when the last byte says that more follow)
    if (p > n || b == 255) return kNoSlot;
  }
  return p;
}

// Exclusive scan of x over the CTA; *total gets the sum.
__device__ __forceinline__ uint32_t cta_exscan(uint32_t x, uint32_t* warp_sum, uint32_t* total) {
  uint32_t inc = x;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, inc, o);
    if (lane_id() >= o) inc += y;
  }
  __syncthreads();  // earlier reads of warp_sum
  if (lane_id() == 31) warp_sum[threadIdx.x >> 5] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (int w = 0; w < kDT / 32; w++) {
    const uint32_t v = warp_sum[w];
    if (w < (int)(threadIdx.x >> 5)) before += v;
    all += v;
  }
  *total = all;
  return before + inc - x;
}

// Decodes the block staged at `in` (n >= 1 bytes) on its own, by the whole CTA, into `out` (global,
// 16-byte aligned, room for cap bytes rounded up to 16); returns its size, or kNoSlot when it is
// malformed, longer than `cap` or reaches back before its first byte.  mem: kPtrRoom + 2 kPosRoom entries.
__device__ uint32_t decode_staged(const uint8_t* in, uint32_t n, uint32_t cap, uint16_t* mem, uint8_t* out) {
  __shared__ uint16_t entry[kSegs], group[kGroups];
  __shared__ uint32_t warp_sum[kDT / 32 + 1];
  const uint32_t t = threadIdx.x, lane = lane_id(), warp = t >> 5;
  uint16_t* const next = mem;              // where a sequence at each position would end
  uint16_t* const leave = mem + kPtrRoom;  // the index where the chain from each position first leaves its segment
  uint16_t* const far = leave + kPosRoom;  // ... its warp's segments
  uint16_t* const ptr = mem;               // over next, later: every output byte's source
  Seq* const seq = reinterpret_cast<Seq*>(leave);  // over leave, later
  uint32_t lit, lp, ml;
  for (uint32_t q = t; q - lane < n; q += kDT) {
    uint32_t x = q < n ? next_seq(in, n, q) : kNoSlot;
    if (q < n) next[swz(q)] = (uint16_t)x;
    const uint32_t end = min(n, (q | 31) + 1);
#pragma unroll
    for (int r = 0; r < 4; r++) {  // a sequence with a match takes three bytes or more: at most 11 in 32
      const uint32_t y = __shfl_sync(kFull, x, x & 31);
      if (x < end) x = y;
    }
    if (q < n) leave[swz(q)] = (uint16_t)(x < n ? swz(x) : x == n ? kChainEnd : kChainBad);
  }
  if (t < kSegs) entry[t] = 0xffff;
  if (t < kGroups) group[t] = 0xffff;
  __syncthreads();
  constexpr uint32_t kIn = kSegs / kGroups;  // segments of a warp
  for (uint32_t s = kIn; s-- > 0;) {
    const uint32_t q = (warp * kIn + s) * 32 + lane;
    if (q < n) {
      const uint32_t x = leave[swz(q)];
      far[swz(q)] = (uint16_t)(x < min((warp + 1) * kIn * 34, kChainEnd) ? far[x] : x);
    }
    __syncwarp();
  }
  __syncthreads();
  // one thread crosses the block group by group, then one a group its segments
  if (t == 0) {
    uint32_t q = 0;
    for (; q < kChainEnd; q = far[q]) group[q / (kIn * 34)] = (uint16_t)q;
    warp_sum[kDT / 32] = q;
  }
  __syncthreads();
  if (warp_sum[kDT / 32] != kChainEnd) return kNoSlot;
  if (lane == 0)
    for (uint32_t q = group[warp]; q < min((warp + 1) * kIn * 34, kChainEnd); q = leave[q]) entry[q / 34] = (uint16_t)q;
  __syncthreads();
  // the chain's positions in order
  uint32_t nseq, total, mine = 0;
  const uint32_t q1 = min(n, 32 * t + 32);
  const uint32_t qe = t < kSegs && entry[t] != 0xffff ? entry[t] - 2 * t : 0xffff;
  for (uint32_t q = qe; q < q1; q = next[swz(q)]) mine++;
  uint32_t k = cta_exscan(mine, warp_sum, &nseq);  // (its barriers: `leave` is read no more)
  if (nseq > kMaxSeq) return kNoSlot;
  for (uint32_t q = qe; q < q1; q = next[swz(q)]) seq[k++].lpos = (uint16_t)q;
  __syncthreads();
  // sizes, output starts, offsets: a thread takes sequences [k0, k1)
  const uint32_t per = (nseq + kDT - 1) / kDT;
  const uint32_t k0 = min(nseq, t * per), k1 = min(nseq, k0 + per);
  uint32_t sum = 0;
  bool bad = false;
  for (k = k0; k < k1; k++) {
    if (parse_seq(in, n, cap, seq[k].lpos, &lit, &lp, &ml) == kNoSlot) {
      bad = true;
      break;
    }
    const uint32_t f = ml ? (uint32_t)in[lp + lit] | (uint32_t)in[lp + lit + 1] << 8 : 0u;
    seq[k] = Seq{(uint16_t)(lit + ml), (uint16_t)lit, (uint16_t)lp, (uint16_t)f};  // lit + ml: at most 2 * cap
    sum += lit + ml;
  }
  if (__syncthreads_or(bad)) return kNoSlot;
  uint32_t o = cta_exscan(sum, warp_sum, &total);
  if (total > cap) return kNoSlot;
  for (k = k0; k < k1; k++) {
    const uint32_t len = seq[k].start, l = seq[k].mst, f = seq[k].offs;
    seq[k].start = (uint16_t)o;
    seq[k].mst = (uint16_t)(o + l);
    if (len > l) bad |= f == 0 || f > o + l;
    o += len;
  }
  if (t == 0) seq[nseq].start = (uint16_t)total;
  if (__syncthreads_or(bad)) return kNoSlot;
  // the sources of the thread's bytes: a literal (bit 15 and its input position) or an earlier output byte
  const uint32_t o0 = kOut * t;
  uint32_t v[kOut];
#pragma unroll
  for (int u = 0; u < kOut; u++) v[u] = 0x8000u;
  if (o0 < total) {
    uint32_t lo = 0, hi = nseq;  // seq[lo].start <= o0 < seq[hi].start
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (seq[mid].start <= o0) lo = mid;
      else hi = mid;
    }
    Seq c = seq[lo], after = seq[lo + 1];
    // byte d of a match repeats byte d mod offset of its source run
    uint32_t d = o0 > c.mst ? o0 - c.mst : 0;
    if (d >= c.offs && d) d %= c.offs;
#pragma unroll
    for (int u = 0; u < kOut; u++) {
      o = o0 + u;
      if (o < total) {
        if (o >= after.start) {  // (only the last sequence can be empty)
          c = after;
          after = seq[++lo + 1];
          d = 0;
        }
        if (o < c.mst) {
          v[u] = 0x8000u | (c.lpos + o - c.start);
        } else {
          v[u] = c.mst - c.offs + d;
          if (++d == c.offs) d = 0;
        }
      }
    }
  }
  uint32_t* const own = reinterpret_cast<uint32_t*>(ptr + swz_out(o0));
#pragma unroll
  for (int u = 0; u < kOut; u += 2) own[u / 2] = v[u] | v[u + 1] << 16;
  __syncthreads();
  // every source followed to its literal (a pointer read while its owner moves it on is an
  // earlier one of the same chain: still right)
  for (bool open = true;;) {
    if (open) {
      open = false;
#pragma unroll
      for (int u = 0; u < kOut; u++)
        if (!(v[u] & 0x8000u)) {
          v[u] = ptr[swz_out(v[u])];
          open |= !(v[u] & 0x8000u);
        }
#pragma unroll
      for (int u = 0; u < kOut; u += 2) own[u / 2] = v[u] | v[u + 1] << 16;
    }
    if (!__syncthreads_or(open)) break;
  }
  if (o0 < total) {
    uint32_t x[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      x[u] = in[v[4 * u] & 0x1fff] | (uint32_t)in[v[4 * u + 1] & 0x1fff] << 8 | (uint32_t)in[v[4 * u + 2] & 0x1fff] << 16 |
             (uint32_t)in[v[4 * u + 3] & 0x1fff] << 24;
    reinterpret_cast<uint4*>(out)[t] = make_uint4(x[0], x[1], x[2], x[3]);
  }
  return total;
}

// One CTA per block.
__global__ void __launch_bounds__(kDT, 2) k_lz4_blocks(const Lz4Frame* __restrict__ frames, Lz4Slot* __restrict__ slots,
                                                       uint8_t* __restrict__ slot_mem, bool early) {
  extern __shared__ __align__(16) uint8_t dsm[];
  if (early) cudaTriggerProgrammaticLaunchCompletion();
  const Lz4Slot sl = slots[blockIdx.x];
  if (sl.state != 3) return;
  const Lz4Frame fr = frames[sl.frame];
  // the aligned 16-byte words that hold the block (they stay inside the stream's allocation)
  const uint8_t* src = fr.src + sl.pos;
  const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
  const uint4* a = reinterpret_cast<const uint4*>(src - phase);
  const uint32_t nw = (phase + sl.size + 15) >> 4;
  for (uint32_t q = threadIdx.x; q < nw; q += kDT) reinterpret_cast<uint4*>(dsm)[q] = __ldg(a + q);
  __syncthreads();
  const uint32_t slot = lz4_slot_bytes(fr.dst_len);
  const uint32_t size = decode_staged(dsm + phase, sl.size, slot, reinterpret_cast<uint16_t*>(dsm + kInStage),
                                      slot_mem + fr.mem0 + (size_t)(blockIdx.x - fr.slot0) * slot);
  if (threadIdx.x == 0) slots[blockIdx.x].size = size;
}

// The whole frame by one warp, its blocks in order (matches may reach back into earlier ones).
__device__ bool decode_frame(const Lz4Frame& fr) {
  const uint8_t* s = fr.src;
  const uint64_t n = fr.src_len;
  uint64_t pos = 0, o = 0;
  bool block_sum = false, content_sum = false;
  bool ok = frame_header(s, n, &pos, &block_sum, &content_sum);
  while (ok) {
    if (n - pos < 4) return false;
    const uint32_t bs = le32(s + pos);
    pos += 4;
    if (bs == 0) break;  // end mark
    const uint32_t sz = bs & 0x7FFFFFFFu;
    if (sz > n - pos || (block_sum && n - pos - sz < 4)) return false;
    if (bs & 0x80000000u) {  // stored
      if (sz > fr.dst_len - o) return false;
      for (uint32_t i = lane_id(); i < sz; i += 32) fr.dst[o + i] = s[pos + i];
      o += sz;
    } else {
      ok = decode_block(s + pos, sz, fr.dst, fr.dst_len, &o);
    }
    pos += sz + (block_sum ? 4 : 0);
    __syncwarp();
  }
  // (content checksums are skipped, not verified)
  if (ok && content_sum && n - pos < 4) ok = false;
  return ok && o == fr.dst_len;
}

__global__ void __launch_bounds__(kWarps * 32) k_lz4_place(const Lz4Frame* __restrict__ frames, const Lz4Slot* __restrict__ slots,
                                                           const uint8_t* __restrict__ slot_mem, int32_t* err) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  const uint32_t g = blockIdx.x, lane = lane_id();
  const Lz4Slot sl = slots[g];
  const Lz4Frame fr = frames[sl.frame];
  const uint32_t i = g - fr.slot0;
  // the frame's blocks: any that could not be decoded on its own, their sizes before this one
  uint64_t before = 0, total = 0;
  bool bad = false;
  for (uint32_t q0 = 0; q0 < fr.n_slots; q0 += 32) {
    const uint32_t q = q0 + lane;
    const uint32_t sz = q < fr.n_slots ? slots[fr.slot0 + q].size : 0u;
    bad |= __any_sync(kFull, sz == kNoSlot);
    uint64_t t = sz, p = q < i ? sz : 0u;
    for (int x = 16; x; x >>= 1) {
      t += __shfl_xor_sync(kFull, t, x);
      p += __shfl_xor_sync(kFull, p, x);
    }
    total += t;
    before += p;
  }
  bad = bad || total != fr.dst_len;
  // a frame with a content checksum is checked for it by decode_frame
  if (bad || (fr.src_len > 4 && (fr.src[4] & 0x04))) {
    if (i != 0 || threadIdx.x >= 32) return;
    const bool ok = decode_frame(fr);
    if (!ok && lane == 0) atomicOr(err, 1);
    return;
  }
  const uint8_t* from = sl.state == 2 ? fr.src + sl.pos : slot_mem + fr.mem0 + (size_t)i * lz4_slot_bytes(fr.dst_len);
  copy_bytes<kWarps * 32>(fr.dst + before, from, sl.size, threadIdx.x);
}

}  // namespace

uint32_t lz4_compress_warps() { return (uint32_t)SmCount() * kCBlocks * kCWarps; }

cudaError_t launch_lz4_compress(const Lz4Chunk* chunks, uint32_t n_chunks, uint32_t* next, uint8_t* scratch,
                                uint8_t* out, unsigned long long* out_used, unsigned long long out_cap,
                                Lz4Block* res, bool skip_stored, int32_t* err, cudaStream_t st) {
  if (n_chunks == 0) return cudaSuccess;
  const uint32_t grid = lz4_compress_warps() / kCWarps;
  const cudaError_t e = AllowSharedMemory((const void*)k_lz4_compress, kCompressSmem);
  if (e != cudaSuccess) return e;
  k_lz4_compress<<<grid, kCWarps * 32, kCompressSmem, st>>>(chunks, n_chunks, next, scratch, out, out_used, out_cap, res, skip_stored, err);
  return cudaGetLastError();
}

// The headers are a chain through the frame, 14 for a wide batch's worded column.  Followed by every
// block's CTA they took it a fifth of its time (5 of 27 thousand cycles, 14 at the end of such a frame), and
// its slots had to be guessed; the host follows them while the device reads the stream, all frames a step
// at a time, the next headers on their way.
void lz4_index(const uint8_t* const* src, Lz4Frame* frames, uint32_t n, std::vector<Lz4Slot>* slots, size_t* mem) {
  struct Walk {
    uint64_t pos = 0;
    size_t first = 0;  // its slots in `found`
    uint32_t room = 0, count = 0;
    bool block_sum = false, bad = false;
  };
  std::vector<Walk> w(n);
  std::vector<uint32_t> active(n);
  size_t room = 0;
  for (uint32_t k = 0; k < n; k++) {
    __builtin_prefetch(src[k]);
    active[k] = k;
    w[k].first = room;
    w[k].room = (uint32_t)std::min<uint64_t>(lz4_frame_slots(frames[k].dst_len), frames[k].src_len / 4 + 1);
    room += w[k].room;
  }
  std::vector<Lz4Slot> found(room);
  for (bool first = true; !active.empty(); first = false) {
    size_t left = 0;
    for (const uint32_t k : active) {
      Walk& x = w[k];
      const uint8_t* s = src[k];
      const uint64_t len = frames[k].src_len;
      if (first) {
        bool content_sum;
        x.bad = len >= (1ull << 31) || !frame_header(s, len, &x.pos, &x.block_sum, &content_sum);
      }
      if (x.bad || len - x.pos < 4) {
        x.bad = true;
        continue;
      }
      const uint32_t bs = le32(s + x.pos), sz = bs & 0x7FFFFFFFu;
      x.pos += 4;
      if (bs == 0) continue;  // end mark
      const bool stored = bs & 0x80000000u;
      if (x.count == x.room || sz > len - x.pos || (x.block_sum && len - x.pos - sz < 4) || (!stored && sz > kLz4MaxBlock)) {
        x.bad = true;
        continue;
      }
      found[x.first + x.count++] = Lz4Slot{(uint32_t)x.pos, k, sz, stored ? 2u : 3u};
      x.pos += sz + (x.block_sum ? 4 : 0);
      __builtin_prefetch(s + x.pos);
      active[left++] = k;
    }
    active.resize(left);
  }
  slots->clear();
  slots->reserve(room + n);
  *mem = 0;
  for (uint32_t k = 0; k < n; k++) {
    frames[k].slot0 = (uint32_t)slots->size();
    frames[k].mem0 = *mem;
    if (w[k].bad) slots->push_back(Lz4Slot{0, k, kNoSlot, 0});
    else if (w[k].count == 0) slots->push_back(Lz4Slot{0, k, 0, 1});
    else slots->insert(slots->end(), found.begin() + (ptrdiff_t)w[k].first, found.begin() + (ptrdiff_t)(w[k].first + w[k].count));
    frames[k].n_slots = (uint32_t)slots->size() - frames[k].slot0;
    *mem += (size_t)frames[k].n_slots * lz4_slot_bytes(frames[k].dst_len);
  }
}

void lz4_index_whole(Lz4Frame* frames, uint32_t n, std::vector<Lz4Slot>* slots) {
  slots->clear();
  for (uint32_t k = 0; k < n; k++) {
    frames[k].slot0 = k;
    frames[k].n_slots = 1;
    frames[k].mem0 = 0;
    slots->push_back(Lz4Slot{0, k, kNoSlot, 0});
  }
}

cudaError_t launch_lz4_decode(const Lz4Frame* frames, Lz4Slot* slots, uint32_t n_slots, uint8_t* slot_mem, int32_t* err,
                              cudaStream_t st) {
  if (n_slots == 0) return cudaSuccess;
  cudaError_t e = AllowSharedMemory((const void*)k_lz4_blocks, kDecodeSmem);
  if (e != cudaSuccess) return e;
  // the second comes up while the first runs, unless there are more blocks than can run at once: it would
  // hold what they wait for
  const bool early = n_slots <= 2u * (uint32_t)SmCount();
  k_lz4_blocks<<<n_slots, kDT, kDecodeSmem, st>>>(frames, slots, slot_mem, early);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = n_slots;
  cfg.blockDim = kWarps * 32;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_lz4_place, frames, (const Lz4Slot*)slots, (const uint8_t*)slot_mem, err);
}

}  // namespace gz
