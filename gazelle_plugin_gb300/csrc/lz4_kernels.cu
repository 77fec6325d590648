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
__device__ uint32_t xxh32_short(const uint8_t* p, uint32_t n) {
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

__device__ __forceinline__ uint32_t le32(const uint8_t* p) {
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
//   k_lz4_blocks  gives every block a CTA that follows no long chain: where the next token would be is
//                 computed for every byte position at once; every thread resolves where a chain leaves
//                 its 32 positions, from the last one back, so one thread crosses the block in at most 256
//                 steps; the threads whose positions it enters list their tokens, the sequences' sizes
//                 are scanned, and every output byte's source is followed to a literal by pointer
//                 jumping.  Bound by instruction issue and shared memory (43 KiB: five CTAs per SM):
//                 67 us when the tokens were found by pointer doubling (ten rounds over all positions) and
//                 every byte was looked at in every round of jumping; 22 us less per map output now.
//                 Where a block's bytes go depends on the sizes of the blocks before it, so they
//                 go to a slot of their own
//   k_lz4_place   adds up the sizes and moves slots (and stored blocks) to their place
// A frame that is anything else (blocks that reach back into earlier ones, larger blocks, more
// blocks than slots, malformed) is decoded as a whole by one warp of k_lz4_place.
constexpr uint32_t kNoSlot = 0xffffffffu;      // the block cannot be decoded on its own
constexpr int kDT = 256;                       // threads per block
constexpr uint32_t kInStage = kLz4MaxBlock + 64;   // + the phase of its first byte
constexpr uint32_t kMaxSeq = kLz4MaxBlock / 4 + 1; // every match yields four bytes or more
constexpr uint32_t kSeqRoom = (kMaxSeq + 1 + 7) & ~7u;
constexpr uint32_t kPtrRoom = kLz4MaxBlock + 2 * (kLz4MaxBlock / 32);
constexpr size_t kDecodeSmem = kInStage + 2 * 2 * kPtrRoom;
static_assert(kLz4MaxBlock == kDT * 32, "32 positions per thread");
static_assert(4 * kSeqRoom <= kPtrRoom, "the sequences' arrays fit over the exits");
static_assert(kDecodeSmem <= 44 * 1024, "five CTAs per SM, no opt-in");
// index of position / output byte o in an array: a thread's 32 entries start in a bank of their own
__device__ __forceinline__ uint32_t swz(uint32_t o) { return o + 2 * (o >> 5); }

// Reads and checks a frame's header; false when malformed.  *pos: its first block.
__device__ bool frame_header(const uint8_t* s, uint64_t n, uint64_t* pos, bool* block_sum, bool* content_sum) {
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
// malformed, longer than `cap` or reaches back before its first byte.
__device__ uint32_t decode_staged(const uint8_t* in, uint32_t n, uint32_t cap, uint16_t* ptr, uint16_t* seq,
                                  uint16_t* entry, uint32_t* warp_sum, uint8_t* out) {
  const uint32_t t = threadIdx.x;
  uint16_t* start = seq;                 // first output byte of each sequence
  uint16_t* mst = seq + kSeqRoom;        // its first match byte
  uint16_t* lpos = seq + 2 * kSeqRoom;   // its literals in the input
  uint16_t* offs = seq + 3 * kSeqRoom;   // its match offset
  uint32_t lit, lp, ml;
  // next: where a sequence at each position would end: n the block's end, 0xffff nowhere
  uint16_t* next = ptr;
  for (uint32_t q = t; q < n; q += kDT) next[swz(q)] = (uint16_t)parse_seq(in, n, cap, q, &lit, &lp, &ml);
  entry[t] = 0xffff;
  __syncthreads();
  // leave: where the chain from each position first leaves its thread's 32 positions
  uint16_t* leave = seq;
  const uint32_t q0 = 32 * t, q1 = min(n, q0 + 32);
  for (uint32_t q = q1; q-- > q0;) {  // (not entered when q1 < q0)
    uint32_t x = next[swz(q)];
    if (x < q1) x = leave[swz(x)];
    leave[swz(q)] = (uint16_t)x;
  }
  __syncthreads();
  if (t == 0) {
    uint32_t q = 0;
    do {
      entry[q >> 5] = (uint16_t)q;
      q = leave[swz(q)];
    } while (q < n);
    warp_sum[kDT / 32] = q;
  }
  __syncthreads();
  if (warp_sum[kDT / 32] != n) return kNoSlot;
  // the chain's positions in order
  uint32_t nseq, total, mine = 0;
  for (uint32_t q = entry[t]; q < q1; q = next[swz(q)]) mine++;
  uint32_t k = cta_exscan(mine, warp_sum, &nseq);  // (its barriers: `leave` is read no more)
  if (nseq > kMaxSeq) return kNoSlot;
  for (uint32_t q = entry[t]; q < q1; q = next[swz(q)]) lpos[k++] = (uint16_t)q;
  __syncthreads();
  // sizes, output starts, offsets: a thread takes sequences [k0, k1)
  const uint32_t per = (nseq + kDT - 1) / kDT;
  const uint32_t k0 = min(nseq, t * per), k1 = min(nseq, k0 + per);
  uint32_t sum = 0;
  for (k = k0; k < k1; k++) {
    parse_seq(in, n, cap, lpos[k], &lit, &lp, &ml);
    lpos[k] = (uint16_t)lp;
    start[k] = (uint16_t)(lit + ml);  // at most 2 * cap
    mst[k] = (uint16_t)lit;
    offs[k] = ml ? (uint16_t)((uint32_t)in[lp + lit] | (uint32_t)in[lp + lit + 1] << 8) : (uint16_t)0;
    sum += lit + ml;
  }
  uint32_t o = cta_exscan(sum, warp_sum, &total);
  if (total > cap) return kNoSlot;
  bool bad = false;
  for (k = k0; k < k1; k++) {
    const uint32_t len = start[k], l = mst[k];
    start[k] = (uint16_t)o;
    mst[k] = (uint16_t)(o + l);
    if (len > l) bad |= offs[k] == 0 || offs[k] > o + l;
    o += len;
  }
  if (t == 0) start[nseq] = (uint16_t)total;
  if (__syncthreads_or(bad)) return kNoSlot;
  // every output byte's source: a literal (bit 15 and its input position) or an earlier output byte
  {
    const uint32_t o0 = 32 * t, o1 = min(total, o0 + 32);
    if (o0 < o1) {
      uint32_t lo = 0, hi = nseq;  // start[lo] <= o0 < start[hi]
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (start[mid] <= o0) lo = mid;
        else hi = mid;
      }
      uint32_t s0 = start[lo], s1 = start[lo + 1], m0 = mst[lo], l0 = lpos[lo], f0 = offs[lo];
      for (o = o0; o < o1; o++) {
        while (o >= s1) {
          lo++;
          s0 = s1;
          s1 = start[lo + 1];
          m0 = mst[lo];
          l0 = lpos[lo];
          f0 = offs[lo];
        }
        uint32_t v;
        if (o < m0) {
          v = 0x8000u | (l0 + o - s0);
        } else {
          // byte d of a match repeats byte d mod offset of its source run
          uint32_t d = o - m0;
          if (d >= f0) d %= f0;
          v = m0 - f0 + d;
        }
        ptr[swz(o)] = (uint16_t)v;
      }
    }
  }
  __syncthreads();
  // every source followed to its literal (a pointer read while its owner moves it on is an
  // earlier one of the same chain: still right); thread t keeps bytes t + 256 j, bit j not there yet
  uint32_t todo = 0;
  for (uint32_t j = 0; j < (total + kDT - 1 - t) / kDT; j++) todo |= 1u << j;
  for (;;) {
    for (uint32_t m = todo; m; m &= m - 1) {
      const uint32_t j = __ffs(m) - 1, q = j * kDT + t;
      uint32_t v = ptr[swz(q)];
      if (!(v & 0x8000u)) {
        v = ptr[swz(v)];
        ptr[swz(q)] = (uint16_t)v;
      }
      if (v & 0x8000u) todo &= ~(1u << j);
    }
    if (!__syncthreads_or(todo)) break;
  }
  for (uint32_t w = t; w < (total + 3) >> 2; w += kDT) {
    // (bytes past the end come from whatever the array holds there, an index inside the stage)
    const uint32_t i = swz(4 * w);
    const uint32_t a = *reinterpret_cast<const uint32_t*>(ptr + i), b = *reinterpret_cast<const uint32_t*>(ptr + i + 2);
    const uint32_t x = in[a & 0x1fff] | (uint32_t)in[(a >> 16) & 0x1fff] << 8 | (uint32_t)in[b & 0x1fff] << 16 |
                       (uint32_t)in[(b >> 16) & 0x1fff] << 24;
    reinterpret_cast<uint32_t*>(out)[w] = x;
  }
  return total;
}

// One CTA per (frame, block ordinal): block `i` of frame `fi` into slot frames[fi].slot0 + i.
__global__ void __launch_bounds__(kDT, 5) k_lz4_blocks(const Lz4Frame* __restrict__ frames, const uint32_t* __restrict__ frame_of,
                                                       Lz4Slot* __restrict__ slots, uint8_t* __restrict__ slot_mem) {
  extern __shared__ __align__(16) uint8_t dsm[];
  __shared__ uint16_t entry[kDT];
  __shared__ uint32_t warp_sum[kDT / 32 + 1];
  const uint32_t g = blockIdx.x;
  const Lz4Frame fr = frames[frame_of[g]];
  const uint32_t i = g - fr.slot0;
  const uint8_t* s = fr.src;
  const uint64_t n = fr.src_len;
  Lz4Slot sl{0, 0, kNoSlot, 0};  // a bad frame, or a block that cannot be decoded on its own
  uint64_t pos = 0;
  bool block_sum = false, content_sum = false;
  bool ok = n < (1ull << 31) && frame_header(s, n, &pos, &block_sum, &content_sum);
  uint32_t sz = 0;
  bool stored = false;
  for (uint32_t b = 0; ok; b++) {  // (every thread walks the headers: uniform loads)
    if (n - pos < 4) {
      ok = false;
      break;
    }
    const uint32_t bs = le32(s + pos);
    pos += 4;
    if (bs == 0) {  // end mark: fewer than i + 1 blocks
      sl.size = 0;
      sl.state = 1;
      ok = false;
      break;
    }
    sz = bs & 0x7FFFFFFFu;
    stored = bs & 0x80000000u;
    if (sz > n - pos || (block_sum && n - pos - sz < 4)) {
      ok = false;
      break;
    }
    if (b == i) break;
    pos += sz + (block_sum ? 4 : 0);
  }
  if (ok && i + 1 == fr.n_slots) {  // the last slot: the end mark must follow
    const uint64_t after = pos + sz + (block_sum ? 4 : 0);
    if (n - after < 4 || le32(s + after) != 0) ok = false;
  }
  if (ok) {
    sl.pos = (uint32_t)pos;
    if (stored) {
      sl.size = sz;
      sl.state = 2;
    } else if (sz > 0 && sz <= kLz4MaxBlock) {
      // the aligned 16-byte words that hold the block (they stay inside the stream's allocation)
      const uint8_t* src = s + pos;
      const uint32_t phase = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15);
      const uint4* a = reinterpret_cast<const uint4*>(src - phase);
      const uint32_t nw = (phase + sz + 15) >> 4;
      for (uint32_t q = threadIdx.x; q < nw; q += kDT) reinterpret_cast<uint4*>(dsm)[q] = __ldg(a + q);
      __syncthreads();
      const uint32_t slot = lz4_slot_bytes(fr.dst_len);
      uint16_t* ptr = reinterpret_cast<uint16_t*>(dsm + kInStage);
      sl.size = decode_staged(dsm + phase, sz, slot, ptr, ptr + kPtrRoom, entry, warp_sum,
                              slot_mem + fr.mem0 + (size_t)i * slot);
      if (sl.size != kNoSlot) sl.state = 3;
    }
  }
  if (threadIdx.x == 0) slots[g] = sl;
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

__global__ void __launch_bounds__(kWarps * 32) k_lz4_place(const Lz4Frame* __restrict__ frames,
                                                           const uint32_t* __restrict__ frame_of, uint32_t n_slots,
                                                           const Lz4Slot* __restrict__ slots,
                                                           const uint8_t* __restrict__ slot_mem, int32_t* err) {
  const uint32_t g = blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (g >= n_slots) return;
  const uint32_t lane = lane_id();
  const Lz4Frame fr = frames[frame_of[g]];
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
    if (i != 0) return;
    const bool ok = decode_frame(fr);
    if (!ok && lane == 0) atomicOr(err, 1);
    return;
  }
  const Lz4Slot sl = slots[g];
  if (sl.state == 2) copy_bytes<32>(fr.dst + before, fr.src + sl.pos, sl.size, lane);
  else if (sl.state == 3) copy_bytes<32>(fr.dst + before, slot_mem + fr.mem0 + (size_t)i * lz4_slot_bytes(fr.dst_len), sl.size, lane);
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 152;
  }
  return sms;
}

}  // namespace

uint32_t lz4_compress_warps() { return (uint32_t)sm_count() * kCBlocks * kCWarps; }

cudaError_t launch_lz4_compress(const Lz4Chunk* chunks, uint32_t n_chunks, uint32_t* next, uint8_t* scratch,
                                uint8_t* out, unsigned long long* out_used, unsigned long long out_cap,
                                Lz4Block* res, bool skip_stored, int32_t* err, cudaStream_t st) {
  if (n_chunks == 0) return cudaSuccess;
  const uint32_t grid = lz4_compress_warps() / kCWarps;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k_lz4_compress, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCompressSmem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  k_lz4_compress<<<grid, kCWarps * 32, kCompressSmem, st>>>(chunks, n_chunks, next, scratch, out, out_used, out_cap, res, skip_stored, err);
  return cudaGetLastError();
}

cudaError_t launch_lz4_decode(const Lz4Frame* frames, const uint32_t* frame_of, uint32_t n_slots, Lz4Slot* slots,
                              uint8_t* slot_mem, int32_t* err, cudaStream_t st) {
  if (n_slots == 0) return cudaSuccess;
  k_lz4_blocks<<<n_slots, kDT, kDecodeSmem, st>>>(frames, frame_of, slots, slot_mem);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_lz4_place<<<(n_slots + kWarps - 1) / kWarps, kWarps * 32, 0, st>>>(frames, frame_of, n_slots, slots, slot_mem, err);
  return cudaGetLastError();
}

}  // namespace gz
