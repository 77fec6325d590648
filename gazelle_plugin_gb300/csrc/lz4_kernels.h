// LZ4_FRAME codec kernels (lz4_kernels.cu): block compression of buffer chunks and frame decoding.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace gz {

constexpr uint32_t kLz4MaxBlock = 8192;  // bytes of input per block (at most the frame's 64 KiB block size)
// worst-case compressed block (all literals: token, length bytes) rounded to 16 bytes
constexpr uint32_t kLz4Slot = ((kLz4MaxBlock + kLz4MaxBlock / 255 + 16) + 15) & ~15u;

struct Lz4Chunk {  // one block's input: 1 .. kLz4MaxBlock bytes (raw: any length, copied as it is)
  const uint8_t* src;
  uint32_t len;
  uint32_t raw;
};

struct Lz4Block {  // where a chunk's block landed in the output arena
  uint64_t pos;      // 16-byte aligned
  uint32_t size;     // payload bytes
  uint32_t stored;   // 1: the payload is the input itself (the frame marks it uncompressed)
};

struct Lz4Frame {  // one frame to decode: src_len bytes into exactly dst_len bytes
  const uint8_t* src;
  uint64_t src_len;
  uint8_t* dst;
  uint64_t dst_len;
  uint32_t slot0;    // its first block slot
  uint32_t n_slots;  // its slots: one a block, at least one
  uint64_t mem0;     // where the slots' memory starts (lz4_slot_bytes each)
};

struct Lz4Slot {  // one block of a frame
  uint32_t pos;    // its payload inside the frame
  uint32_t frame;
  uint32_t size;   // bytes of the payload, once decoded those it gives; kLz4NoSlot: not decodable on its own
  uint32_t state;  // 0: see size, 1: a frame without blocks, 2: stored, 3: compressed
};
constexpr uint32_t kLz4NoSlot = 0xffffffffu;

// Most block slots of a frame of dst_len bytes: blocks of kLz4MaxBlock bytes, and three shorter ones
// inside it (an offsets buffer starts with its own first offset, a batch may continue from an
// earlier device pass); a frame with more blocks is decoded by one warp.
inline uint32_t lz4_frame_slots(uint64_t dst_len) {
  return (uint32_t)((dst_len + kLz4MaxBlock - 1) / kLz4MaxBlock) + 3;
}

// Warps of the compression grid (each needs kLz4Slot bytes of scratch).
uint32_t lz4_compress_warps();

// Compresses every chunk into the arena `out` (out_cap bytes; *out_used is the bump counter,
// *next the work counter, both zero at launch); res[c] tells where chunk c went.  *err gets bit
// 0 when the arena ran out.  skip_stored: a chunk that does not shrink takes no room (its input is
// its payload).
cudaError_t launch_lz4_compress(const Lz4Chunk* chunks, uint32_t n_chunks, uint32_t* next, uint8_t* scratch,
                                uint8_t* out, unsigned long long* out_used, unsigned long long out_cap,
                                Lz4Block* res, bool skip_stored, int32_t* err, cudaStream_t st);

// Memory of one block slot of a frame of dst_len bytes (16-byte units; no block is longer).
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t lz4_slot_bytes(uint64_t dst_len) {
  return dst_len < kLz4MaxBlock ? ((uint32_t)dst_len + 15u) & ~15u : kLz4MaxBlock;
}

// Host: the blocks of n frames from their headers, every frame's slots in a row (slot0, n_slots and mem0
// of each frame are set; *mem gets the bytes of all slots).  src[k]: frame k's bytes in host memory.  A frame that is
// malformed or has more blocks than slots gets one slot that cannot be decoded on its own.
void lz4_index(const uint8_t* const* src, Lz4Frame* frames, uint32_t n, std::vector<Lz4Slot>* slots, size_t* mem);

// The same with one slot a frame that cannot be decoded on its own: the frames are decoded whole, without
// memory for slots (never more slots than lz4_index's).
void lz4_index_whole(Lz4Frame* frames, uint32_t n, std::vector<Lz4Slot>* slots);

// Decodes every frame; *err gets bit 0 for a malformed frame or a size that differs.  `slots` (n_slots of
// them, lz4_index's) are written, `slot_mem` is scratch.  The sources' allocations start and end on 16-byte
// boundaries.
cudaError_t launch_lz4_decode(const Lz4Frame* frames, Lz4Slot* slots, uint32_t n_slots, uint8_t* slot_mem, int32_t* err,
                              cudaStream_t st);

}  // namespace gz
