// Copies between any two byte addresses by a group of threads (k_emit, the reader's k_read).
#pragma once
#include <stdint.h>

namespace gz {

// Bytes 4 * Q + sh / 8 .. + 16 of the 32 bytes a, b.
template <int Q>
__device__ __forceinline__ uint4 shift16(const uint4& a, const uint4& b, uint32_t sh) {
  const uint32_t w[9] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, 0u};
  return make_uint4(__funnelshift_r(w[Q], w[Q + 1], sh), __funnelshift_r(w[Q + 1], w[Q + 2], sh),
                    __funnelshift_r(w[Q + 2], w[Q + 3], sh), __funnelshift_r(w[Q + 3], w[Q + 4], sh));
}

// n 16-byte words of dst from the source bytes at phase s = 4 * Q + sh / 8 of the aligned word a.  Every
// word read holds bytes of the source (with s = 0 the second one of a pair is the first again).
template <int NT, int Q>
__device__ __forceinline__ void copy_words16(uint4* dst, const uint4* a, uint32_t n, uint32_t s, uint32_t t) {
  const uint32_t sh = (s & 3) * 8, up = s ? 1u : 0u;
#pragma unroll 4
  for (uint32_t i = t; i < n; i += NT) {
    const uint4 x = a[i], y = a[i + up];
    dst[i] = shift16<Q>(x, y, sh);
  }
}

// n bytes of src to dst by threads t = 0 .. NT - 1 (NT >= 16): aligned 16-byte words of the destination, each
// shifted together from two aligned source words, and up to 15 bytes at either end.
template <int NT>
__device__ __forceinline__ void copy_bytes(uint8_t* dst, const uint8_t* src, uint32_t n, uint32_t t) {
  const uint32_t head = min(n, (16u - ((uint32_t)reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
  if (t < head) dst[t] = src[t];
  dst += head;
  src += head;
  n -= head;
  const uint32_t s = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15), nw = n >> 4;
  const uint4* a = reinterpret_cast<const uint4*>(src - s);
  uint4* d = reinterpret_cast<uint4*>(dst);
  switch (s >> 2) {  // the same in the whole group
    case 0: copy_words16<NT, 0>(d, a, nw, s, t); break;
    case 1: copy_words16<NT, 1>(d, a, nw, s, t); break;
    case 2: copy_words16<NT, 2>(d, a, nw, s, t); break;
    default: copy_words16<NT, 3>(d, a, nw, s, t); break;
  }
  if (t < (n & 15)) dst[(nw << 4) + t] = src[(nw << 4) + t];
}

}  // namespace gz
