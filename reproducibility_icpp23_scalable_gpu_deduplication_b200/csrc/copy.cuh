// Loads of the chunk copies (diff assembly and restart).
#pragma once
#include <cstring>

#include "common.cuh"

namespace b2d {

// 16 bytes of the buffer from byte s on (s + 16 <= len), whatever its alignment: two aligned
// 16-byte loads and a byte shift, or byte loads where an aligned load would leave the buffer
__device__ __forceinline__ uint4 load_unit(const uint8_t* data, uint64_t len, uint64_t s) {
  const uint8_t* p = data + s;
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 15u);
  if (mis == 0) return __ldg(reinterpret_cast<const uint4*>(p));
  uint4 r;
  if (s < mis || len - s < 32u - mis) {
    uint8_t t[16];
#pragma unroll
    for (int b = 0; b < 16; b++) t[b] = p[b];
    memcpy(&r, t, 16);
    return r;
  }
  const uint4* q = reinterpret_cast<const uint4*>(p - mis);
  const uint4 lo = __ldg(q), hi = __ldg(q + 1);
  uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  if (mis & 8u) {
#pragma unroll
    for (int i = 0; i < 6; i++) w[i] = w[i + 2];
  }
  if (mis & 4u) {
#pragma unroll
    for (int i = 0; i < 5; i++) w[i] = w[i + 1];
  }
  const uint32_t sh = 8u * (mis & 3u);
  r.x = __funnelshift_r(w[0], w[1], sh);
  r.y = __funnelshift_r(w[1], w[2], sh);
  r.z = __funnelshift_r(w[2], w[3], sh);
  r.w = __funnelshift_r(w[3], w[4], sh);
  return r;
}

// an asynchronous copy of a 16-byte piece to shared memory (`bytes` of it, the rest zeros)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// 16 bytes from byte m (< 16) of a piece on, the rest from the next piece
__device__ __forceinline__ uint4 shift_piece(const uint4& lo, const uint4& hi, uint32_t m) {
  uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
  for (int i = 0; i < 6; i++) w[i] = m & 8u ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 5; i++) w[i] = m & 4u ? w[i + 1] : w[i];
  const uint32_t s = 8u * (m & 3u);
  return make_uint4(__funnelshift_r(w[0], w[1], s), __funnelshift_r(w[1], w[2], s), __funnelshift_r(w[2], w[3], s),
                    __funnelshift_r(w[3], w[4], s));
}
}  // namespace b2d
