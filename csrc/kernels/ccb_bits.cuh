// Bit-matrix transpose across a warp, shared by the codecs that store values as bit planes.
#pragma once
#include <stdint.h>

namespace ccb {

// Transposes the 32 x 32 bit matrix whose row i is the word held by lane i: afterwards
// lane j holds column j (bit i of the result = bit j of lane i's input). Five exchange steps;
// in each a lane keeps half of its bits and takes the other half from its partner's word: whole
// halfwords and bytes with one permute, smaller fields with a rotation and a three-input
// logical operation. The selectors depend on the lane alone and are hoisted out of loops:
// 13 instructions a transpose (with two shifts, two selects and the masks it was 30).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
  const uint32_t h = (lane & 16) ? 0x3276u : 0x5410u, b = (lane & 8) ? 0x3715u : 0x6240u;
  x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), h);
  x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), b);
#pragma unroll
  for (int s = 4; s >= 1; s >>= 1) {
    const uint32_t low = s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
    const bool up = (lane & s) != 0;
    const uint32_t keep = up ? ~low : low;
    const uint32_t p = __shfl_xor_sync(0xffffffffu, x, s);
    const uint32_t moved = __funnelshift_l(p, p, up ? 32 - s : s);   // what wraps round falls on kept bits
    x = (x & keep) | (moved & ~keep);
  }
  return x;
}

}  // namespace ccb
