// Bit-matrix transpose across a warp, shared by the codecs that store values as bit planes.
#pragma once
#include <stdint.h>

namespace ccb {

// Transposes the 32 x 32 bit matrix whose row i is the word held by lane i: afterwards
// lane j holds column j (bit i of the result = bit j of lane i's input). Five exchange steps.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const uint32_t m = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t p = __shfl_xor_sync(0xffffffffu, x, s);
    const bool up = (lane & s) != 0;
    const uint32_t moved = up ? (p >> s) : (p << s);
    const uint32_t keep = up ? ~m : m;
    x = (x & keep) | (moved & ~keep);
  }
  return x;
}

}  // namespace ccb
