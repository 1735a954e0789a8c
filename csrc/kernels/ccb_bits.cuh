// Bit-matrix transpose across a warp, shared by the codecs that store values as bit planes.
#pragma once
#include <stdint.h>

namespace ccb {

// Transposes the 32 x 32 bit matrix whose row i is the word held by lane i: afterwards
// lane j holds column j (bit i of the result = bit j of lane i's input). Five exchange steps;
// in each a lane keeps half of its bits and takes the other half from its partner's word: whole
// halfwords and bytes with one permute, smaller fields with a rotation and a three-input
// logical operation: 13 instructions. Selectors, rotations and masks are the lane's own. They are written
// as two operations each, because a choice between two constants is made again at every use
// instead of being kept in a register: 20 instructions a transpose.
struct Transpose32 {
  uint32_t half, byte, rot4, rot2, rot1, keep4, keep2, keep1;
  __device__ __forceinline__ explicit Transpose32(uint32_t lane) {
    half = 0x5410u + (lane >> 4 & 1u) * (0x3276u - 0x5410u);
    byte = 0x6240u + (lane >> 3 & 1u) * (0x3715u - 0x6240u);
    rot4 = 4u + (lane >> 2 & 1u) * 24u;
    rot2 = 2u + (lane >> 1 & 1u) * 28u;
    rot1 = 1u + (lane & 1u) * 30u;
    keep4 = 0x0f0f0f0fu << (lane & 4u);
    keep2 = 0x33333333u << (lane & 2u);
    keep1 = 0x55555555u << (lane & 1u);
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), half);
    x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), byte);
    auto step = [&](int s, uint32_t rot, uint32_t keep) {
      const uint32_t p = __shfl_xor_sync(0xffffffffu, x, s), moved = __funnelshift_l(p, p, rot);   // what wraps round falls on kept bits
      x = (x & keep) | (moved & ~keep);
    };
    step(4, rot4, keep4);
    step(2, rot2, keep2);
    step(1, rot1, keep1);
    return x;
  }
};
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) { return Transpose32((uint32_t)lane)(x); }

}  // namespace ccb
