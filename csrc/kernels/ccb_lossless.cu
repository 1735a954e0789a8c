// Lossless float codec (f32 / bf16 / f16) on local memory, for the compression-hook ABI.
//
// The reference reaches a lossless GPU codec only through the external DietGPU library
// (userconfig/wrapper_code_examples/compression/dietgpu/dietgpu.cu:32-103:
// floatCompress / floatDecompress, exponents entropy-coded, the rest stored raw). This is
// an own sm_100a codec of the same shape: the exponent field of every value is split from
// sign and mantissa; sign and mantissa are stored raw in byte planes; the exponents of a
// block of 512 values are stored as (exponent - block minimum) in as many bit planes as the
// block's exponent range needs (0 to 8). Gradient-like and activation data keep the
// exponents of neighbouring values within a few octaves, so 3 to 5 planes replace 8 bits.
//
// Work decomposition: a warp owns a block of 512 values (16 per lane, like the other
// codecs); the bit planes are built, and read back, by bit-matrix transposes across the warp, one
// 32-bit word per (plane, element-of-lane). A CTA of 8 warps owns a TILE of
// 8 blocks = 4096 values and packs the variable-length exponent planes of its blocks
// back to back inside the tile's fixed-capacity slot:
//
//   container = [32-byte header][slot 0][slot 1]...          slot stride = 32 + 4096 * sizeof(T)
//   header    = u32 magic "CCBL", u32 dtype, u64 count, u64 used bytes (sum over slots), u64 0
//   slot      = u32 used bytes, u8 width[8], u8 kmin[8], 12 bytes 0,
//               rest section (fixed size): f32 3 byte planes of 4096 B (low, middle, sign|high)
//                                          bf16 1 byte plane (sign << 7 | mantissa)
//                                          f16 1 byte plane (mantissa low 8) + 3 bit planes
//                                              (mantissa bits 8, 9 and the sign), 48 words per block
//               exponent section: for block b, width[b] planes of 16 words:
//                                 word[p * 16 + j] bit l = bit p of (exponent - kmin[b]) of value 16 l + j
//
// A slot is never larger than its stride (8 planes = 1 byte per value = the raw exponent),
// so compression needs no size negotiation: a transport that wants the gain sends the
// `used` prefix of every slot, one that cannot (fixed-stride hooks) sends the stride.
#include <cuda_runtime.h>

#include "../rt/ccb_rt_internal.h"
#include "ccb_device.cuh"
#include "ccb_bits.cuh"
#include "ccb_lossless_layout.h"

namespace ccb {

constexpr int kLlThreads = 256;
constexpr int kLlBlocksPerTile = kLlThreads / 32;          // 8
constexpr int kLlTileElems = kLlBlocksPerTile * kWarpElems;  // 4096
constexpr uint32_t kLlMagic = 0x4C424343u;                 // "CCBL"
constexpr int kLlHeader = 32;
constexpr int kLlCtas = 4;   // resident on an SM

template <class T> struct LlTraits;
template <> struct LlTraits<float> {
  static constexpr int kExpShift = 23, kExpBits = 8, kRestBytesPerTile = 3 * kLlTileElems;
};
template <> struct LlTraits<__nv_bfloat16> {
  static constexpr int kExpShift = 7, kExpBits = 8, kRestBytesPerTile = kLlTileElems;
};
template <> struct LlTraits<__half> {
  static constexpr int kExpShift = 10, kExpBits = 5, kRestBytesPerTile = kLlTileElems + 3 * kLlTileElems / 8;
};

template <class T> __host__ __device__ constexpr size_t ll_slot_bytes() { return 32 + (size_t)kLlTileElems * sizeof(T); }

// Byte `k` of four words as one word.
__device__ __forceinline__ uint32_t bytes_of(uint32_t a, uint32_t b, uint32_t c, uint32_t d, int k) {
  const uint32_t pair = (uint32_t)k | ((uint32_t)(k + 4) << 4);
  return __byte_perm(__byte_perm(a, b, pair), __byte_perm(c, d, pair), 0x5410);
}

// Four words as a 4 x 4 matrix of bytes, transposed: its own inverse.
__device__ __forceinline__ void transpose_bytes(uint32_t (&w)[4]) {
  const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);   // bytes 0 and 1 of each
  const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);   // 2 and 3
  w[0] = __byte_perm(a, b, 0x5410);
  w[1] = __byte_perm(a, b, 0x7632);
  w[2] = __byte_perm(c, d, 0x5410);
  w[3] = __byte_perm(c, d, 0x7632);
}

// Bit planes of the 16 small values (8 bits at most) of each lane of a warp. The values 4 r + g
// (r = 0..3) of a lane share the word u[g], value 4 r + g in byte r; a 32 x 32 bit-matrix
// transpose of u[g] across the warp leaves plane p of value 4 r + g in lane 8 r + p. The four
// words of a lane are then the words 16 p + 4 r .. + 3 of the plane section: ONE 16-byte store
// by the lanes whose plane exists. Where four planes are enough, nearly always, two values share a
// byte and two transposes do: plane p of the values 2 s, 2 s + 1 comes to lane 4 s + p.
__device__ __forceinline__ void store_planes(uint32_t* section, uint32_t (&u)[4], int planes, int lane) {
  if (planes <= 4) {
    const uint32_t a = transpose32(u[0] + 16u * u[2], lane), b = transpose32(u[1] + 16u * u[3], lane);
    const int s = lane >> 2, p = lane & 3;
    if (p < planes) *reinterpret_cast<uint2*>(section + 16 * p + 2 * s) = make_uint2(a, b);
    return;
  }
#pragma unroll
  for (int g = 0; g < 4; ++g) u[g] = transpose32(u[g], lane);
  const int r = lane >> 3, p = lane & 7;
  if (p < planes) *reinterpret_cast<uint4*>(section + 16 * p + 4 * r) = make_uint4(u[0], u[1], u[2], u[3]);
}
// The words of a lane, as they lie in memory (two of them where four planes are enough), and the values from them.
__device__ __forceinline__ uint4 fetch_planes(const uint32_t* section, int planes, int lane) {
  uint4 q = make_uint4(0u, 0u, 0u, 0u);
  if (planes <= 4) {
    const int s = lane >> 2, p = lane & 3;
    if (p < planes) {
      const uint2 h = *reinterpret_cast<const uint2*>(section + 16 * p + 2 * s);
      q.x = h.x;
      q.y = h.y;
    }
  } else {
    const int r = lane >> 3, p = lane & 7;
    if (p < planes) q = *reinterpret_cast<const uint4*>(section + 16 * p + 4 * r);
  }
  return q;
}
__device__ __forceinline__ void values_of_planes(const uint4& q, uint32_t (&u)[4], int planes, int lane) {
  u[0] = transpose32(q.x, lane);
  u[1] = transpose32(q.y, lane);
  if (planes <= 4) {
    u[2] = (u[0] >> 4) & 0x0f0f0f0fu;
    u[3] = (u[1] >> 4) & 0x0f0f0f0fu;
    u[0] &= 0x0f0f0f0fu;
    u[1] &= 0x0f0f0f0fu;
  } else {
    u[2] = transpose32(q.z, lane);
    u[3] = transpose32(q.w, lane);
  }
}
// The words u[] of values held in pairs (value 2 k in the low half of w[k], byte `at` of each half), and back.
__device__ __forceinline__ void planes_of_pairs(const uint32_t (&w)[8], int at, uint32_t (&u)[4]) {
  u[0] = bytes_of(w[0], w[2], w[4], w[6], at);
  u[1] = bytes_of(w[0], w[2], w[4], w[6], at + 2);
  u[2] = bytes_of(w[1], w[3], w[5], w[7], at);
  u[3] = bytes_of(w[1], w[3], w[5], w[7], at + 2);
}
__device__ __forceinline__ void pairs_of_planes(const uint32_t (&u)[4], uint32_t (&w)[8]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {   // bytes r of u[0], u[1] are the values 4 r, 4 r + 1
    w[2 * r] = __byte_perm(u[0], u[1], (uint32_t)r | ((uint32_t)(r + 4) << 8)) & 0x00ff00ffu;
    w[2 * r + 1] = __byte_perm(u[2], u[3], (uint32_t)r | ((uint32_t)(r + 4) << 8)) & 0x00ff00ffu;
  }
}

// Both directions are bound by the pipe of the logical and byte operations or by their memory, and work
// on four values at a time as far as they can: the exponents and the bytes of sign and mantissa of four
// values are one word each. A tile's values are requested while the tile before is packed, and one
// barrier per tile passes the widths round. The decoder has the planes of the next tile and the head of
// the one after on their way; adding to fp32 values it has no registers for that (a 4 MiB chunk 5.2 us
// with, 4.4 without). 32 Mi bf16 values, encoding and decoding: 23.1 and 22.6 us (27.2 and 28.7 with two
// values at a time and four transposes a block); 32 Mi fp32 values 42.3 and 40.9. The memory needs 18
// and 38 each way. An fp32 encoder with 64 registers for a fourth CTA takes 43.3 us, on random bits 48 instead
// of 44; five or six CTAs of any kind are slower. (B200.)
template <class T>
__global__ void __launch_bounds__(kLlThreads, sizeof(T) == 4 ? 3 : kLlCtas) lossless_encode_kernel(const T* __restrict__ in, size_t count, char* out, size_t ntiles) {
  after_kernel_before();
  using Tr = LlTraits<T>;
  __shared__ uint2 info[2][kLlBlocksPerTile];   // (width, minimum) of each block, by parity of the tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t lane_at = (size_t)warp * kWarpElems + (size_t)lane * kLaneElems;
  unsigned long long produced = 0;
  size_t t = blockIdx.x;
  Wide16<T> next;
  if (t < ntiles) load16_wide<T>(in, t * kLlTileElems + lane_at, count, next);
  for (int parity = 0; t < ntiles; t += gridDim.x, parity ^= 1) {
    char* slot = out + kLlHeader + t * ll_slot_bytes<T>();
    const Wide16<T> raw = next;
    if (t + gridDim.x < ntiles) load16_wide<T>(in, (t + gridDim.x) * kLlTileElems + lane_at, count, next);
    char* restp = slot + 32 + warp * kWarpElems + lane * 16;
    uint32_t u[4], kmin, kmax;
    // sign and mantissa: raw byte planes (and for f16 three bit planes); then the exponents
    if constexpr (Tr::kExpBits == 8) {
      // high = sign and the exponent's upper seven bits, low = its last bit and seven of the mantissa
      uint32_t high[4], low[4], rest[4];
      [[maybe_unused]] uint32_t b0[4], b1[4];   // fp32: the two bytes below
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if constexpr (sizeof(T) == 4) {
          uint32_t w[4] = {raw.w[4 * r], raw.w[4 * r + 1], raw.w[4 * r + 2], raw.w[4 * r + 3]};
          transpose_bytes(w);
          b0[r] = w[0];
          b1[r] = w[1];
          low[r] = w[2];
          high[r] = w[3];
        } else {
          low[r] = __byte_perm(raw.w[2 * r], raw.w[2 * r + 1], 0x6420);
          high[r] = __byte_perm(raw.w[2 * r], raw.w[2 * r + 1], 0x7531);
        }
        rest[r] = (high[r] & 0x80808080u) | (low[r] & 0x7f7f7f7fu);
        u[r] = ((high[r] * 2u) & 0xfefefefeu) | ((low[r] >> 7) & 0x01010101u);
      }
      if constexpr (sizeof(T) == 4) {
        stg(restp, make_uint4(b0[0], b0[1], b0[2], b0[3]));
        stg(restp + kLlTileElems, make_uint4(b1[0], b1[1], b1[2], b1[3]));
      }
      stg(restp + (sizeof(T) == 4 ? 2 * kLlTileElems : 0), make_uint4(rest[0], rest[1], rest[2], rest[3]));
      // extremes of the bytes two at a time: odd bytes decide a halfword by themselves, even ones once shifted up
      uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t even = u[r] * 256u;
        lo = __vminu2(__vminu2(lo, u[r]), even);
        hi = __vmaxu2(__vmaxu2(hi, u[r]), even);
      }
      kmin = __reduce_min_sync(0xffffffffu, min(lo & 0xffffu, lo >> 16)) >> 8;
      kmax = __reduce_max_sync(0xffffffffu, max(hi & 0xffffu, hi >> 16)) >> 8;
#pragma unroll
      for (int r = 0; r < 4; ++r) u[r] -= kmin * 0x01010101u;
      transpose_bytes(u);
    } else {
      constexpr uint32_t kKey = ((1u << Tr::kExpBits) - 1u) * 0x00010001u;
      constexpr uint32_t kMan = ((1u << Tr::kExpShift) - 1u) * 0x00010001u;
      uint32_t key[8], rest[8], lo = kKey, hi = 0u;
#pragma unroll
      for (int k = 0; k < 8; ++k) {   // two values at a time
        key[k] = (raw.w[k] >> Tr::kExpShift) & kKey;
        rest[k] = (raw.w[k] & kMan) | ((raw.w[k] >> (15 - Tr::kExpShift)) & (0x00010001u << Tr::kExpShift));
        lo = __vminu2(lo, key[k]);
        hi = __vmaxu2(hi, key[k]);
      }
      stg(restp, make_uint4(__byte_perm(rest[0], rest[1], 0x6420), __byte_perm(rest[2], rest[3], 0x6420),
                            __byte_perm(rest[4], rest[5], 0x6420), __byte_perm(rest[6], rest[7], 0x6420)));
      if constexpr (Tr::kExpBits == 5) {
        uint32_t high[4];
        planes_of_pairs(rest, 1, high);
        store_planes(reinterpret_cast<uint32_t*>(slot + 32 + kLlTileElems) + warp * 48, high, 3, lane);
      }
      kmin = __reduce_min_sync(0xffffffffu, min(lo & 0xffffu, lo >> 16));
      kmax = __reduce_max_sync(0xffffffffu, max(hi & 0xffffu, hi >> 16));
#pragma unroll
      for (int k = 0; k < 8; ++k) key[k] -= kmin * 0x00010001u;
      planes_of_pairs(key, 0, u);
    }
    const int w = 32 - __clz((int)(kmax - kmin));   // 0 when all exponents are equal
    if (lane == 0) info[parity][warp] = make_uint2((uint32_t)w, kmin);
    __syncthreads();   // the other parity's words were read before this barrier's predecessor
    const uint2 mine = info[parity][lane & (kLlBlocksPerTile - 1)];
    const uint32_t off = __reduce_add_sync(0xffffffffu, lane < warp ? mine.x : 0u);
    // exponent planes of this block, behind those of the blocks before it
    store_planes(reinterpret_cast<uint32_t*>(slot + 32 + Tr::kRestBytesPerTile) + off * 16, u, w, lane);
    if (warp == 0) {
      const uint32_t all = __reduce_add_sync(0xffffffffu, lane < kLlBlocksPerTile ? mine.x : 0u);
      const uint32_t used = 32u + (uint32_t)Tr::kRestBytesPerTile + all * 64u;
      if (lane == 0) {
        *reinterpret_cast<uint32_t*>(slot) = used;
        produced += used;
      }
      if (lane < kLlBlocksPerTile) {
        reinterpret_cast<unsigned char*>(slot)[4 + lane] = (unsigned char)mine.x;
        reinterpret_cast<unsigned char*>(slot)[12 + lane] = (unsigned char)mine.y;
      }
      if (lane < 3) reinterpret_cast<uint32_t*>(slot)[5 + lane] = 0u;
    }
  }
  // The container's header was cleared before the launch; the byte count is summed over the
  // CTAs (one atomic each, not one per tile), block 0 adds the header's own bytes and the rest.
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      reinterpret_cast<uint32_t*>(out)[0] = kLlMagic;
      reinterpret_cast<uint32_t*>(out)[1] = sizeof(T) == 4 ? CCB_F32 : Tr::kExpBits == 8 ? CCB_BF16 : CCB_F16;
      reinterpret_cast<unsigned long long*>(out)[1] = count;
      produced += kLlHeader;
    }
    atomicAdd(reinterpret_cast<unsigned long long*>(out + 16), produced);
  }
}

// MODE 0: out = decoded values; MODE 1: out += decoded values (in T, one rounding)
template <class T, int MODE>
__global__ void __launch_bounds__(kLlThreads, kLlCtas) lossless_decode_kernel(const char* __restrict__ in, size_t count, T* out, size_t ntiles) {
  after_kernel_before();
  using Tr = LlTraits<T>;
  constexpr int kRest = sizeof(T) == 4 ? 3 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sh = 8 * (warp & 3);
  struct Head { uint4 h; uint32_t high_min; };   // used, widths 0-3, widths 4-7, minima 0-3; minima 4-7
  struct Body { uint4 rest[kRest], planes, high; uint32_t kmin; int w; };
  auto slot_of = [&](size_t t) { return in + kLlHeader + t * ll_slot_bytes<T>(); };
  auto mine = [&](size_t t) { return t < ntiles && t * kLlTileElems + (size_t)warp * kWarpElems < count; };
  auto head_of = [&](size_t t) -> Head {
    return Head{*reinterpret_cast<const uint4*>(slot_of(t)), *reinterpret_cast<const uint32_t*>(slot_of(t) + 16)};
  };
  auto body_of = [&](size_t t, const Head& d) -> Body {
    Body b;
    const char* slot = slot_of(t);
    const uint32_t wsel = warp < 4 ? d.h.y : d.h.z;
    b.w = (int)ccb_ll_planes((wsel >> sh) & 0xffu, Tr::kExpBits);
    b.kmin = ((warp < 4 ? d.h.w : d.high_min) >> sh) & 0xffu;
    const uint32_t off = ccb_ll_first_plane(__dp4a(wsel & ((1u << sh) - 1u), 0x01010101u, warp < 4 ? 0u : __dp4a(d.h.y, 0x01010101u, 0u)), warp, Tr::kExpBits);
    b.planes = fetch_planes(reinterpret_cast<const uint32_t*>(slot + 32 + Tr::kRestBytesPerTile) + off * 16, b.w, lane);
#pragma unroll
    for (int p = 0; p < kRest; ++p) b.rest[p] = *reinterpret_cast<const uint4*>(slot + 32 + warp * kWarpElems + lane * 16 + (size_t)p * kLlTileElems);
    if constexpr (Tr::kExpBits == 5) b.high = fetch_planes(reinterpret_cast<const uint32_t*>(slot + 32 + kLlTileElems) + warp * 48, 3, lane);
    return b;
  };
  size_t t = blockIdx.x;
  if (!mine(t)) return;   // only the last tile has blocks that hold nothing
  constexpr bool kAhead = sizeof(T) == 2 || MODE == 0;
  Head head = head_of(t);
  Body next;
  if (kAhead) {
    next = body_of(t, head);
    if (mine(t + gridDim.x)) head = head_of(t + gridDim.x);
  }
  for (;;) {
    if (!kAhead) next = body_of(t, head);
    const Body b = next;
    const size_t idx = t * kLlTileElems + (size_t)warp * kWarpElems + (size_t)lane * kLaneElems;
    t += gridDim.x;
    const bool more = mine(t);
    if (kAhead && more) {
      next = body_of(t, head);
      if (mine(t + gridDim.x)) head = head_of(t + gridDim.x);
    }
    if (!kAhead && more) head = head_of(t);
    [[maybe_unused]] Wide16<T> have;
    if constexpr (MODE == 1 && sizeof(T) == 2) load16_wide<T>(out, idx, count, have);
    uint32_t u[4];
    values_of_planes(b.planes, u, b.w, lane);
    Wide16<T> raw;
    if constexpr (Tr::kExpBits == 8) {
      transpose_bytes(u);   // values 4 r .. + 3 in word r, as the bytes of sign and mantissa lie
      const uint4 top = b.rest[kRest - 1];
      const uint32_t rest[4] = {top.x, top.y, top.z, top.w};
      [[maybe_unused]] const uint32_t b0[4] = {b.rest[0].x, b.rest[0].y, b.rest[0].z, b.rest[0].w};
      [[maybe_unused]] const uint32_t b1[4] = {b.rest[kRest > 1 ? 1 : 0].x, b.rest[kRest > 1 ? 1 : 0].y, b.rest[kRest > 1 ? 1 : 0].z, b.rest[kRest > 1 ? 1 : 0].w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t key = u[r] + b.kmin * 0x01010101u;
        const uint32_t high = (rest[r] & 0x80808080u) | ((key >> 1) & 0x7f7f7f7fu);
        const uint32_t low = (rest[r] & 0x7f7f7f7fu) | ((key * 128u) & 0x80808080u);
        if constexpr (sizeof(T) == 4) {
          uint32_t w[4] = {b0[r], b1[r], low, high};
          transpose_bytes(w);
#pragma unroll
          for (int j = 0; j < 4; ++j) raw.w[4 * r + j] = w[j];
        } else {
          raw.w[2 * r] = __byte_perm(low, high, 0x5140);
          raw.w[2 * r + 1] = __byte_perm(low, high, 0x7362);
        }
      }
    } else {
      uint32_t key[8], rest[8], high[4], hp[8];
      pairs_of_planes(u, key);
      const uint32_t q[4] = {b.rest[0].x, b.rest[0].y, b.rest[0].z, b.rest[0].w};
      values_of_planes(b.high, high, 3, lane);
      pairs_of_planes(high, hp);
      constexpr uint32_t kMan = ((1u << Tr::kExpShift) - 1u) * 0x00010001u;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        rest[k] = __byte_perm(q[k >> 1], 0u, k & 1 ? 0x4342 : 0x4140) | (hp[k] << 8);
        raw.w[k] = (((rest[k] << (15 - Tr::kExpShift)) & 0x80008000u) | (rest[k] & kMan)) | ((key[k] + b.kmin * 0x00010001u) << Tr::kExpShift);
      }
    }
    if constexpr (MODE == 1) {
      if constexpr (sizeof(T) == 4) load16_wide<T>(out, idx, count, have);
      float x[16], y[16];
      wide16_to_f<T>(raw, x);
      wide16_to_f<T>(have, y);
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] += y[j];
      store16_wide<T>(out, idx, count, x);
    } else {
      store16_wide<T>(out, idx, count, raw);
    }
    if (!more) return;
  }
}

static size_t ll_tiles(size_t count) { return (count + kLlTileElems - 1) / kLlTileElems; }
static size_t ll_slot(int dtype) { return dtype == CCB_F32 ? ll_slot_bytes<float>() : ll_slot_bytes<__half>(); }
// Up to eight tiles an SM each has a CTA. Beyond that CTAs take several in turn, in grids of as many an
// SM as were fastest of 4, 8 and 16 (32 Mi values encoded / decoded, us: bf16 23.1 / 22.6, 23.1 / 22.8 and
// 24.7 / 24.6; f16 31.4 / 30.6, 30.8 / 28.8, 30.8 / 30.0; fp32 46.9 / 44.5, 43.3 / 41.1, 42.3 / 40.9): what
// a first tile costs against a last turn that only some have. B200.
static int ll_grid(size_t ntiles, int dtype) {
  const size_t sms = (size_t)sm_count(), cap = sms * (dtype == CCB_F32 ? 16 : dtype == CCB_F16 ? 8 : 4);
  return (int)(ntiles == 0 ? 1 : ntiles <= 8 * sms || ntiles < cap ? ntiles : cap);
}

}  // namespace ccb

using namespace ccb;

extern "C" uint64_t ccb_lossless_max_bytes(int dtype, uint64_t count) {
  if (dtype != CCB_F32 && dtype != CCB_BF16 && dtype != CCB_F16) return 0;
  return kLlHeader + ll_tiles(count) * ll_slot(dtype);
}

extern "C" int ccb_lossless_encode(int dtype, const void* in, uint64_t count, void* out, void* stream) {
  if (!in || !out || (reinterpret_cast<uintptr_t>(out) & 15)) {
    set_error("ccb_lossless_encode: null or misaligned buffer (the container must be 16-byte aligned)");
    return CCB_ERR_ARG;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dtype != CCB_F32 && dtype != CCB_BF16 && dtype != CCB_F16) return CCB_ERR_UNSUPPORTED;
  // the kernel writes the header (a copy from the host would be a staged transfer per call) and
  // adds up its byte count, which has to start at zero
  if (launch_clear(out, kLlHeader, s) != cudaSuccess) {
    set_error("ccb_lossless_encode: clearing the header failed: %s", cudaGetErrorString(cudaGetLastError()));
    return CCB_ERR_CUDA;
  }
  const size_t nt = ll_tiles(count);
  const int g = ll_grid(nt, dtype);
  if (dtype == CCB_F32) launch_next(lossless_encode_kernel<float>, g, kLlThreads, 0, s, (const float*)in, count, (char*)out, nt);
  else if (dtype == CCB_BF16) launch_next(lossless_encode_kernel<__nv_bfloat16>, g, kLlThreads, 0, s, (const __nv_bfloat16*)in, count, (char*)out, nt);
  else launch_next(lossless_encode_kernel<__half>, g, kLlThreads, 0, s, (const __half*)in, count, (char*)out, nt);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("ccb_lossless_encode: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

extern "C" int ccb_lossless_decode(int dtype, const void* in, uint64_t count, void* out, int accumulate, void* stream) {
  if (!in || !out || (reinterpret_cast<uintptr_t>(in) & 15)) {
    set_error("ccb_lossless_decode: null or misaligned buffer");
    return CCB_ERR_ARG;
  }
  const size_t nt = ll_tiles(count);
  if (nt == 0) return CCB_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int g = ll_grid(nt, dtype);
#define CCB_LL_DEC(T)                                                                                          \
  do {                                                                                                         \
    if (accumulate) launch_next(lossless_decode_kernel<T, 1>, g, kLlThreads, 0, s, (const char*)in, count, (T*)out, nt); \
    else launch_next(lossless_decode_kernel<T, 0>, g, kLlThreads, 0, s, (const char*)in, count, (T*)out, nt);            \
  } while (0)
  if (dtype == CCB_F32) CCB_LL_DEC(float);
  else if (dtype == CCB_BF16) CCB_LL_DEC(__nv_bfloat16);
  else if (dtype == CCB_F16) CCB_LL_DEC(__half);
  else return CCB_ERR_UNSUPPORTED;
#undef CCB_LL_DEC
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("ccb_lossless_decode: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

// Bytes a transport has to move for this container: the header plus the used prefix of
// every slot. Reads 8 bytes back from the device after synchronising `stream`.
extern "C" int ccb_lossless_used_bytes(const void* comp, uint64_t* bytes, void* stream) {
  if (!comp || !bytes) return CCB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned long long v = 0;
  if (cudaMemcpyAsync(&v, static_cast<const char*>(comp) + 16, sizeof(v), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    set_error("ccb_lossless_used_bytes: %s", cudaGetErrorString(cudaGetLastError()));
    return CCB_ERR_CUDA;
  }
  *bytes = v;
  return CCB_OK;
}
