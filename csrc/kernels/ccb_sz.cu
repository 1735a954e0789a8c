// SZ-style error-bounded lossy codec for 3-D fp32 fields, and its fusion with
// AllGather / Broadcast over peer memory.
//
// Codec (format "ccb-sz v2"):
//   1. pre-quantisation   q = rint(x / step), step = 2 eb (1 - 2^-10), corrected by +-1
//                         where fp32 rounding picked the farther grid point; the bound
//                         |x - q * step| <= eb is then checked on the very product the
//                         decoder computes, and a tile that fails it is stored raw;
//   2. 3-D Lorenzo        d = q - (prediction from the 7 already-coded neighbours),
//                         computed on the integers, inside a 32 x 8 x 8 tile (values
//                         outside the tile predict as 0), hence lossless and parallel:
//                         the decoder undoes it with prefix sums along x, y and z;
//   3. bit-packing        zig-zag to unsigned, then per packing row of 32 values the
//                         minimum width w (0..32) and w bit-planes of 32 bits. A row is
//                         element e of the eight consecutive x that each of the 32 threads
//                         of a z plane owns (thread = 4 y + x / 8): row index 8 z + e, bit
//                         t of a plane belongs to thread t. Planes come out of a 32 x 32
//                         bit-matrix transpose across the warp (five shuffle steps), one
//                         transpose for FOUR rows when their widths are at most 8 bits.
// A tile is  [64 row widths (1 B each)][bit-planes of row 0][row 1]...  padded to
// 16 B; a tile whose values do not fit the integer range (or are not finite) is
// stored raw (width byte 0 = 255, then 8 KiB of fp32). Eight consecutive tiles form a
// group that owns a fixed-capacity slot of kGroupStride bytes:
//   [8 x u32 tile sizes][tile 0][tile 1]...
// so a receiver finds every tile without any size exchange, while only the used
// bytes are ever written (and cross NVLink).
//
// Kernel shapes: local buffers (ccb_sz_compress, ccb_sz_decompress) take a CTA a group, a
// warp a tile (sz_pack_kernel, sz_unpack_kernel; fields of few tiles are unpacked by a CTA a
// tile, sz_unpack_few_kernel). The collectives take one thread-block
// cluster of 8 CTAs per group: each CTA fetches its tile with ONE 3-D TMA copy
// (cp.async.bulk.tensor, no multicast) tracked by an mbarrier, packs it in shared memory,
// the cluster exchanges the 8 sizes through distributed shared memory to place the tiles
// back to back, and the packed tile is copied out with 16-byte stores straight into every
// peer's arena, where the same CTAs decode what arrives. Fields whose x extent is not a
// multiple of 4 elements (TMA needs 16-byte row strides) take a plain-load path there.
//
// The reference has no GPU error-bounded codec: it reaches SZ3 through dlopen on the
// CPU (userconfig/wrapper_code_examples/compression/sz3/mpi_sz3_wrapper.c:57-101,
// :138-218) and cuZFP as a library call (zfp_for_gpu_nvidia.cu:130, :179).
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>

#include <map>
#include <mutex>
#include <utility>

#include "../rt/ccb_rt_internal.h"
#include "ccb/ccb_sz.h"
#include "ccb_fastdiv.h"
#include "ccb_sz_layout.h"
#include "ccb_bits.cuh"
#include "ccb_reduce.cuh"

namespace cg = cooperative_groups;

namespace ccb {

constexpr int kTX = 32, kTY = 8, kTZ = 8;
constexpr int kTileVals = kTX * kTY * kTZ;        // 2048
constexpr int kRows = CCB_SZ_ROWS;                // kTY * kTZ
constexpr int kSzThreads = 256;                   // warp = z plane, lane = x
constexpr int kClusterSize = CCB_SZ_TILES;
constexpr int kTileCap = CCB_SZ_TILE_CAP;         // 8256 bytes, worst case (w = 32 everywhere)
constexpr int kGroupHeader = CCB_SZ_GROUP_HEADER;
constexpr int kGroupStride = CCB_SZ_GROUP_STRIDE;   // 66112, multiple of 16
static_assert(kRows == kTY * kTZ && kTileCap == kRows + kTileVals * 4, "the tile that ccb_sz_layout.h describes");
static_assert(kGroupStride % 16 == 0, "slots must keep 16-byte alignment");
constexpr float kQMax = 4194304.f;                // 2^22: |q| beyond this stores the tile raw

struct SzField {
  const float* in;   // compress source (or 0)
  float* out;        // decompress destination (or 0)
};

struct SzArgs {
  CommDev c;
  CUtensorMap tmap[CCB_MAX_RANKS];   // one per local rank, over `in`
  SzField f[CCB_MAX_RANKS];          // per local rank
  unsigned long long* used_bytes;    // per local rank: compressed bytes produced (atomicAdd), or 0
  int nx, ny, nz;
  int tiles_x, tiles_y, tiles_z;
  unsigned int ngroups;
  float eb, two_eb, inv_two_eb;
  int use_tma;
  int mode;                          // 2 all-gather, 3 broadcast
  int root;
  int rank0, nlocal;
  unsigned int bcast_waves;          // progress steps a broadcast root publishes (1..kMaxBcastWaves)
  unsigned long long slot_bytes;     // arena bytes of one source's slot (ngroups * kGroupStride, rounded)
  // Division of a tile index by tiles_x and by tiles_x * tiles_y as a multiplication:
  // (ccb_fastdiv.h; exact for tile < 2^22 and d < 2^18, which the host checks: 0 = use the
  // division). An integer division by a run-time value
  // costs about 25 instructions, and every thread needs three per tile.
  unsigned long long magic_x, magic_xy;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait on an mbarrier phase: false when the copy never completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t spin = 0; spin < (1u << 26); ++spin) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

struct TileCoord { int x0, y0, z0; };
template <class Args>
__device__ __forceinline__ TileCoord tile_coord(const Args& a, unsigned int tile) {
  TileCoord t;
  unsigned int tx, ty, tz;
  if (a.magic_x) {
    const unsigned int txy = a.tiles_x * a.tiles_y;
    tz = ccb_fastdiv(tile, a.magic_xy);
    const unsigned int rem = tile - tz * txy;
    ty = ccb_fastdiv(rem, a.magic_x);
    tx = rem - ty * a.tiles_x;
  } else {
    tx = tile % a.tiles_x, ty = (tile / a.tiles_x) % a.tiles_y, tz = tile / (a.tiles_x * a.tiles_y);
  }
  t.x0 = tx * kTX; t.y0 = ty * kTY; t.z0 = tz * kTZ;
  return t;
}

// Thread mapping of both directions: warp = z plane of the tile, lane = 4 y + xq, and the
// thread owns the eight consecutive values x = 8 xq .. 8 xq + 7 of line (y, z), which sit at
// words 8 * threadIdx.x .. +7 of the tile in shared memory (two 16-byte accesses). A packing
// row is element e of all 32 lanes of a warp: row index 8 z + e.

__device__ __forceinline__ uint32_t bytesum(uint32_t v) { return __dp4a(v, 0x01010101u, 0u); }
// True when every byte of w (each at most 32) is at most 8 / at most 16.
__device__ __forceinline__ bool bytes_le8(uint32_t w) { return ((w + 0x77777777u) & 0x80808080u) == 0; }
__device__ __forceinline__ bool bytes_le16(uint32_t w) { return ((w + 0x6f6f6f6fu) & 0x80808080u) == 0; }

// Bit-planes of four rows with widths of up to 32 bits: `W` holds the widths (one byte each),
// `off` is the word offset of the first row's planes. Widths up to 16 take two bit-matrix
// transposes, wider rows one each. (Up to 8 bits, by far the most common, the four rows share
// one transpose: see the callers.) The byte layout does not depend on which way was taken.
template <bool kStore>
__device__ __forceinline__ void wide_planes4(uint32_t (&u)[4], uint32_t W, uint32_t off, uint32_t* words, int lane) {
  auto pass = [&](int bits, int first_row, int rows) {   // rows * bits == 32
    const int rr = lane / bits, jj = lane % bits, row = first_row + rr;
    const uint32_t w = (W >> (8 * row)) & 0xffu;
    const uint32_t at = off + bytesum(W & ((1u << (8 * row)) - 1u)) + jj;
    if (kStore) {
      uint32_t U = 0;
      for (int r2 = 0; r2 < rows; ++r2) U |= u[first_row + r2] << (bits * r2);
      const uint32_t X = transpose32(U, lane);
      if ((uint32_t)jj < w) words[at] = X;
    } else {
      const uint32_t X = (uint32_t)jj < w ? ldg_cg_u32(words + at) : 0u;
      const uint32_t U = transpose32(X, lane);
      for (int r2 = 0; r2 < rows; ++r2) u[first_row + r2] = bits == 32 ? U : (U >> (bits * r2)) & ((1u << bits) - 1u);
    }
  };
  if (bytes_le16(W)) {
    pass(16, 0, 2);
    pass(16, 2, 2);
  } else {
#pragma unroll
    for (int r2 = 0; r2 < 4; ++r2) pass(32, r2, 1);
  }
}

constexpr float kRoundMagic = 12582912.f;   // 1.5 * 2^23: adding and subtracting it rounds to nearest even

// Packs the tile held in `vals` (fp32, [z][y][x]) into `pk`; returns its byte size.
// The codes overwrite the values in shared memory (each thread its own eight words).
// With `recon` set, the decoder's view of the tile (q * step, or the raw values of a raw
// tile) is also written to its place in that field: the sender's own copy of what every
// receiver will decode, without a decode pass. `failed` (any thread): the tile's copy never came and
// the values are NaN; the tile is stored raw.
__device__ __forceinline__ uint32_t pack_tile(float* vals, unsigned char* pk, int* s_tot, const SzArgs& a, bool failed,
                                              float* recon = nullptr, TileCoord tc = TileCoord{0, 0, 0}) {
  const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
  int4* q4 = reinterpret_cast<int4*>(vals) + 2 * threadIdx.x;
  float x[8];
  {
    const float4 v0 = reinterpret_cast<const float4*>(q4)[0], v1 = reinterpret_cast<const float4*>(q4)[1];
    x[0] = v0.x; x[1] = v0.y; x[2] = v0.z; x[3] = v0.w; x[4] = v1.x; x[5] = v1.y; x[6] = v1.z; x[7] = v1.w;
  }
  int q[8];
  const float half = 0.5f * a.two_eb;
  // s = x / step; adding 1.5 * 2^23 rounds it to nearest even and leaves the integer in the low
  // mantissa bits, subtracting it again gives it as a float; diff = x - q * step with the very
  // product that the decoder computes (every operation rounded by itself: no fused multiply-add).
  // (As packed pairs, mul.rn.f32x2 and add.rn.f32x2, the operations came out fused all the same.)
  float smax = 0.f;
  bool far = false;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float s = __fmul_rn(x[e], a.inv_two_eb), r = __fadd_rn(s, kRoundMagic);
    const float diff = __fsub_rn(x[e], __fmul_rn(__fadd_rn(r, -kRoundMagic), a.two_eb));
    smax = fmaxf(smax, fabsf(s));
    far |= !(fabsf(diff) <= half);
    q[e] = __float_as_int(r) - __float_as_int(kRoundMagic);
  }
  bool bad = failed || !(smax < kQMax);   // infinities too; a NaN is caught below (its difference is NaN)
  // Nearly always |diff| <= step / 2 < eb: the value sits on the nearest grid point and the
  // bound holds, nothing to correct or to re-check. The correction runs only when some lane
  // of the warp needs it (NaN counts as needing it), with the same result either way.
  if (__any_sync(0xffffffffu, far)) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float s = __fmul_rn(x[e], a.inv_two_eb);
      bad |= !(fabsf(s) < kQMax);
      float rf = __fadd_rn(__fadd_rn(s, kRoundMagic), -kRoundMagic);
      const float diff = __fsub_rn(x[e], __fmul_rn(rf, a.two_eb));
      rf += diff > half ? 1.f : 0.f;                              // fp32 rounding picked the farther grid point
      rf -= -diff > half ? 1.f : 0.f;
      // The grid step is a shade under 2 eb, which absorbs the rounding of q * step for
      // |q| < 2^13. Beyond that a value can fall between two grid points that are both more
      // than eb away: such a tile is stored raw, so the bound always holds.
      bad |= fabsf(__fsub_rn(x[e], __fmul_rn(rf, a.two_eb))) > a.eb;
      q[e] = (int)rf;
    }
  }
  q4[0] = make_int4(q[0], q[1], q[2], q[3]);
  q4[1] = make_int4(q[4], q[5], q[6], q[7]);
  const bool raw_tile = __syncthreads_or(bad);   // and the barrier between the codes and their readers
  if (recon) {
    const int gx = tc.x0 + 8 * (lane & 3), gy = tc.y0 + (lane >> 2), gz = tc.z0 + z;
    if (gy < a.ny && gz < a.nz) {
      float* row = recon + ((size_t)gz * a.ny + gy) * a.nx + gx;
      float o[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = raw_tile ? x[e] : __fmul_rn((float)q[e], a.two_eb);
      if (gx + 8 <= a.nx && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
        reinterpret_cast<float4*>(row)[0] = make_float4(o[0], o[1], o[2], o[3]);
        reinterpret_cast<float4*>(row)[1] = make_float4(o[4], o[5], o[6], o[7]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (gx + e < a.nx) row[e] = o[e];
      }
    }
  }
  if (raw_tile) {  // raw tile: marker + the fp32 values, each thread its own eight
    for (int i = threadIdx.x; i < kRows; i += kSzThreads) pk[i] = (i == 0) ? 255 : 0;
    float4* raw = reinterpret_cast<float4*>(pk + kRows) + 2 * threadIdx.x;
    raw[0] = make_float4(x[0], x[1], x[2], x[3]);
    raw[1] = make_float4(x[4], x[5], x[6], x[7]);
    __syncthreads();
    return kRows + kTileVals * 4;
  }
  // Lorenzo residual = the three first differences, in any order: z through shared memory
  // (plane z - 1 belongs to the warp below), y through the lane four below, x in registers.
  if (z > 0) {
    const int4 b0 = q4[-64], b1 = q4[-63];
    q[0] -= b0.x; q[1] -= b0.y; q[2] -= b0.z; q[3] -= b0.w; q[4] -= b1.x; q[5] -= b1.y; q[6] -= b1.z; q[7] -= b1.w;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int up = __shfl_up_sync(0xffffffffu, q[e], 4);
    q[e] -= lane >= 4 ? up : 0;
  }
  int left = __shfl_up_sync(0xffffffffu, q[7], 1);
  if ((lane & 3) == 0) left = 0;
  uint32_t u[8];
#pragma unroll
  for (int e = 7; e >= 0; --e) {
    const int d = q[e] - (e ? q[e - 1] : left);
    u[e] = ((uint32_t)d << 1) ^ (uint32_t)(d >> 31);
  }
  uint32_t* words = reinterpret_cast<uint32_t*>(pk + kRows);
  // Rows of at most 8 bits: four rows share one transpose, after which lane 8 r + j holds bit
  // plane j of row r. Which planes exist is then one vote: the planes up to each row's highest
  // nonzero one (its bits smeared downwards), and a lane's place is the count of those before
  // it. This replaced a warp-wide OR, a count of leading zeros and byte sums for every row
  // (packing a 512^3 field: 459 us before, 419 after, with one barrier of the tile less).
  const bool narrow = !__any_sync(0xffffffffu, (u[0] | u[1] | u[2] | u[3] | u[4] | u[5] | u[6] | u[7]) > 0xffu);
  uint32_t W0 = 0u, W1 = 0u;   // narrow: the planes that exist, one bit a lane; otherwise the widths, one byte a row
  uint32_t tot_lo, tot;        // words of the first four rows, of all eight
  if (narrow) {
    u[0] = transpose32(__byte_perm(__byte_perm(u[0], u[1], 0x0040), __byte_perm(u[2], u[3], 0x0040), 0x5410), lane);
    u[1] = transpose32(__byte_perm(__byte_perm(u[4], u[5], 0x0040), __byte_perm(u[6], u[7], 0x0040), 0x5410), lane);
    W0 = __ballot_sync(0xffffffffu, u[0] != 0u);
    W1 = __ballot_sync(0xffffffffu, u[1] != 0u);
    W0 |= (W0 >> 1) & 0x7f7f7f7fu;
    W1 |= (W1 >> 1) & 0x7f7f7f7fu;
    W0 |= (W0 >> 2) & 0x3f3f3f3fu;
    W1 |= (W1 >> 2) & 0x3f3f3f3fu;
    W0 |= (W0 >> 4) & 0x0f0f0f0fu;
    W1 |= (W1 >> 4) & 0x0f0f0f0fu;
    if (lane < 8) pk[8 * z + lane] = (unsigned char)__popc(((lane < 4 ? W0 : W1) >> (8 * (lane & 3))) & 0xffu);
    tot_lo = __popc(W0);
    tot = tot_lo + __popc(W1);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t w = 32 - __clz((int)__reduce_or_sync(0xffffffffu, u[e]));
      if (e < 4) W0 |= w << (8 * e);
      else W1 |= w << (8 * (e - 4));
    }
    tot_lo = bytesum(W0);
    tot = tot_lo + bytesum(W1);
    if (lane == 0) reinterpret_cast<uint2*>(pk)[z] = make_uint2(W0, W1);   // the eight width bytes of this plane
  }
  if (lane == 0) s_tot[z] = (int)tot;
  __syncthreads();
  const uint32_t t = lane < kTZ ? (uint32_t)s_tot[lane] : 0u;
  const uint32_t total = __reduce_add_sync(0xffffffffu, t), base = __reduce_add_sync(0xffffffffu, lane < z ? t : 0u);
  if (narrow) {
    const uint32_t before = (1u << lane) - 1u;
    if ((W0 >> lane) & 1u) words[base + __popc(W0 & before)] = u[0];
    if ((W1 >> lane) & 1u) words[base + tot_lo + __popc(W1 & before)] = u[1];
  } else {
    uint32_t ua[4] = {u[0], u[1], u[2], u[3]}, ub[4] = {u[4], u[5], u[6], u[7]};
    wide_planes4<true>(ua, W0, base, words, lane);
    wide_planes4<true>(ub, W1, base + tot_lo, words, lane);
  }
  const uint32_t bytes = kRows + 4u * total;
  const uint32_t padded = (bytes + 15u) & ~15u;
  if (threadIdx.x < (padded - bytes) / 4) words[total + threadIdx.x] = 0u;
  __syncthreads();
  return padded;
}

// Decodes a packed tile at `src` (global or arena memory) and writes it to its place in `out`;
// `qs2` is two times 8 KB of shared scratch, of which a packed tile takes the one that the packed
// tile before it did not (`scratch`: 0 or 1). A raw tile takes none and needs no barrier. (512^3
// fields, B200: raw tiles only 407 us, packed tiles only 324; with a scratch for every tile and a
// barrier in the raw ones it was 432 and 321.) A tile whose widths cannot be (or `sound` false: whose
// place cannot) becomes NaN, without an access through its words.
template <class Args>
__device__ __forceinline__ void unpack_tile(const unsigned char* src, bool sound, int* qs2, int& scratch, const Args& a, float* out, const TileCoord& t) {
  const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
  // the 16 words of row widths, one per lane, and their running word count
  const uint32_t hw = sound && lane < 16 ? ldg_cg_u32(src + 4 * lane) : 0u;
  const bool raw_tile = (__shfl_sync(0xffffffffu, hw, 0) & 0xffu) == 255u;
  sound = sound && (raw_tile || !__any_sync(0xffffffffu, !ccb_sz_widths_ok(hw)));
  if (raw_tile || !sound) {
    const float* raw = reinterpret_cast<const float*>(src + kRows);
    for (int i = threadIdx.x; i < kTileVals; i += kSzThreads) {
      const int gx = t.x0 + (i % kTX), gy = t.y0 + (i / kTX) % kTY, gz = t.z0 + i / (kTX * kTY);
      if (gx < a.nx && gy < a.ny && gz < a.nz)
        out[((size_t)gz * a.ny + gy) * a.nx + gx] = __uint_as_float(sound ? ldg_cg_u32(raw + i) : 0x7fffffffu);
    }
    return;
  }
  scratch ^= 1;
  int* qs = qs2 + scratch * kTileVals;
  const uint32_t base = __reduce_add_sync(0xffffffffu, lane < 2 * z ? bytesum(hw) : 0u);
  const uint32_t W0 = __shfl_sync(0xffffffffu, hw, 2 * z), W1 = __shfl_sync(0xffffffffu, hw, 2 * z + 1);
  uint32_t* words = reinterpret_cast<uint32_t*>(const_cast<unsigned char*>(src) + kRows);
  uint32_t ua[4], ub[4];
  // Unpacking a 512^3 field took 373 us with the row offsets by a scan, the longer transpose and
  // a third barrier, and takes 276 (B200).
  if (bytes_le8(W0) && bytes_le8(W1)) {   // lane 8 r + j fetches plane j of row r: one transpose for four rows
    const int sh = lane & 24, j = lane & 7;
    const uint32_t before = (1u << sh) - 1u;
    const uint32_t w0 = (W0 >> sh) & 0xffu, w1 = (W1 >> sh) & 0xffu;
    const uint32_t at0 = base + bytesum(W0 & before) + j, at1 = base + bytesum(W0) + bytesum(W1 & before) + j;
    const uint32_t X0 = (uint32_t)j < w0 ? ldg_cg_u32(words + at0) : 0u, X1 = (uint32_t)j < w1 ? ldg_cg_u32(words + at1) : 0u;
    const uint32_t U0 = transpose32(X0, lane), U1 = transpose32(X1, lane);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      ua[r] = (U0 >> (8 * r)) & 0xffu;
      ub[r] = (U1 >> (8 * r)) & 0xffu;
    }
  } else {
    auto four = [&](uint32_t (&u)[4], uint32_t W, uint32_t off) {
      if (bytes_le8(W)) {
        const int sh = lane & 24, j = lane & 7;
        const uint32_t at = off + bytesum(W & ((1u << sh) - 1u)) + j;
        const uint32_t U = transpose32((uint32_t)j < ((W >> sh) & 0xffu) ? ldg_cg_u32(words + at) : 0u, lane);
#pragma unroll
        for (int r = 0; r < 4; ++r) u[r] = (U >> (8 * r)) & 0xffu;
      } else {
        wide_planes4<false>(u, W, off, words, lane);
      }
    };
    four(ua, W0, base);
    four(ub, W1, base + bytesum(W0));
  }
  int p[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t u = e < 4 ? ua[e & 3] : ub[e & 3];
    const int d = (int)(u >> 1) ^ -(int)(u & 1u);
    p[e] = e ? p[e - 1] + d : d;          // prefix along x inside the thread
  }
  {
    int sum = p[7];                         // then across the four threads of the line
    int v = __shfl_up_sync(0xffffffffu, sum, 1);
    if ((lane & 3) >= 1) sum += v;
    v = __shfl_up_sync(0xffffffffu, sum, 2);
    if ((lane & 3) >= 2) sum += v;
    const int before = sum - p[7];
#pragma unroll
    for (int e = 0; e < 8; ++e) p[e] += before;
  }
  int4* q4 = reinterpret_cast<int4*>(qs) + 2 * threadIdx.x;
  q4[0] = make_int4(p[0], p[1], p[2], p[3]);
  q4[1] = make_int4(p[4], p[5], p[6], p[7]);
  __syncthreads();
  // prefix along y: threads re-mapped to (x = lane, z = warp) walk the eight lines of their plane
  {
    int run = 0;
#pragma unroll
    for (int y = 0; y < kTY; ++y) {
      run += qs[(z * kTY + y) * kTX + lane];
      qs[(z * kTY + y) * kTX + lane] = run;
    }
  }
  __syncthreads();
  // prefix along z: threads re-mapped to (x = lane, y = warp) walk z with a running sum and
  // write each reconstructed row straight to the field (coalesced 128-byte row stores)
  {
    const int y = z;  // this warp now owns line y of every plane
    const int gx = t.x0 + lane, gy = t.y0 + y;
    const size_t plane = (size_t)a.ny * a.nx;
    float* at = out + (size_t)t.z0 * plane + (size_t)gy * a.nx + gx;
    const int planes = gx < a.nx && gy < a.ny ? a.nz - t.z0 : 0;   // planes of the tile that this thread writes
    const int* from = qs + y * kTX + lane;
    int run = 0;
    if (planes >= kTZ) {
#pragma unroll
      for (int zz = 0; zz < kTZ; ++zz) {
        run += from[zz * kTY * kTX];
        *at = __fmul_rn((float)run, a.two_eb);
        at += plane;
      }
    } else {
#pragma unroll
      for (int zz = 0; zz < kTZ; ++zz) {
        run += from[zz * kTY * kTX];
        if (zz < planes) *at = __fmul_rn((float)run, a.two_eb);
        at += plane;
      }
    }
  }
  // No barrier: a thread that writes this scratch again has passed the two barriers of the packed
  // tile between.
}

__device__ __forceinline__ void load_tile_plain(const float* in, float* vals, const TileCoord& t, const SzArgs& a) {
  const int lane = threadIdx.x & 31, z = threadIdx.x >> 5;
#pragma unroll
  for (int y = 0; y < kTY; ++y) {
    const int gx = t.x0 + lane, gy = t.y0 + y, gz = t.z0 + z;
    float v = 0.f;
    if (gx < a.nx && gy < a.ny && gz < a.nz) v = in[((size_t)gz * a.ny + gy) * a.nx + gx];
    vals[(z * kTY + y) * kTX + lane] = v;
  }
}
__device__ __forceinline__ void multimem_st(void* p, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void multimem_st_u32(void* p, uint32_t v) {
  asm volatile("multimem.st.relaxed.sys.global.f32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
constexpr int kStage = kTileCap + 16;
constexpr unsigned int kMaxBcastWaves = 8;   // most progress steps of a broadcast (flag slots 0..7)   // one packed tile, 16-byte granular

// The collectives: mode 2 all-gather, 3 broadcast.
// The cluster shape belongs to the kernel, not to the launch: as a launch attribute it was lost where
// a profiler took over the collectives' cooperative launch, every CTA took itself for tile 0 of
// its group, and seven tiles of eight were never written.
__global__ void __cluster_dims__(kClusterSize, 1, 1) __launch_bounds__(kSzThreads, 5) sz_kernel(const __grid_constant__ SzArgs a) {
  const int mode = a.mode;
  const unsigned int kBcastWaves = a.bcast_waves;
  // Two 8 KB buffers: compress lands the next tile in one while the other is packed;
  // decompress prefixes one tile in one of them and the next in the other.
  __shared__ __align__(128) float vals2[2][kTileVals];
  __shared__ __align__(16) unsigned char pk2[2][kStage];
  __shared__ int s_tot[kTZ];
  __shared__ uint32_t s_size[2];         // this CTA's packed size per group parity, read by the cluster
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ CtaSync sync;

  cg::cluster_group cluster = cg::this_cluster();
  const int k = (int)cluster.block_rank();          // tile within the group
  const unsigned int cl = blockIdx.x / kClusterSize, ncl = gridDim.x / kClusterSize;
  const int lr = blockIdx.y, r = a.rank0 + lr, n = a.c.nranks;
  const int b = blockIdx.x;                         // flag column
  const unsigned int ntiles = (unsigned)a.tiles_x * a.tiles_y * a.tiles_z;
  const bool i_send = mode == 2 || r == a.root;
  const size_t area = CCB_DATA_OFFSET + (size_t)(a.c.epoch & 1u) * a.c.half_bytes;
  if (threadIdx.x == 0) {
    sync.fail = 0;
    mbar_init(&mbar[0], 1);
    mbar_init(&mbar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  uint32_t phases = 0u;     // bit s: parity the next wait on mbarrier s expects
  auto landed = [&](int slot) {   // bounded wait for the copy into buffer `slot`; reports a copy that never came
    const bool ok = mbar_wait(&mbar[slot], (phases >> slot) & 1u);
    phases ^= 1u << slot;
    if (!ok) {
      if (threadIdx.x == 0 && a.c.status) atomicOr(a.c.status + CCB_STATUS_FLAGS, CCB_ST_TIMEOUT);
      sync.fail = 1;
    }
    return ok;
  };

  trace_mark(a.c, 0);
  // ------------------------------------------------------------- compress ----
  if (i_send) {
    const float* in = a.f[lr].in;
    unsigned long long produced = 0;
    // one thread starts the copy of this CTA's tile of group g into landing buffer `slot`
    auto prefetch = [&](unsigned int g, int slot) {
      const unsigned int tile = g * kClusterSize + k;
      if (!a.use_tma || g >= a.ngroups || tile >= ntiles || threadIdx.x != 0) return;
      const TileCoord t = tile_coord(a, tile);
      // earlier generic-proxy accesses to the buffer must be ordered before the TMA write
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&mbar[slot], kTileVals * 4);
      tma_load_3d(vals2[slot], &a.tmap[lr], t.x0, t.y0, t.z0, &mbar[slot]);
    };
    // copies a packed tile out: to every peer's arena one by one, or, where the arenas are bound to an NVLink multicast object, ONCE to the multicast
    // address: the switch replicates it, the sender's link carries the bytes one time.
    // The sender keeps no packed copy of its own field (pack_tile wrote the reconstruction).
    const bool use_mc = a.c.mc_arena != nullptr && a.nlocal == 1;
    auto emit = [&](unsigned int g, uint32_t off, uint32_t size, const unsigned char* pk) {
      const uint4* s4 = reinterpret_cast<const uint4*>(pk);
      auto to = [&](char* slot_base) {
        char* grp = slot_base + (size_t)g * kGroupStride;
        if (threadIdx.x == 0) reinterpret_cast<uint32_t*>(grp)[k] = size;
        char* dst = grp + kGroupHeader + off;
        for (uint32_t i = threadIdx.x; i < size / 16; i += kSzThreads) stg(dst + 16 * i, s4[i]);
      };
      if (use_mc) {
        char* grp = a.c.mc_arena + area + (size_t)r * a.slot_bytes + (size_t)g * kGroupStride;
        if (threadIdx.x == 0) multimem_st_u32(grp + 4 * k, size);
        char* dst = grp + kGroupHeader + off;
        for (uint32_t i = threadIdx.x; i < size / 16; i += kSzThreads) multimem_st(dst + 16 * i, s4[i]);
      } else {
        for (int j = 1; j < n; ++j) to(a.c.arena[(r + j) % n] + area + (size_t)r * a.slot_bytes);
      }
    };
    // broadcast: the root's CTAs publish their progress in kBcastWaves steps (flag slot =
    // wave), so that the receivers decode the first groups while the last are still packed
    const unsigned int my_iters = cl < a.ngroups ? (a.ngroups - cl + ncl - 1) / ncl : 0;
    auto wave_end = [&](unsigned int w) { return (unsigned int)(((unsigned long long)my_iters * (w + 1)) / kBcastWaves); };
    unsigned int wave = 0;
    float* own_out = a.f[lr].out + (mode == 2 ? (size_t)r * a.nx * a.ny * a.nz : 0);
    prefetch(cl, 0);
    uint32_t it = 0, pend_size = 0, pend_off = 0;
    unsigned int pend_g = 0;
    bool pend = false;
    for (unsigned int g = cl; g < a.ngroups; g += ncl, ++it) {
      const int slot = it & 1;
      const unsigned int tile = g * kClusterSize + k;
      uint32_t size = 0;
      prefetch(g + ncl, slot ^ 1);   // that buffer was released by the __syncthreads ending the previous pack
      if (tile < ntiles) {
        float* cur = vals2[slot];
        // No barrier here: every thread waits for the copy itself, and the plain load leaves a
        // plane of the tile to the warp that packs it.
        bool ok = true;
        if (!a.use_tma) {
          load_tile_plain(in, cur, tile_coord(a, tile), a);
        } else if (!(ok = landed(slot))) {   // a tile that never came goes out as NaN (this thread's eight values)
          for (int e = 0; e < 8; ++e) cur[8 * threadIdx.x + e] = __int_as_float(0x7fffffff);
        }
        __syncwarp();
        size = pack_tile(cur, pk2[slot], s_tot, a, !ok, own_out, tile_coord(a, tile));
      } else {
        __syncthreads();   // keeps one CTA barrier per iteration between a copy-out and its signal
      }
      if (threadIdx.x == 0) s_size[slot] = size;
      // One cluster barrier per group, split in two so that the copy-out of the PREVIOUS
      // tile runs while the cluster gathers. s_size[slot] is rewritten two groups later,
      // after every CTA has passed the next barrier, when all reads of it are done.
      cluster_arrive();
      if (mode == 3 && it >= 1) {
        // Tiles 0 .. it-2 were copied out one iteration ago by every thread (the barriers of
        // the pack above order those copies before this point), so their stores have had
        // time to complete and the fence of the signal is short.
        while (wave < kBcastWaves && wave_end(wave) <= it - 1) {
          if (threadIdx.x == 0 && wave_end(wave) > (wave ? wave_end(wave - 1) : 0u))
            signal_peers(a.c, ((1u << n) - 1u) & ~(1u << r), (int)wave, r, b);
          ++wave;
        }
      }
      if (pend) emit(pend_g, pend_off, pend_size, pk2[slot ^ 1]);
      cluster_wait();
      uint32_t off = 0;
      for (int j = 0; j < k; ++j) off += *cluster.map_shared_rank(&s_size[slot], j);
      pend = true; pend_g = g; pend_off = off; pend_size = size;
      produced += size;
    }
    if (pend) emit(pend_g, pend_off, pend_size, pk2[(it - 1) & 1]);
    if (mode == 3) {     // the remaining waves (the last one always ends here)
      __syncthreads();
      if (threadIdx.x == 0)
        for (; wave < kBcastWaves; ++wave)
          if (wave_end(wave) > (wave ? wave_end(wave - 1) : 0u)) signal_peers(a.c, ((1u << n) - 1u) & ~(1u << r), (int)wave, r, b);
    }
    cluster.sync();      // nobody leaves while a neighbour may still read its sizes
    if (a.used_bytes && threadIdx.x == 0 && produced) atomicAdd(a.used_bytes + lr, produced + 0ull);
  }

  // --------------------------------------------------------------- signal ----
  trace_mark(a.c, 1);
  __syncthreads();
  if (mode == 2 && threadIdx.x == 0) signal_peers(a.c, ((1u << n) - 1u) & ~(1u << r), 0, r, b);
  // All-gather waits source by source inside the decode loop; broadcast wave by wave.

  // ------------------------------------------------------------ decompress ---
  // Work items (source, group) of this cluster, flattened; the size words of the next
  // item's group are fetched while this item is decoded.
  const int nsrc = mode == 2 ? n - 1 : (mode == 3 && r == a.root) ? 0 : 1;   // the sender's own copy is already written
  const unsigned int per_src = cl < a.ngroups ? (a.ngroups - cl + ncl - 1) / ncl : 0;
  const unsigned int nitems = per_src * nsrc;
  const int ln = threadIdx.x & 31;
  auto group_of = [&](unsigned int f) -> const char* {
    const int q = mode == 2 ? (r + 1 + (int)(f / per_src)) % n : a.root;
    const char* slot = a.c.arena[r] + area + (size_t)q * a.slot_bytes;
    return slot + (size_t)(cl + (f % per_src) * ncl) * kGroupStride;
  };
  auto valid = [&](unsigned int f) { return f < nitems && (cl + (f % per_src) * ncl) * kClusterSize + k < ntiles; };
  auto sizes_of = [&](unsigned int f) -> uint32_t {   // lane j < k gets the size of tile j of the group
    return (valid(f) && ln < k) ? ldg_cg_u32(group_of(f) + 4 * ln) : 0u;
  };
  trace_mark(a.c, 2);
  auto dwave_end = [&](unsigned int w) { return (unsigned int)(((unsigned long long)per_src * (w + 1)) / kBcastWaves); };
  unsigned int dwave = 0;
  int scratch = 0;
  uint32_t sz_next = 0u;
  for (unsigned int f = 0; f < nitems; ++f) {
    if (per_src && f == per_src) trace_mark(a.c, 3);   // first received field decoded
    if (mode == 2 && f % per_src == 0) {   // first item of the next source: its CTA of the same index must be done
      const int src = (r + 1 + (int)(f / per_src)) % n;
      if (!cta_wait_sources(sync, a.c, a.c.arena[r], 0, r, 1u << src, 0xA0)) return;
      sz_next = sizes_of(f);               // (re)read now that the source's bytes are visible
    }
    if (mode == 3) {                        // first item of the next wave of the root's CTA of the same index
      bool waited = false;
      while (dwave < kBcastWaves && (dwave ? dwave_end(dwave - 1) : 0u) <= f) {
        if (dwave_end(dwave) > (dwave ? dwave_end(dwave - 1) : 0u)) {
          if (!cta_wait_sources(sync, a.c, a.c.arena[r], (int)dwave, r, 1u << a.root, 0xA0)) return;
          waited = true;
        }
        ++dwave;
      }
      if (waited) sz_next = sizes_of(f);
    }
    const uint32_t sz = sz_next;
    // no prefetch across a source or wave boundary: those bytes may not have arrived yet
    const bool boundary = (mode == 2 && (f + 1) % per_src == 0) ||
                          (mode == 3 && dwave < kBcastWaves && (dwave ? dwave_end(dwave - 1) : 0u) <= f + 1);
    sz_next = boundary ? 0u : sizes_of(f + 1);
    if (!valid(f)) continue;
    const uint32_t off = __reduce_add_sync(0xffffffffu, sz);
    const bool sound = ccb_sz_offset_ok(off, k);
    if (!sound && threadIdx.x == 0 && a.c.status) atomicOr(a.c.status + CCB_STATUS_FLAGS, CCB_ST_TIMEOUT);   // damaged size words
    const int q = mode == 2 ? (r + 1 + (int)(f / per_src)) % n : a.root;
    float* out = a.f[lr].out + (mode == 2 ? (size_t)q * a.nx * a.ny * a.nz : 0);
    unpack_tile(reinterpret_cast<const unsigned char*>(group_of(f)) + kGroupHeader + off, sound, reinterpret_cast<int*>(vals2[0]), scratch, a,
                out, tile_coord(a, (cl + (f % per_src) * ncl) * kClusterSize + k));
  }
  trace_mark(a.c, 4);
  if (mode == 3) end_handshake(sync, a.c, r);
}

// ------------------------------------------------------- local buffers, a warp a tile --
// Compression into and decompression from a buffer of this GPU. A warp owns a tile and walks its
// eight planes: a lane holds eight consecutive x of line y = lane / 4 (the mapping above), and the words of a
// plane go behind those of the plane before. So nothing of a tile is exchanged between warps, there is one
// barrier a GROUP (a CTA of eight warps), for the tiles' sizes, and no cluster. (With a CTA a tile, its planes on
// eight warps, three barriers a tile and the sizes sent round a cluster, a 512^3 field, bound 1e-4 of its
// range, took 332 us to pack and 279 to unpack; B200.)
struct SzLocalArgs {
  const float* in;
  float* out;
  char* slots;
  unsigned long long* used_bytes;
  int nx, ny, nz, tiles_x, tiles_y, tiles_z;
  unsigned int ngroups;
  float eb, two_eb, inv_two_eb;
  float one;   // 1, which the compiler must not know: see pack_halves
  unsigned long long magic_x, magic_xy;
};
// How a lane's eight values lie in memory: every line on 32 bytes (kVec 8), on 16 (4), or anywhere
// (1: a plane goes through shared memory, so that the accesses of a warp lie side by side).
template <int kVec>
struct PlaneIO {
  float* at;      // this lane's place in plane 0 of the tile
  size_t stride;  // of a plane
  int planes;     // of the tile that this lane has a part in (the others read as 0 and are not written)
  int width;      // kVec 4: whether the second four are inside; 1: lines of the tile, and
  int line;       //         their distance
  float* sh;      // kVec 1: 256 floats of this warp
  int lane;
  __device__ __forceinline__ PlaneIO(const float* field, const SzLocalArgs& a, TileCoord t, float* shared) {
    lane = threadIdx.x & 31;
    sh = shared;
    line = a.nx;
    stride = (size_t)a.ny * a.nx;
    const int gx = kVec == 1 ? t.x0 + lane : t.x0 + 8 * (lane & 3), gy = kVec == 1 ? t.y0 : t.y0 + (lane >> 2);
    at = const_cast<float*>(field) + ((size_t)t.z0 * a.ny + gy) * a.nx + gx;
    planes = gx < a.nx && gy < a.ny ? min(kTZ, a.nz - t.z0) : 0;
    width = kVec == 1 ? a.ny - t.y0 : gx + 4 < a.nx;
  }
  __device__ __forceinline__ void load(int z, float (&v)[8]) const {   // raw: kVec 1 holds column `lane` of the eight lines
    const float* p = at + z * stride;
    if constexpr (kVec == 1) {
#pragma unroll
      for (int y = 0; y < kTY; ++y) v[y] = z < planes && y < width ? __ldcs(p + (size_t)y * line) : 0.f;
    } else {
      uint32_t w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      if constexpr (kVec == 8) {
        if (z < planes) ldg_stream32(p, w);
      } else {
        if (z < planes) { const uint4 u = ldg_stream(p); w[0] = u.x; w[1] = u.y; w[2] = u.z; w[3] = u.w; }
        if (z < planes && width) { const uint4 u = ldg_stream(p + 4); w[4] = u.x; w[5] = u.y; w[6] = u.z; w[7] = u.w; }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(w[e]);
    }
  }
  __device__ __forceinline__ void settle(float (&v)[8]) const {   // raw -> the lane's eight consecutive x
    if constexpr (kVec == 1) {
#pragma unroll
      for (int y = 0; y < kTY; ++y) sh[kTX * y + lane] = v[y];
      __syncwarp();
      const float4 p = reinterpret_cast<const float4*>(sh)[2 * lane], q = reinterpret_cast<const float4*>(sh)[2 * lane + 1];
      v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
      __syncwarp();
    }
  }
  __device__ __forceinline__ void store(int z, const float (&v)[8]) const {
    float* p = at + z * stride;
    if constexpr (kVec == 1) {
      reinterpret_cast<float4*>(sh)[2 * lane] = make_float4(v[0], v[1], v[2], v[3]);
      reinterpret_cast<float4*>(sh)[2 * lane + 1] = make_float4(v[4], v[5], v[6], v[7]);
      __syncwarp();
#pragma unroll
      for (int y = 0; y < kTY; ++y)
        if (z < planes && y < width) p[(size_t)y * line] = sh[kTX * y + lane];
      __syncwarp();
    } else {
      if (z >= planes) return;
      uint32_t w[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(v[e]);
      if constexpr (kVec == 8) {
        stg_stream32(p, w);
      } else {
        stg_stream(p, make_uint4(w[0], w[1], w[2], w[3]));
        if (width) stg_stream(p + 4, make_uint4(w[4], w[5], w[6], w[7]));
      }
    }
  }
};

// The packer brings the values of a tile to shared memory, [z][y][x] behind the 64 bytes of its widths, all planes under
// way at once, and packs it in place: the words of planes 0 to z end where plane z + 1 begins, or before. Two
// neighbouring pieces of 16 bytes change places on odd lines, for a lane reads two of them and eight lanes at a time
// should find theirs in different banks. What lies outside the field is 0.
template <int kVec>
__device__ __forceinline__ void stage_tile(const SzLocalArgs& a, TileCoord t, unsigned char* tile) {
  const int lane = threadIdx.x & 31, depth = min(kTZ, a.nz - t.z0);
  const size_t stride = (size_t)a.ny * a.nx;
  const uint32_t to = smem_u32(tile + kRows);
  auto bring = [&](auto width, uint32_t dst, const float* src, bool on) {
    constexpr int kBytes = decltype(width)::value;
    const int n = on ? kBytes : 0;
    if constexpr (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  };
  const float* from[2];
  bool on[2];
  if constexpr (kVec != 1) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int x = t.x0 + 4 * (lane & 7), y = t.y0 + (lane >> 3) + 4 * i;
      on[i] = x < a.nx && y < a.ny;
      from[i] = on[i] ? a.in + ((size_t)t.z0 * a.ny + y) * a.nx + x : a.in;
    }
  } else {
    on[0] = t.x0 + lane < a.nx;
    from[0] = on[0] ? a.in + ((size_t)t.z0 * a.ny + t.y0) * a.nx + t.x0 + lane : a.in;
  }
  const size_t step0 = on[0] ? stride : 0;   // what lies outside is not read: its address stays
  [[maybe_unused]] size_t step1 = 0;
  if constexpr (kVec != 1) step1 = on[1] ? stride : 0;
#pragma unroll
  for (int z = 0; z < kTZ; ++z) {
    const bool deep = z < depth;
    if constexpr (kVec != 1) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        bring(Int<16>{}, to + 1024 * z + 512 * i + 16 * (lane ^ (lane >> 3 & 1)), from[i], on[i] && deep);
        if (z + 1 < depth) from[i] += i ? step1 : step0;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kTY; ++i) {
        const bool in = on[0] && deep && t.y0 + i < a.ny;
        bring(Int<4>{}, to + 1024 * z + 128 * i + 4 * (lane ^ (4 * (i & 1))), in ? from[0] + (size_t)i * a.nx : a.in, in);
      }
      if (z + 1 < depth) from[0] += step0;
    }
    if (z == 1 || z + 1 == kTZ) asm volatile("cp.async.commit_group;" ::: "memory");
  }
}
// The lane's eight values of plane z: x = 8 (lane % 4) .. + 7 of line lane / 4. The words of this plane may follow.
__device__ __forceinline__ void staged_plane(const unsigned char* tile, int z, float (&x)[8]) {
  const int lane = threadIdx.x & 31;
  const float4* at = reinterpret_cast<const float4*>(tile + kRows + 1024 * z) + 2 * lane;
  const float4 p = at[lane >> 2 & 1], q = at[~lane >> 2 & 1];
  x[0] = p.x; x[1] = p.y; x[2] = p.z; x[3] = p.w; x[4] = q.x; x[5] = q.y; x[6] = q.z; x[7] = q.w;
  __syncwarp();
}

// Codes of one plane where the nearest grid point may be another or none is near enough: the arithmetic and
// its result are pack_tile's. `base` is added to each.
__device__ __forceinline__ void exact_codes(const float (&x)[8], const SzLocalArgs& a, int base, int (&q)[8], bool& bad) {
  const float half = 0.5f * a.two_eb;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float se = __fmul_rn(x[e], a.inv_two_eb);
    bad |= !(fabsf(se) < kQMax);
    float rf = __fadd_rn(__fadd_rn(se, kRoundMagic), -kRoundMagic);
    const float diff = __fsub_rn(x[e], __fmul_rn(rf, a.two_eb));
    rf += diff > half ? 1.f : 0.f;
    rf -= -diff > half ? 1.f : 0.f;
    bad |= fabsf(__fsub_rn(x[e], __fmul_rn(rf, a.two_eb))) > a.eb;
    q[e] = (int)rf + base;
  }
  bad = __any_sync(0xffffffffu, bad);
}
// Codes of one plane, 2^21 added to each. Codes that far from 0 and values that are not finite show in the
// codes' high bits and take the exact tests.
constexpr int kCodeBias = 1 << 21;
__device__ __forceinline__ void plane_codes(const float (&x)[8], const SzLocalArgs& a, int (&q)[8], bool& bad) {
  const float half = 0.5f * a.two_eb;
  const f32x2 inv2 = pair2(a.inv_two_eb, a.inv_two_eb), step2 = pair2(a.two_eb, a.two_eb), magic2 = pair2(-kRoundMagic, -kRoundMagic);
  float worst = 0.f;
  uint32_t high = 0u;
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    float s0, s1, p0, p1;
    split2(mul2(pair2(x[e], x[e + 1]), inv2), s0, s1);
    const float r0 = __fadd_rn(s0, kRoundMagic), r1 = __fadd_rn(s1, kRoundMagic);
    q[e] = __float_as_int(r0) - (__float_as_int(kRoundMagic) - kCodeBias);
    q[e + 1] = __float_as_int(r1) - (__float_as_int(kRoundMagic) - kCodeBias);
    high |= (uint32_t)q[e] | (uint32_t)q[e + 1];
    split2(mul2(add2(pair2(r0, r1), magic2), step2), p0, p1);
    worst = fmaxf(worst, fmaxf(fabsf(__fsub_rn(x[e], p0)), fabsf(__fsub_rn(x[e + 1], p1))));
  }
  const bool wild = (high >> 22) != 0u;   // NaN and infinities among them, so `worst` may pass them over
  if (__any_sync(0xffffffffu, wild || worst > half)) exact_codes(x, a, kCodeBias, q, bad);
}

// 255 in the bytes whose highest bit is set, 0 in the others.
__device__ __forceinline__ uint32_t byte_signs(uint32_t v) {
  uint32_t m;
  asm("prmt.b32 %0, %1, 0, 0xba98;" : "=r"(m) : "r"(v));
  return m;
}
// A plane of wider residuals to `words`: W0 and W1 become the widths of its rows, a byte each. Returns its words.
__device__ __forceinline__ uint32_t wide_plane(const int (&d)[8], uint32_t* words, uint32_t& W0, uint32_t& W1, int lane) {
  uint32_t u[8];
  W0 = W1 = 0u;
#pragma unroll
  for (int e = 0; e < 8; ++e) u[e] = ((uint32_t)d[e] << 1) ^ (uint32_t)(d[e] >> 31);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t w = 32 - __clz((int)__reduce_or_sync(0xffffffffu, u[e]));
    if (e < 4) W0 |= w << (8 * e);
    else W1 |= w << (8 * (e - 4));
  }
  const uint32_t lo = bytesum(W0);
  uint32_t ua[4] = {u[0], u[1], u[2], u[3]}, ub[4] = {u[4], u[5], u[6], u[7]};
  wide_planes4<true>(ua, W0, 0u, words, lane);
  wide_planes4<true>(ub, W1, lo, words, lane);
  return lo + bytesum(W1);
}

// Which of the planes up to 8 of four rows are stored, from the bits that occur: all up to the highest of a row.
__device__ __forceinline__ uint32_t planes_up_to(uint32_t any) {
  any |= (any >> 1) & 0x7f7f7f7fu;
  any |= (any >> 2) & 0x3f3f3f3fu;
  return any | ((any >> 4) & 0x0f0f0f0fu);
}
__device__ __forceinline__ uint32_t byte_bits(uint32_t v) {   // the bits set in each byte
  v -= (v >> 1) & 0x55555555u;
  v = (v & 0x33333333u) + ((v >> 2) & 0x33333333u);
  return (v + (v >> 4)) & 0x0f0f0f0fu;
}
// Bytes `at` and `at` + 2 of four words that hold elements i and 4 + i: of elements 0 to 3, of 4 to 7.
__device__ __forceinline__ void bytes_of_halves(const uint32_t (&t)[4], int at, uint32_t& u0, uint32_t& u1) {
  const uint32_t sel = 0x6240u + 0x1111u * at, lo = __byte_perm(t[0], t[1], sel), hi = __byte_perm(t[2], t[3], sel);
  u0 = __byte_perm(lo, hi, 0x5410);
  u1 = __byte_perm(lo, hi, 0x7632);
}

// Packs the warp's tile as pack_planes does, if its codes lie within 4094 of the first: then two residuals share a word,
// a + 65536 b, whose sums and differences are those of the pairs whatever carries between the halves, since in
// the end a is below 2^15 either way (8 x 4095). All codes are taken relative to the first, which
// leaves only the first residual other than it is. Returns the tile's words; kNoHalves where a plane is not such a one:
// `left` then says where pack_planes goes on.
// Additions of 1.5 * 2^23 are multiply-adds by a.one, two at a time: as additions they could be fused with the
// products before them (see f32x2).
constexpr uint32_t kNoHalves = 0xffffffffu, kFirstMost = kCodeBias - 4096;   // kFirstMost: of the first code, so that all are below 2^21
struct TileLeft {
  int z;            // planes that are packed
  uint32_t run;     // their words
  int before[8];    // codes of the last of them, 2^21 added
};
__device__ __forceinline__ uint32_t pack_halves(const SzLocalArgs& a, unsigned char* pk, bool& bad, TileLeft& left) {
  const int lane = threadIdx.x & 31;
  uint32_t* words = reinterpret_cast<uint32_t*>(pk + kRows);
  const float half = 0.5f * a.two_eb;
  const f32x2 inv2 = pair2(a.inv_two_eb, a.inv_two_eb), step2 = pair2(a.two_eb, a.two_eb), one2 = pair2(a.one, a.one), less2 = pair2(-a.one, -a.one);
  const f32x2 magic2 = pair2(kRoundMagic, kRoundMagic), back2 = pair2(-kRoundMagic, -kRoundMagic);
  const Transpose32 transposed((uint32_t)lane);
  const int below_line = lane >= 4 ? -1 : 0;
  const uint32_t self = 1u << lane, below = self - 1u, below_row = (1u << (lane & 24)) - 1u, from_mine = 0xffu >> (lane & 7);
  uint32_t before[4], run = 0, wide = 0;   // wide: planes whose rows' widths are stored as such, not yet as the bit planes that they have
  f32x2 first2 = 0;
  bool far = false;   // the first code is not within 16 bits
  auto plane = [&](int z, const float (&x)[8], auto first_too) -> bool {
    int q[8];
    float diff[8], away[8];
    f32x2 r2[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const f32x2 x2 = pair2(x[2 * i], x[2 * i + 1]);
      float r0, r1;
      r2[i] = fma2(mul2(x2, inv2), one2, magic2);
      split2(r2[i], r0, r1);
      q[2 * i] = __float_as_int(r0);
      q[2 * i + 1] = __float_as_int(r1);
      split2(fma2(mul2(add2(r2[i], back2), step2), less2, x2), diff[2 * i], diff[2 * i + 1]);
    }
    uint32_t bias0 = 0x80808080u;
    uint32_t corner = 0;
    if (decltype(first_too)::value && z == 0) {
      const int first = __shfl_sync(0xffffffffu, q[0], 0);
      corner = (uint32_t)first - __float_as_uint(kRoundMagic);
      far = !ccb_sz_code_within(corner, 31999u);
      if (lane == 0) bias0 += far ? 1u << 14 : corner;
#pragma unroll
      for (int i = 0; i < 4; ++i) before[i] = (uint32_t)first * 65537u;
      first2 = pair2(-__int_as_float(first), -__int_as_float(first));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) split2(add2(r2[i], first2), away[2 * i], away[2 * i + 1]);
    const float worst = max3_abs_nan(max3_abs_nan(diff[0], diff[1], diff[2]), max3_abs_nan(diff[3], diff[4], diff[5]), max3_abs_nan(diff[6], diff[7], 0.f));
    const float apart = max3_abs_nan(max3_abs_nan(away[0], away[1], away[2]), max3_abs_nan(away[3], away[4], away[5]), max3_abs_nan(away[6], away[7], 0.f));
    if (__any_sync(0xffffffffu, !(worst <= half && apart <= 4094.f) || !ccb_sz_code_within(corner, kFirstMost))) {
      if (__any_sync(0xffffffffu, !(apart <= 4094.f) || !ccb_sz_code_within(corner, kFirstMost))) return false;
#pragma unroll
      for (int e = 0; e < 8; ++e) {   // the nearest grid point by the decoder's own product, as in exact_codes: nearly always one of 256
        const bool off = fabsf(diff[e]) > half;
        if (__any_sync(0xffffffffu, off) && off) {
          q[e] += diff[e] > 0.f ? 1 : -1;
          bad |= !(fabsf(__fsub_rn(x[e], __fmul_rn(__fadd_rn(__int_as_float(q[e]), -kRoundMagic), a.two_eb))) <= a.eb);
        }
      }
      bad = __any_sync(0xffffffffu, bad);
      if (bad) return false;
    }
    uint32_t d[4], t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t w = (uint32_t)q[4 + i] * 65536u + (uint32_t)q[i];
      d[i] = w - before[i];
      before[i] = w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] += (uint32_t)below_line * __shfl_up_sync(0xffffffffu, d[i], 4);
    // what stands left of elements 0 and 4: the left lane's 7 and this lane's 3
    const uint32_t last = d[3] + 0x80008000u;
    uint32_t left = __shfl_up_sync(0xffffffffu, last, 1);
    if ((lane & 3) == 0) left = 0x80000000u;
    t[0] = d[0] - __byte_perm(left, last, 0x5432) + bias0;
#pragma unroll
    for (int i = 1; i < 4; ++i) t[i] = d[i] - d[i - 1] + 0x00800080u;
    if (!__any_sync(0xffffffffu, ((t[0] | t[1] | t[2] | t[3]) & 0xff00ff00u) != 0u)) {
      // nearly always: residuals as bytes d + 128, whose zig-zag is twice d, complemented where d is negative
      uint32_t u0, u1;
      bytes_of_halves(t, 0, u0, u1);
      u0 = ((u0 + u0) & 0xfefefefeu) ^ ~byte_signs(u0);
      u1 = ((u1 + u1) & 0xfefefefeu) ^ ~byte_signs(u1);
      const uint32_t any0 = __reduce_or_sync(0xffffffffu, u0), any1 = __reduce_or_sync(0xffffffffu, u1);
      // a lane, plane j of its row, is stored if any plane from j up of that row holds a bit
      const uint32_t W0 = __ballot_sync(0xffffffffu, ((any0 >> lane) & from_mine) != 0u), W1 = __ballot_sync(0xffffffffu, ((any1 >> lane) & from_mine) != 0u);
      u0 = transposed(u0);
      u1 = transposed(u1);
      if (lane == 0) reinterpret_cast<uint2*>(pk)[z] = make_uint2(W0, W1);
      const uint32_t mid = run + __popc(W0);
      if (W0 & self) words[run + __popc(W0 & below)] = u0;
      if (W1 & self) words[mid + __popc(W1 & below)] = u1;
      run = mid + __popc(W1);
    } else if (!(decltype(first_too)::value && far && z == 0)) {
      // up to 16 bits: the same in halves, whose lower and upper bytes are transposed by themselves
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t v = t[i] + 0x7f807f80u;
        uint32_t minus;
        asm("prmt.b32 %0, %1, 0, 0xbb99;" : "=r"(minus) : "r"(v));
        t[i] = ((v + v) & 0xfffefffeu) ^ ~minus;
      }
      uint32_t u0, u1, y0, y1;
      bytes_of_halves(t, 0, u0, u1);
      bytes_of_halves(t, 1, y0, y1);
      const uint32_t V0 = planes_up_to(__reduce_or_sync(0xffffffffu, y0)), V1 = planes_up_to(__reduce_or_sync(0xffffffffu, y1));
      // a row with an upper plane has all the lower ones
      const uint32_t W0 = planes_up_to(__reduce_or_sync(0xffffffffu, u0)) | (V0 & 0x01010101u) * 0xffu;
      const uint32_t W1 = planes_up_to(__reduce_or_sync(0xffffffffu, u1)) | (V1 & 0x01010101u) * 0xffu;
      u0 = transposed(u0);
      u1 = transposed(u1);
      y0 = transposed(y0);
      y1 = transposed(y1);
      const uint32_t mid = run + __popc(W0) + __popc(V0);
      uint32_t* row0 = words + run + __popc(W0 & below_row) + __popc(V0 & below_row) + (lane & 7);
      uint32_t* row1 = words + mid + __popc(W1 & below_row) + __popc(V1 & below_row) + (lane & 7);
      if (W0 & self) row0[0] = u0;
      if (V0 & self) row0[8] = y0;
      if (W1 & self) row1[0] = u1;
      if (V1 & self) row1[8] = y1;
      run = mid + __popc(W1) + __popc(V1);
      if (lane == 0) reinterpret_cast<uint2*>(pk)[z] = make_uint2(byte_bits(W0) + byte_bits(V0), byte_bits(W1) + byte_bits(V1));
      wide |= 1u << z;
    } else {
      int e[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int lo = (int)(t[i] << 16) >> 16;
        e[i] = lo - 128;
        e[4 + i] = ((int)(t[i] - (uint32_t)lo) >> 16) - 128;
      }
      if (lane == 0) e[0] += (int)corner - (1 << 14);
      uint32_t W0, W1;
      run = wide_plane(e, words, W0, W1, lane);
      if (lane == 0) reinterpret_cast<uint2*>(pk)[0] = make_uint2(W0, W1);
      wide = 1u;
    }
    return true;
  };
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncwarp();
#pragma unroll 1
  for (int z = 0; z < kTZ; z += 2) {
    float x[8];
    if (z == 2) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
    }
    left.z = z;
    staged_plane(pk, z, x);
    if (!plane(z, x, Int<1>{})) break;
    left.z = z + 1;
    staged_plane(pk, z + 1, x);
    if (!plane(z + 1, x, Int<0>{})) break;
    left.z = z + 2;
  }
  if (bad) return 0;
  __syncwarp();
  if (lane < 2 * left.z && !((wide >> (lane >> 1)) & 1u)) {
    uint32_t* rows = reinterpret_cast<uint32_t*>(pk) + lane;
    *rows = byte_bits(*rows);
  }
  if (left.z < kTZ) {
    left.run = run;
    float first, unused;
    split2(first2, first, unused);
    const uint32_t code = __float_as_uint(-first);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t two = before[i] - code * 65537u;
      const int lo = (int)(two << 16) >> 16, hi = (int)(two - (uint32_t)lo) >> 16, base = (int)(code - __float_as_uint(kRoundMagic) + kCodeBias);
      left.before[i] = left.z ? base + lo : kCodeBias;
      left.before[4 + i] = left.z ? base + hi : kCodeBias;
    }
    return kNoHalves;
  }
  const uint32_t pad = (0u - run) & 3u;
  if ((uint32_t)lane < pad) words[run + lane] = 0u;
  return run;
}

// Planes of four rows of at most eight bits each, the zig-zag residuals of a lane in the bytes of u: the words, one
// bit plane a lane, and which lanes hold one that is stored.
__device__ __forceinline__ uint32_t row_planes(uint32_t& u, int lane) {
  const uint32_t stored = planes_up_to(__reduce_or_sync(0xffffffffu, u));
  u = transpose32(u, lane);
  return stored;
}

// Packs what is left of the warp's tile to `pk` (64 width bytes, then the planes). Returns the tile's words, or 0 and `bad` as
// soon as a plane shows that it has to be stored raw.
__device__ __forceinline__ uint32_t pack_planes(const SzLocalArgs& a, unsigned char* pk, bool& bad, const TileLeft& left) {
  const int lane = threadIdx.x & 31;
  uint32_t* words = reinterpret_cast<uint32_t*>(pk + kRows);
  int before[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) before[e] = left.before[e];
  uint32_t run = left.run;
#pragma unroll 1
  for (int z = left.z; z < kTZ; ++z) {
    float x[8];
    staged_plane(pk, z, x);
    int q[8], d[8];
    plane_codes(x, a, q, bad);
    if (bad) return 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      d[e] = q[e] - before[e];
      before[e] = q[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int up = __shfl_up_sync(0xffffffffu, d[e], 4);
      if (lane >= 4) d[e] -= up;
    }
    const int left = __shfl_up_sync(0xffffffffu, d[7], 1);
#pragma unroll
    for (int e = 7; e >= 1; --e) d[e] -= d[e - 1];
    if (lane & 3) d[0] -= left;
    // Residuals of eight bits or less, nearly always: as bytes d + 128, four to a word. The zig-zag of
    // four bytes is five operations; rows, planes and widths as in pack_tile.
    uint32_t t[8], high = 0u;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      t[e] = (uint32_t)(d[e] + 128);
      high |= t[e];
    }
    uint32_t W0, W1, tot;
    if (!__any_sync(0xffffffffu, high > 0xffu)) {
      uint32_t u[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t b = __byte_perm(__byte_perm(t[4 * k], t[4 * k + 1], 0x0040), __byte_perm(t[4 * k + 2], t[4 * k + 3], 0x0040), 0x5410);
        u[k] = ((b + b) & 0xfefefefeu) ^ ~byte_signs(b);
      }
      W0 = row_planes(u[0], lane);
      W1 = row_planes(u[1], lane);
      if (lane < 8) pk[8 * z + lane] = (unsigned char)__popc(((lane < 4 ? W0 : W1) >> (8 * (lane & 3))) & 0xffu);
      const uint32_t tot_lo = __popc(W0), below = (1u << lane) - 1u;
      tot = tot_lo + __popc(W1);
      if ((W0 >> lane) & 1u) words[run + __popc(W0 & below)] = u[0];
      if ((W1 >> lane) & 1u) words[run + tot_lo + __popc(W1 & below)] = u[1];
    } else {
      tot = wide_plane(d, words + run, W0, W1, lane);
      if (lane == 0) reinterpret_cast<uint2*>(pk)[z] = make_uint2(W0, W1);
    }
    run += tot;
  }
  const uint32_t pad = (0u - run) & 3u;   // the tile ends on 16 bytes (64 width bytes before the words)
  if ((uint32_t)lane < pad) words[run + lane] = 0u;
  return run;
}

// A warp stages the whole of its tile, 8256 bytes at most, three CTAs an SM; with less of it, tiles that were larger
// went through the codec a second time, to their places (512^3 values of white noise, bound 1e-5 of their range,
// 470 us). Bound by instructions at 24 warps an SM: ncu, 384^3, 48.8 M of them, 221 a plane with all that a tile needs
// besides, 73 % of the issue slots, 60 % of the pipe of logical operations. With planes loaded to registers one ahead,
// residuals one to a word and planes of 9 to 16 bits a row at a time it was 62.3 M (B200, us, that / so: 512^3 field, bound
// 1e-4 of its range, 173 / 138; 1e-3 168 / 132; 1e-5 190 / 166; 300 x 300 x 404 55.6 / 49.4, x 403 68 / 61; 130 x 201 x 258
// 22.8 / 16; white noise 512^3, 1e-6 265 / 245, 1e-7, all raw, 239 / 206). Two planes at a time 135.5 at 1e-4 but 202 at 1e-5.
template <int kVec>
__global__ void __launch_bounds__(kSzThreads, 3) sz_pack_kernel(const __grid_constant__ SzLocalArgs a) {
  after_kernel_before();
  extern __shared__ __align__(16) unsigned char stages[];   // kClusterSize * kTileCap
  __shared__ uint32_t s_size[kClusterSize];
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  const unsigned int tile = blockIdx.x * kClusterSize + k;
  char* group = a.slots + (size_t)blockIdx.x * kGroupStride;
  unsigned char* stage = stages + k * kTileCap;
  const TileCoord coord = tile_coord(a, tile);
  uint32_t size = 0;
  bool raw = false;
  if (tile < (unsigned)a.tiles_x * a.tiles_y * a.tiles_z) {
    stage_tile<kVec>(a, coord, stage);
    TileLeft left;
    uint32_t words = pack_halves(a, stage, raw, left);
    if (words == kNoHalves) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      words = pack_planes(a, stage, raw, left);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // of a tile that was left early
    size = raw ? kTileCap : (kRows + 4u * words + 15u) & ~15u;
  }
  if (lane == 0) s_size[k] = size;
  __syncthreads();
  const uint32_t of = lane < kClusterSize ? s_size[lane] : 0u;
  const uint32_t off = __reduce_add_sync(0xffffffffu, lane < k ? of : 0u);
  if (k == 0) {
    const uint32_t all = __reduce_add_sync(0xffffffffu, of);
    if (lane < kClusterSize) reinterpret_cast<uint32_t*>(group)[lane] = of;
    if (lane == 0 && a.used_bytes) atomicAdd(a.used_bytes, (unsigned long long)all);
  }
  if (size == 0) return;
  char* dst = group + kGroupHeader + off;
  if (!raw) {
    for (uint32_t i = lane; i < size / 16; i += 32) stg(dst + 16 * i, reinterpret_cast<const uint4*>(stage)[i]);
    return;
  }
  reinterpret_cast<uint16_t*>(dst)[lane] = lane == 0 ? 255 : 0;   // marker, then the fp32 values
  __syncwarp();
  const PlaneIO<kVec> io(a.in, a, coord, reinterpret_cast<float*>(stage + kRows));
  float ahead[8];
  io.load(0, ahead);
#pragma unroll 2
  for (int z = 0; z < kTZ; ++z) {
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = ahead[e];
    if (z + 1 < kTZ) io.load(z + 1, ahead);
    io.settle(x);
    float4* to = reinterpret_cast<float4*>(dst + kRows) + 2 * (32 * z + lane);
    to[0] = make_float4(x[0], x[1], x[2], x[3]);
    to[1] = make_float4(x[4], x[5], x[6], x[7]);
  }
}

// Unpacking sums a plane's residuals along x and y and adds the plane before: with the plane as a matrix D (8
// lines of 32) and triangular matrices of ones, L D U + previous. The tensor cores do it. As fp16 pairs a
// lane's eight residuals of its line are the fragment of D^T (k = x, n = y) that it has to hold. U^T D^T, for
// the two halves of x apart, comes out in fp16 (sums of 16 residuals of 8 bits, 2048 at most: exact), is the
// left operand of the product with L^T as it stands, and that adds to the codes of the plane before in fp32
// (whole numbers, exact). Residuals of 9 to 15 bits go through in two digits, 7 bits and the rest, those of up to
// 22 that a first plane has where the values are far from 0 in three.
__device__ __forceinline__ void mma_x(uint32_t& d0, uint32_t& d1, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f16.f16.f16.f16 {%0, %1}, {%2, %3, %4, %5}, {%6, %7}, {%8, %8};"
      : "=r"(d0), "=r"(d1) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_y(float (&c)[4], const uint32_t (&a)[4], uint32_t b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %8}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b));
}
struct PlanePrefix {
  // [x_in <= x_out] for x_in = 8 t .. + 7 and x_out = 4 g .. + 3 (g = lane / 4, t = lane % 4) as pairs of fp16 ones
  // and zeros: what the difference of 8 t and 4 g, a multiple of 4, leaves of it.
  uint32_t p0, p4, p8, q0, q4;
  uint32_t lines;     // [y_in <= y_out], L^T
  float code[2][4];   // [m][2 h + j]: x = 4 g + 2 m + h, y = 2 t + j
  __device__ __forceinline__ explicit PlanePrefix(int lane) {
    const int g = lane >> 2, t = lane & 3, e = 8 * t - 4 * g;
    auto ones = [](bool lo, bool hi) { return (lo ? 0x3c00u : 0u) | (hi ? 0x3c000000u : 0u); };
    p0 = ones(e <= 0, e <= 0);
    p4 = ones(e <= -4, e <= -4);
    p8 = ones(e <= -8, e <= -8);
    q0 = ones(e <= 0, e <= -4);
    q4 = ones(e <= -4, e <= -8);
    lines = ones(2 * t <= g, 2 * t + 1 <= g);
#pragma unroll
    for (int i = 0; i < 8; ++i) code[i >> 2][i & 3] = 0.f;
  }
  // h[i]: residuals 2 i and 2 i + 1 of the lane's eight; `weighted`: L^T times the weight of the digit that they are.
  __device__ __forceinline__ void add(float (&to)[2][4], const uint32_t (&h)[4], uint32_t weighted) const {
    uint32_t d[4], f[4];
    mma_x(d[0], d[1], q0, p0, p4, p4, h[0], h[1]);
    mma_x(d[2], d[3], q4, p4, p8, p8, h[2], h[3]);
    mma_x(f[0], f[1], p0, p0, q0, p0, h[0], h[1]);
    mma_x(f[2], f[3], p4, p4, q4, p4, h[2], h[3]);
    mma_y(to[0], d, weighted);
    mma_y(to[1], f, weighted);
  }
};
// fp16 pairs of a lane's eight residuals, held as bytes plus a bias in b[0] and b[1]: a byte is the low mantissa of 1024.
__device__ __forceinline__ void halves_of(const uint32_t (&b)[2], uint32_t bias, uint32_t (&h)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w = __byte_perm(b[i >> 1], 0x64646464u, i & 1 ? 0x4342 : 0x4140);
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&w), *reinterpret_cast<const __half2*>(&bias));
    h[i] = *reinterpret_cast<const uint32_t*>(&d);
  }
}

// Where a lane writes the codes of PlanePrefix: x = 4 g .. + 3 of the lines y = 2 t and 2 t + 1. kAligned: every line
// on 16 bytes, a warp writes four of 128 bytes at a time; otherwise a plane goes through shared memory, line by line.
template <bool kAligned>
struct PlaneOut {
  float* at;
  size_t stride;     // of a plane
  int line;          // of a line
  int planes, more;  // planes of the tile that the lane writes; kAligned: of its second line; otherwise lines of the tile
  float* sh;
  __device__ __forceinline__ PlaneOut(const SzLocalArgs& a, TileCoord t, float* shared) {
    const int lane = threadIdx.x & 31;
    sh = shared;
    line = a.nx;
    stride = (size_t)a.ny * a.nx;
    const int gx = kAligned ? t.x0 + (lane & ~3) : t.x0 + lane, gy = kAligned ? t.y0 + 2 * (lane & 3) : t.y0;
    at = a.out + ((size_t)t.z0 * a.ny + gy) * a.nx + gx;
    const int depth = gx < a.nx ? min(kTZ, a.nz - t.z0) : 0;
    planes = gy < a.ny ? depth : 0;
    more = !kAligned ? a.ny - t.y0 : gy + 1 < a.ny ? depth : 0;
  }
  // The planes in turn: the address moves on.
  __device__ __forceinline__ void store(int z, const float (&code)[2][4], f32x2 step2) {
    float* p = at;
    at += stride;
    float4 v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      split2(mul2(pair2(code[0][j], code[0][2 + j]), step2), v[j].x, v[j].y);
      split2(mul2(pair2(code[1][j], code[1][2 + j]), step2), v[j].z, v[j].w);
    }
    if constexpr (kAligned) {
      if (z < planes) stg_stream(p, *reinterpret_cast<const uint4*>(&v[0]));
      if (z < more) stg_stream(p + line, *reinterpret_cast<const uint4*>(&v[1]));
    } else {
      const int lane = threadIdx.x & 31;
#pragma unroll
      for (int j = 0; j < 2; ++j) reinterpret_cast<float4*>(sh)[8 * (2 * (lane & 3) + j) + (lane >> 2)] = v[j];
      __syncwarp();
#pragma unroll
      for (int y = 0; y < kTY; ++y)
        if (z < planes && y < more) p[(size_t)y * line] = sh[kTX * y + lane];
      __syncwarp();
    }
  }
};

// Bytes of a packed tile that a warp holds in shared memory: with residuals of at most 8 bits, those of the first plane
// 22, all of it; with at most 15 bits its planes in two turns.
constexpr int kUnpackStage = 2816, kDigitsMost = kRows + 4 * (8 * 22 + 7 * 8 * 15);
static_assert(kRows + 4 * (8 * 22 + 7 * 8 * 8) <= kUnpackStage && kDigitsMost % 16 == 0, "tiles of small residuals are held whole");
static_assert(kDigitsMost - (kUnpackStage - 4 * 8 * 22) + 16 <= kUnpackStage - kRows, "what a first turn leaves fits a second one");
__device__ __forceinline__ void bring_tile(unsigned char* to, const unsigned char* from, uint32_t bytes, int lane) {
  for (uint32_t i = 16u * lane; i < bytes; i += 512u) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to) + i), "l"(from + i) : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// A packed tile whose residuals have at most 15 bits, those of its first plane 22, in shared memory; kWhole false: the first
// kUnpackStage bytes of it, of the `size` at `src`.
template <bool kWhole, bool kAligned>
__device__ __forceinline__ void unpack_digits(PlaneOut<kAligned>& io, unsigned char* tile, const unsigned char* src, uint32_t size, uint32_t small, float step) {
  const int lane = threadIdx.x & 31, j = lane & 7;
  const uint32_t* words = reinterpret_cast<const uint32_t*>(tile + kRows);
  // Lane 8 r + j fetches bit planes of row r: for j = 7 the first, which holds the signs, so that it comes to the
  // highest bit of a byte; else plane j + 1, and of wider rows j + 8.
  const uint32_t below = (1u << (lane & 24)) - 1u, first = (uint32_t)(j + 1) & 7u, pick = 0x4440u | (uint32_t)(lane >> 3);
  PlanePrefix sums(lane);
  const f32x2 step2 = pair2(step, step);
  uint32_t run = 0;   // words before the plane
  auto plane = [&](int z, auto narrow) {
    const uint2 W = reinterpret_cast<const uint2*>(tile)[z];
    const uint32_t half = __dp4a(W.x, 0x01010101u, run);
    const uint32_t at0 = __dp4a(W.x & below, 0x01010101u, run) + first, at1 = __dp4a(W.y & below, 0x01010101u, half) + first;
    const uint32_t w0 = __byte_perm(W.x, 0u, pick), w1 = __byte_perm(W.y, 0u, pick);
    run = __dp4a(W.y, 0x01010101u, half);
    const uint32_t X0 = first < w0 ? words[at0] : 0u, X1 = first < w1 ? words[at1] : 0u;
    const uint32_t x0 = transpose32(X0, lane), x1 = transpose32(X1, lane), s0 = byte_signs(x0), s1 = byte_signs(x1);
    uint32_t h[4];
    if (decltype(narrow)::value || ((small >> (2 * z)) & 3u) == 3u) {   // zig-zag undone: a negative residual is the complement; plus 128
      const uint32_t b[2] = {(x0 | 0x80808080u) ^ s0, (x1 | 0x80808080u) ^ s1};
      halves_of(b, 0x64806480u, h);
      sums.add(sums.code, h, sums.lines);
    } else {   // the low seven bits, and 128 times the others with the sign
      uint32_t y0 = X0, y1 = X1;
      if (j < 7) {
        y0 = first + 7u < w0 ? words[at0 + 7u] : 0u;
        y1 = first + 7u < w1 ? words[at1 + 7u] : 0u;
      }
      const uint32_t lo[2] = {(x0 ^ s0) & 0x7f7f7f7fu, (x1 ^ s1) & 0x7f7f7f7fu};
      halves_of(lo, 0x64006400u, h);
      sums.add(sums.code, h, sums.lines);
      y0 = transpose32(y0, lane);
      y1 = transpose32(y1, lane);
      const bool third = z == 0 && __any_sync(0xffffffffu, max(w0, w1) > 15u);
      const uint32_t mid[2] = {third ? (y0 ^ s0) & 0x7f7f7f7fu : (y0 | 0x80808080u) ^ s0, third ? (y1 ^ s1) & 0x7f7f7f7fu : (y1 | 0x80808080u) ^ s1};
      halves_of(mid, third ? 0x64006400u : 0x64806480u, h);
      sums.add(sums.code, h, (sums.lines & 0x04000400u) * 0x16u);   // 128 for 1
      if (third) {   // 16384 times these in one rounding of what is a whole number below 2^23 again
        y0 = X0;
        y1 = X1;
        if (j < 7) {
          y0 = first + 14u < w0 ? words[at0 + 14u] : 0u;
          y1 = first + 14u < w1 ? words[at1 + 14u] : 0u;
        }
        const uint32_t hi[2] = {(transpose32(y0, lane) | 0x80808080u) ^ s0, (transpose32(y1, lane) | 0x80808080u) ^ s1};
        halves_of(hi, 0x64806480u, h);
        float top[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        sums.add(top, h, sums.lines);
#pragma unroll
        for (int e = 0; e < 8; ++e) sums.code[e >> 2][e & 3] = __fmaf_rn(top[e >> 2][e & 3], 16384.f, sums.code[e >> 2][e & 3]);
      }
    }
    io.store(z, sums.code, step2);
  };
  if constexpr (!kWhole) {
    uint32_t held = (kUnpackStage - kRows) / 4;   // words before the end of what is in shared memory
#pragma unroll 1
    for (int z = 0; z < kTZ; ++z) {
      const uint2 W = reinterpret_cast<const uint2*>(tile)[z];
      if (__dp4a(W.y, 0x01010101u, __dp4a(W.x, 0x01010101u, run)) > held) {
        const uint32_t gone = run & ~3u, at = kRows + 4u * gone;
        __syncwarp();
        bring_tile(tile + kRows, src + at, min(size - at, (uint32_t)(kUnpackStage - kRows)), lane);
        words = reinterpret_cast<const uint32_t*>(tile + kRows) - gone;
        held = size;
      }
      plane(z, Int<0>{});
    }
  } else if ((small | 3u) == 0xffffffffu) {   // nearly always: beyond the first plane no residual of more than 8 bits
    plane(0, Int<0>{});
#pragma unroll
    for (int z = 1; z < kTZ; ++z) plane(z, Int<1>{});
  } else {
#pragma unroll 1
    for (int z = 0; z < kTZ; ++z) plane(z, Int<0>{});
  }
}

// A warp brings a packed tile to shared memory, all of it under way at once or, above 2816 bytes, in two turns, and
// takes its planes from there by the tensor cores; raw ones, and those with residuals of more than 15 bits, are read
// where they are, from L2 where a prefetch puts them, and summed by shuffles. (B200, us, the whole by shuffles with
// one plane requested ahead / so: 512^3 field, bound 1e-4 of its range, 163 / 111; 1e-3 154 / 105; 3e-6 242 / 175; 300 x 300
// x 404 49.5 / 32, x 403 62 / 51; 512^3 of white noise, 1e-6 190 / 173. Stages of 3328 and 4608 bytes cost the noise 10 and
// 12 us and give the fields nothing; five CTAs of 48 registers spill, +10, three of 80 +18; lanes that hold 32 bytes of a
// line 45 instead of 33 where lines lie on 16; resident CTAs with the next tile under way 209 instead of 119.) ncu, 384^3:
// 30.8 M instructions, 58.2 M by shuffles. What is left of the 94 us that the memory needs is the latency of a tile's size,
// then its words.
template <int kVec>
__global__ void __launch_bounds__(kSzThreads, 4) sz_unpack_kernel(const __grid_constant__ SzLocalArgs a) {
  after_kernel_before();
  __shared__ __align__(16) float plane[kVec == 1 ? kClusterSize : 1][kVec == 1 ? kTX * kTY : 4];
  __shared__ __align__(16) unsigned char stages[kClusterSize][kUnpackStage];
  const int lane = threadIdx.x & 31, k = threadIdx.x >> 5;
  const unsigned int tile = blockIdx.x * kClusterSize + k;
  if (tile >= (unsigned)a.tiles_x * a.tiles_y * a.tiles_z) return;
  const char* group = a.slots + (size_t)blockIdx.x * kGroupStride;
  const uint32_t size_word = lane < kClusterSize ? ldg_cg_u32(group + 4 * lane) : 0u;
  const TileCoord coord = tile_coord(a, tile);
  uint32_t off = __reduce_add_sync(0xffffffffu, lane < k ? size_word : 0u);
  const uint32_t size = __shfl_sync(0xffffffffu, size_word, k);
  const bool there = ccb_sz_offset_ok(off, k);
  if (!there) off = 0;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(group) + kGroupHeader + off;
  // (a buffer is promised to start on 4 bytes, no more)
  const bool staged = size >= kRows && size <= kDigitsMost && (size & 15u) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (staged) {
    if (kUnpackStage + 128u * lane < size) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + kUnpackStage + 128 * lane));
    bring_tile(stages[k], src, min(size, (uint32_t)kUnpackStage), lane);
  } else {
    for (uint32_t i = 128u * lane; i < min(size, (uint32_t)kTileCap); i += 4096u) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + i));
  }
  uint32_t hw = 0u;   // the row widths, four a word
  if (lane < 16) hw = staged ? reinterpret_cast<const uint32_t*>(stages[k])[lane] : ldg_cg_u32(src + 4 * lane);
  if (!there) hw = 0xfefefefeu;
  if (staged && !__any_sync(0xffffffffu, ((hw + (lane < 2 ? 0x69696969u : 0x70707070u)) | hw) & 0x80808080u) && kRows + 4u * __reduce_add_sync(0xffffffffu, bytesum(hw)) <= size) {
    PlaneOut<kVec != 1> out(a, coord, plane[kVec == 1 ? k : 0]);
    const uint32_t small = __ballot_sync(0xffffffffu, bytes_le8(hw));
    if (size <= kUnpackStage) unpack_digits<true>(out, stages[k], src, size, small, a.two_eb);
    else unpack_digits<false>(out, stages[k], src, size, small, a.two_eb);
    return;
  }
  const PlaneIO<kVec> io(a.out, a, coord, plane[kVec == 1 ? k : 0]);
  if ((__shfl_sync(0xffffffffu, hw, 0) & 0xffu) == 255u) {
    const uint32_t* raw = reinterpret_cast<const uint32_t*>(src + kRows) + 8 * lane;
    const bool wide = (reinterpret_cast<uintptr_t>(raw) & 15) == 0;
    constexpr int kRawTurns = kVec == 1 ? 2 : 4;
#pragma unroll kRawTurns
    for (int z = 0; z < kTZ; ++z, raw += kTX * kTY) {
      uint32_t w[8];
      if (wide) {
        const uint4 p = ldg_cg(raw), q = ldg_cg(raw + 4);
        w[0] = p.x; w[1] = p.y; w[2] = p.z; w[3] = p.w; w[4] = q.x; w[5] = q.y; w[6] = q.z; w[7] = q.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = ldg_cg_u32(raw + e);
      }
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(w[e]);
      io.store(z, v);
    }
    return;
  }
  if (__any_sync(0xffffffffu, !ccb_sz_widths_ok(hw))) {   // a tile whose place or widths cannot be: NaN, nothing is read through its words
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = __int_as_float(0x7fffffff);
#pragma unroll 1
    for (int z = 0; z < kTZ; ++z) io.store(z, v);
    return;
  }
  uint32_t* words = reinterpret_cast<uint32_t*>(const_cast<unsigned char*>(src) + kRows);
  // the words of a plane with widths of eight bits or less: lane 8 r + j fetches plane j of row r
  struct Ahead { uint32_t W0, W1, X0, X1; bool narrow; };
  uint32_t run = 0, next_run = 0;
  auto fetch = [&](int z) -> Ahead {
    Ahead h;
    h.W0 = __shfl_sync(0xffffffffu, hw, 2 * z);
    h.W1 = __shfl_sync(0xffffffffu, hw, 2 * z + 1);
    h.narrow = bytes_le8(h.W0) && bytes_le8(h.W1);
    h.X0 = h.X1 = 0u;
    const uint32_t lo = bytesum(h.W0);
    if (h.narrow) {
      const int sh = lane & 24, j = lane & 7;
      const uint32_t below = (1u << sh) - 1u;
      if ((uint32_t)j < ((h.W0 >> sh) & 0xffu)) h.X0 = ldg_cg_u32(words + next_run + bytesum(h.W0 & below) + j);
      if ((uint32_t)j < ((h.W1 >> sh) & 0xffu)) h.X1 = ldg_cg_u32(words + next_run + lo + bytesum(h.W1 & below) + j);
    }
    next_run += lo + bytesum(h.W1);
    return h;
  };
  int acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};   // the plane before, then this one
  // A narrow plane's residuals are summed along x and y as bytes d + 128 in halves of a word: 256 of
  // them fit 16 bits, and what the 128s come to at (x, y) is known.
  const int bias0 = 128 * (8 * (lane & 3) + 1) * ((lane >> 2) + 1), bias_step = 128 * ((lane >> 2) + 1);
  const f32x2 step2 = pair2(a.two_eb, a.two_eb);
  Ahead ahead = fetch(0);
#pragma unroll 1
  for (int z = 0; z < kTZ; ++z) {
    const Ahead h = ahead;
    const uint32_t at = run;
    run = next_run;
    if (z + 1 < kTZ) ahead = fetch(z + 1);
    if (h.narrow) {
      uint32_t A[2], B[2];   // elements (0, 2) and (1, 3) of each four
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t U = transpose32(i ? h.X1 : h.X0, lane);
        const uint32_t b = ((U >> 1) & 0x7f7f7f7fu) ^ (0x80808080u - (U & 0x01010101u));   // zig-zag undone, plus 128
        A[i] = b & 0x00ff00ffu;
        B[i] = ((b >> 8) & 0x00ff00ffu) + A[i];
        const uint32_t lower = B[i] << 16;
        A[i] += lower;
        B[i] += lower;
      }
      uint32_t c = (B[0] >> 16) * 0x00010001u;
      A[1] += c;
      B[1] += c;
      const uint32_t line = B[1] >> 16;   // then across the four threads of the line
      uint32_t sum = line, v = __shfl_up_sync(0xffffffffu, sum, 1);
      if ((lane & 3) >= 1) sum += v;
      v = __shfl_up_sync(0xffffffffu, sum, 2);
      if ((lane & 3) >= 2) sum += v;
      c = (sum - line) * 0x00010001u;
      uint32_t p[4] = {A[0] + c, B[0] + c, A[1] + c, B[1] + c};
#pragma unroll
      for (int s = 4; s < 32; s <<= 1) {   // and down the eight lines
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t w = __shfl_up_sync(0xffffffffu, p[i], s);
          if (lane >= s) p[i] += w;
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t w = p[(e >> 2) * 2 + (e & 1)];
        acc[e] += (int)(e & 2 ? w >> 16 : w & 0xffffu) - (bias0 + e * bias_step);
      }
    } else {
      uint32_t u[8];
      auto four = [&](int first, uint32_t W, uint32_t from) {
        uint32_t f[4];
        if (bytes_le8(W)) {
          const int sh = lane & 24, j = lane & 7;
          const uint32_t U = transpose32((uint32_t)j < ((W >> sh) & 0xffu) ? ldg_cg_u32(words + from + bytesum(W & ((1u << sh) - 1u)) + j) : 0u, lane);
#pragma unroll
          for (int r = 0; r < 4; ++r) f[r] = (U >> (8 * r)) & 0xffu;
        } else {
          wide_planes4<false>(f, W, from, words, lane);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) u[first + r] = f[r];
      };
      four(0, h.W0, at);
      four(4, h.W1, at + bytesum(h.W0));
      int p[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int d = (int)(u[e] >> 1) ^ -(int)(u[e] & 1u);
        p[e] = e ? p[e - 1] + d : d;
      }
      int sum = p[7], v = __shfl_up_sync(0xffffffffu, sum, 1);
      if ((lane & 3) >= 1) sum += v;
      v = __shfl_up_sync(0xffffffffu, sum, 2);
      if ((lane & 3) >= 2) sum += v;
      const int before = sum - p[7];
#pragma unroll
      for (int e = 0; e < 8; ++e) p[e] += before;
#pragma unroll
      for (int s = 4; s < 32; s <<= 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int w = __shfl_up_sync(0xffffffffu, p[e], s);
          if (lane >= s) p[e] += w;
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += p[e];
    }
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; e += 2) split2(mul2(pair2((float)acc[e], (float)acc[e + 1]), step2), f[e], f[e + 1]);
    io.store(z, f);
  }
}

// A field of few tiles leaves most of the chip idle with a warp a tile, and what counts is how long a
// tile takes: here a CTA a tile, a plane a warp (unpack_tile), six CTAs an SM.
__global__ void __launch_bounds__(kSzThreads, 6) sz_unpack_few_kernel(const __grid_constant__ SzLocalArgs a) {
  after_kernel_before();
  __shared__ __align__(16) int codes[kTileVals];
  const unsigned int k = blockIdx.x % kClusterSize, lane = threadIdx.x & 31;
  const char* group = a.slots + (size_t)(blockIdx.x / kClusterSize) * kGroupStride;
  const uint32_t off = __reduce_add_sync(0xffffffffu, lane < k ? ldg_cg_u32(group + 4 * lane) : 0u);
  int scratch = 1;
  unpack_tile(reinterpret_cast<const unsigned char*>(group) + kGroupHeader + off, ccb_sz_offset_ok(off, k), codes, scratch, a, a.out, tile_coord(a, blockIdx.x));
}

// ----------------------------------------------------------------- container ----
// The contiguous form of a compressed field: [40-byte header][u32 used bytes of each group]
// [the used bytes of every group]. Packing and unpacking are a scan over the groups' sizes and
// one copy of the used bytes. As tensor operations (a mask over the group slots, a boolean
// index into them) they passed over the slots' whole capacity, eight times the payload,
// several times: a field of 130 x 201 x 258 took 819 us through compress, pack, unpack and
// decompress, 159 us since (B200).

struct ContainerHead {   // 40 bytes, as in a file
  uint32_t magic, version;
  int nx, ny, nz;
  float eb, step;
  uint32_t ngroups;
  unsigned long long payload;
};
static_assert(sizeof(ContainerHead) == 40, "container header layout");

// offsets[g] = sum of the (clipped) sizes before group g; offsets[ngroups] = their total,
// offsets[ngroups + 1] = the largest size as it stands, or 2^32 - 1 where a group's tiles cannot have the
// sizes that its header gives them. `sizes` (u32 each) or, without them, the
// groups' own headers in `slots`. One CTA: a few thousand groups at most in use, and the copy
// that follows is the larger part. The last two go to `sums` as well, if given, to be read back.
// With `head` (the start of a container, the sizes behind it) the number of groups is what the header
// says, if no more than `ngroups`; otherwise nothing is scanned. The header then goes to `found`, and the groups' headers, in the `bytes` bytes from
// `head` on, are held against the list.
constexpr int kScanThreads = 1024;
__device__ __forceinline__ bool sizes_sound(const uint4& x, const uint4& y) {
  return ccb_sz_size_ok(x.x) && ccb_sz_size_ok(x.y) && ccb_sz_size_ok(x.z) && ccb_sz_size_ok(x.w) && ccb_sz_size_ok(y.x) && ccb_sz_size_ok(y.y) &&
         ccb_sz_size_ok(y.z) && ccb_sz_size_ok(y.w);
}
__device__ __forceinline__ uint32_t sizes_sum(const uint4& x, const uint4& y) { return x.x + x.y + x.z + x.w + y.x + y.y + y.z + y.w; }
__global__ void __launch_bounds__(kScanThreads) container_scan_kernel(const char* __restrict__ slots, const uint32_t* __restrict__ sizes,
                                                                      unsigned int ngroups, unsigned long long* offsets,
                                                                      const uint32_t* __restrict__ head, uint32_t* found, unsigned long long bytes,
                                                                      unsigned long long* sums) {
  after_kernel_before();
  if (head) {
    const uint32_t said = head[7];
    ngroups = said <= ngroups ? said : 0u;
    if (threadIdx.x < 10) found[threadIdx.x] = head[threadIdx.x];
  }
  __shared__ unsigned long long part[kScanThreads / 32];
  __shared__ uint32_t largest[kScanThreads / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long carry = 0;
  uint32_t most = 0;
  for (unsigned int g0 = 0; g0 < ngroups; g0 += kScanThreads) {
    const unsigned int g = g0 + threadIdx.x;
    uint32_t size = 0;
    if (g < ngroups) {
      if (sizes) {
        size = sizes[g];
      } else {
        const uint4* h = reinterpret_cast<const uint4*>(slots + (size_t)g * kGroupStride);
        const uint4 x = h[0], y = h[1];
        size = sizes_sum(x, y) + kGroupHeader;
        if (!sizes_sound(x, y)) most = 0xffffffffu;
      }
    }
    most = max(most, size);
    const uint32_t clipped = min(size, (uint32_t)kGroupStride);
    unsigned long long incl = clipped;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    unsigned long long before = carry, all = 0;
    for (int k = 0; k < kScanThreads / 32; ++k) {
      if (k < warp) before += part[k];
      all += part[k];
    }
    if (g < ngroups) offsets[g] = before + incl - clipped;
    if (head && g < ngroups) {   // (a list that does not add up to what is there is refused by its total)
      const unsigned long long at = sizeof(ContainerHead) + 4ull * ngroups + before + incl - clipped;
      if ((at & 3u) == 0 && at + kGroupHeader <= bytes) {
        const uint32_t* h = head + at / 4;
        const uint4 x = make_uint4(h[0], h[1], h[2], h[3]), y = make_uint4(h[4], h[5], h[6], h[7]);
        if (!sizes_sound(x, y) || sizes_sum(x, y) + kGroupHeader != size) most = 0xffffffffu;
      } else {
        most = 0xffffffffu;
      }
    }
    carry += all;
    __syncthreads();
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) largest[warp] = most;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kScanThreads / 32; ++k) most = max(most, largest[k]);
    offsets[ngroups] = carry;
    offsets[ngroups + 1] = most;
    if (sums) {   // of a container: behind the header in `found`
      sums[0] = carry;
      sums[1] = most;
    }
  }
}

// n bytes from src to dst by the CTA, in the widest accesses that both addresses allow (a group
// slot starts on 16 bytes, its place in a container on 4).
__device__ __forceinline__ void copy_bytes(char* dst, const char* src, uint32_t n) {
  const uint32_t low = (uint32_t)(reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u;
  uint32_t done = 0;
  if ((low & 15u) == 0) {
    for (uint32_t i = threadIdx.x; i < n / 16; i += blockDim.x) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    done = n & ~15u;
  } else if ((low & 7u) == 0) {
    for (uint32_t i = threadIdx.x; i < n / 8; i += blockDim.x) reinterpret_cast<uint2*>(dst)[i] = reinterpret_cast<const uint2*>(src)[i];
    done = n & ~7u;
  } else if ((low & 3u) == 0) {
    for (uint32_t i = threadIdx.x; i < n / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
    done = n & ~3u;
  }
  for (uint32_t i = done + threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

constexpr uint32_t kContainerMagic = 0x5A534343u, kContainerVersion = 2u;

__global__ void __launch_bounds__(256) container_pack_kernel(const char* __restrict__ slots, const unsigned long long* __restrict__ offsets,
                                                             ContainerHead head, char* out) {
  after_kernel_before();
  char* payload = out + sizeof(ContainerHead) + 4 * (size_t)head.ngroups;
  for (unsigned int g = blockIdx.x; g < head.ngroups; g += gridDim.x) {
    const char* slot = slots + (size_t)g * kGroupStride;
    const unsigned long long at = offsets[g];
    if (threadIdx.x == 0) {
      uint32_t size = kGroupHeader;
      for (int k = 0; k < kClusterSize; ++k) size += reinterpret_cast<const uint32_t*>(slot)[k];
      reinterpret_cast<uint32_t*>(out + sizeof(ContainerHead))[g] = size;
    }
    copy_bytes(payload + at, slot, (uint32_t)(offsets[g + 1] - at));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    head.payload = offsets[head.ngroups];
    const uint32_t* h = reinterpret_cast<const uint32_t*>(&head);
    for (int k = 0; k < (int)(sizeof(ContainerHead) / 4); ++k) reinterpret_cast<uint32_t*>(out)[k] = h[k];
  }
}

// The inverse; the rest of every slot is cleared.
__global__ void __launch_bounds__(256) container_unpack_kernel(const char* __restrict__ payload, const unsigned long long* __restrict__ offsets,
                                                               unsigned int ngroups, char* slots) {
  after_kernel_before();
  for (unsigned int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    char* slot = slots + (size_t)g * kGroupStride;
    const unsigned long long at = offsets[g];
    const uint32_t n = (uint32_t)(offsets[g + 1] - at);
    copy_bytes(slot, payload + at, n);
    const uint32_t up = (n + 15u) & ~15u;
    for (uint32_t i = n + threadIdx.x; i < up; i += blockDim.x) slot[i] = 0;
    for (uint32_t i = up / 16 + threadIdx.x; i < kGroupStride / 16; i += blockDim.x)
      reinterpret_cast<uint4*>(slot)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// --------------------------------------------------------------------- host --
typedef CUresult (*encode_tiled_t)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static encode_tiled_t tensor_map_encoder() {
  static encode_tiled_t fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<encode_tiled_t>(p);
    (void)cudaGetLastError();
  }
  return fn;
}

static bool make_tmap(CUtensorMap* m, const float* base, int nx, int ny, int nz) {
  encode_tiled_t enc = tensor_map_encoder();
  if (!enc || (nx % 4) != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
  cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
  cuuint64_t strides[2] = {(cuuint64_t)nx * 4, (cuuint64_t)nx * ny * 4};
  cuuint32_t box[3] = {kTX, kTY, kTZ};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class Args>
static void fill_geometry(Args& a, int nx, int ny, int nz, float eb) {
  a.nx = nx; a.ny = ny; a.nz = nz;
  a.tiles_x = (nx + kTX - 1) / kTX;
  a.tiles_y = (ny + kTY - 1) / kTY;
  a.tiles_z = (nz + kTZ - 1) / kTZ;
  const unsigned long long tiles = (unsigned long long)a.tiles_x * a.tiles_y * a.tiles_z;
  a.ngroups = (unsigned int)((tiles + kClusterSize - 1) / kClusterSize);
  const unsigned long long txy = (unsigned long long)a.tiles_x * a.tiles_y;
  // tile indices run up to ngroups * kClusterSize (the last group may be partly empty)
  const unsigned long long max_tile = (unsigned long long)a.ngroups * kClusterSize;
  a.magic_x = ccb_fastdiv_magic(max_tile, (unsigned long long)a.tiles_x);
  a.magic_xy = ccb_fastdiv_magic(max_tile, txy);
  if (!a.magic_x || !a.magic_xy) a.magic_x = a.magic_xy = 0;
  a.eb = eb;
  a.two_eb = 2.f * eb * (1.f - 0.0009765625f);  // quantisation step: 2 eb (1 - 2^-10)
  a.inv_two_eb = 1.f / a.two_eb;
}

// How the last waiting launch went: 1 = cooperative launch of the clusters accepted, 2 = refused
// and launched plainly (co-residency then rests on the occupancy bound).
static int g_sz_launch_path = 0;

// Asking for the occupancy of a cluster launch costs more than the launch: once per kernel and device.
static int resident_clusters(void (*kernel)(const SzArgs), const cudaLaunchConfig_t& cfg, int num_sms) {
  static std::mutex lock;
  static std::map<std::pair<void (*)(const SzArgs), int>, int> known;
  int dev = 0, clusters = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> hold(lock);
  auto at = known.find(std::make_pair(kernel, dev));
  if (at != known.end()) return at->second;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
    (void)cudaGetLastError();
    return num_sms / kClusterSize;   // not kept: the next call asks again
  }
  known[std::make_pair(kernel, dev)] = clusters;
  return clusters;
}

// Launch of clusters of 8 CTAs (__cluster_dims__), cooperative: the kernel waits on peers.
static int sz_launch(SzArgs& a, int nlocal, int num_sms, cudaStream_t stream) {
  void (*kernel)(const SzArgs) = sz_kernel;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cudaLaunchAttribute attr;
  cfg.blockDim = dim3(kSzThreads, 1, 1);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = stream;
  cfg.gridDim = dim3(kClusterSize, 1, 1);
  const int max_clusters = resident_clusters(kernel, cfg, num_sms);
  // CTAs that wait on peers must all be resident: stay within the resident clusters
  unsigned int clusters = a.ngroups;
  const unsigned int cap = (unsigned)(max_clusters / nlocal > 0 ? max_clusters / nlocal : 1);
  if (clusters > cap) clusters = cap;
  if (clusters * kClusterSize > CCB_MAX_CTAS) clusters = CCB_MAX_CTAS / kClusterSize;
  cfg.gridDim = dim3(clusters * kClusterSize, (unsigned)nlocal, 1);
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
  g_sz_launch_path = 1;
  if (e != cudaSuccess) {  // some drivers refuse cluster + cooperative: the bounded grid still fits
    (void)cudaGetLastError();
    cfg.numAttrs = 0;
    g_sz_launch_path = 2;
    e = cudaLaunchKernelEx(&cfg, kernel, a);
  }
  if (e != cudaSuccess) {
    set_error("sz kernel launch failed: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

// Eight CTAs of 256 threads fill an SM; a group is a few KB, so a CTA takes several in turn.
static unsigned int container_grid(uint64_t ngroups) {
  const uint64_t most = (uint64_t)sm_count() * 8;
  return (unsigned int)(ngroups < most ? ngroups : most);
}
// See PlaneIO.
static int line_width(const void* field, int nx) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(field);
  return nx % 8 == 0 && at % 32 == 0 ? 8 : nx % 4 == 0 && at % 16 == 0 ? 4 : 1;
}
// More shared memory than a kernel may have unasked: allowed once for each device.
template <int kVec>
static void launch_pack(const SzLocalArgs& a, cudaStream_t stream) {
  constexpr int kBytes = kClusterSize * kTileCap;
  static std::atomic<uint64_t> allowed{0};
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
  if (!(allowed.load(std::memory_order_relaxed) & bit)) {
    if (cudaFuncSetAttribute(sz_pack_kernel<kVec>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes) == cudaSuccess)
      allowed.fetch_or(bit, std::memory_order_relaxed);
  }
  launch_next(sz_pack_kernel<kVec>, a.ngroups, kSzThreads, kBytes, stream, a);
}
// Tiles up to which a CTA a tile unpacks a field faster than a warp a tile, or loses less at loose bounds than it gains at
// tight ones. B200, us, CTA / warp at bounds of 1e-4, 1e-5 and 1e-6 of the range (0.6, 1 and 2.1 bytes a value; 1e-3 as 1e-4, or
// up to 2 us less for the warp):
//   lines on 32 bytes  64 x 64 x 64 (128 tiles)   3.5 / 6.2   3.5 / 7.0   3.7 / 11.9
//                      128 x 128 x 256 (2048)     8.7 / 8.0   9.1 / 9.2   10.0 / 10.2
//                      144 x 136 x 256 (2448)     9.9 / 8.7   10.3 / 10.7 11.2 / 12.9
//                      160 x 160 x 256 (3200)     12.2 / 8.8  12.7 / 11.5 13.7 / 14.9
//   on 16              128 x 128 x 260 (2304)     9.8 / 7.5   10.2 / 8.7  10.9 / 10.1
//                      144 x 136 x 260 (2754)     11.2 / 8.4  11.7 / 10.9 12.8 / 12.7
//   anywhere           144 x 136 x 258 (2754)     11.4 / 11.7 11.9 / 14.0 12.6 / 15.5
//                      176 x 200 x 258 (4950)     18.3 / 17.8 19.1 / 21.1 20.4 / 24.0
//                      200 x 208 x 258 (5850)     21.2 / 18.2 22.0 / 23.4 23.4 / 26.1
static unsigned int few_tiles(int width) { return width == 1 ? 5120u : 2560u; }
static int launched(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: %s", what, cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

}  // namespace ccb

using namespace ccb;

extern "C" int ccb_sz_launch_path(void) { return g_sz_launch_path; }

extern "C" uint64_t ccb_sz_capacity(int nx, int ny, int nz) {
  SzArgs a;
  memset(&a, 0, sizeof(a));
  fill_geometry(a, nx, ny, nz, 1.f);
  return (uint64_t)a.ngroups * kGroupStride;
}

extern "C" int ccb_sz_compress(const float* in, int nx, int ny, int nz, float eb, void* out, unsigned long long* d_used,
                               ccb_stream_t stream) {
  if (!in || !out || nx < 1 || ny < 1 || nz < 1 || !(eb > 0.f)) {
    set_error("ccb_sz_compress: bad arguments");
    return CCB_ERR_ARG;
  }
  SzLocalArgs a;
  memset(&a, 0, sizeof(a));
  fill_geometry(a, nx, ny, nz, eb);
  a.in = in;
  a.one = 1.f;
  a.slots = static_cast<char*>(out);
  a.used_bytes = d_used;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (d_used) launch_clear(d_used, sizeof(unsigned long long), s);
  switch (line_width(in, nx)) {
    case 8: launch_pack<8>(a, s); break;
    case 4: launch_pack<4>(a, s); break;
    default: launch_pack<1>(a, s);
  }
  return launched("ccb_sz_compress");
}

extern "C" int ccb_sz_decompress(const void* in, int nx, int ny, int nz, float eb, float* out, ccb_stream_t stream) {
  if (!in || !out || nx < 1 || ny < 1 || nz < 1 || !(eb > 0.f)) {
    set_error("ccb_sz_decompress: bad arguments");
    return CCB_ERR_ARG;
  }
  SzLocalArgs a;
  memset(&a, 0, sizeof(a));
  fill_geometry(a, nx, ny, nz, eb);
  a.out = out;
  a.slots = const_cast<char*>(static_cast<const char*>(in));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const unsigned int ntiles = (unsigned)a.tiles_x * a.tiles_y * a.tiles_z;
  const int width = line_width(out, nx);
  if (ntiles <= few_tiles(width)) {
    launch_next(sz_unpack_few_kernel, ntiles, kSzThreads, 0, s, a);
    return launched("ccb_sz_decompress");
  }
  switch (width) {
    case 8: launch_next(sz_unpack_kernel<8>, a.ngroups, kSzThreads, 0, s, a); break;
    case 4: launch_next(sz_unpack_kernel<4>, a.ngroups, kSzThreads, 0, s, a); break;
    default: launch_next(sz_unpack_kernel<1>, a.ngroups, kSzThreads, 0, s, a);
  }
  return launched("ccb_sz_decompress");
}

static int container_scan(const void* slots, const uint32_t* sizes, uint64_t ngroups, unsigned long long* offsets, unsigned long long* sums, ccb_stream_t stream) {
  if (!offsets || (slots != nullptr) == (sizes != nullptr) || ngroups == 0 || (ngroups >> 31) || (reinterpret_cast<uintptr_t>(slots) & 15) ||
      (reinterpret_cast<uintptr_t>(sizes) & 3) || (reinterpret_cast<uintptr_t>(sums) & 7)) {
    set_error("ccb_sz_container_scan: bad arguments");
    return CCB_ERR_ARG;
  }
  launch_next(container_scan_kernel, 1, kScanThreads, 0, static_cast<cudaStream_t>(stream), static_cast<const char*>(slots), sizes, (unsigned int)ngroups, offsets, nullptr, nullptr,
              0ull, sums);
  return launched("ccb_sz_container_scan");
}
// offsets: ngroups + 2 words of 64 bits (see container_scan_kernel). Exactly one of slots and
// sizes is given.
extern "C" int ccb_sz_container_scan(const void* slots, const uint32_t* sizes, uint64_t ngroups, unsigned long long* offsets, ccb_stream_t stream) {
  return container_scan(slots, sizes, ngroups, offsets, nullptr, stream);
}
extern "C" int ccb_sz_container_sums(const void* slots, uint64_t ngroups, unsigned long long* offsets, unsigned long long* sums, ccb_stream_t stream) {
  return container_scan(slots, nullptr, ngroups, offsets, sums, stream);
}

// The scan of a container of `bytes` bytes whose header is still on the device: offsets for at most
// `room` groups (room + 2 words); found (56 bytes, 8-byte aligned) takes the header, the sum of the
// group sizes and the largest. Nothing is scanned where the header speaks of more groups than `room`.
extern "C" int ccb_sz_container_open(const void* blob, uint64_t bytes, uint64_t room, unsigned long long* offsets, void* found, ccb_stream_t stream) {
  if (!blob || !offsets || !found || room == 0 || (room >> 31) || bytes < sizeof(ContainerHead) + 4 * room || (reinterpret_cast<uintptr_t>(blob) & 3) ||
      (reinterpret_cast<uintptr_t>(found) & 7)) {
    set_error("ccb_sz_container_open: bad arguments");
    return CCB_ERR_ARG;
  }
  const uint32_t* head = static_cast<const uint32_t*>(blob);
  launch_next(container_scan_kernel, 1, kScanThreads, 0, static_cast<cudaStream_t>(stream), nullptr, head + sizeof(ContainerHead) / 4, (unsigned int)room, offsets, head,
              static_cast<uint32_t*>(found), bytes, static_cast<unsigned long long*>(found) + 5);
  return launched("ccb_sz_container_open");
}

// out: 40 + 4 * ngroups + offsets[ngroups] bytes, 4-byte aligned.
extern "C" int ccb_sz_container_pack(const void* slots, const unsigned long long* offsets, int nx, int ny, int nz, float eb, uint64_t ngroups, void* out,
                                     ccb_stream_t stream) {
  if (!slots || !offsets || !out || ngroups == 0 || (ngroups >> 31) || (reinterpret_cast<uintptr_t>(slots) & 15) || (reinterpret_cast<uintptr_t>(out) & 3)) {
    set_error("ccb_sz_container_pack: bad arguments");
    return CCB_ERR_ARG;
  }
  const ContainerHead head = {kContainerMagic, kContainerVersion, nx, ny, nz, eb, 2.f * eb * (1.f - 0.0009765625f), (uint32_t)ngroups, 0};
  launch_next(container_pack_kernel, container_grid(ngroups), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const char*>(slots), offsets, head, static_cast<char*>(out));
  return launched("ccb_sz_container_pack");
}

// payload: offsets[ngroups] bytes; slots: ngroups * kGroupStride bytes, 16-byte aligned.
extern "C" int ccb_sz_container_unpack(const void* payload, const unsigned long long* offsets, uint64_t ngroups, void* slots, ccb_stream_t stream) {
  if (!payload || !offsets || !slots || ngroups == 0 || (ngroups >> 31) || (reinterpret_cast<uintptr_t>(slots) & 15)) {
    set_error("ccb_sz_container_unpack: bad arguments");
    return CCB_ERR_ARG;
  }
  launch_next(container_unpack_kernel, container_grid(ngroups), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const char*>(payload), offsets,
                                                                                                   (unsigned int)ngroups, static_cast<char*>(slots));
  return launched("ccb_sz_container_unpack");
}

// Error-bounded AllGather (root < 0) or Broadcast (root >= 0) of one nx*ny*nz field per
// rank. AllGather: recv holds nranks fields in rank order. d_used (optional, one
// counter per local rank, device memory) receives the compressed bytes each rank sent
// to ONE destination.
extern "C" int ccb_sz_collective(ccb_comm* c, const float* const* send, float* const* recv, int nx, int ny, int nz, float eb,
                                 int root, unsigned long long* d_used, ccb_stream_t stream_) {
  int rc = check_alive(c);
  if (rc) return rc;
  if (!send || !recv || nx < 1 || ny < 1 || nz < 1 || !(eb > 0.f)) {
    set_error("ccb_sz_collective: bad arguments");
    return CCB_ERR_ARG;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int n = ccb_comm_nranks(c), nlocal = ccb_comm_nlocal(c);
  SzArgs a;
  memset(&a, 0, sizeof(a));
  fill_geometry(a, nx, ny, nz, eb);
  a.slot_bytes = ((unsigned long long)a.ngroups * kGroupStride + 255ull) & ~255ull;
  a.c = comm_dev(c, 0);
  const int nslots = n;
  if ((unsigned long long)nslots * a.slot_bytes > a.c.half_bytes) {
    set_error("arena too small: an error-bounded collective of %d x %d x %d needs %llu bytes of staging (CCB_ARENA_MB)", nx, ny, nz,
              (unsigned long long)nslots * a.slot_bytes * 2 + CCB_DATA_OFFSET);
    return CCB_ERR_CAPACITY;
  }
  a.c = comm_dev(c, next_epoch(c));
  bool tma = true;
  for (int i = 0; i < nlocal; ++i) {
    a.f[i].in = send[i];
    a.f[i].out = recv[i];
    const bool sender = root < 0 || (ccb_comm_rank(c) + i) == root;
    if (sender && !make_tmap(&a.tmap[i], send[i], nx, ny, nz)) tma = false;
  }
  a.use_tma = tma ? 1 : 0;
  a.used_bytes = d_used;
  a.mode = root < 0 ? 2 : 3;
  a.root = root < 0 ? 0 : root;
  a.rank0 = ccb_comm_rank(c);
  a.nlocal = nlocal;
  {  // progress steps of a broadcast: every step costs the root a system fence
    static int waves = 0;
    if (!waves) {
      const char* e = getenv("CCB_SZ_BCAST_WAVES");
      waves = e ? atoi(e) : 2;
      if (waves < 1) waves = 1;
      if (waves > (int)kMaxBcastWaves) waves = (int)kMaxBcastWaves;
    }
    a.bcast_waves = (unsigned int)waves;
  }
  if (d_used) cudaMemsetAsync(d_used, 0, sizeof(unsigned long long) * nlocal, stream);
  return sz_launch(a, nlocal, sm_count(), stream);
}
