// The collectives of ranks that share one GPU and one process (Communicator.local): every rank's
// buffers are in this GPU's memory, so nothing has to pass through an arena. A warp takes 512
// elements of a block, reads them from every rank that contributes, passes each contribution
// through the codec in registers (the same encode and decode, in the same order, as the kernels
// that talk over peer memory, hence the same results bit for bit) and writes every rank's result.
// No staging, no flags, no cooperative launch: each input is read once and each output written
// once. The kernels of ccb_reduce.cuh, ccb_pipe.cuh, ccb_ring.cuh and ccb_exchange.cuh remain the
// ones for ranks on several GPUs, and a local communicator takes them where their schedule is
// asked for (a phase trace, a grid cap, waves, a pipeline mode) and where the ranks' buffers
// overlap: see ranks_in_registers() and its callers in the runtime.
//
// All of them are bound by memory, or by the instructions of the codec where many ranks contribute.
// A warp does one unit and ends: nothing is carried, registers stay few, and the hardware hands out
// CTAs in the order of the addresses.
#pragma once
#include "ccb_codec.cuh"
#include "ccb_grid.h"

namespace ccb {

constexpr int kLocalThreads = 128;   // with 256 the slots of an SM come free in larger pieces (B200, us, 256 / 128: reduce-scatter of 8 x 32 MiB of bf16 in int8 53.2 / 52.3, tree of 3 x 40 MiB of f16 51.0 / 49.3, gather of 8 x 400,003 fp32 21.7 / 20.9)

enum { kLocalTwoShot = 0, kLocalOneShot = 1, kLocalRing = 2, kLocalTree = 3, kLocalScatter = 4 };

struct LocalReduceArgs {
  const void* send[CCB_MAX_RANKS];
  void* recv[CCB_MAX_RANKS];
  float* ef[CCB_MAX_RANKS];    // residuals, or 0
  uint64_t count;              // elements of the message (kLocalScatter: of one shard)
  uint64_t shard_elems;        // distance of the shards in the send buffers
  uint32_t units;              // warps' units of 512 elements in the whole call
  uint32_t shard_units;        // units of one shard
  int n, op, root;             // root: kLocalScatter delivers to this rank alone (>= 0), or shard s to rank s (< 0)
};

// Ranks whose values are requested before the first is used, and CTAs of 128 threads on an SM: what
// was fastest of one, two and four ranks at 40 to 128 registers a thread. (At these nothing spills but 4
// to 8 bytes in one-shots and trees of 16-bit types.)
// (B200. 4 ranks of 64 MiB of bf16, two-shot int8: two ranks at 64 registers 82.4 us, at 48, which
// spill, 105, four at 80 123. 8 ranks of 25 MiB to their owners: 43.3; one rank at 48 53. Shards at
// odd places: one at 64 registers 66, two 70. 2 ranks of 5,000,011 fp32 values: one at 64 10.5, two
// at 128 12.6. 4 ranks of 25 MiB of bf16 with residuals: two at 128 registers 96.7, one 100.6.)
template <class T, int ALGO, bool kEf, bool kAnyOffset> struct LocalShape {
  static constexpr int kBatch = sizeof(T) == 4 || kAnyOffset ? 1 : 2;
  static constexpr int kCtas = kEf ? 4 : (ALGO == kLocalTree ? 6 : 8) - (sizeof(T) == 4 && (kAnyOffset || ALGO == kLocalTree) ? 2 : 0);
};

template <class T>
__device__ __forceinline__ void store_elem(T* p, uint32_t word, int half) {
  if constexpr (sizeof(T) == 4) *reinterpret_cast<uint32_t*>(p) = word;
  else *reinterpret_cast<unsigned short*>(p) = (unsigned short)(word >> (16 * half));
}

// Every buffer starts on 32 bytes (kAnyOffset: anywhere). `inside`: the unit lies inside the message,
// the same in all lanes. At the ragged end a lane reads the 32-byte sectors that hold any of its
// elements (which stay inside their allocation) and clears the rest; 16 loads one by one took as
// long as a call of a few thousand units. The callers have a body for each: with the two in one the
// reduce-scatter of 8 x 25 MiB took 58 us instead of 49.
template <class T, bool kAnyOffset = false>
__device__ __forceinline__ void local_load(const T* base, size_t idx, size_t limit, bool inside, Wide16<T>& raw) {
  constexpr int W = 4 * (int)sizeof(T), kPer = 4 / (int)sizeof(T);
  const char* p = reinterpret_cast<const char*>(base + idx);
  const uint32_t off = kAnyOffset ? (uint32_t)(reinterpret_cast<uintptr_t>(p) & 31) : 0u;
  constexpr int kWords = kAnyOffset ? W + 8 : W;
  uint32_t w[kWords];
  if (inside) {
#pragma unroll
    for (int k = 0; k < W; k += 8) ldg_stream32(p - off + 4 * k, w + k);
    if (kAnyOffset && off) ldg_stream32(p - off + 4 * W, w + kWords - 8);
  } else {
    const uint32_t bytes = idx < limit ? (uint32_t)min((size_t)16, limit - idx) * (uint32_t)sizeof(T) : 0u;
#pragma unroll
    for (int k = 0; k < kWords; k += 8) {
      if (bytes && 4u * k < off + bytes) {
        ldg_stream32(p - off + 4 * k, w + k);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) w[k + i] = 0u;
      }
    }
  }
  if constexpr (kAnyOffset) shift_down<T>(w, off / (uint32_t)sizeof(T));
#pragma unroll
  for (int k = 0; k < W; ++k) raw.w[k] = w[k];
  if (!inside) {
    const uint32_t n = idx < limit ? (uint32_t)min((size_t)16, limit - idx) : 0u;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      if ((uint32_t)(kPer * k) >= n) raw.w[k] = 0u;
      else if (kPer == 2 && (uint32_t)(2 * k + 1) >= n) raw.w[k] &= 0xffffu;
    }
  }
}
template <class T, bool kAnyOffset = false>
__device__ __forceinline__ void local_store(T* base, size_t idx, size_t limit, bool inside, const Wide16<T>& raw) {
  constexpr int W = 4 * (int)sizeof(T), kPer = 4 / (int)sizeof(T);
  if (inside && kAnyOffset) {
    store16_wide<T, true>(base, idx, limit, raw);
  } else if (!kAnyOffset && (inside || idx + 16 <= limit)) {
#pragma unroll
    for (int k = 0; k < W; k += 8) stg_stream32(reinterpret_cast<char*>(base + idx) + 4 * k, raw.w + k);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (idx + i < limit) store_elem<T>(base + idx + i, raw.w[i / kPer], i % kPer);
  }
}

// Units of 512 elements on 32 bytes by way of shared memory: what a warp has under way does not take registers
// there. kUnitPieces pieces of 16 bytes each; a lane reads sizeof(T) of them that follow one another, and they change
// places so that eight lanes at a time find theirs in different banks.
template <class T> constexpr int kUnitPieces = 32 * (int)sizeof(T);
template <class T> __device__ __forceinline__ uint32_t unit_piece(uint32_t c) { return c ^ (c >> 3 & (sizeof(T) == 4 ? 3u : 1u)); }
template <class T>
__device__ __forceinline__ void bring_unit(uint4* to, const T* from) {   // to be waited for by the lane, then met by the warp
  const uint32_t lane = threadIdx.x & 31, at = (uint32_t)__cvta_generic_to_shared(to);
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at + 16u * unit_piece<T>(lane + 32 * i)), "l"(reinterpret_cast<const char*>(from) + 16 * (lane + 32 * i)) : "memory");
}
template <class T>
__device__ __forceinline__ void brought_unit(const uint4* unit, float (&v)[16]) {   // the lane's 16 elements
  const uint32_t lane = threadIdx.x & 31;
  Wide16<T> raw;
#pragma unroll
  for (int i = 0; i < (int)sizeof(T); ++i) {
    const uint4 p = unit[unit_piece<T>(sizeof(T) * lane + i)];
    raw.w[4 * i] = p.x; raw.w[4 * i + 1] = p.y; raw.w[4 * i + 2] = p.z; raw.w[4 * i + 3] = p.w;
  }
  wide16_to_f<T>(raw, v);
}

template <class T>
__device__ __forceinline__ void pack16(const float (&v)[16], Wide16<T>& o) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < 16; ++i) o.w[i] = __float_as_uint(v[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) o.w[i] = pack2<T>(v[2 * i], v[2 * i + 1]);
  }
}

// Lossy codecs add and do nothing else (the entry points refuse the rest).
template <class C>
__device__ __forceinline__ void combine16(int op, float (&a)[16], const float (&d)[16]) {
  if (C::kId != CCB_CODEC_NONE || op == CCB_OP_SUM) {   // never fused with the decoder's product: same bits as the kernels over peer memory
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = __fadd_rn(a[i], d[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = apply_op(op, a[i], d[i]);
  }
}

// v becomes what a receiver of the packet decodes; with a residual, v - that is kept for the next call.
// kSentOnly: where the kernels over peer memory decode this packet for the residual alone (see residual_of_sent).
template <class C, bool kEf, bool kAnyOffset = false, bool kSentOnly = false>
__device__ __forceinline__ void through_codec(float (&v)[16], float* ef, size_t idx, size_t limit, bool inside) {
  if constexpr (!kEf) {
    C::round_trip(v);
  } else {
    float d[16], r[16];
    if constexpr (kSentOnly && C::kId == CCB_CODEC_INT4) {
      typename C::Packet pk;
      C::encode(v, pk);
      C::decode(pk, d);
      C::residual(pk, v, r);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) d[i] = v[i];
      C::round_trip(d);
#pragma unroll
      for (int i = 0; i < 16; ++i) r[i] = __fsub_rn(v[i], d[i]);
    }
    if (ef) {
      Wide16<float> e;
      pack16<float>(r, e);
      local_store<float, kAnyOffset>(ef, idx, limit, inside, e);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = d[i];
  }
}
template <bool kEf, bool kAnyOffset = false>
__device__ __forceinline__ void add_residual(float (&v)[16], const float* ef, size_t idx, size_t limit, bool inside) {
  if constexpr (kEf) {
    if (ef) {
      Wide16<float> e;
      local_load<float, kAnyOffset>(ef, idx, limit, inside, e);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(e.w[i]);
    }
  }
}

// The binomial tree below rank r with kRounds rounds: v = what r's parent decodes.
template <class T, class C, bool kEf, bool kAnyOffset, int kRounds>
__device__ __forceinline__ void local_subtree(const LocalReduceArgs& a, int r, size_t idx, bool inside, float (&v)[16]) {
  Wide16<T> raw;
  local_load<T, kAnyOffset>(static_cast<const T*>(a.send[r]), idx, a.count, inside, raw);
  wide16_to_f<T>(raw, v);
  auto child = [&](auto round) {
    constexpr int k = decltype(round)::value;
    if constexpr (k < kRounds) {
      if (r + (1 << k) < a.n) {
        float d[16];
        local_subtree<T, C, kEf, kAnyOffset, k>(a, r + (1 << k), idx, inside, d);
        combine16<C>(a.op, v, d);
      }
    }
  };
  child(Int<0>{});
  child(Int<1>{});
  child(Int<2>{});
  add_residual<kEf, kAnyOffset>(v, a.ef[r], idx, a.count, inside);
  through_codec<C, kEf, kAnyOffset>(v, a.ef[r], idx, a.count, inside);
}

// One unit of 512 elements: element idx (of the message; kLocalScatter: of shard s) and the 15 after it.
template <class T, class C, int ALGO, bool kEf, bool kAnyOffset, bool inside>
__device__ __forceinline__ void local_reduce_unit(const LocalReduceArgs& a, uint32_t s, size_t idx) {
  const int n = a.n;
  const int owner = ALGO == kLocalScatter && a.root >= 0 ? a.root : (int)s;
  float acc[16];
  if constexpr (ALGO == kLocalTree) {
    static_assert(CCB_MAX_RANKS <= 8, "three rounds");
    local_subtree<T, C, kEf, kAnyOffset, 3>(a, 0, idx, inside, acc);
  } else {
    const size_t at = ALGO == kLocalScatter ? (size_t)s * a.shard_elems : 0;
    // the order in which contributions enter the sum: the owner, then ascending ranks (two-shot,
    // reduce-scatter); ascending ranks (one-shot); once round from the shard's number (ring)
    auto rank_of = [&](int j) -> int {
      if (ALGO == kLocalOneShot) return j;
      if (ALGO == kLocalRing) return (int)s + j < n ? (int)s + j : (int)s + j - n;
      return j == 0 ? owner : j - (j <= owner ? 1 : 0);
    };
    auto take = [&](auto batch, int j0) {   // ranks rank_of(j0), ... into the sum
      constexpr int kN = decltype(batch)::value;
      Wide16<T> raw[kN];
      [[maybe_unused]] Wide16<float> e[kEf ? kN : 1];
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        const int q = rank_of(j0 + i);
        local_load<T, kAnyOffset>(static_cast<const T*>(a.send[q]) + at, idx, a.count, inside, raw[i]);
        if constexpr (kEf)
          if (a.ef[q]) local_load<float, kAnyOffset>(a.ef[q] + at, idx, a.count, inside, e[i]);
      }
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        const int j = j0 + i;
        float v[16];
        wide16_to_f<T>(raw[i], v);
        if ((ALGO == kLocalTwoShot || ALGO == kLocalScatter) && j == 0) {   // the owner's own values: not compressed
#pragma unroll
          for (int k = 0; k < 16; ++k) acc[k] = v[k];
          continue;
        }
        const int q = rank_of(j);
        if (ALGO == kLocalRing && j > 0) combine16<C>(a.op, v, acc);
        if constexpr (kEf) {
          if (a.ef[q]) {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] += __uint_as_float(e[i].w[k]);
          }
        }
        through_codec<C, kEf, kAnyOffset, ALGO != kLocalRing>(v, kEf && a.ef[q] ? a.ef[q] + at : nullptr, idx, a.count, inside);
        if (ALGO == kLocalRing || (ALGO == kLocalOneShot && j == 0)) {
#pragma unroll
          for (int k = 0; k < 16; ++k) acc[k] = v[k];
        } else {
          combine16<C>(a.op, acc, v);
        }
      }
    };
    // whole batches without a test for each rank (reduce-scatter of 8 x 25 MiB: 43 us, 49 with one)
    constexpr int kBatch = inside ? LocalShape<T, ALGO, kEf, kAnyOffset>::kBatch : 1;
    int j0 = 0;
#pragma unroll 1
    for (; j0 + kBatch <= n; j0 += kBatch) take(Int<kBatch>{}, j0);
    if constexpr (kBatch > 1) {
#pragma unroll 1
      for (; j0 < n; ++j0) take(Int<1>{}, j0);
    }
    if constexpr (ALGO == kLocalTwoShot) {   // the owner compresses the sum once more; everybody decodes that
      add_residual<kEf, kAnyOffset>(acc, a.ef[owner], idx, a.count, inside);
      through_codec<C, kEf, kAnyOffset>(acc, a.ef[owner], idx, a.count, inside);
    }
  }
  Wide16<T> o;
  pack16<T>(acc, o);
  if constexpr (ALGO == kLocalScatter) {
    local_store<T, kAnyOffset>(static_cast<T*>(a.recv[owner]), idx, a.count, inside, o);
  } else {
#pragma unroll 1
    for (int p = 0; p < n; ++p) local_store<T, kAnyOffset>(static_cast<T*>(a.recv[p]), idx, a.count, inside, o);
  }
}

template <class T, class C, int ALGO, bool kEf, bool kAnyOffset>
__global__ void __launch_bounds__(kLocalThreads, LocalShape<T, ALGO, kEf, kAnyOffset>::kCtas) local_reduce_kernel(const __grid_constant__ LocalReduceArgs a) {
  after_kernel_before();
  const uint32_t u = ccb_grid_warp(blockIdx.x, blockDim.x, threadIdx.x);
  if (u >= a.units) return;
  const uint32_t s = ALGO == kLocalTwoShot || ALGO == kLocalRing || ALGO == kLocalScatter ? u / a.shard_units : 0u;
  const size_t e0 = (size_t)(ALGO == kLocalScatter ? u - s * a.shard_units : u) * kWarpElems, idx = e0 + (threadIdx.x & 31) * kLaneElems;
  if (e0 + kWarpElems <= a.count) local_reduce_unit<T, C, ALGO, kEf, kAnyOffset, true>(a, s, idx);
  else local_reduce_unit<T, C, ALGO, kEf, kAnyOffset, false>(a, s, idx);
}

// ----------------------------------------------------------------------- one rank --
// An all-reduce of one rank: a round trip through the codec, one unit a warp. With nothing carried
// from unit to unit a thread has 32 registers (16-bit types) and an SM all of its 64 warps, each
// waits once, and CTAs are handed out in the order of the addresses, which is what the memory likes
// best: 256 MiB of bf16 in int8 81 us, 6.6 TB/s, the rate of a plain copy, where resident CTAs that
// looped over the message with a unit requested ahead took 100 (and 88 at 46 registers a thread). B200.
template <class T, class C, bool kEf, bool kAnyOffset, bool inside>
__device__ __forceinline__ void local_solo_unit(const LocalReduceArgs& a, size_t idx) {
  Wide16<T> raw;
  local_load<T, kAnyOffset>(static_cast<const T*>(a.send[0]), idx, a.count, inside, raw);
  [[maybe_unused]] Wide16<float> e;
  if constexpr (kEf) local_load<float, kAnyOffset>(a.ef[0], idx, a.count, inside, e);
  float v[16];
  wide16_to_f<T>(raw, v);
  if constexpr (kEf) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(e.w[i]);
  }
  through_codec<C, kEf, kAnyOffset>(v, kEf ? a.ef[0] : nullptr, idx, a.count, inside);
  Wide16<T> o;
  pack16<T>(v, o);
  local_store<T, kAnyOffset>(static_cast<T*>(a.recv[0]), idx, a.count, inside, o);
}
template <class T, class C, bool kEf, bool kAnyOffset>
__global__ void __launch_bounds__(kLocalThreads, kEf ? 8 : sizeof(T) == 4 ? (kAnyOffset ? 8 : 12) : kAnyOffset ? 12 : 16) local_solo_kernel(const __grid_constant__ LocalReduceArgs a) {
  after_kernel_before();
  const size_t e0 = (((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kWarpElems, idx = e0 + (threadIdx.x & 31) * kLaneElems;
  if (e0 >= a.count) return;
  if (e0 + kWarpElems <= a.count) local_solo_unit<T, C, kEf, kAnyOffset, true>(a, idx);
  else local_solo_unit<T, C, kEf, kAnyOffset, false>(a, idx);
}

// ------------------------------------------------------------------------- exchange --
// One block per (source, destination), or one per source where all its destinations get the same
// elements (all-gather, broadcast): those are read and encoded once. A warp takes a run of `run`
// consecutive units of a block.
struct LocalExchangeArgs {
  const void* src[CCB_MAX_RANKS * CCB_MAX_RANKS];
  uint64_t cnt[CCB_MAX_RANKS * CCB_MAX_RANKS];
  void* dst[CCB_MAX_RANKS * CCB_MAX_RANKS];                // of all blocks, in their order
  uint32_t first_run[CCB_MAX_RANKS * CCB_MAX_RANKS + 1];   // runs before each block
  uint8_t first_dst[CCB_MAX_RANKS * CCB_MAX_RANKS + 1];
  uint64_t in_place;   // blocks that are their own destination, a bit each
  int nblocks;
  uint32_t run;
};

// kAnyOffset: blocks may start anywhere. Where the destinations of a block lie alike on their
// 32-byte sectors the warp rotates a unit once for all of them, and the first sector of a unit is
// completed with what the unit before left over; a run begins with that unit, of which it stores nothing
// else, so that only the ends of a block are written element by element. (With the ends of runs of four written so,
// 64 stores of an element for eight of a lane's 32 bytes, an all-gather of 8 x 1,638,401 bf16 in fp8 took 50 us, 46 so; B200.)
// A block in place keeps to its own units: the one before may have been written. (Without kAnyOffset a run is one unit.)
template <class T, class C, bool kAnyOffset>
__global__ void __launch_bounds__(kLocalThreads, kAnyOffset ? (sizeof(T) == 4 ? 4 : 6) : 12) local_exchange_kernel(const __grid_constant__ LocalExchangeArgs a) {
  after_kernel_before();
  constexpr int W = 4 * (int)sizeof(T), kPer = 4 / (int)sizeof(T);   // words of a lane, elements of a word
  const int lane = threadIdx.x & 31;
  const uint32_t w = ccb_grid_warp(blockIdx.x, blockDim.x, threadIdx.x);
  if (w >= a.first_run[a.nblocks]) return;
  int b = 0;
  while (w >= a.first_run[b + 1]) ++b;
  const T* src = static_cast<const T*>(a.src[b]);
  const size_t cnt = a.cnt[b];
  const int d0 = a.first_dst[b], d1 = a.first_dst[b + 1];
  auto plain = [&](size_t e0, auto whole) {   // a unit by itself
    constexpr bool inside = decltype(whole)::value != 0;
    const size_t idx = e0 + lane * kLaneElems;
    Wide16<T> o;
    local_load<T, kAnyOffset>(src, idx, cnt, inside, o);
    float v[16];
    wide16_to_f<T>(o, v);
    C::round_trip(v);
    pack16<T>(v, o);
#pragma unroll 1
    for (int d = d0; d < d1; ++d) local_store<T, kAnyOffset>(static_cast<T*>(a.dst[d]), idx, cnt, inside, o);
  };
  if constexpr (!kAnyOffset) {
    const size_t e0 = (size_t)(w - a.first_run[b]) * kWarpElems;
    if (e0 + kWarpElems <= cnt) plain(e0, Int<1>{});
    else plain(e0, Int<0>{});
  } else {
    const size_t u0 = (size_t)(w - a.first_run[b]) * a.run, whole = cnt / kWarpElems;
    const size_t u1 = u0 + a.run < whole ? u0 + a.run : whole;   // the run's whole units; a ragged one may follow
    const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(a.dst[d0]) & 31);   // a unit is a whole number of sectors
    const uint32_t mis = off / (uint32_t)sizeof(T);
    bool alike = true;
    for (int d = d0 + 1; d < d1; ++d) alike = alike && (uint32_t)(reinterpret_cast<uintptr_t>(a.dst[d]) & 31) == off;
    if (!alike) {
#pragma unroll 1
      for (size_t u = u0; u < u1; ++u) plain(u * kWarpElems, Int<1>{});
    } else if (u0 < u1) {
      Wide16<T> next, left;   // left, in lane 0: the last `mis` elements of the unit before
      const bool apart = !(a.in_place >> b & 1u);
      const size_t start = apart && mis && u0 ? u0 - 1 : u0;
      size_t u = start;
      local_load<T, true>(src, u * kWarpElems + lane * kLaneElems, cnt, true, next);
#pragma unroll 1
      for (; u < u1; ++u) {
        const size_t idx = u * kWarpElems + lane * kLaneElems;
        float v[16];
        wide16_to_f<T>(next, v);
        if (u + 1 < u1) local_load<T, true>(src, idx + kWarpElems, cnt, true, next);
        C::round_trip(v);
        Wide16<T> o;
        pack16<T>(v, o);
        rotate_up<T>(o.w, mis, lane);
        const Wide16<T> mine = o;   // lane 0: this unit's last `mis` elements, then its first 16 - mis
        if (lane == 0 && u > start) {
#pragma unroll
          for (int k = 0; k < W; ++k) {
            if ((uint32_t)(kPer * k + kPer - 1) < mis) o.w[k] = left.w[k];
            else if (kPer == 2 && (uint32_t)(2 * k) < mis) o.w[k] = __byte_perm(left.w[k], o.w[k], 0x7610);
          }
        }
        const bool sector = lane != 0 || u > start || mis == 0;
#pragma unroll 1
        for (int d = u < u0 ? d1 : d0; d < d1; ++d) {
          T* p = static_cast<T*>(a.dst[d]) + idx - mis;
          if (sector) {
#pragma unroll
            for (int k = 0; k < W; k += 8) stg_stream32(reinterpret_cast<char*>(p) + 4 * k, o.w + k);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if ((uint32_t)i >= mis) store_elem<T>(p + i, o.w[(i / kPer) & (W - 1)], i % kPer);
          }
        }
        left = mine;
      }
      if (lane == 0 && (u1 == whole || !apart)) {   // behind the last whole unit of the block
#pragma unroll 1
        for (int d = d0; d < d1; ++d) {
          T* p = static_cast<T*>(a.dst[d]) + u1 * kWarpElems - mis;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if ((uint32_t)i < mis) store_elem<T>(p + i, left.w[(i / kPer) & (W - 1)], i % kPer);
        }
      }
    }
    if (u1 == whole && u0 + a.run > whole && whole * kWarpElems < cnt) plain(whole * kWarpElems, Int<0>{});
  }
}

}  // namespace ccb
