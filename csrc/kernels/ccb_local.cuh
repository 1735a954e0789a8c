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
#pragma once
#include "ccb_codec.cuh"

namespace ccb {

constexpr int kLocalThreads = 256;

enum { kLocalTwoShot = 0, kLocalOneShot = 1, kLocalRing = 2, kLocalTree = 3, kLocalScatter = 4 };

struct LocalReduceArgs {
  const void* send[CCB_MAX_RANKS];
  void* recv[CCB_MAX_RANKS];
  float* ef[CCB_MAX_RANKS];    // residuals, or 0
  uint64_t count;              // elements of the message (kLocalScatter: of one shard)
  uint64_t shard_elems;        // distance of the shards in the send buffers
  uint32_t units;              // warps' units of 512 elements in the whole call
  uint32_t shard_units;        // units of one shard
  int wide;                    // every buffer starts on 32 bytes (or kAnyOffset)
  int n, op, root;             // root: kLocalScatter delivers to this rank alone (>= 0), or shard s to rank s (< 0)
};

// Ranks whose values are requested before the first is used, and CTAs of 256 threads on an SM: what
// was fastest of one to four ranks at 64, 80 and 128 registers a thread. (B200; 4 ranks of 64 MiB
// of bf16, ring, fp8: two ranks at 64 registers 83 us, four at 80 registers 98, one 92. 8 ranks of
// 25 MiB to their owners in int8: 51, 70, 57. Shards at odd places, one rank at a time 70 us, two
// 76. 2 ranks of 5,000,011 fp32 values: two at 128 registers 12.6, at 64 17.3. 4 ranks of 25 MiB
// with residuals: one at 128 registers 102, two 112, one at 80 114: those spill.)
template <class T, int ALGO, bool kEf, bool kAnyOffset> struct LocalShape {
  static constexpr int kBatch = kEf || kAnyOffset ? 1 : 2;
  static constexpr int kCtas = kEf || sizeof(T) == 4 ? 2 : ALGO == kLocalTree ? 3 : 4;
};

// kInside: the unit lies inside the message, and (but for kAnyOffset) on 32 bytes. One access a
// lane and 32 bytes then, without the branches and the element loop of the general form.
template <class T, bool kInside, bool kAnyOffset = false>
__device__ __forceinline__ void local_load(const T* base, size_t idx, size_t limit, Wide16<T>& raw) {
  constexpr int W = 4 * (int)sizeof(T);
  if constexpr (!kInside) {
    load16_wide<T, kAnyOffset>(base, idx, limit, raw);
  } else {
    const char* p = reinterpret_cast<const char*>(base + idx);
    if constexpr (kAnyOffset) {
      const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 31);
      uint32_t w[W + 8];
#pragma unroll
      for (int k = 0; k < W; k += 8) ldg_stream32(p - off + 4 * k, w + k);
      if (off) ldg_stream32(p - off + 4 * W, w + W);
      shift_down<T>(w, off / (uint32_t)sizeof(T));
#pragma unroll
      for (int k = 0; k < W; ++k) raw.w[k] = w[k];
    } else {
#pragma unroll
      for (int k = 0; k < W; k += 8) ldg_stream32(p + 4 * k, raw.w + k);
    }
  }
}
template <class T, bool kInside, bool kAnyOffset = false>
__device__ __forceinline__ void local_store(T* base, size_t idx, size_t limit, const Wide16<T>& raw) {
  if constexpr (kInside && !kAnyOffset) {
#pragma unroll
    for (int k = 0; k < 4 * (int)sizeof(T); k += 8) stg_stream32(reinterpret_cast<char*>(base + idx) + 4 * k, raw.w + k);
  } else {
    store16_wide<T, kAnyOffset>(base, idx, limit, raw);
  }
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
template <class T>
__device__ __forceinline__ void store_elem(T* p, uint32_t word, int half) {
  if constexpr (sizeof(T) == 4) *reinterpret_cast<uint32_t*>(p) = word;
  else *reinterpret_cast<unsigned short*>(p) = (unsigned short)(word >> (16 * half));
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
// kSentOnly: the kernels over peer memory decode this packet for the residual alone (see CodecInt4::residual).
template <class C, bool kEf, bool kInside, bool kSentOnly = false>
__device__ __forceinline__ void through_codec(float (&v)[16], float* ef, size_t idx, size_t limit) {
  typename C::Packet pk;
  C::encode(v, pk);
  float d[16];
  C::decode(pk, d);
  if constexpr (kEf) {
    if (ef) {
      float r[16];
      if constexpr (kSentOnly && C::kId == CCB_CODEC_INT4) {
        C::residual(pk, v, r);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = __fsub_rn(v[i], d[i]);
      }
      Wide16<float> e;
      pack16<float>(r, e);
      local_store<float, kInside>(ef, idx, limit, e);
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = d[i];
}
template <bool kEf, bool kInside>
__device__ __forceinline__ void add_residual(float (&v)[16], const float* ef, size_t idx, size_t limit) {
  if constexpr (kEf) {
    if (ef) {
      Wide16<float> e;
      local_load<float, kInside>(ef, idx, limit, e);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(e.w[i]);
    }
  }
}

// The binomial tree below rank r with kRounds rounds: v = what r's parent decodes.
template <class T, class C, bool kEf, bool kInside, int kRounds>
__device__ __forceinline__ void local_subtree(const LocalReduceArgs& a, int r, size_t idx, float (&v)[16]) {
  Wide16<T> raw;
  local_load<T, kInside>(static_cast<const T*>(a.send[r]), idx, a.count, raw);
  wide16_to_f<T>(raw, v);
  auto child = [&](auto round) {
    constexpr int k = decltype(round)::value;
    if constexpr (k < kRounds) {
      if (r + (1 << k) < a.n) {
        float d[16];
        local_subtree<T, C, kEf, kInside, k>(a, r + (1 << k), idx, d);
        combine16<C>(a.op, v, d);
      }
    }
  };
  child(Int<0>{});
  child(Int<1>{});
  child(Int<2>{});
  add_residual<kEf, kInside>(v, a.ef[r], idx, a.count);
  through_codec<C, kEf, kInside>(v, a.ef[r], idx, a.count);
}

// One unit: element idx of the message (kLocalScatter: of shard s) and the 15 after it.
template <class T, class C, int ALGO, bool kEf, bool kAnyOffset, bool kInside>
__device__ __forceinline__ void local_reduce_unit(const LocalReduceArgs& a, uint32_t s, size_t idx) {
  const int n = a.n;
  const int owner = ALGO == kLocalScatter && a.root >= 0 ? a.root : (int)s;
  float acc[16];
  if constexpr (ALGO == kLocalTree) {
    static_assert(CCB_MAX_RANKS <= 8, "three rounds");
    local_subtree<T, C, kEf, kInside, 3>(a, 0, idx, acc);
  } else {
    constexpr int kBatch = kInside ? LocalShape<T, ALGO, kEf, kAnyOffset>::kBatch : 1;
    const size_t at = ALGO == kLocalScatter ? (size_t)s * a.shard_elems : 0;
    // the order in which contributions enter the sum: the owner, then ascending ranks (two-shot,
    // reduce-scatter); ascending ranks (one-shot); once round from the shard's number (ring)
    auto rank_of = [&](int j) -> int {
      if (ALGO == kLocalOneShot) return j;
      if (ALGO == kLocalRing) return (int)s + j < n ? (int)s + j : (int)s + j - n;
      return j == 0 ? owner : j - (j <= owner ? 1 : 0);
    };
#pragma unroll 1
    for (int j0 = 0; j0 < n; j0 += kBatch) {
      Wide16<T> raw[kBatch];
      Wide16<float> e[kEf ? kBatch : 1];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        if (j0 + i < n) {
          const int q = rank_of(j0 + i);
          local_load<T, kInside, kAnyOffset>(static_cast<const T*>(a.send[q]) + at, idx, a.count, raw[i]);
          if constexpr (kEf)
            if (a.ef[q]) local_load<float, kInside && !kAnyOffset, kAnyOffset>(a.ef[q] + at, idx, a.count, e[i]);
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int j = j0 + i;
        if (j < n) {
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
          through_codec<C, kEf, kInside && !kAnyOffset, ALGO != kLocalRing>(v, kEf && a.ef[q] ? a.ef[q] + at : nullptr, idx, a.count);
          if (ALGO == kLocalRing || (ALGO == kLocalOneShot && j == 0)) {
#pragma unroll
            for (int k = 0; k < 16; ++k) acc[k] = v[k];
          } else {
            combine16<C>(a.op, acc, v);
          }
        }
      }
    }
    if constexpr (ALGO == kLocalTwoShot) {   // the owner compresses the sum once more; everybody decodes that
      add_residual<kEf, kInside>(acc, a.ef[owner], idx, a.count);
      through_codec<C, kEf, kInside>(acc, a.ef[owner], idx, a.count);
    }
  }
  Wide16<T> o;
  pack16<T>(acc, o);
  if constexpr (ALGO == kLocalScatter) {
    local_store<T, kInside, kAnyOffset>(static_cast<T*>(a.recv[owner]), idx, a.count, o);
  } else {
#pragma unroll 1
    for (int p = 0; p < n; ++p) local_store<T, kInside>(static_cast<T*>(a.recv[p]), idx, a.count, o);
  }
}

// The ragged end of a message, and buffers off the 32-byte boundaries: out of line, because its
// branches and element loops cost the common unit registers.
template <class T, class C, int ALGO, bool kEf, bool kAnyOffset>
__device__ __noinline__ void local_reduce_ragged(const LocalReduceArgs& a, uint32_t s, size_t idx) {
  local_reduce_unit<T, C, ALGO, kEf, kAnyOffset, false>(a, s, idx);
}

template <class T, class C, int ALGO, bool kEf, bool kAnyOffset>
__global__ void __launch_bounds__(kLocalThreads, LocalShape<T, ALGO, kEf, kAnyOffset>::kCtas) local_reduce_kernel(const __grid_constant__ LocalReduceArgs a) {
  const int lane = threadIdx.x & 31;
  const uint32_t step = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < a.units; u += step) {
    const uint32_t s = ALGO == kLocalTwoShot || ALGO == kLocalRing || ALGO == kLocalScatter ? u / a.shard_units : 0u;
    const size_t e0 = (size_t)(ALGO == kLocalScatter ? u - s * a.shard_units : u) * kWarpElems;
    if (a.wide && e0 + kWarpElems <= a.count) local_reduce_unit<T, C, ALGO, kEf, kAnyOffset, true>(a, s, e0 + lane * kLaneElems);
    else local_reduce_ragged<T, C, ALGO, kEf, kAnyOffset>(a, s, e0 + lane * kLaneElems);
  }
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
  int nblocks;
  uint32_t run;
};

// kAnyOffset: blocks may start anywhere. Where the destinations of a block lie alike on their
// 32-byte sectors the warp rotates a unit once for all of them, and the first sector of a unit is
// completed with what the unit before left over, so that only the ends of a run are written
// element by element.
template <class T, class C, bool kAnyOffset>
__global__ void __launch_bounds__(kLocalThreads, kAnyOffset || sizeof(T) == 4 ? 3 : 4) local_exchange_kernel(const __grid_constant__ LocalExchangeArgs a) {
  constexpr int W = 4 * (int)sizeof(T), kPer = 4 / (int)sizeof(T);   // words of a lane, elements of a word
  const int lane = threadIdx.x & 31;
  const uint32_t step = (gridDim.x * blockDim.x) >> 5, runs = a.first_run[a.nblocks];
  int b = 0;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < runs; w += step) {
    while (w >= a.first_run[b + 1]) ++b;
    const T* src = static_cast<const T*>(a.src[b]);
    const size_t cnt = a.cnt[b];
    const int d0 = a.first_dst[b], d1 = a.first_dst[b + 1];
    const size_t u0 = (size_t)(w - a.first_run[b]) * a.run;
    size_t u1 = u0 + a.run;
    const size_t all = (cnt + kWarpElems - 1) / kWarpElems;
    if (u1 > all) u1 = all;
    uint32_t mis = 0;
    Wide16<T> left;   // lane 0: the last `mis` elements of the unit before
    if constexpr (kAnyOffset) {
      const uint32_t off = (uint32_t)(reinterpret_cast<uintptr_t>(a.dst[d0]) & 31);   // a unit is a whole number of sectors
      if (off & 15) {
        mis = off / (uint32_t)sizeof(T);
        for (int d = d0 + 1; d < d1; ++d)
          if ((uint32_t)(reinterpret_cast<uintptr_t>(a.dst[d]) & 31) != off) mis = 0;
      }
    }
    Wide16<T> next;
    load16_wide<T, kAnyOffset>(src, u0 * kWarpElems + lane * kLaneElems, cnt, next);
    bool carried = false;
    for (size_t u = u0; u < u1; ++u) {
      const size_t idx = u * kWarpElems + lane * kLaneElems;
      float v[16];
      wide16_to_f<T>(next, v);
      if (u + 1 < u1) load16_wide<T, kAnyOffset>(src, idx + kWarpElems, cnt, next);
      through_codec<C, false, true>(v, nullptr, 0, 0);
      Wide16<T> o;
      pack16<T>(v, o);
      if constexpr (kAnyOffset) {
        const bool whole = mis && (u + 1) * kWarpElems <= cnt;   // the same in all lanes
        if (whole) {
          rotate_up<T>(o.w, mis, lane);
          const Wide16<T> mine = o;   // lane 0: this unit's last `mis` elements, then its first 16 - mis
          if (lane == 0 && carried) {
#pragma unroll
            for (int k = 0; k < W; ++k) {
              if ((uint32_t)(kPer * k + kPer - 1) < mis) o.w[k] = left.w[k];
              else if (kPer == 2 && (uint32_t)(2 * k) < mis) o.w[k] = __byte_perm(left.w[k], o.w[k], 0x7610);
            }
          }
          const bool sector = lane != 0 || carried;
          for (int d = d0; d < d1; ++d) {
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
          carried = true;
          continue;
        }
      }
      for (int d = d0; d < d1; ++d) store16_wide<T, kAnyOffset>(static_cast<T*>(a.dst[d]), idx, cnt, o);
    }
    if constexpr (kAnyOffset) {
      if (carried && lane == 0) {   // behind the last whole unit of the run
        const size_t end = (u1 * kWarpElems <= cnt ? u1 : u1 - 1) * kWarpElems;
        for (int d = d0; d < d1; ++d) {
          T* p = static_cast<T*>(a.dst[d]) + end - mis;
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if ((uint32_t)i < mis) store_elem<T>(p + i, left.w[(i / kPer) & (W - 1)], i % kPer);
        }
      }
    }
  }
}

}  // namespace ccb
