// MoE dispatch and combine over peer memory with per-destination compression
// (fp8 e4m3 + ue8m0 block scales by default): see include/ccb/ccb_moe.h.
//
// Work unit = 512 consecutive elements of one row (a warp); a CTA tile = 16 units.
// Unit u of the block (src -> dst) is always handled by CTA ((u / 16) mod G) on both
// sides, so dispatch needs only per-CTA flags. The combine's receive side gathers
// rows by token, which may have been written by any CTA of the source, so it waits
// for ALL CTA flags of every source before reading.
#include <cuda_runtime.h>
#include <string.h>

#include "../rt/ccb_rt_internal.h"
#include "ccb/ccb_moe.h"
#include "ccb_local.cuh"
#include "ccb_reduce.cuh"

namespace ccb {

struct MoeArgs {
  CommDev c;
  const void* src[CCB_MAX_RANKS];        // x (dispatch) or y (combine), per local rank
  void* dst[CCB_MAX_RANKS];              // recv rows (dispatch) or out tokens (combine)
  const int32_t* perm[CCB_MAX_RANKS];    // dispatch: send order -> token row
  const int32_t* dest_rank[CCB_MAX_RANKS];
  const int32_t* pos[CCB_MAX_RANKS];
  const float* gate[CCB_MAX_RANKS];
  uint64_t cnt[CCB_MAX_RANKS][CCB_MAX_RANKS];   // rows [src][dst] (dispatch direction)
  uint64_t hidden, tokens;
  uint64_t slot_pad, slot_bytes;          // per (src,dst) slot, elements / bytes
  int topk;
  int rank0, nlocal;
};

// One body, two instantiations: each direction has registers of its own (as one kernel, fp32
// without a codec spilled 92 bytes with the unit ahead; so no more than 20 anywhere, in fp32 combines).
template <class T, class C, bool kCombine>
__global__ void __launch_bounds__(kThreads, 2) moe_kernel(const __grid_constant__ MoeArgs a) {
  __shared__ CtaSync sync;
  const CommDev& c = a.c;
  const int lr = blockIdx.y, r = a.rank0 + lr, n = c.nranks;
  const int b = blockIdx.x, G = gridDim.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const T* src = static_cast<const T*>(a.src[lr]);
  T* dst = static_cast<T*>(a.dst[lr]);
  char* my = c.arena[r];
  const size_t area = CCB_DATA_OFFSET + (size_t)(c.epoch & 1u) * c.half_bytes;
  const size_t H = a.hidden;
  const unsigned int upr = (unsigned int)(H / kWarpElems);  // units per row (constant divisor above: a shift)
  // unit -> (row, column) without a 64-bit division per unit: a shift when a row is a power
  // of two of units (the usual hidden sizes), else a 32-bit division
  const int upr_shift = (upr & (upr - 1u)) == 0 ? __ffs((int)upr) - 1 : -1;
  auto row_of = [&](size_t u, size_t& col) -> size_t {
    const unsigned int u32 = (unsigned int)u;
    const unsigned int j = upr_shift >= 0 ? (u32 >> upr_shift) : (u32 / upr);
    col = (size_t)(u32 - j * upr) * kWarpElems + (size_t)lane * kLaneElems;
    return j;
  };
  const size_t pad = a.slot_pad;
  if (threadIdx.x == 0) sync.fail = 0;
  __syncthreads();

  // ---- send: block (r -> p). Dispatch gathers rows through perm; combine sends the
  // ---- contiguous block of rows that came from origin p (transposed counts).
  // Destinations are visited starting with the next rank, (r + 1) % n, ..., r: at any moment
  // every rank stores to a different peer, so no inbound link takes all the traffic. In both send
  // phases and in a dispatch's receive the next unit is requested before the one in hand is
  // converted: a unit's address may hang on an index load, and a warp that did one unit at a time
  // waited for both in turn. A dispatch decodes its own rows where it encoded them, after the
  // peers have been told. (8 ranks, 8192 x 4096 bf16, top 2, fp8: dispatch 583 us one unit at a
  // time, 517 so. With the combine's 508 that is 5.4 GB of staged rows, 820 us at 6.55 TB/s.)
  auto send_block = [&](int p, auto&& deliver) {
    const size_t rows = kCombine ? a.cnt[p][r] : a.cnt[r][p];
    size_t base_row = 0, send_row_off = 0;  // combine: first row of origin p; dispatch: offset into perm
    for (int s = 0; s < p; ++s) {
      base_row += a.cnt[s][r];
      send_row_off += a.cnt[r][s];
    }
    const size_t units = rows * upr;
    size_t u = (size_t)b * kWarps + warp, idx = 0;
    Wide16<T> raw;
    auto request = [&]() {
      size_t col;
      const size_t j = row_of(u, col);
      const size_t srow = kCombine ? base_row + j : (size_t)a.perm[lr][send_row_off + j];
      load16_wide<T>(src + srow * H, col, H, raw);
      idx = j * H + col;
    };
    if (u < units) request();
    while (u < units) {
      const size_t at = idx;
      float v[16];
      wide16_to_f<T>(raw, v);
      u += (size_t)G * kWarps;
      if (u < units) request();
      typename C::Packet pk;
      C::encode(v, pk);
      deliver(at, pk);
    }
  };
  for (int jd = 1; jd <= (kCombine ? n : n - 1); ++jd) {
    const int p = r + jd < n ? r + jd : r + jd - n;
    char* slot = c.arena[p] + area + (size_t)r * a.slot_bytes;
    send_block(p, [&](size_t at, const typename C::Packet& pk) { C::store(slot, pad, at, pk); });
  }
  __syncthreads();
  // the combine's receiver gathers rows written by any CTA, its own rank's included,
  // so there the flag goes to this rank's own arena as well
  if (threadIdx.x == 0) signal_peers(c, kCombine ? (1u << n) - 1u : ((1u << n) - 1u) & ~(1u << r), 0, r, b);

  if constexpr (!kCombine) {
    // ---- dispatch receive: rows of source q land at recv row (sum_{s<q} cnt[s][r]) + j
    // own rows first (nothing to wait for), then each source as its flag arrives, in the
    // order in which the sources reach this rank
    auto first_row = [&](int q) {
      size_t row0 = 0;
      for (int s = 0; s < q; ++s) row0 += a.cnt[s][r];
      return row0;
    };
    {
      // index and column of a unit make one offset into the slot and, with H elements a row, into dst
      T* mine = dst + first_row(r) * H;
      send_block(r, [&](size_t at, const typename C::Packet& pk) {
        float d[16];
        C::decode(pk, d);
        store16_wide<T>(mine, at, at + 16, d);
      });
    }
    for (int jq = 1; jq < n; ++jq) {
      const int q = (r - jq + n) % n;
      if (!cta_wait_sources(sync, c, my, 0, r, 1u << q, 0xB0)) return;
      const size_t units = a.cnt[q][r] * upr;
      const char* slot = my + area + (size_t)q * a.slot_bytes;
      T* to = dst + first_row(q) * H;
      size_t u = (size_t)b * kWarps + warp;
      const size_t step = (size_t)G * kWarps;
      typename C::Packet nxt;
      // unit u of a block of whole rows starts at element 512 u
      if (u < units) C::load(slot, pad, u * kWarpElems + (size_t)lane * kLaneElems, nxt);
      while (u < units) {
        const size_t at = u * kWarpElems + (size_t)lane * kLaneElems;
        const typename C::Packet pk = nxt;
        u += step;
        if (u < units) C::load(slot, pad, u * kWarpElems + (size_t)lane * kLaneElems, nxt);
        float d[16];
        C::decode(pk, d);
        store16_wide<T>(to, at, at + 16, d);
      }
    }
  } else {
    // ---- combine receive: wait for every CTA of every source, then gather per token
    for (int i = threadIdx.x; i < n * G; i += kThreads) {
      const int q = i / G, cb = i % G;
      if (!wait_flag(flag_ptr(my, 0, q, cb), c.epoch, c, my, 0xC0 | (q << 8))) sync.fail = 1;
    }
    __syncthreads();
    if (sync.fail) {
      if (threadIdx.x == 0) broadcast_abort(c, c.epoch);
      return;
    }
    const size_t units = a.tokens * upr;
    // One pair at a time: the 16 warps of a CTA hide the loads of one another, and an index sequence
    // that ran ahead of the packets cost more than it hid (8 ranks of 2048 x 2048 bf16 in fp8: 138
    // us with it and 131 without at top 4, 83 and 80 at top 2, 52 and 54 at top 1).
    for (size_t u = (size_t)b * kWarps + warp; u < units; u += (size_t)G * kWarps) {
      size_t col;
      const size_t tok = row_of(u, col);
      float acc[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[i] = 0.f;
      for (int k = 0; k < a.topk; ++k) {
        const uint32_t q = (uint32_t)a.dest_rank[lr][tok * a.topk + k], j = (uint32_t)a.pos[lr][tok * a.topk + k];
        const float g = a.gate[lr][tok * a.topk + k];
        // For a dropped pair no row was sent; it fetches one that lies in the arena and adds nothing. (With
        // a branch round the fetch a combine of 2048 x 2048 rows, top 1, took 58.7 us and not 53.5.)
        const bool sent = q < (uint32_t)n && j < (uint32_t)a.cnt[r][q < (uint32_t)n ? q : 0u];
        typename C::Packet pk;
        C::load(my + area + (size_t)(sent ? q : 0u) * a.slot_bytes, pad, (size_t)(sent ? j : 0u) * H + col, pk);
        float d[16];
        C::decode(pk, d);
        if (sent) {
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i] += g * d[i];
        }
      }
      store16_wide<T>(dst + tok * H, col, H, acc);
    }
  }
}

// Ranks that share one GPU (see ccb_local.cuh): rows go from the senders' tensors to the receivers'
// through the codec in registers, without staging and flags.
struct MoeLocalArgs {
  const void* src[CCB_MAX_RANKS];
  void* dst[CCB_MAX_RANKS];
  const int32_t* perm[CCB_MAX_RANKS];
  const int32_t* dest_rank[CCB_MAX_RANKS];
  const int32_t* pos[CCB_MAX_RANKS];
  const float* gate[CCB_MAX_RANKS];
  uint32_t cnt[CCB_MAX_RANKS][CCB_MAX_RANKS];      // rows [src][dst]
  uint32_t first_in[CCB_MAX_RANKS][CCB_MAX_RANKS];   // [holder][origin]: first row of that origin in the holder's buffer
  uint32_t first_out[CCB_MAX_RANKS][CCB_MAX_RANKS];  // [src][dst]: first entry of that block in perm
  uint64_t hidden;
  uint32_t tokens, row_units, chunk_rows, chunks;   // a chunk of a block: its rows for one CTA
  uint32_t batch_units, groups;                     // units of a row for a warp, such groups of units in a row
  int topk, n;
};
// Both ways a warp brings what it works on to shared memory first, up to 4 KiB under way at once.
constexpr int kMoeLocalThreads = 128, kMoeStage = 4096;
template <class T> constexpr int kMoeSlots = kMoeStage / 16 / kUnitPieces<T>;   // units of 512 elements in it
template <class T>
__device__ __forceinline__ void moe_bring(uint4* stage, const char* from, uint32_t units) {   // consecutive units
#pragma unroll 1
  for (uint32_t u = 0; u < units; ++u, from += kWarpElems * sizeof(T), stage += kUnitPieces<T>) bring_unit<T>(stage, reinterpret_cast<const T*>(from));
}
__device__ __forceinline__ void moe_brought() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// Dispatch. The rows of a rank are sorted by destination, and within one by token. A CTA takes
// `chunk_rows` rows of one block, a warp some units of a row at a time; the blocks of a rank take turns chunk by
// chunk, so that the topk copies of a token, which lie at about the same depth of their blocks, are
// read from memory once and from L2 after that.
template <class T, class C>
__global__ void __launch_bounds__(kMoeLocalThreads, 12) moe_local_dispatch_kernel(const __grid_constant__ MoeLocalArgs a) {
  after_kernel_before();
  __shared__ uint4 stages[kMoeLocalThreads / 32][kMoeStage / 16];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t n = (uint32_t)a.n, p = blockIdx.x % n, c = blockIdx.x / n % a.chunks, r = blockIdx.x / n / a.chunks;
  const uint32_t j0 = c * a.chunk_rows, rows = a.cnt[r][p];
  if (j0 >= rows) return;
  const uint32_t items = min(a.chunk_rows, rows - j0) * a.groups;
  const int32_t* perm = a.perm[r] + a.first_out[r][p] + j0;
  T* dst = static_cast<T*>(a.dst[p]) + (size_t)(a.first_in[p][r] + j0) * a.hidden;
#pragma unroll 1
  for (uint32_t i = warp; i < items; i += blockDim.x / 32) {
    const uint32_t j = i / a.groups, u0 = (i - j * a.groups) * a.batch_units, units = min(a.batch_units, a.row_units - u0);
    moe_bring<T>(stages[warp], reinterpret_cast<const char*>(static_cast<const T*>(a.src[r]) + (size_t)perm[j] * a.hidden + (size_t)u0 * kWarpElems), units);
    moe_brought();
    T* out = dst + (size_t)j * a.hidden + (size_t)u0 * kWarpElems;
#pragma unroll 1
    for (uint32_t u = 0; u < units; ++u) {
      float v[16];
      brought_unit<T>(stages[warp] + u * kUnitPieces<T>, v);
      C::round_trip(v);
      Wide16<T> o;
      pack16<T>(v, o);
      local_store<T>(out, (size_t)u * kWarpElems + lane * kLaneElems, 0, true, o);
    }
    __syncwarp();
  }
}

// Combine: a warp takes some units of 512 elements of one token and brings them from all rows that hold the token to
// shared memory, 4 KiB under way at once, where a row at a time in registers left a warp waiting for one row after
// the other, 1 KiB each. An index outside its block (the entry of a dropped pair) contributes nothing.
// (8 ranks, 8192 x 4096 bf16, top 2, fp8: 328 us a row at a time with 40 warps an SM, 267 so, of 246 that the memory
// needs; top 4 of 2048 x 2048 in int8, bound by its codec, 84 and 84. 36 warps an SM, 56 registers: with 40, which spill, 265
// but 98 at top 4, with 32 276. B200.)
template <class T, class C>
__global__ void __launch_bounds__(kMoeLocalThreads, 9) moe_local_combine_kernel(const __grid_constant__ MoeLocalArgs a) {
  after_kernel_before();
  constexpr int kSlots = kMoeSlots<T>;
  __shared__ uint4 stages[kMoeLocalThreads / 32][kMoeStage / 16];
  const uint32_t lane = threadIdx.x & 31;
  uint4* stage = stages[threadIdx.x >> 5];
  const uint32_t w = ccb_grid_warp(blockIdx.x, blockDim.x, threadIdx.x), per_rank = a.tokens * a.groups;
  if (w >= per_rank * (uint32_t)a.n) return;
  const uint32_t r = w / per_rank, item = w - r * per_rank, tok = item / a.groups, u0 = (item - tok * a.groups) * a.batch_units;
  const uint32_t units = min(a.batch_units, a.row_units - u0);
  const size_t pair0 = (size_t)tok * a.topk;
  const int32_t* dest = a.dest_rank[r] + pair0;
  const int32_t* pos = a.pos[r] + pair0;
  const float* gate = a.gate[r] + pair0;
  T* out = static_cast<T*>(a.dst[r]) + (size_t)tok * a.hidden + (size_t)u0 * kWarpElems;
  float acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  int k0 = 0;
#pragma unroll 1
  do {   // more than one turn: units is 1; one all the same where a token has no rows, whose sum is 0
    const uint32_t rows = (uint32_t)min(kSlots, a.topk - k0);
    const char* row = nullptr;   // lane k: the k-th row from the unit on
    float gate_k = 0.f;
    bool held = false;
    if (lane < rows) {
      const uint32_t q = (uint32_t)dest[k0 + lane], j = (uint32_t)pos[k0 + lane];
      gate_k = gate[k0 + lane];
      held = q < (uint32_t)a.n && j < a.cnt[r][q];
      if (held) row = reinterpret_cast<const char*>(static_cast<const T*>(a.src[q]) + (size_t)(a.first_in[q][r] + j) * a.hidden + (size_t)u0 * kWarpElems);
    }
    const uint32_t all = __ballot_sync(0xffffffffu, held);
#pragma unroll 1
    for (uint32_t k = 0; k < rows; ++k) {
      const char* from = reinterpret_cast<const char*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(row), k));
      if (all >> k & 1u) moe_bring<T>(stage + k * a.batch_units * kUnitPieces<T>, from, units);
    }
    moe_brought();
#pragma unroll 1
    for (uint32_t u = 0; u < units; ++u) {
#pragma unroll 1
      for (uint32_t k = 0; k < rows; ++k) {
        const float g = __shfl_sync(0xffffffffu, gate_k, k);
        if (!(all >> k & 1u)) continue;
        float d[16];
        brought_unit<T>(stage + (k * a.batch_units + u) * kUnitPieces<T>, d);
        C::round_trip(d);
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] += g * d[e];
      }
      if (k0 + kSlots >= a.topk) {
        Wide16<T> o;
        pack16<T>(acc, o);
        local_store<T>(out + (size_t)u * kWarpElems, lane * kLaneElems, 0, true, o);
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = 0.f;
      }
    }
    __syncwarp();
    k0 += kSlots;
  } while (k0 < a.topk);
}

template <template <class, class> class K>
static const void* moe_by_type(int dtype, int codec) {
#define CCB_MOE_CODEC(T)                                                  \
  switch (codec) {                                                        \
    case CCB_CODEC_NONE: return K<T, CodecNone<T>>::fn();                 \
    case CCB_CODEC_INT8: return K<T, CodecInt8<128>>::fn();               \
    case CCB_CODEC_INT8_G256: return K<T, CodecInt8<256>>::fn();          \
    case CCB_CODEC_FP8: return K<T, CodecFp8>::fn();                      \
    case CCB_CODEC_INT4: return K<T, CodecInt4>::fn();                    \
    default: return nullptr;                                              \
  }
  switch (dtype) {
    case CCB_F32: CCB_MOE_CODEC(float)
    case CCB_BF16: CCB_MOE_CODEC(__nv_bfloat16)
    case CCB_F16: CCB_MOE_CODEC(__half)
  }
#undef CCB_MOE_CODEC
  return nullptr;
}
template <class T, class C> struct MoeDispatch { static const void* fn() { return reinterpret_cast<const void*>(&moe_kernel<T, C, false>); } };
template <class T, class C> struct MoeCombine { static const void* fn() { return reinterpret_cast<const void*>(&moe_kernel<T, C, true>); } };
template <class T, class C> struct MoeLocalDispatch { static const void* fn() { return reinterpret_cast<const void*>(&moe_local_dispatch_kernel<T, C>); } };
template <class T, class C> struct MoeLocalCombine { static const void* fn() { return reinterpret_cast<const void*>(&moe_local_combine_kernel<T, C>); } };

static int moe_local_launch(ccb_comm* c, const MoeArgs& m, bool combine, int dtype, int codec, uint64_t max_rows, cudaStream_t stream) {
  MoeLocalArgs a;
  memset(&a, 0, sizeof(a));
  a.n = ccb_comm_nranks(c);
  for (int i = 0; i < a.n; ++i) {
    a.src[i] = m.src[i];
    a.dst[i] = m.dst[i];
    a.perm[i] = m.perm[i];
    a.dest_rank[i] = m.dest_rank[i];
    a.pos[i] = m.pos[i];
    a.gate[i] = m.gate[i];
    for (int k = 0; k < a.n; ++k) {
      a.cnt[i][k] = (uint32_t)m.cnt[i][k];
      for (int s = 0; s < k; ++s) {
        a.first_in[i][k] += (uint32_t)m.cnt[s][i];
        a.first_out[i][k] += (uint32_t)m.cnt[i][s];
      }
    }
  }
  a.hidden = m.hidden;
  a.row_units = (uint32_t)(m.hidden / kWarpElems);
  a.tokens = (uint32_t)m.tokens;
  a.topk = m.topk > 0 ? m.topk : 0;
  const uint32_t slots = dtype == CCB_F32 ? kMoeSlots<float> : kMoeSlots<__half>, rows = combine ? (uint32_t)a.topk < slots ? (uint32_t)a.topk : slots : 1u;
  a.batch_units = rows ? slots / rows : 1u;
  if (a.batch_units > a.row_units) a.batch_units = a.row_units;
  a.groups = (a.row_units + a.batch_units - 1) / a.batch_units;
  uint64_t ctas, warps = kMoeLocalThreads / 32;
  if (combine) {
    const uint64_t items = (uint64_t)a.n * m.tokens * a.groups, sms = (uint64_t)comm_sms(c);
    while (warps > 1 && items / warps < sms) --warps;
    ctas = (items + warps - 1) / warps;
  } else {
    a.chunk_rows = warps > a.groups ? (uint32_t)(warps / a.groups) : 1u;   // about an item a warp
    a.chunks = (uint32_t)((max_rows + a.chunk_rows - 1) / a.chunk_rows);
    ctas = (uint64_t)a.n * a.n * a.chunks;
  }
  if (ctas == 0) return CCB_OK;
  const void* fn = combine ? moe_by_type<MoeLocalCombine>(dtype, codec) : moe_by_type<MoeLocalDispatch>(dtype, codec);
  void* params[] = {&a};
  const cudaError_t e = launch_next(fn, dim3((unsigned)ctas), dim3((unsigned)(32 * warps)), params, 0, stream);
  if (e != cudaSuccess) {
    set_error("kernel launch failed: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

static int moe_launch(ccb_comm* c, const void* fn, MoeArgs& a, bool combine, int dtype, int codec, uint64_t max_rows, uint64_t work_rows, cudaStream_t stream) {
  if (!fn) {
    set_error("unsupported dtype %d / codec %d", dtype, codec);
    return CCB_ERR_UNSUPPORTED;
  }
  if (a.hidden == 0 || a.hidden % kWarpElems) {
    set_error("hidden size must be a multiple of %d", kWarpElems);
    return CCB_ERR_ARG;
  }
  const int n = ccb_comm_nranks(c);
  a.slot_pad = (max_rows ? max_rows : 1) * a.hidden;
  a.slot_bytes = codec_slot_bytes(codec, dtype, a.slot_pad);
  a.c = comm_dev(c, 0);
  if ((uint64_t)n * a.slot_bytes > a.c.half_bytes) {
    set_error("arena too small: MoE blocks of %llu rows need %llu bytes of staging", (unsigned long long)max_rows,
              (unsigned long long)((uint64_t)n * a.slot_bytes * 2));
    return CCB_ERR_CAPACITY;
  }
  const size_t units = (size_t)work_rows * (a.hidden / kWarpElems);
  if (units >> 32 || ((uint64_t)max_rows * (a.hidden / kWarpElems)) >> 32) {  // the kernel indexes units with 32 bits
    set_error("MoE block too large: %llu rows of %llu elements", (unsigned long long)work_rows, (unsigned long long)a.hidden);
    return CCB_ERR_CAPACITY;
  }
  // The kernels above index all ranks' units, and the rows of a buffer, with 32 bits. A combine over
  // the arena has read all rows before it writes a token, so there its results may lie on the rows.
  // (A dispatch has not, there or here: its results may not lie on what the ranks send.)
  uint64_t all_rows = 0;
  bool apart = true, aligned = true;
  for (int s = 0; s < n; ++s) {
    aligned = aligned && ((reinterpret_cast<uintptr_t>(a.src[s]) | reinterpret_cast<uintptr_t>(a.dst[s])) & 31) == 0;
    uint64_t rows = 0;
    for (int d = 0; d < n; ++d) rows += a.cnt[d][s];
    all_rows += rows;
    const uint64_t row_bytes = a.hidden * elem_size(dtype);
    for (int d = 0; combine && d < n; ++d) {
      const uintptr_t y = reinterpret_cast<uintptr_t>(a.src[s]), out = reinterpret_cast<uintptr_t>(a.dst[d]);
      apart = apart && !(y < out + a.tokens * row_bytes && out < y + rows * row_bytes);
    }
  }
  if (ranks_in_registers(c) && apart && aligned && !(((all_rows + (uint64_t)n * a.tokens) * (a.hidden / kWarpElems)) >> 31))
    return moe_local_launch(c, a, combine, dtype, codec, max_rows, stream);
  a.c = comm_dev(c, next_epoch(c));
  a.rank0 = ccb_comm_rank(c);
  a.nlocal = ccb_comm_nlocal(c);
  size_t tiles = (units + kWarps - 1) / kWarps;
  int cap = grid_cap(c, fn);
  if (tiles < 1) tiles = 1;
  return launch(c, fn, tiles < (size_t)cap ? (int)tiles : cap, &a, stream);
}

}  // namespace ccb

using namespace ccb;

extern "C" int ccb_moe_dispatch(ccb_comm* c, const void* const* x, void* const* recv, const int32_t* const* perm,
                                const uint64_t* counts, uint64_t hidden, int dtype, int codec, ccb_stream_t stream) {
  int rc = check_alive(c);
  if (rc) return rc;
  const int n = ccb_comm_nranks(c), nl = ccb_comm_nlocal(c);
  MoeArgs a;
  memset(&a, 0, sizeof(a));
  uint64_t mx = 0;
  for (int s = 0; s < n; ++s)
    for (int d = 0; d < n; ++d) {
      a.cnt[s][d] = counts[s * n + d];
      if (a.cnt[s][d] > mx) mx = a.cnt[s][d];
    }
  for (int i = 0; i < nl; ++i) {
    a.src[i] = x[i];
    a.dst[i] = recv[i];
    a.perm[i] = perm[i];
  }
  a.hidden = hidden;
  return moe_launch(c, moe_by_type<MoeDispatch>(dtype, codec), a, false, dtype, codec, mx, mx, static_cast<cudaStream_t>(stream));
}

extern "C" int ccb_moe_combine(ccb_comm* c, const void* const* y, void* const* out, const int32_t* const* dest_rank,
                               const int32_t* const* pos, const float* const* gate, const uint64_t* counts, uint64_t tokens,
                               int topk, uint64_t hidden, int dtype, int codec, ccb_stream_t stream) {
  int rc = check_alive(c);
  if (rc) return rc;
  const int n = ccb_comm_nranks(c), nl = ccb_comm_nlocal(c);
  MoeArgs a;
  memset(&a, 0, sizeof(a));
  uint64_t mx = 0;
  for (int s = 0; s < n; ++s)
    for (int d = 0; d < n; ++d) {
      a.cnt[s][d] = counts[s * n + d];
      if (a.cnt[s][d] > mx) mx = a.cnt[s][d];
    }
  for (int i = 0; i < nl; ++i) {
    a.src[i] = y[i];
    a.dst[i] = out[i];
    a.dest_rank[i] = dest_rank[i];
    a.pos[i] = pos[i];
    a.gate[i] = gate[i];
  }
  a.hidden = hidden;
  a.tokens = tokens;
  a.topk = topk;
  return moe_launch(c, moe_by_type<MoeCombine>(dtype, codec), a, true, dtype, codec, mx, tokens > mx ? tokens : mx, static_cast<cudaStream_t>(stream));
}
