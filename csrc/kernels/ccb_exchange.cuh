// Fused codec + data-movement collectives over peer memory: AllGather(v),
// Broadcast, Scatter(v), Gather and AlltoAll(v) are all one "exchange": rank r
// compresses cnt[r][p] elements for peer p in registers, stores them into p's
// arena, flags; p decompresses every slot it was sent into its receive buffer.
//
// The reference builds each of these from per-peer quantize kernel + ncclSend /
// ncclRecv + dequantize kernel sequences with a host sync per step
// (plain_nccl_compress.cu:779-834 Broadcast, :917-965 AllGather, :1081-1147
// AllToAll; run_codes/wrappers/src/nccl/nccl_extensions.c:28-250 Scatter, Gather,
// AllGatherv, Scatterv as uncompressed byte-typed send/recv loops).
#pragma once
#include "ccb_reduce.cuh"

namespace ccb {

// kOwnDirect: a rank's own block need not go through its arena, the packet is decoded where it was
// encoded. Where buffers of the ranks of one process lie in one another (see the host) it is not
// so: then a rank's own block too is read before its flag and written after the others'. Two
// instantiations, because the choice as an argument cost up to 2 % of an all-gather at odd
// offsets (registers: 8 ranks, 2,097,153 fp32 values in int8, 173 against 176 us).
// kAnyOffset: blocks may start anywhere. Where all of them start on 16 bytes the form without it
// is smaller and spills nothing in fp32 (24 to 52 bytes with it): all-gather of 8 ranks of 2 Mi
// fp32 values in int8 167 us with it, 158 without, a broadcast of 4096 values among 4 ranks 10.4
// and 8.9.
template <class T, class C, bool kOwnDirect, bool kAnyOffset>
__global__ void __launch_bounds__(kThreads, 2) exchange_kernel(const __grid_constant__ ExchangeArgs a) {
  __shared__ CtaSync sync;
  const CommDev& c = a.c;
  const int lr = blockIdx.y, r = a.rank0 + lr, n = c.nranks;
  const int b = blockIdx.x, G = gridDim.x;
  const int lane_off = (threadIdx.x >> 5) * kWarpElems + (threadIdx.x & 31) * kLaneElems;
  const int warp_off = (threadIdx.x >> 5) * kWarpElems;
  // A tile is tile_warps x 512 elements: mid-size messages use narrow tiles so that they
  // still spread over all CTAs; warps beyond tile_warps only take part in the barriers.
  const size_t tile_elems = (size_t)a.tile_warps * kWarpElems;
  const bool active_warp = (int)(threadIdx.x >> 5) < a.tile_warps;
  const T* send = static_cast<const T*>(a.send[lr]);
  T* recv = static_cast<T*>(a.recv[lr]);
  char* my = c.arena[r];
  const size_t area = CCB_DATA_OFFSET + (size_t)(c.epoch & 1u) * c.half_bytes;
  const size_t pad = a.slot_pad;
  if (threadIdx.x == 0) sync.fail = 0;
  __syncthreads();

  // Same block for every destination (AllGather, Broadcast): encode once, store n times.
  bool same = true;
  uint32_t dstmask = 0;
  for (int p = 0; p < n; ++p) {
    if (a.cnt[r][p] == 0) continue;
    dstmask |= 1u << p;
    const int f = __ffs(dstmask) - 1;
    if (a.cnt[r][p] != a.cnt[r][f] || a.send_off[r][p] != a.send_off[r][f]) same = false;
  }

  // One tile is requested ahead of the one in work, so that a warp waits for memory once per
  // tile and not once per access. (All-gather among 8 ranks of 1,638,401 bf16 values each
  // in fp8: 673 us before, most of it element-wise stores at odd offsets, 100 after.)
  // (In fp32 a tile ahead is 16 registers more than the kernel has: there the load stays where it is used.)
  constexpr bool kAhead = sizeof(T) == 2, kPacketAhead = sizeof(typename C::Packet) <= 32;
  auto encode_block = [&](const T* src, size_t valid, auto&& deliver) {
    size_t t = b;
    Wide16<T> raw;
    bool have = active_warp && t * tile_elems + warp_off < valid;
    if (have && kAhead) load16_wide<T, kAnyOffset>(src, t * tile_elems + lane_off, valid, raw);
    while (have) {
      const size_t idx = t * tile_elems + lane_off;
      if (!kAhead) load16_wide<T, kAnyOffset>(src, idx, valid, raw);
      float v[16];
      wide16_to_f<T>(raw, v);
      t += G;
      have = t * tile_elems + warp_off < valid;
      if (have && kAhead) load16_wide<T, kAnyOffset>(src, t * tile_elems + lane_off, valid, raw);
      typename C::Packet pk;
      C::encode(v, pk);
      deliver(idx, pk);
    }
  };
  auto keep_own = [&](size_t idx, const typename C::Packet& pk) {
    float d[16];
    C::decode(pk, d);
    store16_wide<T, kAnyOffset>(recv + a.recv_off[r][r], idx, a.cnt[r][r], d);
  };
  const uint32_t staged = kOwnDirect ? dstmask & ~(1u << r) : dstmask;   // blocks that go through an arena
  const bool own = kOwnDirect && ((dstmask >> r) & 1u);
  constexpr int kFirst = kOwnDirect ? 1 : 0;
  if (dstmask && same) {
    const int f = __ffs(dstmask) - 1;
    encode_block(send + a.send_off[r][f], a.cnt[r][f], [&](size_t idx, const typename C::Packet& pk) {
      for (int j = kFirst; j < n; ++j) {
        const int p = r + j < n ? r + j : r + j - n;
        if ((staged >> p) & 1u) C::store(c.arena[p] + area + (size_t)r * a.slot_bytes, pad, idx, pk);
      }
      if (own) keep_own(idx, pk);
    });
  } else if (staged) {
    for (int j = kFirst; j < n; ++j) {
      const int p = r + j < n ? r + j : r + j - n;
      if (!((staged >> p) & 1u)) continue;
      char* dst = c.arena[p] + area + (size_t)r * a.slot_bytes;
      encode_block(send + a.send_off[r][p], a.cnt[r][p], [&](size_t idx, const typename C::Packet& pk) { C::store(dst, pad, idx, pk); });
    }
  }
  __syncthreads();
  const uint32_t peers = dstmask & ~(1u << r);
  if (threadIdx.x == 0 && peers) signal_peers(c, peers, 0, r, b);
  // The own block of an exchange with several different blocks comes after the others have
  // been read (its place in recv may be another block's place in send), while they travel.
  if (own && !same) encode_block(send + a.send_off[r][r], a.cnt[r][r], keep_own);

  uint32_t srcmask = 0;
  for (int q = 0; q < n; ++q)
    if (q != r && a.cnt[q][r]) srcmask |= 1u << q;   // what this CTA put into its own arena it reads back itself
  if (srcmask && !cta_wait_sources(sync, c, my, 0, r, srcmask, 0x30)) return;
  for (int j = kFirst; j < n; ++j) {
    const int q = r + j < n ? r + j : r + j - n;
    const size_t valid = a.cnt[q][r];
    const char* slot = my + area + (size_t)q * a.slot_bytes;
    T* dst = recv + a.recv_off[r][q];
    size_t t = b;
    typename C::Packet nxt;
    bool have = active_warp && t * tile_elems + warp_off < valid;
    if (have && kPacketAhead) C::load(slot, pad, t * tile_elems + lane_off, nxt);
    while (have) {
      const size_t idx = t * tile_elems + lane_off;
      if (!kPacketAhead) C::load(slot, pad, idx, nxt);
      const typename C::Packet pk = nxt;
      t += G;
      have = t * tile_elems + warp_off < valid;
      if (have && kPacketAhead) C::load(slot, pad, t * tile_elems + lane_off, nxt);
      float d[16];
      C::decode(pk, d);
      store16_wide<T, kAnyOffset>(dst, idx, valid, d);
    }
  }
  if (a.ack) end_handshake(sync, c, r);
}

}  // namespace ccb
