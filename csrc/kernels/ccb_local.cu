// Instantiations and launches of the kernels for ranks that share one GPU (ccb_local.cuh).
#include <string.h>

#include "../rt/ccb_rt_internal.h"
#include "ccb_local.cuh"

namespace ccb {

template <class T, int ALGO, bool kEf, bool kAnyOffset>
static const void* reduce_by_codec(int codec) {
  switch (codec) {
    case CCB_CODEC_NONE: return reinterpret_cast<const void*>(&local_reduce_kernel<T, CodecNone<T>, ALGO, kEf, kAnyOffset>);
    case CCB_CODEC_INT8: return reinterpret_cast<const void*>(&local_reduce_kernel<T, CodecInt8<128>, ALGO, kEf, kAnyOffset>);
    case CCB_CODEC_FP8: return reinterpret_cast<const void*>(&local_reduce_kernel<T, CodecFp8, ALGO, kEf, kAnyOffset>);
    case CCB_CODEC_INT8_G256: return reinterpret_cast<const void*>(&local_reduce_kernel<T, CodecInt8<256>, ALGO, kEf, kAnyOffset>);
    case CCB_CODEC_INT4: return reinterpret_cast<const void*>(&local_reduce_kernel<T, CodecInt4, ALGO, kEf, kAnyOffset>);
    default: return nullptr;
  }
}
template <class T>
static const void* reduce_by_algo(int algo, int codec, bool ef, bool aligned) {
  switch (algo) {
    case kLocalTwoShot: return ef ? reduce_by_codec<T, kLocalTwoShot, true, false>(codec) : reduce_by_codec<T, kLocalTwoShot, false, false>(codec);
    case kLocalOneShot: return ef ? reduce_by_codec<T, kLocalOneShot, true, false>(codec) : reduce_by_codec<T, kLocalOneShot, false, false>(codec);
    case kLocalRing: return ef ? reduce_by_codec<T, kLocalRing, true, false>(codec) : reduce_by_codec<T, kLocalRing, false, false>(codec);
    case kLocalTree: return ef ? reduce_by_codec<T, kLocalTree, true, false>(codec) : reduce_by_codec<T, kLocalTree, false, false>(codec);
    case kLocalScatter:
      if (ef) return reduce_by_codec<T, kLocalScatter, true, true>(codec);
      return aligned ? reduce_by_codec<T, kLocalScatter, false, false>(codec) : reduce_by_codec<T, kLocalScatter, false, true>(codec);
    default: return nullptr;
  }
}
template <class T, bool kAnyOffset>
static const void* exchange_by_codec(int codec) {
  switch (codec) {
    case CCB_CODEC_NONE: return reinterpret_cast<const void*>(&local_exchange_kernel<T, CodecNone<T>, kAnyOffset>);
    case CCB_CODEC_INT8: return reinterpret_cast<const void*>(&local_exchange_kernel<T, CodecInt8<128>, kAnyOffset>);
    case CCB_CODEC_FP8: return reinterpret_cast<const void*>(&local_exchange_kernel<T, CodecFp8, kAnyOffset>);
    case CCB_CODEC_INT8_G256: return reinterpret_cast<const void*>(&local_exchange_kernel<T, CodecInt8<256>, kAnyOffset>);
    case CCB_CODEC_INT4: return reinterpret_cast<const void*>(&local_exchange_kernel<T, CodecInt4, kAnyOffset>);
    default: return nullptr;
  }
}

// CTAs of up to 256 threads; a call of few units gets narrower ones, so that it is spread over the
// chip all the same. One unit (or run) a warp: nothing is carried from one to the next, and the
// hardware hands out CTAs as others end (ring case above: 83 us so, 97 with resident CTAs that loop).
static int local_launch(ccb_comm* c, const void* fn, void* args, uint64_t warps, cudaStream_t stream) {
  const uint64_t sms = (uint64_t)comm_sms(c);
  uint64_t per = (warps + sms - 1) / sms;
  per = per < 1 ? 1 : per > kLocalThreads / 32 ? kLocalThreads / 32 : per;
  uint64_t ctas = (warps + per - 1) / per;
  if (ctas > (1u << 20)) ctas = 1u << 20;
  void* params[] = {args};
  const cudaError_t e = cudaLaunchKernel(fn, dim3((unsigned)(ctas ? ctas : 1)), dim3((unsigned)(32 * per)), params, 0, stream);
  if (e != cudaSuccess) {
    set_error("kernel launch failed: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}

static bool on32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }

int local_reduce(ccb_comm* c, const ReduceArgs& r, int algo, int dtype, int codec, cudaStream_t stream) {
  LocalReduceArgs a;
  memset(&a, 0, sizeof(a));
  a.n = r.c.nranks;
  a.op = r.op;
  a.root = -1;
  bool ef = false, aligned = true;
  for (int i = 0; i < a.n; ++i) {
    a.send[i] = r.send[i];
    a.recv[i] = r.recv[i];
    a.ef[i] = r.ef[i];
    ef = ef || r.ef[i];
    aligned = aligned && on32(r.send[i]) && on32(r.recv[i]) && on32(r.ef[i]);
  }
  a.shard_elems = r.shard_elems;
  uint64_t units = (r.count + kWarpElems - 1) / kWarpElems, shard_units = (r.shard_elems + kWarpElems - 1) / kWarpElems;
  a.count = r.count;
  if (algo == kLocalScatter) {
    if (r.mode == CCB_MODE_REDUCE) {
      a.root = r.root;
      a.shard_elems = 0;
      shard_units = units;
    } else {
      a.count = r.shard_elems;
      units = shard_units * (uint64_t)a.n;
      aligned = aligned && r.shard_elems * elem_size(dtype) % 32 == 0;
    }
  }
  if (units >> 31) {
    set_error("%llu elements in one call", (unsigned long long)r.count);
    return CCB_ERR_CAPACITY;
  }
  a.wide = aligned || algo == kLocalScatter;
  a.units = (uint32_t)units;
  a.shard_units = (uint32_t)shard_units;
  const void* fn = dtype == CCB_F32    ? reduce_by_algo<float>(algo, codec, ef, aligned)
                   : dtype == CCB_BF16 ? reduce_by_algo<__nv_bfloat16>(algo, codec, ef, aligned)
                   : dtype == CCB_F16  ? reduce_by_algo<__half>(algo, codec, ef, aligned)
                                       : nullptr;
  if (!fn) {
    set_error("unsupported dtype %d / codec %d", dtype, codec);
    return CCB_ERR_UNSUPPORTED;
  }
  return local_launch(c, fn, &a, units, stream);
}

int local_exchange(ccb_comm* c, const ExchangeArgs& x, bool aligned, int dtype, int codec, cudaStream_t stream) {
  const int n = x.c.nranks;
  const size_t es = elem_size(dtype);
  LocalExchangeArgs a;
  memset(&a, 0, sizeof(a));
  uint64_t units = 0;
  int dsts = 0;
  for (int r = 0; r < n; ++r) {
    int first = -1;
    bool same = true;
    for (int p = 0; p < n; ++p) {
      if (!x.cnt[r][p]) continue;
      if (first < 0) first = p;
      same = same && x.cnt[r][p] == x.cnt[r][first] && x.send_off[r][p] == x.send_off[r][first];
    }
    bool open = false;
    for (int p = 0; p < n; ++p) {
      if (!x.cnt[r][p]) continue;
      if (!open || !same) {   // a block of its own, or the one that all destinations share
        a.src[a.nblocks] = static_cast<const char*>(x.send[r]) + x.send_off[r][p] * es;
        a.cnt[a.nblocks] = x.cnt[r][p];
        a.first_dst[a.nblocks] = (uint8_t)dsts;
        units += (x.cnt[r][p] + kWarpElems - 1) / kWarpElems;
        ++a.nblocks;
        open = true;
      }
      a.dst[dsts++] = static_cast<char*>(x.recv[p]) + x.recv_off[p][r] * es;
    }
  }
  a.first_dst[a.nblocks] = (uint8_t)dsts;
  // Aligned blocks gain nothing by runs but the next unit's load ahead of this one's stores; at any
  // offset every run ends in element stores. Runs as long as leave every warp slot of the chip its own.
  const uint64_t slots = (uint64_t)comm_sms(c) * 24;
  a.run = 1;
  while (a.run < (aligned ? 2u : 8u) && units / (2 * a.run) >= slots) a.run *= 2;
  uint64_t runs = 0;
  for (int b = 0; b < a.nblocks; ++b) {
    a.first_run[b] = (uint32_t)runs;
    const uint64_t of = (a.cnt[b] + kWarpElems - 1) / kWarpElems;
    runs += (of + a.run - 1) / a.run;
  }
  a.first_run[a.nblocks] = (uint32_t)runs;
  if (units >> 31) {
    set_error("%llu units in one exchange", (unsigned long long)units);
    return CCB_ERR_CAPACITY;
  }
  const void* fn = nullptr;
  switch (dtype) {
    case CCB_F32: fn = aligned ? exchange_by_codec<float, false>(codec) : exchange_by_codec<float, true>(codec); break;
    case CCB_BF16: fn = aligned ? exchange_by_codec<__nv_bfloat16, false>(codec) : exchange_by_codec<__nv_bfloat16, true>(codec); break;
    case CCB_F16: fn = aligned ? exchange_by_codec<__half, false>(codec) : exchange_by_codec<__half, true>(codec); break;
  }
  if (!fn) {
    set_error("unsupported dtype %d / codec %d", dtype, codec);
    return CCB_ERR_UNSUPPORTED;
  }
  return local_launch(c, fn, &a, runs, stream);
}

}  // namespace ccb
