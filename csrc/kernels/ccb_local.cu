// Launches of the kernels for ranks that share one GPU (ccb_local.cuh).
#include <string.h>

#include "../rt/ccb_rt_internal.h"
#include "ccb_local_table.cuh"

namespace ccb {

extern template const void* local_kernel<float>(const LocalKey&);
extern template const void* local_kernel<__nv_bfloat16>(const LocalKey&);
extern template const void* local_kernel<__half>(const LocalKey&);

static const void* find(int dtype, const LocalKey& k) {
  switch (dtype) {
    case CCB_F32: return local_kernel<float>(k);
    case CCB_BF16: return local_kernel<__nv_bfloat16>(k);
    case CCB_F16: return local_kernel<__half>(k);
    default: return nullptr;
  }
}

// One unit (or run) a warp (ring, 4 ranks of 64 MiB of bf16 in fp8: 83 us so, 97 with resident CTAs
// that loop). CTAs of up to 128 threads; a call of few units gets narrower ones, to be spread over
// the chip all the same.
static int local_launch(ccb_comm* c, const void* fn, void* args, uint64_t warps, cudaStream_t stream) {
  const uint64_t sms = (uint64_t)comm_sms(c);
  uint64_t per = (warps + sms - 1) / sms;
  per = per < 1 ? 1 : per > kLocalThreads / 32 ? kLocalThreads / 32 : per;
  const uint64_t ctas = (warps + per - 1) / per;
  void* params[] = {args};
  const cudaError_t e = launch_next(fn, dim3((unsigned)(ctas ? ctas : 1)), dim3((unsigned)(32 * per)), params, 0, stream);
  if (e != cudaSuccess) {
    set_error("kernel launch failed: %s", cudaGetErrorString(e));
    return CCB_ERR_CUDA;
  }
  count_launch();
  return CCB_OK;
}
static int no_kernel(int dtype, int codec, uint64_t units) {
  if (units >> 31) {
    set_error("%llu units of 512 elements in one call", (unsigned long long)units);
    return CCB_ERR_CAPACITY;
  }
  set_error("unsupported dtype %d / codec %d", dtype, codec);
  return CCB_ERR_UNSUPPORTED;
}

static bool on32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }

static bool reduce_aligned(const ReduceArgs& r, size_t es, bool* ef) {
  bool aligned = r.mode != CCB_MODE_REDUCESCATTER || r.shard_elems * es % 32 == 0;
  *ef = false;
  for (int i = 0; i < r.c.nranks; ++i) {
    *ef = *ef || r.ef[i];
    aligned = aligned && on32(r.send[i]) && on32(r.recv[i]) && on32(r.ef[i]);
  }
  return aligned;
}

// Residuals want every buffer on 32 bytes; the others have forms for any offset. (4 ranks of 25 MiB of
// bf16 in int8 with residuals: 96 us so; by the kernels over peer memory 159 with values on 16 bytes,
// 326 with residuals on 4, 490 with values on 2. Without residuals, values on 2 bytes, 58 here. B200.)
bool local_reduce_takes(const ReduceArgs& r, int dtype) {
  bool ef;
  return reduce_aligned(r, elem_size(dtype), &ef) || !ef;
}

int local_reduce(ccb_comm* c, const ReduceArgs& r, int algo, int dtype, int codec, cudaStream_t stream) {
  LocalKey key = {LocalKey::kReduce, algo, codec, false, false};
  key.aligned = reduce_aligned(r, elem_size(dtype), &key.ef);
  LocalReduceArgs a;
  memset(&a, 0, sizeof(a));
  a.n = r.c.nranks;
  a.op = r.op;
  a.root = -1;
  for (int i = 0; i < a.n; ++i) {
    a.send[i] = r.send[i];
    a.recv[i] = r.recv[i];
    a.ef[i] = r.ef[i];
  }
  a.shard_elems = r.shard_elems;
  uint64_t units = (r.count + kWarpElems - 1) / kWarpElems, shard_units = (r.shard_elems + kWarpElems - 1) / kWarpElems;
  a.count = r.count;
  if (r.mode == CCB_MODE_REDUCE) {
    a.root = r.root;
    a.shard_elems = 0;
    shard_units = units;
  } else if (r.mode == CCB_MODE_REDUCESCATTER) {
    a.count = r.shard_elems;
    units = shard_units * (uint64_t)a.n;
  }
  const void* fn = find(dtype, key);
  if (!fn || units >> 31) return no_kernel(dtype, codec, units);
  a.units = (uint32_t)units;
  a.shard_units = (uint32_t)shard_units;
  return local_launch(c, fn, &a, units, stream);
}

bool local_solo_takes(const void* send, const void* recv, const float* ef) { return !ef || (on32(send) && on32(recv) && on32(ef)); }

int local_solo(ccb_comm* c, const void* send, void* recv, float* ef, uint64_t count, int dtype, int codec, cudaStream_t stream) {
  LocalReduceArgs a;
  memset(&a, 0, sizeof(a));
  a.n = 1;
  a.send[0] = send;
  a.recv[0] = recv;
  a.ef[0] = ef;
  a.count = count;
  const void* fn = find(dtype, LocalKey{LocalKey::kSolo, 0, codec, ef != nullptr, on32(send) && on32(recv) && on32(ef)});
  const uint64_t units = (count + kWarpElems - 1) / kWarpElems;
  if (!fn || units >> 31) return no_kernel(dtype, codec, units);
  return local_launch(c, fn, &a, units, stream);
}

int local_exchange(ccb_comm* c, const ExchangeArgs& x, int dtype, int codec, cudaStream_t stream) {
  const int n = x.c.nranks;
  const size_t es = elem_size(dtype);
  LocalExchangeArgs a;
  memset(&a, 0, sizeof(a));
  uint64_t units = 0;
  int dsts = 0;
  bool aligned = true;
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
        aligned = aligned && on32(a.src[a.nblocks]);
        units += (x.cnt[r][p] + kWarpElems - 1) / kWarpElems;
        ++a.nblocks;
        open = true;
      }
      a.dst[dsts] = static_cast<char*>(x.recv[p]) + x.recv_off[p][r] * es;
      aligned = aligned && on32(a.dst[dsts]);
      if (a.dst[dsts] == a.src[a.nblocks - 1]) a.in_place |= 1ull << (a.nblocks - 1);
      ++dsts;
    }
  }
  a.first_dst[a.nblocks] = (uint8_t)dsts;
  // At any offset a run reads the unit before it once more: runs as long as leave every warp slot of the chip
  // its own. Aligned units have nothing to do with one another.
  const uint64_t slots = (uint64_t)comm_sms(c) * 24;
  a.run = 1;
  while (!aligned && a.run < 8u && units / (2 * a.run) >= slots) a.run *= 2;
  uint64_t runs = 0;
  for (int b = 0; b < a.nblocks; ++b) {
    a.first_run[b] = (uint32_t)runs;
    const uint64_t of = (a.cnt[b] + kWarpElems - 1) / kWarpElems;
    runs += (of + a.run - 1) / a.run;
  }
  a.first_run[a.nblocks] = (uint32_t)runs;
  const void* fn = find(dtype, LocalKey{LocalKey::kExchange, 0, codec, false, aligned});
  if (!fn || units >> 31) return no_kernel(dtype, codec, units);
  return local_launch(c, fn, &a, runs, stream);
}

}  // namespace ccb
