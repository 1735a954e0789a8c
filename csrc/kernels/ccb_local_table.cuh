// The kernels of ccb_local.cuh by what a call asks for. One translation unit for each element type
// (ccb_local_f32.cu and so on) instantiates the table, so that they compile side by side.
#pragma once
#include "ccb_local.cuh"

namespace ccb {

struct LocalKey {
  enum { kReduce, kSolo, kExchange } kind;
  int algo;       // kReduce: kLocalTwoShot ...
  int codec;
  bool ef;        // some rank has a residual
  bool aligned;   // every address that a unit starts at is a multiple of 32 bytes
};

template <class T, class C>
const void* local_kernel_of(const LocalKey& k) {
#define CCB_FN(...) reinterpret_cast<const void*>(&__VA_ARGS__)
#define CCB_ALGO(A)                                                                           \
  case A:                                                                                     \
    if (k.ef) return k.aligned ? CCB_FN(local_reduce_kernel<T, C, A, true, false>) : nullptr; \
    return k.aligned ? CCB_FN(local_reduce_kernel<T, C, A, false, false>) : CCB_FN(local_reduce_kernel<T, C, A, false, true>);
  if (k.kind == LocalKey::kExchange) return k.aligned ? CCB_FN(local_exchange_kernel<T, C, false>) : CCB_FN(local_exchange_kernel<T, C, true>);
  if (k.kind == LocalKey::kSolo) {
    if (k.ef) return k.aligned ? CCB_FN(local_solo_kernel<T, C, true, false>) : nullptr;
    return k.aligned ? CCB_FN(local_solo_kernel<T, C, false, false>) : CCB_FN(local_solo_kernel<T, C, false, true>);
  }
  switch (k.algo) {
    CCB_ALGO(kLocalTwoShot)
    CCB_ALGO(kLocalOneShot)
    CCB_ALGO(kLocalRing)
    CCB_ALGO(kLocalTree)
    CCB_ALGO(kLocalScatter)
    default: return nullptr;
  }
#undef CCB_ALGO
#undef CCB_FN
}

// Null where there is no such kernel: residuals want aligned buffers.
template <class T>
const void* local_kernel(const LocalKey& k) {
  switch (k.codec) {
    case CCB_CODEC_NONE: return local_kernel_of<T, CodecNone<T>>(k);
    case CCB_CODEC_INT8: return local_kernel_of<T, CodecInt8<128>>(k);
    case CCB_CODEC_FP8: return local_kernel_of<T, CodecFp8>(k);
    case CCB_CODEC_INT8_G256: return local_kernel_of<T, CodecInt8<256>>(k);
    case CCB_CODEC_INT4: return local_kernel_of<T, CodecInt4>(k);
    default: return nullptr;
  }
}

}  // namespace ccb
