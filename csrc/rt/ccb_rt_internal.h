// Declarations shared between the translation units of libccb.so.
#pragma once
#include <cuda_runtime.h>

#include "ccb/ccb.h"

struct ccb_comm;

namespace ccb {

struct LaunchPlace;   // ccb_overlap.h
void set_error(const char* fmt, ...);
void count_launch();
int sm_count();   // of the current device
CommDev comm_dev(ccb_comm* c, uint32_t epoch);
uint32_t next_epoch(ccb_comm* c);
int grid_cap(ccb_comm* c, const void* kernel, int threads = 512);
int launch(ccb_comm* c, const void* kernel, int ctas, void* args, cudaStream_t stream, int threads = 512, const LaunchPlace* overlapping = nullptr);
// A launch that is got ready while the kernel before it on the stream still runs: for kernels that begin with
// after_kernel_before() (ccb_device.cuh). Kernels behind one another on a stream begin about 2 us sooner (B200, us, launched
// plainly / so: three chunks of 3,000,001 values compressed, reduced and decompressed, five kernels, 30.7 / 20.5; a
// reduce-scatter of 4 x 87,113 bf16 6.2 / 4.0, of 8 x 25 MiB 43.8 / 41.9).
cudaError_t launch_next(const void* kernel, dim3 grid, dim3 block, void** params, size_t shared, cudaStream_t stream);
template <class... P, class... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, int block, size_t shared, cudaStream_t stream, A... a) {
  return [&](P... p) {
    void* params[] = {const_cast<void*>(static_cast<const void*>(&p))...};
    return launch_next(reinterpret_cast<const void*>(kernel), grid, dim3((unsigned)block), params, shared, stream);
  }(a...);
}
// Up to 128 bytes, on four, set to zero by such a launch: behind a memset the next kernel begins 1 us later.
cudaError_t launch_clear(void* words, size_t bytes, cudaStream_t stream);
int check_alive(ccb_comm* c);
size_t elem_size(int dtype);
size_t codec_slot_bytes(int codec, int dtype, size_t pad);
// The pipelined two-shot kernel for this element type and codec (csrc/kernels/ccb_pipe.cu),
// or null; its CTAs have pipe_kernel_threads() threads and own runs of kPipeChunkElems elements.
constexpr int kPipeChunkElems = 4096;
const void* pipe_kernel_fn(int dtype, int codec);
int pipe_kernel_threads();
// Ranks that share one GPU (csrc/kernels/ccb_local.cu). ranks_in_registers(): all ranks of the
// communicator are this process's and nothing asks for the schedule of ranks on several GPUs.
bool ranks_in_registers(const ccb_comm* c);
int comm_sms(const ccb_comm* c);
bool local_reduce_takes(const ReduceArgs& r, int dtype);   // residuals want buffers on 32 bytes
bool local_solo_takes(const void* send, const void* recv, const float* ef);
int local_reduce(ccb_comm* c, const ReduceArgs& r, int algo, int dtype, int codec, cudaStream_t stream);
int local_solo(ccb_comm* c, const void* send, void* recv, float* ef, uint64_t count, int dtype, int codec, cudaStream_t stream);
int local_exchange(ccb_comm* c, const ExchangeArgs& x, int dtype, int codec, cudaStream_t stream);
int nvls_all_reduce(ccb_comm* c, const void* const* send, void* const* recv, uint64_t count, int dtype, int op,
                    cudaStream_t stream);
}  // namespace ccb
