/* SZ-style error-bounded lossy codec for 3-D fp32 fields ("ccb-sz v2": pre-quantise
 * under an absolute bound, 3-D Lorenzo prediction on the integers inside 32x8x8
 * tiles, per-row bit-plane packing) and its fusion with AllGather / Broadcast.
 * Fields are [nz][ny][nx] with x fastest. The format and the kernels are described
 * in csrc/kernels/ccb_sz.cu. The reference reaches SZ3 only on the CPU through
 * dlopen (userconfig/wrapper_code_examples/compression/sz3/mpi_sz3_wrapper.c). */
#ifndef CCB_SZ_H
#define CCB_SZ_H

#include <stdint.h>

#include "ccb.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Bytes a compressed buffer must provide for an nx*ny*nz field (fixed-capacity group
 * slots; the bytes actually used are reported by ccb_sz_compress). */
uint64_t ccb_sz_capacity(int nx, int ny, int nz);
/* How the last collective launch of this process went: 0 = none yet, 1 = the driver took the
 * kernel's clusters and the cooperative attribute together, 2 = it refused the pair and the kernel
 * was launched plainly (grid bounded by the resident-cluster count). */
int ccb_sz_launch_path(void);
/* |in - decompress(compress(in))| <= eb for every finite element. `out` starts on 16 bytes, the fields
 * and a buffer to be read on 4. `d_used` (device memory, optional) receives the number of compressed
 * bytes produced (those of the tiles, without the groups' size words). A tile of a damaged buffer whose
 * size words put it outside its group, or whose rows are wider than 32 bits, is decompressed to NaN;
 * what else a damaged buffer holds is decoded as it stands, from inside its slots, to values that may differ
 * with the size and the alignment of the field. */
int ccb_sz_compress(const float* in, int nx, int ny, int nz, float eb, void* out, unsigned long long* d_used,
                    ccb_stream_t stream);
int ccb_sz_decompress(const void* in, int nx, int ny, int nz, float eb, float* out, ccb_stream_t stream);
/* The packed container of a compressed buffer: a 40-byte header, the used bytes of each group as u32,
 * then the used bytes of every group. All pointers device memory.
 * scan: offsets[g] = used bytes before group g, offsets[ngroups] their total, offsets[ngroups + 1]
 * the largest group's (ngroups + 2 words; 2^32 - 1 where a group's header holds sizes that tiles cannot
 * have); from the groups' own headers (slots) or from a list of
 * sizes, exactly one of the two given. pack writes 40 + 4 * ngroups + offsets[ngroups] bytes;
 * unpack takes the payload behind a container's size list and fills ngroups whole slots.
 * open: the scan of a container of `bytes` bytes whose header has not been read yet. `found` (56 bytes, on
 * 8) takes the header, then the total and the largest as u64 (2^32 - 1 also where a group's header does not
 * add up to its size in the list); offsets has room + 2 words, and nothing is
 * scanned where the header speaks of more than `room` groups (40 + 4 * room <= bytes). */
int ccb_sz_container_open(const void* blob, uint64_t bytes, uint64_t room, unsigned long long* offsets, void* found, ccb_stream_t stream);
int ccb_sz_container_scan(const void* slots, const uint32_t* sizes, uint64_t ngroups, unsigned long long* offsets, ccb_stream_t stream);
/* The scan of slots, its last two words to `sums` as well: device memory or pinned host memory, 8-byte aligned. */
int ccb_sz_container_sums(const void* slots, uint64_t ngroups, unsigned long long* offsets, unsigned long long* sums, ccb_stream_t stream);
int ccb_sz_container_pack(const void* slots, const unsigned long long* offsets, int nx, int ny, int nz, float eb, uint64_t ngroups, void* out,
                          ccb_stream_t stream);
int ccb_sz_container_unpack(const void* payload, const unsigned long long* offsets, uint64_t ngroups, void* slots, ccb_stream_t stream);
/* root < 0: AllGather (recv holds nranks fields in rank order); root >= 0: Broadcast.
 * One fused kernel: compress, store into the peers' arenas, decode on arrival.
 * `d_used`: optional device counters, one per local rank, of the compressed bytes a
 * rank sent to one destination. */
int ccb_sz_collective(ccb_comm* c, const float* const* send, float* const* recv, int nx, int ny, int nz, float eb, int root,
                      unsigned long long* d_used, ccb_stream_t stream);

#ifdef __cplusplus
}
#endif
#endif
