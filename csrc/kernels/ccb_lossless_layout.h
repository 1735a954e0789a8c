/* Where the exponent planes of a block lie in a slot of the lossless container: behind those of the
 * blocks before it, 64 bytes a plane. The widths come from the container, which may be damaged, so
 * each counts for `bits` (of the type's exponent) at most: then the planes of eight blocks fit the
 * slot whatever the bytes say. Plain C, shared by the kernel and the CPU test. */
#ifndef CCB_LOSSLESS_LAYOUT_H
#define CCB_LOSSLESS_LAYOUT_H

#include <stdint.h>

#if defined(__CUDACC__)
#define CCB_LL_FN __host__ __device__ static inline
#else
#define CCB_LL_FN static inline
#endif

/* first: planes of the blocks 0 .. block - 1, as their width bytes add up; width: this block's own byte. */
CCB_LL_FN uint32_t ccb_ll_first_plane(uint32_t first, uint32_t block, uint32_t bits) { return first < block * bits ? first : block * bits; }
CCB_LL_FN uint32_t ccb_ll_planes(uint32_t width, uint32_t bits) { return width < bits ? width : bits; }

#endif
