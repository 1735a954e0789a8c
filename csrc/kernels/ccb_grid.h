/* The number of a warp in a grid whose warps each take one unit. Formed from the warps of a block and
 * not from its threads, whose number passes 2^32 at 2^27 warps: right up to 2^32 warps, twice what the
 * launches let through. Plain C, shared by kernels and the CPU test. */
#ifndef CCB_GRID_H
#define CCB_GRID_H

#include <stdint.h>

#if defined(__CUDACC__)
#define CCB_GRID_FN __host__ __device__ static inline
#else
#define CCB_GRID_FN static inline
#endif

CCB_GRID_FN uint32_t ccb_grid_warp(uint32_t block, uint32_t block_threads, uint32_t thread) { return block * (block_threads >> 5) + (thread >> 5); }

#endif
