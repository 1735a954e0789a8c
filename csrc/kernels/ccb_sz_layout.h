/* What a tile of a compressed group may look like, for everything that reads one. A group slot is
 * [8 x u32 tile sizes][tiles back to back]; a packed tile is 64 row widths (a byte each, 32 bits at
 * most) and as many words as they add up to, or the marker 255, 63 zero bytes and 2048 fp32 values;
 * both padded to 16 bytes. A buffer may come from a file or a message, so its words are checked
 * before they become addresses: a tile that passes lies inside its slot whatever else its words say
 * (GROUP_HEADER + 7 * TILE_CAP + TILE_CAP < GROUP_STRIDE). Plain C, shared by host code, kernels and
 * the CPU test. */
#ifndef CCB_SZ_LAYOUT_H
#define CCB_SZ_LAYOUT_H

#include <stdint.h>

#if defined(__CUDACC__)
#define CCB_SZ_LAYOUT_FN __host__ __device__ static inline
#else
#define CCB_SZ_LAYOUT_FN static inline
#endif

#define CCB_SZ_TILES 8                               /* of a group */
#define CCB_SZ_ROWS 64                               /* of a tile, 32 values each */
#define CCB_SZ_TILE_CAP (CCB_SZ_ROWS + 4 * 2048)     /* bytes; raw, or 32 bits everywhere */
#define CCB_SZ_GROUP_HEADER (4 * CCB_SZ_TILES)
#define CCB_SZ_GROUP_STRIDE (CCB_SZ_GROUP_HEADER + CCB_SZ_TILES * CCB_SZ_TILE_CAP + 32)

/* May tile k of a group lie `off` bytes behind the header, off being the sum of the sizes before it? */
CCB_SZ_LAYOUT_FN int ccb_sz_offset_ok(uint32_t off, unsigned k) { return off <= k * (uint32_t)CCB_SZ_TILE_CAP && (off & 15u) == 0; }
/* May a tile have this size? (0: beyond the end of the field.) */
CCB_SZ_LAYOUT_FN int ccb_sz_size_ok(uint32_t size) { return size == 0 || (size >= CCB_SZ_ROWS && size <= CCB_SZ_TILE_CAP && (size & 15u) == 0); }
/* Is every byte of a word of four row widths at most 32? */
CCB_SZ_LAYOUT_FN int ccb_sz_widths_ok(uint32_t four) { return ((four | ((four & 0x7f7f7f7fu) + 0x5f5f5f5fu)) & 0x80808080u) == 0; }
/* The packer adds 1.5 * 2^23 to a value in steps and takes how far the sum's bits are above that number's as the
 * code (mod 2^32): is it within `most` (below 2^22) of 0? Without a sign, because -1.5 * 2^23, the sum of a value 1.5 * 2^24
 * steps below 0, lies 2^31 away, which has no magnitude in 32 bits. */
CCB_SZ_LAYOUT_FN int ccb_sz_code_within(uint32_t code, uint32_t most) { return code + most <= 2u * most; }

#endif
