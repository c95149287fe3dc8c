// f32_split.h -- how many blocks share the depth of a tile in the 32-bit products of portions (k_gemm_f32_async)
#pragma once
#include <stdint.h>

namespace nb {

// Doubled, up to 8, while the blocks of all tiles of 64 x 64 still find a place at once at two to a place, and a block keeps 64 columns of the depth at least.  rows: of a group,
// its share where they are dealt out.  places: two for each SM, which holds four blocks (128 threads of 128 registers, 31 KB).  Two layers of Famudra's width 1024, us a portion, two blocks to an SM / four:
// 5 rows 298 / 221, 11 316 / 257, 40 360 / 314, 100 479 / 398, 203 612 / 517.  (Before, with whole row tiles counted / rows in 64ths of a tile: 37 rows 424 / 455, 203 1131 / 1170 in four layers.)
inline uint32_t f32_split(uint32_t col_tiles, uint32_t rows, uint32_t groups, uint32_t K, uint32_t places) {
    const uint64_t tiles = (uint64_t)col_tiles * ((rows + 63u) / 64u) * groups;
    uint32_t split = 1;
    while (split < 8u && tiles * split * 2u <= 2u * places && K >= split * 2u * 64u) split *= 2u;
    return split;
}

}  // namespace nb
