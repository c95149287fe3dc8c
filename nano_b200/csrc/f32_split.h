// f32_split.h -- how many blocks share the depth of a tile in the 32-bit products of portions (k_gemm_f32_async)
#pragma once
#include <stdint.h>

namespace nb {

// Doubled, up to 8, while the blocks of all tiles of 64 x 64 still find a place at once at two to an SM, and a block keeps 64 columns of the depth at least.  rows: of a group,
// its share where they are dealt out.  Two layers of Famudra's width 1024, 16 tiles wide, us a portion, with whole row tiles counted / rows in 64ths of a tile (which gave 70 to 127
// rows 3 tiles instead of 2): 37 rows 424 / 455, 64 523 / 561, 100 698 / 740, 127 786 / 834, 170 1014 / 1066, 203 1131 / 1170.
// (At four to an SM, which the kernel's registers allow, the same portions took 380, 490, 630, 730, 905 and 1051.)
inline uint32_t f32_split(uint32_t col_tiles, uint32_t rows, uint32_t groups, uint32_t K, uint32_t sms) {
    const uint64_t tiles = (uint64_t)col_tiles * ((rows + 63u) / 64u) * groups;
    uint32_t split = 1;
    while (split < 8u && tiles * split * 2u <= 2u * sms && K >= split * 2u * 64u) split *= 2u;
    return split;
}

}  // namespace nb
