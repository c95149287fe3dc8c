// f32_split.h -- how many blocks share the depth of a tile in the 32-bit products of portions (k_gemm_f32_async)
#pragma once
#include <stdint.h>

namespace nb {

// Doubled, up to 8, while the blocks of all tiles of 64 x 64 still find a place at once, four to an SM (128 threads of 128 registers, 31 KB), and a block keeps 64 columns of the depth at
// least.  rows: of a group, its share where they are dealt out; they count as whole tiles.  Two layers, us a portion, two blocks to an SM / four: Famudra width 1024, 5 rows 302 / 243, 24
// 366 / 316, 100 468 / 407, 203 662 / 580, 700 1556 / 1456; Kadesun width 2048, 64 1093 / 910, 700 5378 / 5358; Fidatar width 1024, 203 934 / 593.  Where a row has 512 columns the shares are
// short: Famudra 100 234 / 238, Kadesun 385 638 / 650, but 203 503 / 431.
constexpr uint32_t kF32BlocksPerSm = 4;
inline uint32_t f32_split(uint32_t col_tiles, uint32_t rows, uint32_t groups, uint32_t K, uint32_t sms) {
    const uint64_t tiles = (uint64_t)col_tiles * ((rows + 63u) / 64u) * groups;
    uint32_t split = 1;
    while (split < 8u && tiles * split * 2u <= (uint64_t)kF32BlocksPerSm * sms && K >= split * 2u * 64u) split *= 2u;
    return split;
}

}  // namespace nb
