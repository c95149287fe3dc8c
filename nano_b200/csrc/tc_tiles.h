// tc_tiles.h -- the tiles of a portion's tensor-core product (layered_tc.cu) and where it reads its rows.  Plain arithmetic, for the host and a test without a GPU.
#pragma once
#include <stdint.h>

namespace nb {

// each: how many rows a group has on average
inline uint32_t tc_tile_tokens(uint32_t each) { return each <= 32u ? 32u : each <= 64u ? 64u : 128u; }

// Does the product read its fp32 rows itself (one launch), or a rounded copy that a launch of its own makes before it.  Groups of at most 64 rows on average, whose tiles are 32 or 64
// tokens, and only while the tiles read less than 32 MB of them: every tile of weights reads the rows again.  Two layers, us a portion, copy / rows: Famudra width 1024 (eight layers) 5 tokens
// 616 / 470, 11 535 / 490, 40 718 / 677, 64 783 / 708; Fidatar width 1024 5 162 / 147, 64 184 / 180; Kadesun width 2048 5 220 / 207, 40 257 / 245, but 64 (50 MB for 12288 columns) 254 / 260 and
// Fidatar width 2048 64 (33 MB) 258 / 264.  More rows than 64 would go in two tiles of 64: faster at width 1024 (four layers of Famudra, 300 tokens 471 / 409), slower at others (two of Famudra's width
// 2048, 160 279 / 287; eight of Vumunex' width 1024, 384 2796 / 3010), and another split of the depth, so other sums.
constexpr uint64_t kTcRawBytes = 32u << 20;
inline bool tc_reads_rows(uint32_t N, uint32_t groups, uint32_t each, uint32_t K) { return each <= 64u && (uint64_t)((N + 127u) / 128u) * groups * each * K * 4u <= kTcRawBytes; }

}  // namespace nb
