// stream_groups.h -- how many query heads an attention item of the streaming kernel takes (stream.cuh).  Plain arithmetic, for the host and a test without a GPU.
#pragma once
#include <stdint.h>

namespace nb {

// An item is a group of query heads that share a key/value head, and a split of the keys.  Fewer heads make an item's chain shorter (scores, merges and their shuffles go with the heads) and read the
// keys once more for every group; the splits get fewer, so an item has more rows.  That is the better way while an item's keys and values stay in the ring: up to 20480 coordinates of each, 160 KB.
// us a token by heads of an item, at a position: Nano-168M (16 heads over 8) two / one head 365 / 350 at 16, 414 / 397 at 480; four layers of Qwen3-0.6B (the same of 128) 78.7 / 76.2 at 16, 93.3 / 88.1 at
// 1000, 100.7 / 102.5 at 2000; two of 4B (32 over 8) four / two / one 94.4 / 92.2 / 90.9 at 16, 106.3 / 106.3 / 114.9 at 1500, 126 / 135 / 158 at 4000.  Q4K takes all of them (Qwen3-0.6B 116 / 118 at 16).
constexpr uint32_t kStItemCoords = 20480;
inline uint32_t st_splits(uint32_t groups, uint32_t sms) { const uint32_t n = sms / groups; return n < 1u ? 1u : n > 64u ? 64u : n; }
// kv: key/value heads, kv_mul (1, 2 or 4): query heads of each, range: keys that a token sees at most
inline uint32_t st_group_heads(uint32_t kv, uint32_t kv_mul, uint32_t hd, bool q4k, uint32_t range, uint32_t sms) {
    for (uint32_t h = 1; h < kv_mul && !q4k; h *= 2u)
        if (kv * (kv_mul / h) <= sms && (uint64_t)range * hd <= (uint64_t)kStItemCoords * st_splits(kv * (kv_mul / h), sms)) return h;
    return kv_mul;
}

}  // namespace nb
