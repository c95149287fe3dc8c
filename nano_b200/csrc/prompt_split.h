// prompt_split.h -- how the blocks of a cluster share the depth of a prompt product (prefill.cu).  Plain arithmetic, for the host, the kernel and a test
// without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define NB_HD __host__ __device__ __forceinline__
#else
#define NB_HD inline
#endif

namespace nb {

// a block's part: the stages [s0, s0 + steps) of 128 (Q80) or 64 (F32) of the depth; Q80: the groups [g0, g0 + groups) that lie in them
struct PromptPart { uint32_t s0, steps, g0, groups; };

// what a part is a whole number of: a stage, or the stages of a group wider than one
NB_HD uint32_t prompt_unit_stages(bool q80, uint32_t gs) { return q80 && gs > 128u ? gs / 128u : 1u; }
// units of a depth of n (Q80: the last stage of an n that is no multiple of 128 is a short one) or np (F32: n padded to 64)
NB_HD uint32_t prompt_units(bool q80, uint32_t n, uint32_t np, uint32_t gs) {
    const uint32_t us = prompt_unit_stages(q80, gs);
    return ((q80 ? (n + 127u) / 128u : np / 64u) + us - 1u) / us;
}
// The last parts of a cluster can be empty (9 units over 4 blocks: 3, 3, 3, 0): no stages and, whatever the depth, no groups
NB_HD PromptPart prompt_part(bool q80, uint32_t n, uint32_t np, uint32_t gs, uint32_t ks, uint32_t part) {
    const uint32_t us = prompt_unit_stages(q80, gs), units = prompt_units(q80, n, np, gs), per = (units + ks - 1u) / ks, u0 = part * per < units ? part * per : units;
    PromptPart p;
    p.s0 = u0 * us;
    p.steps = (per < units - u0 ? per : units - u0) * us;
    p.g0 = p.groups = 0;
    if (q80) {
        const uint32_t a = p.s0 * 128u, b = (p.s0 + p.steps) * 128u;
        p.g0 = (a < n ? a : n) / gs;
        p.groups = (b < n ? b : n) / gs - p.g0;
    }
    return p;
}
// Blocks of a cluster: twice as many while fewer than half of the SMs would have a block, down to two units each
NB_HD uint32_t prompt_parts(uint32_t units, uint32_t tiles, uint32_t sms) {
    uint32_t ks = 1;
    while (ks < 8u && tiles * ks * 2u <= sms && units >= ks * 4u) ks *= 2u;
    return ks;
}

}  // namespace nb
