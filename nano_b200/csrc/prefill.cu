// prefill.cu -- the prompt of a model file in portions of up to 1024 positions (F32 and Q80 files, one GPU, fast mode).
//
// A decode step streams every weight for one position; here a weight tile meets 64 or 128 positions.  The arithmetic is the decode path's: RMS norm and
// Q80 activation codes by the same expressions, exact integer group dots, their fp32 terms summed per group; only the order of fp32 sums
// differs, as it does between the decode paths.  What a prompt leaves behind is its K and V rows, so the last layer stops there.
//
//   k_prompt_embed     token rows
//   k_prompt_rows      a position's activation: RMS norm with gain, plain, or SwiGLU of interleaved pairs; then Q80 codes + group scales, or
//                      (F32) three bfloat16 parts
//   k_weight_parts     F32: a matrix in three bfloat16 parts, into one workspace for all of them (its bytes pass through memory four times
//                      for that; a copy that stays would hold half again as much as the file)
//   k_prompt_gemm      C[t][n] (+)= sum over groups: tcgen05.mma on 128 weight rows x TN positions, the accumulator of a GROUP in tensor memory (two
//                      buffers), added to fp32 registers by the threads that own the rows while the next group multiplies.
//                      Q80: kind::i8, int32 exact, times weight scale x activation scale.  F32: kind::f16 on three bfloat16 parts of both
//                      operands, which are all of their 24 bits; of the nine products of parts the three that are left out (small x
//                      smallest, smallest x smallest) are 2^-26 of the whole at most.  The tensor cores cut what they add, so they
//                      add over 16 of the depth only, the small products first, and what they leave is added up with its rounding error carried along.
//   k_prompt_rope      head norm (Qwen3), rotary positions, K and V rows into the cache
//   attention          attn_tc.cu; k_prompt_attn for few positions
#include "prefill.h"

#include <cuda_bf16.h>

#include <algorithm>

#include "family.h"
#define NB_K static
#include "kernels.cuh"
#include "prompt_split.h"
#include "tc_ptx.cuh"

namespace nb {
namespace {

constexpr uint32_t kChunk = 1024, kRows = 128;
// Positions up to which a prompt's first portion has k_prompt_attn; longer ones, and what remains behind a whole portion (its walk of the keys is serial: 1 position behind 1024
// of them 2 to 4 times as slow), have the tensor cores.  Eight layers, us, k_prompt_attn / tensor cores at 16, 33, 40, 50 and 64 positions: 16 heads of 48 323 / 402, 383 / 439,
// 394 / 440, 419 / 449, 440 / 460; 8 of 64 310 / 389, 371 / 429, 375 / 430, 382 / 432, 407 / 445; 64 of 64 415 / 485, 480 / 510, 507 / 505, 533 / 514, 565 / 521; 16 of 128
// 401 / 494, 476 / 533, 530 / 537, 606 / 551, 656 / 568; 32 of 128 633 / 734, 766 / 788, 814 / 803, 859 / 801; 64 of 128 522 / 618, 611 / 638, 658 / 631, 703 / 642.
constexpr uint32_t kPromptAttnFew = 50, kPromptAttnFewWide = 36;          // heads of at most 64 values and at most 16 of them; others
enum { PREP_NORM = 0, PREP_PLAIN = 1, PREP_SWIGLU = 2 };

__device__ __forceinline__ void dep_enter() { asm volatile("griddepcontrol.launch_dependents;\ngriddepcontrol.wait;" ::: "memory"); }

struct PromptEmbedArgs { const void *w, *aux; float *x; const uint32_t *ids; uint32_t E, gs, quant; };
__global__ void __launch_bounds__(256) k_prompt_embed(const PromptEmbedArgs a) {
    dep_enter();
    const size_t tok = a.ids[blockIdx.x];
    float *x = a.x + (size_t)blockIdx.x * a.E;
    for (uint32_t i = threadIdx.x; i < a.E; i += 256u) {
        if (a.quant == 0x00u) x[i] = static_cast<const float *>(a.w)[tok * a.E + i];
        else x[i] = __fmul_rn((float)static_cast<const int8_t *>(a.w)[tok * a.E + i], static_cast<const float *>(a.aux)[(tok * a.E + i) / a.gs]);
    }
}

// x = p[0] + p[1] + p[2], three times 8 bits: exact as long as the last part is no smaller than 2^-133.  A number that has no neighbour in bfloat16 (the
// largest ones would round to infinity) is cut; infinities and NaN stay in the first part
__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        __nv_bfloat16 h = __float2bfloat16_rn(x);
        if (fabsf(__bfloat162float(h)) == INFINITY && fabsf(x) < INFINITY) h = __float2bfloat16_rz(x);
        p[i] = h;
        x = fabsf(x) < INFINITY ? x - __bfloat162float(h) : 0.0f;
    }
}

// codes [T][n] and scales [n / gs][lds] (Q80), or parts [T][3][np] (F32)
struct PromptPrepArgs { const float *src; uint32_t ld; const float *gain; uint32_t n, gs, mode; int8_t *codes; float *scales; uint32_t lds; __nv_bfloat16 *parts; uint32_t np; };
__device__ __forceinline__ float prep_value(const PromptPrepArgs &a, const float *s, float inv, uint32_t i) {
    if (a.mode == PREP_NORM) return __fmul_rn(a.gain[i], __fmul_rn(inv, s[i]));
    if (a.mode == PREP_PLAIN) return s[i];
    const float2 v = *reinterpret_cast<const float2 *>(s + 2u * i);
    return __fmul_rn(__fmul_rn(v.x, __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-v.x)))), v.y);
}
constexpr uint32_t kPrepThreads = 512;
// groups of 256: every other size runs on k_prompt_rows
__global__ void __launch_bounds__(kPrepThreads) k_prompt_prep(const PromptPrepArgs a) {
    dep_enter();
    __shared__ float red[32];
    const uint32_t t = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const float *s = a.src + (size_t)t * a.ld;
    float inv = 1.0f;
    if (a.mode == PREP_NORM) {
        float acc = 0.0f;
        for (uint32_t i = threadIdx.x; i < a.n; i += kPrepThreads) acc = fmaf(s[i], s[i], acc);
        acc = block_sum<kPrepThreads>(acc, red);
        inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(acc, (float)a.n), 1e-5f)));
    }
    for (uint32_t g = warp; g < a.n / 256u; g += kPrepThreads / 32u) {
        float v[8], amax = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) { v[j] = prep_value(a, s, inv, g * 256u + j * 32u + lane); amax = fmaxf(amax, fabsf(v[j])); }
        amax = warp_max(amax);
        const float sc = __fdiv_rn(amax, 127.0f), rinv = __frcp_rn(sc);
#pragma unroll
        for (uint32_t j = 0; j < 8; j++) a.codes[(size_t)t * a.n + g * 256u + j * 32u + lane] = (int8_t)((sc == 0.0f) ? 0 : q80_code(v[j], sc, rinv));
        if (lane == 0) a.scales[(size_t)g * a.lds + t] = sc;
    }
}
// The same for groups of 32, 64 and 128 (8, 16 and 32 lanes) and for F32: a thread holds runs of 4 neighbours, 4 of them in registers, gains are there before the
// wait, codes and parts leave in 4- and 8-byte pieces.  A row is one trip to memory, one sum and one store; a prompt of 250 positions spent 5.1 us in each of its 109
// walks of single values, now 4.3 (16 positions: 3.6, now 2.7).
constexpr uint32_t kRowThreads = 256, kRowRuns = 4, kRowTurn = kRowThreads * 4u * kRowRuns;
template <bool Q80>
__global__ void __launch_bounds__(kRowThreads) k_prompt_rows(const PromptPrepArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ float red[32];
    const uint32_t t = blockIdx.x, lane = threadIdx.x & 31u;
    const float *s = a.src + (size_t)t * a.ld;
    const bool norm = a.mode == PREP_NORM;
    float4 v[kRowRuns], g[kRowRuns];
    auto at = [&](uint32_t base, uint32_t j) { return base + (threadIdx.x + j * kRowThreads) * 4u; };
    auto gains = [&](uint32_t base) {
#pragma unroll
        for (uint32_t j = 0; j < kRowRuns; j++) { const uint32_t i = at(base, j); g[j] = norm && i < a.n ? __ldg(reinterpret_cast<const float4 *>(a.gain + i)) : make_float4(1, 1, 1, 1); }
    };
    auto load = [&](uint32_t base) {
#pragma unroll
        for (uint32_t j = 0; j < kRowRuns; j++) {
            const uint32_t i = at(base, j);
            v[j] = make_float4(0, 0, 0, 0);
            if (i >= a.n) continue;
            if (a.mode == PREP_SWIGLU) {
                const float4 p = *reinterpret_cast<const float4 *>(s + 2u * i), q = *reinterpret_cast<const float4 *>(s + 2u * i + 4u);
                auto glu = [](float x, float y) { return __fmul_rn(__fmul_rn(x, __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x)))), y); };
                v[j] = make_float4(glu(p.x, p.y), glu(p.z, p.w), glu(q.x, q.y), glu(q.z, q.w));
            } else v[j] = *reinterpret_cast<const float4 *>(s + i);
        }
    };
    gains(0);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    load(0);
    float inv = 1.0f;
    if (norm) {
        float acc = 0.0f;
        for (uint32_t base = 0;;) {
#pragma unroll
            for (uint32_t j = 0; j < kRowRuns; j++) acc = fmaf(v[j].x, v[j].x, fmaf(v[j].y, v[j].y, fmaf(v[j].z, v[j].z, fmaf(v[j].w, v[j].w, acc))));
            base += kRowTurn;
            if (base >= a.n) break;
            load(base);
        }
        acc = block_sum<kRowThreads>(acc, red);
        inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(acc, (float)a.n), 1e-5f)));
    }
    const uint32_t LG = Q80 ? a.gs / 4u : 1u, end = Q80 ? a.n : a.np;
    for (uint32_t base = 0; base < end; base += kRowTurn) {
        if (base || (norm && a.n > kRowTurn)) { gains(base); load(base); }
#pragma unroll
        for (uint32_t j = 0; j < kRowRuns; j++) {
            const uint32_t i = at(base, j);
            if (i - lane * 4u >= end) continue;          // the same for the whole warp
            float4 x = v[j];
            if (norm) x = make_float4(__fmul_rn(g[j].x, __fmul_rn(inv, x.x)), __fmul_rn(g[j].y, __fmul_rn(inv, x.y)), __fmul_rn(g[j].z, __fmul_rn(inv, x.z)), __fmul_rn(g[j].w, __fmul_rn(inv, x.w)));
            if (Q80) {
                float amax = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w)));
                for (uint32_t o = 1; o < LG; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
                // rounded by adding 1.5 * 2^23; what lies within 1e-4 of a .5 boundary takes the exact division (the product is at most 2.3e-5 from the quotient), and so
                // does what is no number or out of range (the sum's low bits say nothing then)
                const float sc = __fdiv_rn(amax, 127.0f), rinv = __frcp_rn(sc), magic = 12582912.0f;
                const float q[4] = {x.x * rinv, x.y * rinv, x.z * rinv, x.w * rinv}, xv[4] = {x.x, x.y, x.z, x.w};
                uint32_t pk = 0;
                if (sc != 0.0f)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const float r = q[e] + magic;
                        const uint32_t c = fabsf(q[e] - (r - magic)) <= 0.4999f ? __float_as_uint(r) : (uint32_t)q80_code_slow(xv[e], sc);
                        pk |= (c & 0xffu) << (8 * e);
                    }
                if (i < a.n) {
                    *reinterpret_cast<uint32_t *>(a.codes + (size_t)t * a.n + i) = pk;
                    if ((lane & (LG - 1u)) == 0) a.scales[(size_t)(i / a.gs) * a.lds + t] = sc;
                }
            } else if (i < a.np) {
                __nv_bfloat16 *to = a.parts + (size_t)t * 3u * a.np + i;
                const float xv[4] = {x.x, x.y, x.z, x.w};
                __align__(8) __nv_bfloat16 o[3][4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    __nv_bfloat16 p[3];
                    split3(xv[e], p);
#pragma unroll
                    for (int k = 0; k < 3; k++) o[k][e] = p[k];
                }
#pragma unroll
                for (int k = 0; k < 3; k++) *reinterpret_cast<uint2 *>(to + (size_t)k * a.np) = *reinterpret_cast<const uint2 *>(o[k]);
            }
        }
    }
}

// F32 weights [rows][n] in parts [rows][3][np]; n and np are multiples of 8, a thread makes 8 columns
struct WeightPartsArgs { const float *w; uint32_t rows, n, np; __nv_bfloat16 *parts; };
__global__ void __launch_bounds__(256) k_weight_parts(const WeightPartsArgs a) {
    dep_enter();
    const uint32_t n8 = a.np / 8u;
    const size_t total = (size_t)a.rows * n8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / n8), c = (uint32_t)(i % n8) * 8u;
        __align__(16) __nv_bfloat16 o[3][8];
#pragma unroll
        for (uint32_t q = 0; q < 2; q++) {
            const float4 v = c < a.n ? __ldcs(reinterpret_cast<const float4 *>(a.w + (size_t)r * a.n + c) + q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                __nv_bfloat16 p[3];
                split3(x[j], p);
#pragma unroll
                for (int k = 0; k < 3; k++) o[k][q * 4u + j] = p[k];
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < 3; k++) *reinterpret_cast<uint4 *>(a.parts + (size_t)r * 3u * a.np + k * a.np + c) = *reinterpret_cast<const uint4 *>(o[k]);
    }
}

// add: C += (the residual stream), else C =
struct alignas(64) PromptGemmArgs {
    CUtensorMap wmap, amap; const float *ws, *xs; uint32_t ldx;
    uint32_t N, T, n, gs, np; float *C; uint32_t ldc, add, ks; uint32_t *err;      // ks: blocks of a cluster (along z) that share a tile's depth
};
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add) : "memory");
}
// a stage holds 128 bytes of the depth of 128 weight rows and TN positions: 128 int8, or 64 bfloat16 of all three parts
template <bool Q80, int TN> __host__ __device__ constexpr uint32_t gemm_stage() { return (kRows + (uint32_t)TN) * 128u * (Q80 ? 1u : 3u); }
template <bool Q80, int TN> __host__ __device__ constexpr uint32_t gemm_stages() { return !Q80 ? 3u : TN == 128 ? 6u : 4u; }
template <bool Q80, int TN> constexpr size_t gemm_smem() { return (size_t)gemm_stages<Q80, TN>() * gemm_stage<Q80, TN>() + 1024u; }

template <bool Q80, int TN>
__global__ void __launch_bounds__(192, Q80 && TN == 64 ? 2 : 1) k_prompt_gemm(const __grid_constant__ PromptGemmArgs a) {
    constexpr uint32_t ST = gemm_stages<Q80, TN>(), SB = gemm_stage<Q80, TN>(), WB = kRows * 128u, XB = TN * 128u;
    extern __shared__ uint8_t tc_raw[];
    __shared__ __align__(8) uint64_t bars[2 * ST + 4];
    __shared__ uint32_t tmem_s;
    __shared__ volatile uint32_t bad_s;
    __shared__ __align__(16) float xs_s[Q80 ? 3 : 1][TN];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, ring = (smem_u32(tc_raw) + 1023u) & ~1023u;
    const uint32_t n0 = blockIdx.x * kRows, m0 = blockIdx.y * TN;
    const uint32_t full = smem_u32(bars), empty = full + ST * 8u, tfull = empty + ST * 8u, tfree = tfull + 16u;
    // this block's share of the depth; groups: the depth that one tensor-memory accumulator takes before it is added up in fp32
    const PromptPart part = prompt_part(Q80, a.n, a.np, a.gs, a.ks, blockIdx.z);
    const uint32_t s0 = part.s0, steps = part.steps, g0 = part.g0, groups = Q80 ? part.groups : steps * 4u, all_groups = Q80 ? a.n / a.gs : 0u;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < ST; i++) { mbar_init(full + i * 8u, 1); mbar_init(empty + i * 8u, 1); }
        for (uint32_t i = 0; i < 2; i++) { mbar_init(tfull + i * 8u, 1); mbar_init(tfree + i * 8u, 4); }
        bad_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { tc_alloc(smem_u32(&tmem_s), 2 * TN); tc_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Only now may the next kernels' blocks come: one that waits for this grid while it holds tensor memory must not be in the way of an allocation here
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem = tmem_s, npre = Q80 ? min(ST, steps) : 0u;
    auto weights = [&](uint32_t i) {
        const uint32_t dst = ring + (i % ST) * SB, bar = full + (i % ST) * 8u;
        mbar_expect(bar, SB);
        if (Q80) tma_2d(dst, &a.wmap, (s0 + i) * 128u, n0, bar);
        else for (uint32_t p = 0; p < 3; p++) tma_2d(dst + p * WB, &a.wmap, p * a.np + (s0 + i) * 64u, n0, bar);
    };
    if (warp == 0 && lane == 0) for (uint32_t i = 0; i < npre; i++) weights(i);          // Q80 weights do not depend on the kernels before
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float *mine = reinterpret_cast<float *>(tc_raw + (ring - smem_u32(tc_raw)));          // [TN][128]: a part's sums, once the ring is free
    if (warp == 0 && lane == 0) {
        for (uint32_t i = 0; i < steps; i++) {
            const uint32_t st = i % ST, bar = full + st * 8u, dst = ring + st * SB + (Q80 ? WB : 3u * WB);
            if (i >= ST && !mbar_wait(empty + st * 8u, ((i / ST) - 1u) & 1u)) { bad_s = 1; break; }
            if (!Q80 || i >= npre) weights(i);
            if (Q80) tma_2d(dst, &a.amap, (s0 + i) * 128u, m0, bar);
            else for (uint32_t p = 0; p < 3; p++) tma_2d(dst + p * XB, &a.amap, p * a.np + (s0 + i) * 64u, m0, bar);
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t shape = ((uint32_t)(TN >> 3) << 17) | ((kRows >> 4) << 24);
        constexpr uint32_t idesc = Q80 ? ((2u << 4) | (1u << 7) | (1u << 10) | shape) : ((1u << 4) | (1u << 7) | (1u << 10) | shape);          // int32 += int8 x int8; fp32 += bf16 x bf16
        bool ok = true;
        uint32_t gi = 0;
        auto open = [&]() { const bool w = gi < 2u || mbar_wait(tfree + (gi & 1u) * 8u, ((gi >> 1) - 1u) & 1u); tc_fence_after(); return w; };
        auto close = [&]() { tc_commit(tfull + (gi & 1u) * 8u); gi++; };
        for (uint32_t i = 0; i < steps && ok; i++) {
            ok = mbar_wait(full + (i % ST) * 8u, (i / ST) & 1u);
            if (!ok) break;
            tc_fence_after();
            const uint32_t base = ring + (i % ST) * SB;
            if (Q80) {
                const uint64_t wd = tc_desc(base), xd = tc_desc(base + WB);
                const uint32_t depth = min(128u, a.n - (s0 + i) * 128u);
                if (a.gs >= 128u) {
                    const uint32_t per = a.gs / 128u, at = i % per;          // stages of a group
                    if (at == 0 && !(ok = open())) break;
                    for (uint32_t k = 0; k < depth / 32u; k++) tc_mma_i8(tmem + (gi & 1u) * TN, wd + 2u * k, xd + 2u * k, idesc, at > 0 || k > 0);
                    if (at + 1u == per) close();
                } else {
                    const uint32_t per = a.gs / 32u;
                    for (uint32_t k0 = 0; k0 < depth / 32u && ok; k0 += per) {
                        if (!(ok = open())) break;
                        for (uint32_t k = 0; k < per; k++) tc_mma_i8(tmem + (gi & 1u) * TN, wd + 2u * (k0 + k), xd + 2u * (k0 + k), idesc, k > 0);
                        close();
                    }
                }
            } else {
                const uint32_t xb = base + 3u * WB;
                for (uint32_t k = 0; k < 4u; k++) {
                    if (!(ok = open())) break;
#pragma unroll
                    for (uint32_t p = 0; p < 6; p++) {          // the smallest products first, large x large last
                        constexpr uint32_t wp[6] = {0, 2, 1, 0, 1, 0}, xp[6] = {2, 0, 1, 1, 0, 0};
                        tc_mma_ss(tmem + (gi & 1u) * TN, tc_desc(base + wp[p] * WB) + 2u * k, tc_desc(xb + xp[p] * XB) + 2u * k, idesc, p > 0);
                    }
                    close();
                }
            }
            if (ok) tc_commit(empty + (i % ST) * 8u);
        }
        if (!ok) bad_s = 2;
    } else if (warp >= 2) {
        const uint32_t quad = warp & 3u, n = n0 + quad * 32u + lane, nr = min(n, a.N - 1u), lanes = (quad * 32u) << 16;
        float acc[TN], low[Q80 ? 1 : TN];          // low: what acc is too large by (F32)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[j] = 0.0f;
        if (!Q80) {
#pragma unroll
            for (int j = 0; j < TN; j++) low[Q80 ? 0 : j] = 0.0f;
        }
        bool ok = true;
        // the scales of a group are fetched two groups ahead: the row's own into a register, the positions' into shared memory (a global load per group
        // between a full accumulator and its sums cost 2.5 us a group: 250 x 1024 x 3072 took 62 us)
        const float *ws = Q80 ? a.ws + (size_t)nr * all_groups + g0 : nullptr;
        const uint32_t et = threadIdx.x - 64u;
        auto weight_scale = [&](uint32_t g) { return Q80 && g < groups ? __ldg(ws + g) : 0.0f; };
        auto act_scale = [&](uint32_t g) { return Q80 && g < groups && et < (uint32_t)TN ? __ldcg(a.xs + (size_t)(g0 + g) * a.ldx + m0 + et) : 0.0f; };
        float w0 = weight_scale(0), w1 = weight_scale(1);
        if (Q80) {
            const float x0 = act_scale(0), x1 = act_scale(1);
            if (et < (uint32_t)TN) { xs_s[0][et] = x0; xs_s[1][et] = x1; }
            bar_any(1, 128, false);
        }
        uint32_t slot = 0;
        for (uint32_t g = 0; g < groups; g++) {
            const float w = w0, x2 = act_scale(g + 2u);
            w0 = w1; w1 = weight_scale(g + 2u);
            ok = mbar_wait_warp(tfull + (g & 1u) * 8u, (g >> 1) & 1u);          // (when it ran out: what is added up below is not used)
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < TN; c += 32) {
                uint32_t v[32];
                tc_ld32(tmem + lanes + (g & 1u) * TN + c, v);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    if (Q80) {
                        const float4 x = *reinterpret_cast<const float4 *>(&xs_s[slot][c + j]);
                        acc[c + j] = fmaf((float)(int)v[j], w * x.x, acc[c + j]); acc[c + j + 1] = fmaf((float)(int)v[j + 1], w * x.y, acc[c + j + 1]);
                        acc[c + j + 2] = fmaf((float)(int)v[j + 2], w * x.z, acc[c + j + 2]); acc[c + j + 3] = fmaf((float)(int)v[j + 3], w * x.w, acc[c + j + 3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            float &lo = low[Q80 ? 0 : c + j + q];
                            const float y = __fsub_rn(__uint_as_float(v[j + q]), lo), sum = __fadd_rn(acc[c + j + q], y);
                            lo = __fsub_rn(__fsub_rn(sum, acc[c + j + q]), y);
                            acc[c + j + q] = sum;
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tfree + (g & 1u) * 8u);
            if (Q80) {
                if (et < (uint32_t)TN) xs_s[slot == 0 ? 2 : slot - 1][et] = x2;          // the buffer of the group before this one
                ok = !bar_any(1, 128, !ok);          // the four warps leave together: none is left at this barrier
                slot = slot == 2 ? 0 : slot + 1;
            }
            if (!ok) break;
        }
        if (!ok) bad_s = 3;
        else if (a.ks > 1u) {
#pragma unroll
            for (int j = 0; j < TN; j++) mine[j * kRows + quad * 32u + lane] = acc[j];
        } else if (n < a.N) {
            float *dst = a.C + (size_t)m0 * a.ldc + n;
            const uint32_t live = min((uint32_t)TN, a.T - m0);
            if (a.add) {          // all loads before the first store: one after the other they were 30 us of a product
#pragma unroll
                for (int j = 0; j < TN; j++) if ((uint32_t)j < live) acc[j] += __ldcg(dst + (size_t)j * a.ldc);
            }
#pragma unroll
            for (int j = 0; j < TN; j++) if ((uint32_t)j < live) dst[(size_t)j * a.ldc] = acc[j];
        }
    }
    __syncwarp();
    if (a.ks > 1u) {          // every block of the cluster finishes TN / ks positions: its own and its peers' parts, added in the order of the depth
        cluster_sync_all();
        const uint32_t quad = warp & 3u, n = n0 + quad * 32u + lane, span = TN / a.ks, j0 = blockIdx.z * span, j1 = min(j0 + span, a.T - m0);
        if (warp >= 2 && n < a.N && !bad_s) {
            const uint32_t at = smem_u32(mine + quad * 32u + lane);
            float *dst = a.C + (size_t)m0 * a.ldc + n;
            for (uint32_t j = j0; j < j1; j += 8u) {
                float f[8];
#pragma unroll
                for (int i = 0; i < 8; i++) f[i] = 0.0f;
#pragma unroll 2
                for (uint32_t p = 0; p < a.ks; p++) {
                    uint32_t peer;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at + j * kRows * 4u), "r"(p));
#pragma unroll
                    for (uint32_t i = 0; i < 8; i++) f[i] += ld_cluster_f32(peer + i * kRows * 4u);
                }
                if (a.add) {
#pragma unroll
                    for (uint32_t i = 0; i < 8; i++) if (j + i < j1) f[i] += __ldcg(dst + (size_t)(j + i) * a.ldc);
                }
#pragma unroll
                for (uint32_t i = 0; i < 8; i++) if (j + i < j1) dst[(size_t)(j + i) * a.ldc] = f[i];
            }
        }
        cluster_sync_all();          // no block leaves while another reads its part
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (bad_s) {
        if (threadIdx.x == 0) {
            *a.err = 0x300u + bad_s;
            __threadfence_system();
            const long long t0 = clock64();
            while (clock64() - t0 < 20000000ll) __nanosleep(1000);          // copies still in flight land in this block's shared memory before it is given back
        }
        __syncthreads();
    }
    if (warp == 1) tc_dealloc(tmem, 2 * TN);
}

// head norm (Qwen3) and rotary positions of the rows [q | k | v] of a portion: q to its own buffer, k and v into the cache rows of their positions
struct PromptRopeArgs { const float *p; uint32_t ld, H, KV, pos0; float *q, *kc, *vc; const float *qn, *kn, *cos_, *sin_; Dims d; };
__global__ void __launch_bounds__(256) k_prompt_rope(const PromptRopeArgs a) {
    dep_enter();
    __shared__ float buf[8][128];
    const uint32_t t = blockIdx.x, pos = a.pos0 + t, hd = a.d.hd, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const float *row = a.p + (size_t)t * a.ld, *cr = a.cos_ + (size_t)pos * (hd / 2u), *ci = a.sin_ + (size_t)pos * (hd / 2u);
    for (uint32_t h = warp; h < a.H + 2u * a.KV; h += 8u) {
        const bool isq = h < a.H, isk = !isq && h < a.H + a.KV;
        const uint32_t g = isq ? 0u : (h - a.H) % a.KV;
        float *dst = isq ? a.q + (size_t)t * a.H * hd + (size_t)h * hd : (isk ? a.kc : a.vc) + ((size_t)g * a.d.max_seq + pos) * hd;
        for (uint32_t i = lane; i < hd; i += 32u) buf[warp][i] = row[(size_t)h * hd + i];
        __syncwarp();
        if (isq || isk) head_norm_rope(buf[warp], isq ? a.qn : a.kn, cr, ci, a.d, false);
        for (uint32_t i = lane; i < hd; i += 32u) dst[i] = buf[warp][i];
        __syncwarp();
    }
}

// A head per warp and four of its values per lane, table and gains before the wait: heads of 4, 8, .. 128 values with a norm, of any multiple of 4 without.  (k_prompt_rope
// walks its heads through shared memory, four for every warp: 9.5 us for 250 positions of 32 heads, now 3.4.)
__global__ void __launch_bounds__(256) k_prompt_rope_warp(const PromptRopeArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t t = blockIdx.x, pos = a.pos0 + t, hd = a.d.hd, lane = threadIdx.x & 31u, h = blockIdx.y * 8u + (threadIdx.x >> 5);
    if (h >= a.H + 2u * a.KV) return;
    uint32_t lpr = 1;
    while (lpr * 4u < hd) lpr <<= 1;
    const uint32_t col = (lane & (lpr - 1u)) * 4u;
    const bool on = col < hd, isq = h < a.H, isk = !isq && h < a.H + a.KV;
    const uint32_t g = isq ? 0u : (h - a.H) % a.KV;
    const RopeTab rt = rope_tab_load(a.cos_ + (size_t)pos * (hd / 2u), a.sin_ + (size_t)pos * (hd / 2u), a.d, col, on);
    float4 gn = make_float4(0, 0, 0, 0), v = gn;
    if (a.d.arch == 3u && on && (isq || isk)) gn = __ldg(reinterpret_cast<const float4 *>((isq ? a.qn : a.kn) + col));
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (on) v = *reinterpret_cast<const float4 *>(a.p + (size_t)t * a.ld + (size_t)h * hd + col);
    if (isq || isk) v = norm_rope_apply(v, gn, rt, a.d, lpr, col, on);
    if (on && lane < lpr) {
        float *dst = isq ? a.q + (size_t)t * a.H * hd + (size_t)h * hd : (isk ? a.kc : a.vc) + ((size_t)g * a.d.max_seq + pos) * hd;
        *reinterpret_cast<float4 *>(dst + col) = v;
    }
}

// Attention of a short portion in fp32: a warp per query and head, lane = key for the scores, = columns for the values, 32 keys a turn.  The tensor-core kernels
// take 18 us for as little as 16 positions of Nano's 16 heads (images of keys and values, then one wave of tiles); this one 6, growing with positions x keys.
struct PromptAttnArgs { const float *q, *kc, *vc; float *out; uint32_t H, KV, hd, max_seq, pos0; float scale; };
__global__ void __launch_bounds__(256) k_prompt_attn(const PromptAttnArgs a) {
    dep_enter();
    __shared__ __align__(16) float q_s[8][128];
    const uint32_t t = blockIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, h = blockIdx.y * 8u + warp, hd = a.hd, nkeys = a.pos0 + t + 1u;
    if (h >= a.H) return;
    const uint32_t g = h / (a.H / a.KV);
    const float *K = a.kc + (size_t)g * a.max_seq * hd, *V = a.vc + (size_t)g * a.max_seq * hd, *q = a.q + ((size_t)t * a.H + h) * hd;
    if (lane * 4u < hd) *reinterpret_cast<float4 *>(&q_s[warp][lane * 4u]) = *reinterpret_cast<const float4 *>(q + lane * 4u);
    __syncwarp();
    float m = -FLT_MAX, l = 0.0f;          // (finite, so that a turn whose keys all score minus infinity weighs nothing: -inf - -inf would be no number)
    float4 o = make_float4(0, 0, 0, 0);
    for (uint32_t k0 = 0; k0 < nkeys; k0 += 32u) {
        const uint32_t n = min(32u, nkeys - k0);
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
        const float4 *kr = reinterpret_cast<const float4 *>(K + (size_t)(k0 + min(lane, n - 1u)) * hd);
#pragma unroll 8
        for (uint32_t c = 0; c < hd / 4u; c++) {
            const float4 k = kr[c], x = *reinterpret_cast<const float4 *>(&q_s[warp][c * 4u]);
            s0 = fmaf(k.x, x.x, s0); s1 = fmaf(k.y, x.y, s1); s2 = fmaf(k.z, x.z, s2); s3 = fmaf(k.w, x.w, s3);
        }
        const float s = lane < n ? ((s0 + s1) + (s2 + s3)) * a.scale : -INFINITY, mn = fmaxf(m, warp_max(s)), keep = expf(m - mn), p = lane < n ? expf(s - mn) : 0.0f;
        l = fmaf(l, keep, warp_sum(p));
        m = mn;
        o.x *= keep; o.y *= keep; o.z *= keep; o.w *= keep;
        const float *vr = V + (size_t)k0 * hd + lane * 4u;
#pragma unroll 8
        for (uint32_t j = 0; j < 32u; j++) {
            const float w = __shfl_sync(0xffffffffu, p, j);
            if (j < n && lane * 4u < hd) { const float4 v = *reinterpret_cast<const float4 *>(vr + (size_t)j * hd); o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w); }
        }
    }
    const float inv = 1.0f / l;
    if (lane * 4u < hd) *reinterpret_cast<float4 *>(a.out + ((size_t)t * a.H + h) * hd + lane * 4u) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
}

template <typename A>
int launch(void (*k)(const A), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, const A &args, uint32_t cluster_z = 1) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster_z > 1u) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 1; attr[cfg.numAttrs].val.clusterDim.y = 1; attr[cfg.numAttrs++].val.clusterDim.z = cluster_z;
    }
    NB_CK(cudaLaunchKernelEx(&cfg, k, args));
    return 0;
}
template <bool Q80, int TN>
int optin() { NB_CK(nb::smem_at_least((const void *)k_prompt_gemm<Q80, TN>, (int)gemm_smem<Q80, TN>())); return 0; }
}  // namespace

struct Product { PrefillMat m; CUtensorMap wmap; uint32_t np = 0; };      // np: F32 depth padded to 64
struct PrefillState {
    PrefillModel m; uint32_t sms = 148; bool pdl = true;
    decltype(&cuTensorMapEncodeTiled) encode = nullptr;
    std::vector<Product> qkv, wo, w13, w2;
    float *x = nullptr, *p = nullptr, *q = nullptr, *o = nullptr;      // residual rows, products, turned queries, attention output
    unsigned char *act = nullptr; float *scales = nullptr;             // codes or parts; group scales [G][kChunk]
    __nv_bfloat16 *parts = nullptr;                                    // F32: the matrix that is multiplied by, in parts
    struct AMap { uint32_t n, tn; CUtensorMap map; };
    std::vector<AMap> amaps;
    TcAttnState attn; uint32_t *err_host = nullptr, *err_dev = nullptr;
    std::vector<void *> allocs;
};

namespace {
int dmalloc(PrefillState *s, void **p, size_t bytes) {
    if (cudaMalloc(p, bytes ? bytes : 16) != cudaSuccess) return fail(NB200_ENOMEM, "cudaMalloc(%zu) failed", bytes);
    s->allocs.push_back(*p);
    return 0;
}
#define PM(ptr, bytes) do { int r_ = dmalloc(s, (void **)&(ptr), (bytes)); if (r_) return r_; } while (0)
bool map_2d(const PrefillState *s, CUtensorMap *m, bool q80, const void *base, uint64_t width, uint64_t rows, uint32_t box) {
    const cuuint64_t dims[2] = {width, rows}, strides[1] = {width * (q80 ? 1u : 2u)};
    const cuuint32_t b[2] = {q80 ? 128u : 64u, box}, step[2] = {1, 1};
    return s->encode(m, q80 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, b, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
int add_product(PrefillState *s, std::vector<Product> *list, const PrefillMat &m) {
    Product p;
    p.m = m;
    const bool q80 = s->m.quant == 0x80u;
    p.np = q80 ? 0u : (m.n + 63u) & ~63u;
    const void *base = q80 ? m.w : s->parts;
    const uint32_t width = q80 ? m.n : 3u * p.np;
    if (!map_2d(s, &p.wmap, q80, base, width, m.rows, kRows)) return fail(NB200_ECUDA, "cuTensorMapEncodeTiled refused a matrix of %u x %u", m.rows, m.n);
    list->push_back(p);
    return 0;
}
int create(PrefillState *s, const PrefillModel &m) {
    const bool q80 = m.quant == 0x80u;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult got;
    NB_CK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &got));
    if (got != cudaDriverEntryPointSuccess || !fn) return fail(NB200_ECUDA, "the driver has no cuTensorMapEncodeTiled");
    s->encode = reinterpret_cast<decltype(s->encode)>(fn);
    const uint32_t C = std::min(kChunk, (m.max_seq + 127u) & ~127u), wide = std::max(std::max(m.E, m.q_dim), m.F), wp = std::max(m.q_dim + 2 * m.kv_dim, 2 * m.F);
    const size_t act = (size_t)C * (q80 ? wide : ((wide + 63u) & ~63u) * 6u), scales = q80 ? (size_t)(wide / m.gs) * kChunk : 0u, tiles = attn_tc_tiles(m.max_seq, m.KV);
    size_t parts = 0;          // F32: the largest matrix
    if (!q80) for (const auto *list : {&m.qkv, &m.wo, &m.w13, &m.w2}) for (const PrefillMat &a : *list) parts = std::max(parts, (size_t)a.rows * ((a.n + 63u) & ~63u) * 6u);
    // images of keys and values for max_seq positions, up to 1 GB and to what is allowed (longer prompts run position by position)
    const size_t rest = parts + (size_t)C * (m.E + wp + 2 * m.q_dim) * 4u + act + scales * 4u + tiles * 8u, room = optional_room();
    if (rest >= room) return fail(NB200_ENOMEM, "prompts run position by position: portions need a workspace of %zu bytes, %zu are allowed", rest, room);
    const size_t images = std::min(std::min(attn_tc_bytes(m.max_seq, m.KV, m.hd, m.hd), (size_t)1 << 30), room - rest);
    int r;
    if (parts) PM(s->parts, parts);
    for (uint32_t l = 0; l < m.L; l++) {
        if ((r = add_product(s, &s->qkv, m.qkv[l]))) return r;
        if (l + 1u < m.L && ((r = add_product(s, &s->wo, m.wo[l])) || (r = add_product(s, &s->w13, m.w13[l])) || (r = add_product(s, &s->w2, m.w2[l])))) return r;
    }
    PM(s->x, (size_t)C * m.E * 4); PM(s->p, (size_t)C * wp * 4); PM(s->q, (size_t)C * m.q_dim * 4); PM(s->o, (size_t)C * m.q_dim * 4);
    PM(s->act, act); PM(s->scales, scales * 4);
    NB_CK(cudaMemset(s->act, 0, act));
    if (q80) NB_CK(cudaMemset(s->scales, 0, scales * 4));
    for (uint32_t n : {m.E, m.q_dim, m.F})
        for (uint32_t tn : {64u, 128u}) {
            PrefillState::AMap a{n, tn, {}};
            if (!map_2d(s, &a.map, q80, s->act, q80 ? n : 3u * ((n + 63u) & ~63u), C, tn)) return fail(NB200_ECUDA, "cuTensorMapEncodeTiled refused rows of %u", n);
            s->amaps.push_back(a);
        }
    NB_CK(cudaHostAlloc(&s->err_host, 64, cudaHostAllocMapped));
    *s->err_host = 0;
    NB_CK(cudaHostGetDevicePointer(&s->err_dev, s->err_host, 0));
    if ((r = attn_tc_setup(&s->attn, images, tiles, s->err_dev))) return r;
    if (q80 ? ((r = optin<true, 64>()) || (r = optin<true, 128>())) : (r = optin<false, 64>())) return r;
    NB_CK(cudaDeviceSynchronize());
    return 0;
}
int prep(PrefillState *s, const float *src, uint32_t ld, const float *gain, uint32_t n, uint32_t mode, uint32_t T, cudaStream_t stream) {
    const PromptPrepArgs a{src, ld, gain, n, s->m.gs, mode, reinterpret_cast<int8_t *>(s->act), s->scales, kChunk, reinterpret_cast<__nv_bfloat16 *>(s->act), (n + 63u) & ~63u};
    const bool q80 = s->m.quant == 0x80u;
    if (q80 && s->m.gs > 128u) return launch<PromptPrepArgs>(k_prompt_prep, dim3(T), dim3(kPrepThreads), 0, stream, s->pdl, a);
    return launch<PromptPrepArgs>(q80 ? k_prompt_rows<true> : k_prompt_rows<false>, dim3(T), dim3(kRowThreads), 0, stream, s->pdl, a);
}
int product(PrefillState *s, const Product &w, float *C, uint32_t ldc, bool add, uint32_t T, cudaStream_t stream) {
    // 64 positions per tile where tiles of 128 leave SMs without a block (1024 rows of the O product: 8 blocks for 128 positions), and in F32, whose
    // sums take two registers each
    const uint32_t rt = (w.m.rows + kRows - 1u) / kRows, tn = s->m.quant != 0x80u || T <= 64u || rt * ((T + 127u) / 128u) < s->sms ? 64u : 128u;
    PromptGemmArgs a{};
    a.wmap = w.wmap;
    for (const auto &m : s->amaps) if (m.n == w.m.n && m.tn == tn) a.amap = m.map;
    a.ws = static_cast<const float *>(w.m.aux); a.xs = s->scales; a.ldx = kChunk;
    a.N = w.m.rows; a.T = T; a.n = w.m.n; a.gs = s->m.gs; a.np = w.np; a.C = C; a.ldc = ldc; a.add = add ? 1u : 0u; a.err = s->err_dev;
    // clusters share a tile's depth while fewer than half of the SMs have a block
    const uint32_t tiles = rt * ((T + tn - 1u) / tn), ks = prompt_parts(prompt_units(s->m.quant == 0x80u, w.m.n, w.np, s->m.gs), tiles, s->sms);
    a.ks = ks;
    const dim3 grid(rt, (T + tn - 1u) / tn, ks), block(192);
#define GEMM(q, t) launch<PromptGemmArgs>(k_prompt_gemm<q, t>, grid, block, gemm_smem<q, t>(), stream, s->pdl, a, ks)
    if (s->m.quant == 0x80u) return tn == 64u ? GEMM(true, 64) : GEMM(true, 128);
    int r;
    const WeightPartsArgs wa{static_cast<const float *>(w.m.w), w.m.rows, w.m.n, w.np, s->parts};
    const size_t blocks = ((size_t)w.m.rows * (w.np / 8u) + 255u) / 256u;
    if ((r = launch<WeightPartsArgs>(k_weight_parts, dim3((uint32_t)std::min<size_t>(blocks, s->sms * 8u)), dim3(256), 0, stream, s->pdl, wa))) return r;
    return GEMM(false, 64);
#undef GEMM
}
}  // namespace

int prefill_create(PrefillState **out, const PrefillModel &m, uint32_t sms) {
    *out = nullptr;
    const bool q80 = m.quant == 0x80u;
    if (!q80 && m.quant != 0x00u) return 0;
    if (q80 && (m.gs != 32u && m.gs != 64u && m.gs != 128u && m.gs != 256u)) return 0;
    if (m.hd > 128u || m.hd % 4u || m.E % 8u || m.q_dim % 8u || m.F % 8u || m.q_dim != m.H * m.hd || m.kv_dim != m.KV * m.hd || m.H % m.KV || std::max(std::max(m.E, m.q_dim), m.F) > 32768u) return 0;
    if (q80 && (m.E % 16u || m.q_dim % 16u || m.F % 16u || m.E % m.gs || m.q_dim % m.gs || m.F % m.gs)) return 0;
    PrefillState *s = new PrefillState();
    s->m = m; s->sms = sms;
    const int r = create(s, m);
    if (r) { prefill_destroy(s); return r; }
    *out = s;
    return 0;
}
void prefill_destroy(PrefillState *s) {
    if (!s) return;
    attn_tc_free(&s->attn);
    for (void *p : s->allocs) cudaFree(p);
    if (s->err_host) cudaFreeHost(s->err_host);
    delete s;
}
int prefill_check(PrefillState *s) {
    if (!s || !s->err_host || !*static_cast<volatile uint32_t *>(s->err_host)) return 0;
    const uint32_t code = *s->err_host;
    *s->err_host = 0;
    return fail(NB200_ECUDA, "a wait inside a prompt kernel ran out (code 0x%x): the results of this call are not valid", code);
}
int prefill_run(PrefillState *s, const uint32_t *ids, uint32_t n, cudaStream_t stream, bool pdl, uint64_t *launches) {
    s->pdl = pdl;
    const PrefillModel &m = s->m;
    const uint32_t W = m.q_dim + 2 * m.kv_dim, extra = m.quant == 0x80u ? 0u : 1u;
    const size_t kvl = (size_t)m.KV * m.max_seq * m.hd;
    Dims d{};
    d.arch = m.arch; d.hd = m.hd; d.max_seq = m.max_seq;
    const bool by_warp = m.arch != 3u || (m.hd & (m.hd - 1u)) == 0;          // the norm's exchange of halves between lanes wants 4 x 2^k values
    int r;
    for (uint32_t p0 = 0; p0 < n; p0 += kChunk) {
        const uint32_t T = std::min(kChunk, n - p0);
        if ((r = launch<PromptEmbedArgs>(k_prompt_embed, dim3(T), dim3(256), 0, stream, pdl, PromptEmbedArgs{m.emb.w, m.emb.aux, s->x, ids + p0, m.E, m.gs, m.quant}))) return r;
        (*launches)++;
        for (uint32_t l = 0; l < m.L; l++) {
            const PromptRopeArgs ra{s->p, W, m.H, m.KV, p0, s->q, m.kc + l * kvl, m.vc + l * kvl, m.qnorm ? m.qnorm + (size_t)l * m.hd : nullptr, m.knorm ? m.knorm + (size_t)l * m.hd : nullptr, m.rope_cos, m.rope_sin, d};
            if ((r = prep(s, s->x, m.E, m.norm_attn + (size_t)l * m.E, m.E, PREP_NORM, T, stream)) || (r = product(s, s->qkv[l], s->p, W, false, T, stream)) ||
                (r = by_warp ? launch<PromptRopeArgs>(k_prompt_rope_warp, dim3(T, (m.H + 2u * m.KV + 7u) / 8u), dim3(256), 0, stream, pdl, ra)
                             : launch<PromptRopeArgs>(k_prompt_rope, dim3(T), dim3(256), 0, stream, pdl, ra))) return r;
            *launches += 3u + extra;
            if (l + 1u == m.L) break;          // nothing reads what the last layer would make of these positions
            TcAttn a{};
            a.q = s->q; a.ldq = m.q_dim; a.q_head = m.hd; a.k = m.kc + l * kvl; a.v = m.vc + l * kvl; a.ldk = a.ldv = m.hd; a.k_head = a.v_head = (uint64_t)m.max_seq * m.hd;
            a.out = s->o; a.T = T; a.H = m.H; a.G = m.KV; a.D = a.VD = m.hd; a.pos0 = p0; a.scale = (float)(1.0 / sqrt((double)m.hd));
            const bool few = p0 == 0 && T <= (m.hd <= 64u && m.H <= 16u ? kPromptAttnFew : kPromptAttnFewWide);
            const PromptAttnArgs pa{s->q, m.kc + l * kvl, m.vc + l * kvl, s->o, m.H, m.KV, m.hd, m.max_seq, p0, a.scale};
            if (!few && !attn_tc_fits(&s->attn, a)) return fail(NB200_EINVAL, "a prompt of %u positions does not fit the attention's buffers", n);
            if ((r = few ? launch<PromptAttnArgs>(k_prompt_attn, dim3(T, (m.H + 7u) / 8u), dim3(256), 0, stream, pdl, pa) : attn_tc_launch(&s->attn, a, stream, pdl)) || (r = prep(s, s->o, m.q_dim, nullptr, m.q_dim, PREP_PLAIN, T, stream)) || (r = product(s, s->wo[l], s->x, m.E, true, T, stream)) ||
                (r = prep(s, s->x, m.E, m.norm_ffn + (size_t)l * m.E, m.E, PREP_NORM, T, stream)) || (r = product(s, s->w13[l], s->p, 2 * m.F, false, T, stream)) ||
                (r = prep(s, s->p, 2 * m.F, nullptr, m.F, PREP_SWIGLU, T, stream)) || (r = product(s, s->w2[l], s->x, m.E, true, T, stream))) return r;
            *launches += (few ? 7u : 8u) + 3u * extra;
        }
    }
    return 0;
}
// whether a prompt of n positions fits
bool prefill_fits(const PrefillState *s, uint32_t n) { return s && attn_tc_bytes(n, s->m.KV, s->m.hd, s->m.hd) <= s->attn.bytes; }

}  // namespace nb
