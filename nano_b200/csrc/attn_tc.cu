// attn_tc.cu -- softmax attention of long portions on the fifth-generation tensor cores: fp32 queries, keys and values, products of 32-bit precision.
//
// An fp32 number x is the sum of two f16 numbers to 2^-23 of it, h = f16(x) and l = f16(x - h) (23 of its 24 bits: a quarter of all numbers are off by the last
// one), as long as it lies within 2^-17 of the largest number of its tile (a tile is brought to just under 2^15 by a power of two); a smaller one is
// off by 2^-40 of that largest.  a b = ha hb + ha lb + la hb, three f16 products with fp32 accumulators, leaves out la lb, 2^-22 at most and 2^-25 as a root mean
// square: each the size of one fp32 rounding, where a pass of FMAs makes one per term.  A tile in which one number is more than 2^17 times another holds
// the small ones in fewer bits than fp32 does; an infinity or a NaN in a tile of values makes every row of the tile NaN (as in the FMA kernel, whose tiles are 64 keys).
// The tensor cores cut what they add instead of rounding it, so sums are kept short: the two small products go first, and a
// tile's weighted values join the running sum by ordinary fp32 arithmetic.
// (mma.sync with three bfloat16 parts was built first: 550 us for 976 queries x 16 heads on 1512 keys on average, against 600 for the FMA kernel; the
// old tensor path of this chip does some 600 multiply-adds per cycle and SM.)
//
//   k_attn_images   a tile of 128 keys of one head: its scale, then keys and transposed values in two planes each, in the byte order of
//                   the swizzled shared-memory operand: the attention kernel fetches a tile with two bulk copies
//   k_attn_tc       a block owns 128 rows (query token, query head) of one key/value head.  Warp 0 fetches, warp 1 issues tcgen05.mma, two threads of warps
//                   2..9 own one row, 64 keys of a tile and half of the values each: scores come out of tensor memory with a lane per row, and what the two tell each other is
//                   the tile's maximum; its weights go back into tensor memory as the A operand of the second product.  Scores are double buffered and a
//                   tile's values are added while the next tile's scores are made, so the tensor cores (busy for 11 % of the time) work under the softmax
//                   of eight warps, two per scheduler, which bounds the kernel: with a thread per row, one warp per scheduler, its chain of loads, exponentials and splits
//                   issued in 26 % of the cycles.
// 1024 queries x 16 heads over 4 key/value heads of 128 on 1536 keys on average: 102 us, 606 by the FMA kernel (k_gqa_attn), with softcap 130 and 640; error
// against float64 on normal numbers 0.4e-6 .. 1.1e-6 of a row's norm where the FMA kernel has 0.75e-6 .. 1.6e-6.
#include "attn_tc.h"

#include <cuda_fp16.h>
#include <math.h>

#include "family.h"
#include "tc_ptx.cuh"

namespace nb {
namespace {

constexpr uint32_t kTile = 128, kPageKeys = 32;          // keys of a tile = rows of a block
constexpr float kWeightScale = 16384.0f;                 // weights (0..1) before they are split

// a power of two that brings `big` to [2^14, 2^15)
__device__ __forceinline__ float tile_scale(float big) {
    const int e = (int)(__float_as_uint(big) >> 23) - 127;
    if (!(big > 0.0f) || e > 127) return 1.0f;           // nothing but zeros; with an infinity a tile is not brought anywhere
    return __uint_as_float((uint32_t)(127 + max(-113, min(100, 14 - e))) << 23);
}
__device__ __forceinline__ uint32_t pack2(__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); }
// (x, y) as pairs of the large and of the small parts
__device__ __forceinline__ void split2(float x, float y, uint32_t &h, uint32_t &l) {
    const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
    h = pack2(hx, hy);
    l = pack2(__float2half_rn(x - __half2float(hx)), __float2half_rn(y - __half2float(hy)));
}
__device__ __forceinline__ void split8(const float (&x)[8], float s, uint4 &h, uint4 &l) {
    split2(x[0] * s, x[1] * s, h.x, l.x); split2(x[2] * s, x[3] * s, h.y, l.y); split2(x[4] * s, x[5] * s, h.z, l.z); split2(x[6] * s, x[7] * s, h.w, l.w);
}
__host__ __device__ constexpr uint32_t padded(uint32_t d) { return d <= 64u ? 64u : 128u; }
// byte of the 16-byte piece c8 (8 f16) of row r in an operand of 64-wide blocks of `rows` rows, 128-byte swizzle
__device__ __forceinline__ uint32_t op_byte(uint32_t rows, uint32_t r, uint32_t c8) { return (c8 >> 3) * rows * 128u + r * 128u + (((c8 & 7u) ^ (r & 7u)) << 4); }
__device__ __forceinline__ float max8(const float (&x)[8]) {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) m = fmaxf(m, fabsf(x[i]));
    return m;
}
__device__ __forceinline__ void load8(const float *p, uint32_t n, float (&x)[8]) {          // n: how many exist (a multiple of 4)
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f), a = n >= 4u ? *reinterpret_cast<const float4 *>(p) : z, b = n >= 8u ? *reinterpret_cast<const float4 *>(p + 4) : z;
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
template <int NT>
__device__ __forceinline__ float block_max(float v, float *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = red[0];
    for (int w = 1; w < NT / 32; w++) m = fmaxf(m, red[w]);
    return m;
}
__host__ __device__ inline uint32_t oldest(const TcAttn &a, uint32_t pos) {          // the first key that position pos sees
    uint32_t f = a.block ? pos - pos % a.block : 0u;
    if (a.window && pos + 1u > a.window && pos + 1u - a.window > f) f = pos + 1u - a.window;
    return f;
}

struct ImageArgs { TcAttn a; unsigned char *images; float *scales; uint32_t tile0, tiles, nkeys; };
// image (g, tile): [keys: 2 planes][DP / 64][128 keys][64] then [values: 2 planes][2][VP][64 keys], f16; scales (g, tile): the inverse scales of both.
// blockIdx.z 0: the keys, 1: the values
constexpr uint32_t kImageThreads = 512;
__global__ void __launch_bounds__(kImageThreads) k_attn_images(const ImageArgs ia) {
    asm volatile("griddepcontrol.launch_dependents;\ngriddepcontrol.wait;" ::: "memory");
    __shared__ float red[kImageThreads / 32];
    __shared__ size_t row_s[kTile];
    const TcAttn &a = ia.a;
    const uint32_t tile = ia.tile0 + blockIdx.x, g = blockIdx.y, key0 = tile * kTile, nk = min(kTile, ia.nkeys - key0), DP = padded(a.D), VP = padded(a.VD);
    const bool keys = blockIdx.z == 0;
    if (threadIdx.x < nk) {
        const uint32_t j = key0 + threadIdx.x;
        row_s[threadIdx.x] = (a.table ? (size_t)a.table[j / kPageKeys] * kPageKeys + j % kPageKeys : j - a.first_row) * (keys ? a.ldk : a.ldv);
    }
    __syncthreads();
    const float *src = keys ? a.k + g * a.k_head : a.v + g * a.v_head;
    const uint32_t W = keys ? a.D : a.VD, W4 = W / 4u;
    unsigned char *img = ia.images + ((size_t)g * ia.tiles + blockIdx.x) * (DP + VP) * 512u + (keys ? 0u : DP * 512u);
    float x[8], m = 0.0f;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < nk * W4; i += kImageThreads) {
        const float4 q = *reinterpret_cast<const float4 *>(src + row_s[i / W4] + i % W4 * 4u);
        m = fmaxf(m, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))));
    }
    const float s = tile_scale(block_max<kImageThreads>(m, red));
    if (threadIdx.x == 0) ia.scales[((size_t)g * ia.tiles + blockIdx.x) * 2u + blockIdx.z] = 1.0f / s;
    if (keys) {
        const uint32_t d8 = DP / 8u;
#pragma unroll 2
        for (uint32_t i = threadIdx.x; i < kTile * d8; i += kImageThreads) {          // rows past the last key and columns past D are zeros
            const uint32_t r = i / d8, c = i % d8;
            load8(src + (r < nk ? row_s[r] : 0u) + c * 8u, r < nk && c * 8u < W ? W - c * 8u : 0u, x);
            uint4 h, l;
            split8(x, s, h, l);
            const uint32_t at = op_byte(kTile, r, c);
            *reinterpret_cast<uint4 *>(img + at) = h; *reinterpret_cast<uint4 *>(img + DP * 256u + at) = l;
        }
    } else {
#pragma unroll 2
        for (uint32_t i = threadIdx.x; i < VP * (kTile / 8u); i += kImageThreads) {          // 8 keys of one value column
            const uint32_t d = i % VP, c = i / VP;
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) x[j] = (d < W && c * 8u + j < nk) ? src[row_s[c * 8u + j] + d] : 0.0f;
            uint4 h, l;
            split8(x, s, h, l);
            const uint32_t at = op_byte(VP, d, c);
            *reinterpret_cast<uint4 *>(img + at) = h; *reinterpret_cast<uint4 *>(img + VP * 256u + at) = l;
        }
    }
}

struct AttnTcArgs { TcAttn a; const unsigned char *images; const float *scales; uint32_t tile0, tiles; uint32_t *err; };

constexpr uint32_t kAttnThreads = 320;
template <int DP, int VP> constexpr size_t attn_smem() { return (size_t)(DP + DP + VP) * 512u + 1024u; }          // queries, keys, values

template <int DP, int VP>
__global__ void __launch_bounds__(kAttnThreads, 1) k_attn_tc(const AttnTcArgs ta) {
    extern __shared__ uint8_t tc_raw[];
    enum { KFULL, KFREE, VFULL, VFREE, SFULL0, SFULL1, PREADY, OREADY, NBAR };
    __shared__ __align__(8) uint64_t bars[NBAR];
    __shared__ uint32_t tmem_s, bad_s;
    __shared__ float red[16], top_s[2][2][kTile], sum_s[2][kTile];          // of a row's halves: the largest score of a tile (tiles alternate), the sum of weights
    const TcAttn &a = ta.a;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t qs = (smem_u32(tc_raw) + 1023u) & ~1023u, ksm = qs + DP * 512u, vsm = ksm + DP * 512u;
    unsigned char *q_s = tc_raw + (qs - smem_u32(tc_raw));
    const uint32_t b0 = smem_u32(bars);
    auto bar = [&](uint32_t i) { return b0 + i * 8u; };
    if (tid == 0) {
        for (uint32_t i = 0; i < NBAR; i++) mbar_init(bar(i), i == PREADY ? 8 : 1);
        bad_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { tc_alloc(smem_u32(&tmem_s), 512); tc_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Only now may the next kernel's blocks come: one that waits for this grid while it holds tensor memory must not be in the way of an allocation here
    asm volatile("griddepcontrol.launch_dependents;\ngriddepcontrol.wait;" ::: "memory");
    const uint32_t tmem = tmem_s;
    const uint32_t rep = a.H / a.G, rows = a.T * rep, g = blockIdx.y, r0 = (gridDim.x - 1u - blockIdx.x) * kTile;      // the longest rows first
    const uint32_t last = min(rows, r0 + kTile) - 1u;
    const uint32_t first_pos = a.pos0 + r0 / rep, last_pos = a.pos0 + last / rep, lo = oldest(a, first_pos) / kTile, hi = last_pos / kTile + 1u, n = hi - lo;
    const unsigned char *img = ta.images + ((size_t)g * ta.tiles + (lo - ta.tile0)) * (DP + VP) * 512u;
    const float *scales = ta.scales + ((size_t)g * ta.tiles + (lo - ta.tile0)) * 2u;
    // the block's queries, split, in operand order
    float qinv;
    {
        constexpr uint32_t d8 = DP / 8;
        const uint32_t D8 = (a.D + 7u) / 8u;
        float x[8], m = 0.0f;
        for (uint32_t i = tid; i < (last - r0 + 1u) * D8; i += kAttnThreads) {
            const uint32_t rr = r0 + i / D8, c = i % D8 * 8u;
            load8(a.q + (size_t)(rr / rep) * a.ldq + (size_t)(g * rep + rr % rep) * a.q_head + c, a.D - c, x);
            m = fmaxf(m, max8(x));
        }
        float s = tile_scale(block_max<kAttnThreads>(m, red));
        qinv = 1.0f / s;
        if (a.scale < 0.0f) s = -s;          // the largest raw score is to be the largest score: the sign of a negative scale goes with the query
        for (uint32_t i = tid; i < kTile * d8; i += kAttnThreads) {
            const uint32_t r = i / d8, c = i % d8, rr = min(r0 + r, last);
            load8(a.q + (size_t)(rr / rep) * a.ldq + (size_t)(g * rep + rr % rep) * a.q_head + c * 8u, c * 8u < a.D ? a.D - c * 8u : 0u, x);
            uint4 h, l;
            split8(x, s, h, l);
            const uint32_t at = op_byte(kTile, r, c);
            *reinterpret_cast<uint4 *>(q_s + at) = h; *reinterpret_cast<uint4 *>(q_s + DP * 256 + at) = l;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    // tensor memory: scores (two buffers of 128), where a tile's weights take the place of its scores (32 columns of scores: 16 of the large parts, 16 of the
    // small), and a tile's weighted values.  Heads of 64 values have room for a sum per 32 keys: the tensor cores cut what they add, always towards zero, and a
    // quarter of the additions cut a quarter as much (four layers of width 768 behind 200 / 487 positions, logits against 64 bits by those of single
    // positions: 1.00 / 1.00 with four sums a tile, 1.01 / 1.02 with two)
    constexpr uint32_t SCOL = 0, OCOL = 256, SUMS = VP == 64 ? 4 : 1;
    if (warp == 0 && lane == 0) {
        for (uint32_t i = 0; i < n; i++) {
            if (i && !mbar_wait(bar(KFREE), (i - 1u) & 1u)) { bad_s = 1; break; }
            mbar_expect(bar(KFULL), DP * 512u);
            bulk_load(ksm, img + (size_t)i * (DP + VP) * 512u, DP * 512u, bar(KFULL));
            if (i && !mbar_wait(bar(VFREE), (i - 1u) & 1u)) { bad_s = 2; break; }
            mbar_expect(bar(VFULL), VP * 512u);
            bulk_load(vsm, img + (size_t)i * (DP + VP) * 512u + DP * 512u, VP * 512u, bar(VFULL));
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t id_s = (1u << 4) | ((kTile >> 3) << 17) | ((kTile >> 4) << 24), id_o = (1u << 4) | ((uint32_t)(VP >> 3) << 17) | ((kTile >> 4) << 24);      // fp32 += f16 x f16
        auto scores = [&](uint32_t i) {
            if (!mbar_wait(bar(KFULL), i & 1u)) return false;
            tc_fence_after();
            const uint32_t d = tmem + SCOL + (i & 1u) * kTile;
            bool add = false;
#pragma unroll
            for (uint32_t p = 0; p < 3; p++)          // small x large, large x small, large x large
#pragma unroll
                for (uint32_t ks = 0; ks < DP / 16; ks++) {
                    const uint32_t off = (ks >> 2) * kTile * 128u + (ks & 3u) * 32u;
                    tc_mma_ss(d, tc_desc(qs + (p == 0 ? DP * 256u : 0u) + off), tc_desc(ksm + (p == 1 ? DP * 256u : 0u) + off), id_s, add);
                    add = true;
                }
            tc_commit(bar(KFREE)); tc_commit(bar(SFULL0 + (i & 1u)));
            return true;
        };
        bool ok = scores(0) && (n < 2 || scores(1));
        for (uint32_t i = 0; i < n && ok; i++) {
            ok = mbar_wait(bar(PREADY), i & 1u) && mbar_wait(bar(VFULL), i & 1u);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (uint32_t p = 0; p < 3; p++)
#pragma unroll
                for (uint32_t ks = 0; ks < kTile / 16; ks++) {
                    const uint32_t off = (ks >> 2) * VP * 128u + (ks & 3u) * 32u;
                    const uint32_t w = SCOL + (i & 1u) * kTile + (ks >> 1) * 32u + (ks & 1u) * 8u + (p == 0 ? 16u : 0u);
                    tc_mma_ts(tmem + OCOL + (SUMS > 1 ? (ks >> 1) * VP : 0u), tmem + w, tc_desc(vsm + (p == 1 ? VP * 256u : 0u) + off), id_o, p > 0 || (SUMS > 1 ? ks & 1u : ks) > 0);
                }
            tc_commit(bar(VFREE)); tc_commit(bar(OREADY));
            if (i + 2u < n) ok = mbar_wait(bar(OREADY), i & 1u) && scores(i + 2u);          // they overwrite the weights that the products before read (tile i + 1's scores are there meanwhile)
        }
        if (!ok) bad_s = 3;
    } else if (warp >= 2) {
        const uint32_t quad = warp & 3u, r = quad * 32u + lane, rr = min(r0 + r, last), t = rr / rep, h = g * rep + rr % rep;
        const uint32_t pos = a.pos0 + t, low = oldest(a, pos), low_last = oldest(a, last_pos), lane_base = (quad * 32u) << 16;
        // a row belongs to two threads, of warps that reach the same lanes of tensor memory: each has 64 keys of a tile and half of the values.  They share the row's
        // maximum once a tile (the barrier of their two warps, which also says whether both go on) and their sums at the end.
        constexpr int VH = VP / 2;
        const uint32_t half = (warp - 2u) >> 2, c_lo = half * (kTile / 2u), v_lo = half * (uint32_t)VH;
        float m = a.sink ? a.sink[h] : -INFINITY, l = a.sink && half == 0 ? 1.0f : 0.0f, o[VH];
#pragma unroll
        for (int d = 0; d < VH; d++) o[d] = 0.0f;
        bool ok = true;
        float vinv = 0.0f;
        // the values of the tile before join the sum, which then moves to the new maximum
        auto collect = [&](uint32_t i, float corr) {
            ok = mbar_wait_warp(bar(OREADY), i & 1u);
            if (!ok) return;
            tc_fence_after();
            const float f = vinv * corr;
#pragma unroll
            for (int c = 0; c < VH; c += 32) {
                uint32_t w[32];
                tc_ld32(tmem + lane_base + OCOL + v_lo + c, w);
#pragma unroll
                for (int j = 0; j < 32; j++) o[c + j] = fmaf(__uint_as_float(w[j]), f, o[c + j] * corr);
#pragma unroll
                for (uint32_t q = 1; q < SUMS; q++) {
                    tc_ld32(tmem + lane_base + OCOL + q * VP + v_lo + c, w);
#pragma unroll
                    for (int j = 0; j < 32; j++) o[c + j] = fmaf(__uint_as_float(w[j]), f, o[c + j]);
                }
            }
        };
        for (uint32_t i = 0; i < n; i++) {
            const uint32_t key0 = (lo + i) * kTile, s_at = tmem + lane_base + SCOL + (i & 1u) * kTile;
            const float kc = qinv * scales[2u * i] * (a.softcap > 0.0f ? fabsf(a.scale) / a.softcap : fabsf(a.scale));
            const bool whole = key0 + kTile <= first_pos + 1u && key0 >= low_last;          // every row of the block sees every key of the tile
            ok = ok && mbar_wait_warp(bar(SFULL0 + (i & 1u)), (i >> 1) & 1u);
            tc_fence_after();
            const uint32_t j0 = low > key0 ? low - key0 : 0u, j1 = pos < key0 ? 0u : min(kTile, pos - key0 + 1u);          // the keys this row sees
            float top = -INFINITY;
            if (ok)
#pragma unroll 1
            for (uint32_t c = c_lo; c < c_lo + kTile / 2u; c += 32u) {
                uint32_t w[32];
                tc_ld32(s_at + c, w);
                if (whole) {
#pragma unroll
                    for (uint32_t j = 0; j < 32; j++) top = fmaxf(top, __uint_as_float(w[j]));
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 32; j++) top = c + j >= j0 && c + j < j1 ? fmaxf(top, __uint_as_float(w[j])) : top;
                }
            }
            top_s[i & 1u][half][r] = top;
            if (bar_any(1u + quad, 64u, !ok)) { ok = false; break; }
            top = fmaxf(top, top_s[i & 1u][half ^ 1u][r]) * kc;
            if (a.softcap > 0.0f && top != -INFINITY) top = a.softcap * tanhf(top);
            const float mn = fmaxf(m, top), corr = mn == -INFINITY ? 1.0f : expf(m - mn);
            if (i) collect(i - 1u, corr);
            if (!ok) continue;          // both warps leave at the next barrier, or after the last tile
            vinv = scales[2u * i + 1u] / kWeightScale;
            float sum = 0.0f;
#pragma unroll 1          // (a tile's whole code does not fit the instruction cache)
            for (uint32_t c = c_lo; c < c_lo + kTile / 2u; c += 32u) {
                uint32_t w[32], wh[16], wl[16];
                tc_ld32(s_at + c, w);
                float p[32];
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) p[j] = __uint_as_float(w[j]) * kc;
                if (a.softcap > 0.0f) {
#pragma unroll
                    for (uint32_t j = 0; j < 32; j++) p[j] = a.softcap * tanhf(p[j]);
                }
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) p[j] = expf(p[j] - mn);
                if (!whole) {
#pragma unroll
                    for (uint32_t j = 0; j < 32; j++) p[j] = c + j >= j0 && c + j < j1 ? p[j] : 0.0f;
                }
                float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) s4[j & 3u] += p[j];
                sum += (s4[0] + s4[1]) + (s4[2] + s4[3]);
#pragma unroll
                for (uint32_t j = 0; j < 16; j++) split2(p[2 * j] * kWeightScale, p[2 * j + 1] * kWeightScale, wh[j], wl[j]);
                tc_st16(s_at + c, wh);
                tc_st16(s_at + c + 16u, wl);
            }
            l = fmaf(l, corr, sum);
            m = mn;
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(PREADY));
        }
        if (ok) collect(n - 1u, 1.0f);
        sum_s[half][r] = l;
        ok = !bar_any(1u + quad, 64u, !ok);
        if (!ok) bad_s = 4;
        if (ok && r0 + r <= last) {
            float f = 1.0f / (sum_s[0][r] + sum_s[1][r]);
            if (a.gate) f *= 1.0f / (1.0f + expf(-a.gate[(size_t)t * a.ldg + h]));
            float *dst = a.out + ((size_t)t * a.H + h) * a.VD + v_lo;
            const float *mul = a.mul ? a.mul + (size_t)t * a.ldm + (size_t)h * a.VD + v_lo : nullptr;
#pragma unroll
            for (int d = 0; d < VH; d += 4)
                if (v_lo + d < a.VD) {
                    float4 y = make_float4(o[d] * f, o[d + 1] * f, o[d + 2] * f, o[d + 3] * f);
                    if (mul) { y.x *= mul[d]; y.y *= mul[d + 1]; y.z *= mul[d + 2]; y.w *= mul[d + 3]; }
                    *reinterpret_cast<float4 *>(dst + d) = y;
                }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (bad_s) {
        if (tid == 0) {
            *ta.err = 0x200u + bad_s;
            __threadfence_system();
            const long long t0 = clock64();
            while (clock64() - t0 < 20000000ll) __nanosleep(1000);          // copies still in flight land in this block's shared memory before it is given back
        }
        __syncthreads();
    }
    if (warp == 1) tc_dealloc(tmem, 512);
}

template <typename A>
int launch(void (*k)(const A), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl, const A &args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.attrs = attr;
    if (pdl) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    NB_CK(cudaLaunchKernelEx(&cfg, k, args));
    return 0;
}
template <int DP, int VP>
int optin() { NB_CK(nb::smem_at_least((const void *)k_attn_tc<DP, VP>, (int)attn_smem<DP, VP>())); return 0; }
bool aligned16(const float *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
}  // namespace

size_t attn_tc_bytes(uint32_t keys, uint32_t G, uint32_t D, uint32_t VD) { return D <= 128u && VD <= 128u ? attn_tc_tiles(keys, G) * (padded(D) + padded(VD)) * 512u : 0u; }
int attn_tc_setup(TcAttnState *s, size_t bytes, size_t tiles, uint32_t *err_dev) {
    int r;
    s->err_dev = err_dev;
    if (!bytes) return 0;
    if (cudaMalloc(&s->images, bytes) != cudaSuccess) { s->images = nullptr; return fail(NB200_ENOMEM, "cudaMalloc(%zu) failed", bytes); }
    if (cudaMalloc(&s->scales, tiles * 8u) != cudaSuccess) { s->scales = nullptr; return fail(NB200_ENOMEM, "cudaMalloc(%zu) failed", tiles * 8u); }
    s->bytes = bytes; s->tiles = tiles;
    if ((r = optin<64, 64>()) || (r = optin<64, 128>()) || (r = optin<128, 64>()) || (r = optin<128, 128>())) return r;
    return 0;
}
void attn_tc_free(TcAttnState *s) {
    if (s->images) cudaFree(s->images);
    if (s->scales) cudaFree(s->scales);
    s->images = nullptr; s->scales = nullptr; s->bytes = s->tiles = 0;
}
uint32_t attn_tc_first(const TcAttn &a) { return oldest(a, a.pos0) / kTile * kTile; }
bool attn_tc_fits(const TcAttnState *s, const TcAttn &a) {
    const uint32_t keys = a.pos0 + a.T - attn_tc_first(a);
    return s->images && a.D && a.VD && a.D <= 128u && a.VD <= 128u && ((a.D | a.VD | a.ldk | a.ldv | a.k_head | a.v_head | a.ldq | a.q_head) & 3u) == 0 && aligned16(a.k) && aligned16(a.v) &&
           aligned16(a.q) && aligned16(a.out) && a.H % a.G == 0 && attn_tc_tiles(keys, a.G) <= s->tiles && attn_tc_bytes(keys, a.G, a.D, a.VD) <= s->bytes;
}
int attn_tc_launch(TcAttnState *s, const TcAttn &a, cudaStream_t stream, bool pdl) {
    const uint32_t tile0 = attn_tc_first(a) / kTile, nkeys = a.pos0 + a.T, tiles = (nkeys + kTile - 1u) / kTile - tile0;
    int r;
    if ((r = launch<ImageArgs>(k_attn_images, dim3(tiles, a.G, 2), dim3(kImageThreads), 0, stream, pdl, ImageArgs{a, s->images, s->scales, tile0, tiles, nkeys}))) return r;
    const AttnTcArgs ta{a, s->images, s->scales, tile0, tiles, s->err_dev};
    const dim3 grid((a.T * (a.H / a.G) + kTile - 1u) / kTile, a.G), block(kAttnThreads);
    if (a.D <= 64u) return a.VD <= 64u ? launch<AttnTcArgs>(k_attn_tc<64, 64>, grid, block, attn_smem<64, 64>(), stream, pdl, ta) : launch<AttnTcArgs>(k_attn_tc<64, 128>, grid, block, attn_smem<64, 128>(), stream, pdl, ta);
    return a.VD <= 64u ? launch<AttnTcArgs>(k_attn_tc<128, 64>, grid, block, attn_smem<128, 64>(), stream, pdl, ta) : launch<AttnTcArgs>(k_attn_tc<128, 128>, grid, block, attn_smem<128, 128>(), stream, pdl, ta);
}

}  // namespace nb
