// layered_gqa_one.cuh -- grouped-query attention of a single token (the captured decode step), in the argument block of layered_mixers4.cuh.
//
// What bounds it is the chain between the joint product and the output product: the cache rows of all earlier tokens lie ready long before the queries do, so they are on
// their way to shared memory before the wait; after it every warp walks its own keys, four at a time, without a barrier between scores, softmax and values; and the blocks of a
// key/value head are one cluster, which hands its partial sums round through shared memory (no partials in memory, no fence, no ticket).
// k_gqa_decode, which takes one to four tokens and any alignment (92 KB of code, a page at a time, a barrier after each step, merge by the last block), took 7.5 us of a token of 16 heads of
// 64 at 10 positions, 12.2 and 21.9 of 128 at 1030 and 1780; this 5.1, 7.9 and 11.5.  (Four query heads a block, four keys a turn: 7.0, 14.2 and 19.4.)
#pragma once
#include "layered_mixers4.cuh"

namespace nb {
namespace lm {

constexpr uint32_t kGqaOneBlocks = 8, kGqaOneWarps = 8, kGqaOneHeads = 2, kGqaOneDim = 128, kGqaOneStages = 2, kGqaOneKeys = 8;
// Shared memory: per warp and stage eight rows of keys and values (afterwards the warps' partial sums)
inline size_t gqa_one_smem(uint32_t D, uint32_t VD) { return std::max((size_t)kGqaOneWarps * kGqaOneStages * kGqaOneKeys * (D + VD), (size_t)kGqaOneWarps * kGqaOneHeads * kGqaOneDim) * 4u; }

// The keys the token sees are dealt out in groups of eight: group i to block i % 8, warp i / 8 % 8.  8 lanes share a key's coordinates (of two keys); a lane has 4 value columns of all
// keys.  The group that holds the token itself takes its key and value from the product's row; its block writes them to the cache.
// grid = (kGqaOneBlocks, G x pairs of query heads), clusters of kGqaOneBlocks; 256 threads: one per query head of the pair and coordinate outside the walk over the keys.
// *pos_ptr, the page table and the cache rows before the token are read before the wait: they are written before the kernel that embeds the token, which is launched without overlap.
template <int NH>
__global__ void __launch_bounds__(256) k_gqa_one(const GqaArgs a) {
    pdl_launch_next();
    cluster_arrive();                          // waited for before the first access to another block's shared memory
    constexpr uint32_t CK = kGqaOneDim / 32u, ST = kGqaOneStages, KG = kGqaOneKeys, SLICE = NH * kGqaOneDim / kGqaOneBlocks, NP = kGqaOneBlocks;
    extern __shared__ __align__(16) float gqa_sm[];
    __shared__ __align__(16) float q_s[2][kGqaOneDim], kn_s[kGqaOneDim], vn_s[kGqaOneDim];
    __shared__ float red[2][8], m_s[NH][8], l_s[NH][8], in_o[NP][SLICE], in_m[NP][NH], in_l[NP][NH];
    const uint32_t D = a.D, VD = a.VD, row_f = D + VD, rep = a.H / a.G, hgs = (rep + NH - 1u) / NH, g = blockIdx.y / hgs, h0 = g * rep + blockIdx.y % hgs * NH, nh = min((uint32_t)NH, (g + 1u) * rep - h0);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, sub = lane & 7u, key = lane >> 3, rank = blockIdx.x, half = a.tab ? a.half : 0u;
    const uint32_t pos = a.pos0 + (a.pos_ptr ? *a.pos_ptr : 0u), low = gqa_first(pos, a.block), base = low & ~(KG - 1u);
    const uint32_t groups = (pos - base) / KG + 1u, own = groups - 1u, mine = warp * NP + rank, step = NP * kGqaOneWarps;
    float *ring = gqa_sm + warp * ST * KG * row_f;
    const float *kv = a.cache + g * D;
    const uint32_t to_v = a.G * D + g * VD - g * D;
    auto page_of = [&](uint32_t grp) { return grp < groups ? a.table[(base + grp * KG) / kPage] : 0u; };
    auto fetch = [&](uint32_t grp, uint32_t page, uint32_t st) {          // this lane's part of its two keys' rows; zeros where there is no earlier token
        if (grp < groups) {
            const uint32_t k0 = base + grp * KG + key;
            const float *row = kv + ((size_t)page * kPage + k0 % kPage) * a.RL;
            float *dst = ring + (st * KG + key) * row_f;
#pragma unroll
            for (uint32_t j = 0; j < 2u; j++) {
                const bool ok = k0 + 4u * j >= low && k0 + 4u * j < pos;
                const float *r = row + (ok ? j * 4u * a.RL : 0u);
#pragma unroll
                for (uint32_t c = 0; c < CK; c++) {
                    const uint32_t d = (sub + 8u * c) * 4u;
                    if (d < D) cp_async16(dst + j * 4u * row_f + d, r + d, ok);
                    if (d < VD) cp_async16(dst + j * 4u * row_f + D + d, r + to_v + d, ok);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint32_t page[ST];
#pragma unroll
    for (uint32_t i = 0; i < ST; i++) page[i] = page_of(mine + i * step);
#pragma unroll
    for (uint32_t i = 0; i < ST; i++) fetch(mine + i * step, page[i], i);
    uint32_t next_page = page_of(mine + ST * step);
    // this thread's coordinate d of query head h0 + hq (and of the token's key): gains and the turn's angle
    const uint32_t hq = min(tid >> 7, nh - 1u), d = tid & 127u, dp = d < half ? d + half : d < 2u * half ? d - half : d;
    const bool owner = own % NP == rank, in = d < D, turned = in && d < 2u * half;
    const float *wq = a.wq && !a.head_norm ? a.wq + (h0 + hq) * D : a.wq, *wk = a.wk && !a.head_norm ? a.wk + g * D : a.wk;
    float2 cs = make_float2(1.0f, 0.0f), gq = make_float2(1.0f, 1.0f), gk = gq;
    if (turned) { cs = a.tab[(size_t)pos * half + (d < half ? d : dp)]; if (d < half) cs.y = -cs.y; }
    if (in && wq) gq = make_float2(__ldg(wq + d), __ldg(wq + dp));
    if (in && wk && owner) gk = make_float2(__ldg(wk + d), __ldg(wk + dp));
    pdl_wait();
    // queries and the key, gained and turned; their norms' factors (of whole rows, or of a head) join the scores
    const float *q = a.p + a.q0 + (h0 + hq) * D, *k = a.p + a.k0 + g * D;
    float2 xq = make_float2(0.0f, 0.0f), xk = xq;
    float xv = 0.0f, sq = 0.0f, sk = 0.0f;
    if (in) xq = make_float2(q[d], q[dp]);
    if (owner) { if (in) xk = make_float2(k[d], k[dp]); if (d < VD) xv = a.p[a.v0 + g * VD + d]; }
    if (a.head_norm) { sq = xq.x * xq.x; sk = xk.x * xk.x; }
    else {
        if (a.wq)
#pragma unroll 2
            for (uint32_t i = tid * 4u; i < a.H * D; i += 1024u) { const float4 u = *reinterpret_cast<const float4 *>(a.p + a.q0 + i); sq = fmaf(u.x, u.x, fmaf(u.y, u.y, fmaf(u.z, u.z, fmaf(u.w, u.w, sq)))); }
        if (a.wk && owner)
#pragma unroll 2
            for (uint32_t i = tid * 4u; i < a.G * D; i += 1024u) { const float4 u = *reinterpret_cast<const float4 *>(a.p + a.k0 + i); sk = fmaf(u.x, u.x, fmaf(u.y, u.y, fmaf(u.z, u.z, fmaf(u.w, u.w, sk)))); }
    }
    sq = warp_sum(sq); sk = warp_sum(sk);
    if (lane == 0) { red[0][warp] = sq; red[1][warp] = sk; }
    const float nq = xq.x * gq.x, nk = xk.x * gk.x;
    q_s[tid >> 7][d] = turned ? nq * cs.x + xq.y * gq.y * cs.y : nq;
    const float kn = turned ? nk * cs.x + xk.y * gk.y * cs.y : nk;
    __syncthreads();
    auto sum = [&](const float *r, uint32_t from, uint32_t n) { float v = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < 8u; w++) v += w >= from && w < from + n ? r[w] : 0.0f;
        return v; };
    float qf[NH];
#pragma unroll
    for (uint32_t h = 0; h < NH; h++)
        qf[h] = a.scale * (!a.wq ? 1.0f : a.head_norm ? 1.0f / sqrtf(sum(red[0], 4u * h, 4u) / (float)D + a.eps) : 1.0f / sqrtf(sum(red[0], 0u, 8u) / (float)(a.H * D) + a.eps));
    if (owner) {          // (every block of the key/value head's pairs holds the token; the first pair's writes the cache row)
        const float kf = !a.wk ? 1.0f : a.head_norm ? 1.0f / sqrtf(sum(red[1], 0u, 4u) / (float)D + a.eps) : 1.0f / sqrtf(sum(red[1], 0u, 8u) / (float)(a.G * D) + a.eps);
        if (tid < 128u) { kn_s[d] = kn * kf; vn_s[d] = xv; }
        if (blockIdx.y % hgs == 0 && tid < 128u) {
            float *row = a.cache + ((size_t)a.table[pos / kPage] * kPage + pos % kPage) * a.RL;
            if (in) row[g * D + d] = kn * kf;
            if (d < VD) row[a.G * D + g * VD + d] = xv;
        }
        __syncthreads();
    }
    float4 qr[NH][CK];
    float o[NH][4], m[NH], l[NH];
#pragma unroll
    for (uint32_t h = 0; h < NH; h++) {
        m[h] = -INFINITY; l[h] = 0.0f;
#pragma unroll
        for (uint32_t c = 0; c < CK; c++) qr[h][c] = *reinterpret_cast<const float4 *>(&q_s[h][(sub + 8u * c) * 4u]);
#pragma unroll
        for (uint32_t i = 0; i < 4u; i++) o[h][i] = 0.0f;
    }
    uint32_t st = 0;
#pragma unroll 1
    for (uint32_t grp = mine; grp < groups; grp += step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kGqaOneStages - 1) : "memory");
        __syncwarp();
        const uint32_t kp = base + grp * KG + key;
        float *tile = ring + st * KG * row_f;
        if (grp == own) {          // the token itself
#pragma unroll 1
            for (uint32_t i = lane * 4u; i < row_f; i += 128u) *reinterpret_cast<float4 *>(tile + (pos % KG) * row_f + i) = *reinterpret_cast<const float4 *>(i < D ? kn_s + i : vn_s + i - D);
            __syncwarp();
        }
        float s[2][NH];
#pragma unroll
        for (uint32_t j = 0; j < 2u; j++) {
            const float *row = tile + (key + 4u * j) * row_f;
#pragma unroll
            for (uint32_t h = 0; h < NH; h++) s[j][h] = 0.0f;
#pragma unroll
            for (uint32_t c = 0; c < CK; c++)
                if ((sub + 8u * c) * 4u < D) {
                    const float4 kk = *reinterpret_cast<const float4 *>(row + (sub + 8u * c) * 4u);
#pragma unroll
                    for (uint32_t h = 0; h < NH; h++) s[j][h] = fmaf(qr[h][c].w, kk.w, fmaf(qr[h][c].z, kk.z, fmaf(qr[h][c].y, kk.y, fmaf(qr[h][c].x, kk.x, s[j][h]))));
                }
        }
#pragma unroll
        for (int off = 4; off > 0; off >>= 1)
#pragma unroll
            for (uint32_t j = 0; j < 2u; j++)
#pragma unroll
                for (uint32_t h = 0; h < NH; h++) s[j][h] += __shfl_xor_sync(0xffffffffu, s[j][h], off);
#pragma unroll
        for (uint32_t h = 0; h < NH; h++) {
#pragma unroll
            for (uint32_t j = 0; j < 2u; j++) {
                s[j][h] *= qf[h];
                if (a.softcap > 0.0f) s[j][h] = a.softcap * tanhf(s[j][h] / a.softcap);
                if (kp + 4u * j < low || kp + 4u * j > pos) s[j][h] = -INFINITY;
            }
            float tm = fmaxf(s[0][h], s[1][h]);
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 8)); tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 16));
            const float mn = fmaxf(m[h], tm), mr = mn == -INFINITY ? 0.0f : mn, corr = expf(m[h] - mr);          // (scores of minus infinity weigh nothing)
            s[0][h] = expf(s[0][h] - mr); s[1][h] = expf(s[1][h] - mr);
            float ps = s[0][h] + s[1][h];
            ps += __shfl_xor_sync(0xffffffffu, ps, 8); ps += __shfl_xor_sync(0xffffffffu, ps, 16);
            l[h] = fmaf(l[h], corr, ps); m[h] = mn;
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++) o[h][i] *= corr;
        }
        const float *vt = tile + D + (lane * 4u < VD ? lane * 4u : 0u);          // (lanes past the values: another column's, which nobody reads)
#pragma unroll
        for (uint32_t j = 0; j < KG; j++) {
            const float4 v = *reinterpret_cast<const float4 *>(vt + j * row_f);
#pragma unroll
            for (uint32_t h = 0; h < NH; h++) {
                const float p = __shfl_sync(0xffffffffu, s[j >> 2][h], (j & 3u) * 8u);
                o[h][0] = fmaf(p, v.x, o[h][0]); o[h][1] = fmaf(p, v.y, o[h][1]); o[h][2] = fmaf(p, v.z, o[h][2]); o[h][3] = fmaf(p, v.w, o[h][3]);
            }
        }
        __syncwarp();                          // the stage has been read
        fetch(grp + ST * step, next_page, st);
        next_page = page_of(grp + (ST + 1u) * step);
        st = st + 1u == ST ? 0u : st + 1u;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();                           // every warp is done with its rows
    // the warps' sums, then the blocks': out = gate sum e^{m_i - M} o_i / (sum e^{m_i - M} l_i + e^{sink - M})
    float *o_s = gqa_sm;                       // [warps][NH][128]
#pragma unroll
    for (uint32_t h = 0; h < NH; h++) {
        *reinterpret_cast<float4 *>(o_s + (warp * NH + h) * kGqaOneDim + lane * 4u) = make_float4(o[h][0], o[h][1], o[h][2], o[h][3]);
        if (lane == 0) { m_s[h][warp] = m[h]; l_s[h][warp] = l[h]; }
    }
    __syncthreads();
    cluster_wait();
    if (tid < NH * kGqaOneDim) {
        const uint32_t h = tid / kGqaOneDim;
        float M = -INFINITY, w[8], L = 0.0f, v = 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < 8u; i++) { w[i] = m_s[h][i]; M = fmaxf(M, w[i]); }
        const float mr = M == -INFINITY ? 0.0f : M;
#pragma unroll
        for (uint32_t i = 0; i < 8u; i++) { w[i] = expf(w[i] - mr); L = fmaf(w[i], l_s[h][i], L); v = fmaf(w[i], o_s[(i * NH + h) * kGqaOneDim + d], v); }
        st_cluster(&in_o[rank][tid % SLICE], tid / SLICE, v);
        if (d < NP) { st_cluster(&in_m[rank][h], d, M); st_cluster(&in_l[rank][h], d, L); }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (tid >= SLICE) return;
    const uint32_t at = rank * SLICE + tid, h = at / kGqaOneDim, c = at % kGqaOneDim;
    if (h >= nh || c >= VD) return;
    float M = a.sink ? a.sink[h0 + h] : -INFINITY, w[NP], L = 0.0f, v = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < NP; i++) { w[i] = in_m[i][h]; M = fmaxf(M, w[i]); }
    const float mr = M == -INFINITY ? 0.0f : M;
#pragma unroll
    for (uint32_t i = 0; i < NP; i++) { w[i] = expf(w[i] - mr); L = fmaf(w[i], in_l[i][h], L); v = fmaf(w[i], in_o[i][tid], v); }
    if (a.sink) L += expf(a.sink[h0 + h] - mr);
    a.out[(size_t)(h0 + h) * VD + c] = v * (a.has_gate ? sigmoidf_(a.p[a.g0 + h0 + h]) : 1.0f) / L;
}

}  // namespace lm
}  // namespace nb
