// layered_one.cuh -- the matrix-vector products of a single token (the captured decode step), in the argument block of layered_common.cuh.
//
// What bounds a step is the chain of its launches, and of a link the latency of what it does after the kernel before it has finished (an empty link of this
// chain takes 0.5 us, one load and store 1.0).  So everything that does not depend on that kernel happens before the wait: a warp's first weight row is in
// registers by then, constants of the epilogue too.  After it the block brings the activation row into shared memory ONCE, normed and rounded there, with a
// single trip to L2, and the epilogue's operands travel at the same time; what is left is the row's dot from registers and shared memory.
// k_gemv, which serves up to four rows and any alignment, reads the row in every warp, converts it there, and its epilogue starts a trip of its own.
// A chain of 1024 x 1024 products from HBM, us a link: k_gemv 4.5, weights in registers 2.9, this 2.1 (with two
// running sums; one, in k_gemv's order, makes a whole step of eight routed layers bit for bit that of the general kernels: 290 us a token, 265 with two, 364 before).
// What is left of a link is then the instructions it passes, 620 a warp for a row of 1024, most of them for steps that such a row does not have: a warp leaves a run of steps at its own
// last one, checks lanes only in rows that end inside a step, and loads an activation row of up to 8 KB at once.  Call to call, a token of eight Famudra layers of width 1024 249 -> 232 us.
#pragma once
#include "layered_kernels.cuh"
#include "layered_mixers3.cuh"

namespace nb {
namespace lm {

constexpr uint32_t kOneThreads = 256, kOneWarps = kOneThreads / 32;
constexpr uint32_t kOneMaxK = 11264;          // the row in shared memory (fp32) and the static part stay below 48 KB
template <typename WT> constexpr __host__ __device__ uint32_t one_step() { return 512u / sizeof(WT); }          // columns a warp covers with one 16-byte load a lane
template <typename WT> inline uint32_t one_smem(uint32_t K) { return (K + one_step<WT>() - 1u) / one_step<WT>() * one_step<WT>() * 4u; }

// a load that stays in front of the wait (the compiler may move an ordinary read-only load behind it, to where its value is used)
__device__ __forceinline__ uint4 load_now(const void *p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float load_now_f(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
// where 4-column chunk c of the activation row lies in shared memory: a lane of the dot reads the 8 columns of its 16 bytes of bf16 weights as two loads,
// each of them over 32 neighbouring chunks
template <typename WT> __device__ __forceinline__ uint32_t one_place(uint32_t c) {
    return sizeof(WT) == 2 ? (c & ~63u) + ((c & 1u) << 5) + ((c & 63u) >> 1) : c;
}
// (one running sum in the order of the columns: the same bits as k_gemv where a row has one warp)
template <typename WT> __device__ __forceinline__ void one_fma(const uint4 &w, const float4 *x, uint32_t step, uint32_t lane, float &acc) {
    if (sizeof(WT) == 2) {
        const float4 p = x[step * 64u + lane], q = x[step * 64u + 32u + lane];
        acc = fmaf(__uint_as_float(w.x << 16), p.x, acc); acc = fmaf(__uint_as_float(w.x & 0xffff0000u), p.y, acc);
        acc = fmaf(__uint_as_float(w.y << 16), p.z, acc); acc = fmaf(__uint_as_float(w.y & 0xffff0000u), p.w, acc);
        acc = fmaf(__uint_as_float(w.z << 16), q.x, acc); acc = fmaf(__uint_as_float(w.z & 0xffff0000u), q.y, acc);
        acc = fmaf(__uint_as_float(w.w << 16), q.z, acc); acc = fmaf(__uint_as_float(w.w & 0xffff0000u), q.w, acc);
    } else {
        const float4 p = x[step * 32u + lane];
        acc = fmaf(__uint_as_float(w.x), p.x, acc); acc = fmaf(__uint_as_float(w.y), p.y, acc);
        acc = fmaf(__uint_as_float(w.z), p.z, acc); acc = fmaf(__uint_as_float(w.w), p.w, acc);
    }
}
__device__ __forceinline__ float4 round4(float4 v) { return make_float4(round_bf16(v.x), round_bf16(v.y), round_bf16(v.z), round_bf16(v.w)); }
__device__ __forceinline__ float sum_sq4(float4 v, float s) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, s)))); }

// The activation row, as the product uses it, into shared memory (chunks past K zero).  Ends with a barrier.
template <typename WT, int EXT>
__device__ __forceinline__ void one_stage(const GemmArgs &a, const float *row, float4 *x, float *red) {
    const uint32_t K4 = a.K / 4u, P4 = (a.K + one_step<WT>() - 1u) / one_step<WT>() * one_step<WT>() / 4u;
    const float4 *src = reinterpret_cast<const float4 *>(row), *nw = reinterpret_cast<const float4 *>(a.a_norm_w);
    const bool poly = EXT == 2 && a.a_poly, raw = nw || poly;
    float s2 = 0.0f, s4 = 0.0f, s6 = 0.0f;
    for (uint32_t c0 = threadIdx.x; c0 - threadIdx.x < P4; c0 += 2u * kOneThreads) {          // two loads at a time, also of a short row
        float4 vs[2];
#pragma unroll
        for (uint32_t j = 0; j < 2u; j++) vs[j] = c0 + j * kOneThreads < K4 ? src[c0 + j * kOneThreads] : make_float4(0, 0, 0, 0);
#pragma unroll
        for (uint32_t j = 0; j < 2u; j++) {
            const uint32_t c = c0 + j * kOneThreads;
            if (c - threadIdx.x >= P4) break;
            float4 v = vs[j];
            if (EXT == 2) s2 = sum_sq4(v, s2);
            if (EXT == 2) {
                const float q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; j++) { const float v2 = q[j] * q[j], v3 = v2 * q[j]; s4 = fmaf(v2, v2, s4); s6 = fmaf(v3, v3, s6); }
            }
            if (c < P4) x[one_place<WT>(c)] = !raw && a.round_a ? round4(v) : v;
        }
    }
    if (raw) {
        float sc = 1.0f;
        PolyRow pc{0.0f, 0.0f, 0.0f, 0.0f};
        __shared__ float gsc[EXT == 4 ? 32 : 1];
        const uint32_t plen = EXT == 4 ? a.K / a.a_parts : 1u;
        if (EXT == 4) {          // a warp per part: the part's root mean square
            __syncthreads();
            const uint32_t lane = threadIdx.x & 31u;
            for (uint32_t p = threadIdx.x >> 5; p < a.a_parts; p += kOneWarps) {
                float s = 0.0f;
                for (uint32_t c = p * plen / 4u + lane; c < (p + 1u) * plen / 4u; c += 32u) s = sum_sq4(x[one_place<WT>(c)], s);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) gsc[p] = 1.0f / sqrtf(s / (float)plen + a.a_eps);
            }
            __syncthreads();
        } else {
            if (EXT != 2) {          // single values in k_gemv's order
                __syncthreads();
                const float *xf = reinterpret_cast<const float *>(x);
                for (uint32_t k = threadIdx.x; k < a.K; k += kOneThreads) { const float v = xf[one_place<WT>(k / 4u) * 4u + (k & 3u)]; s2 = fmaf(v, v, s2); }
            }
            s2 = block_sum(s2, red);
            if (EXT == 2 && poly) {
                s4 = block_sum(s4, red); s6 = block_sum(s6, red);
                pc.r1 = a.a_poly[0] / sqrtf(s2 / (float)a.K + a.a_eps); pc.r2 = a.a_poly[1] / sqrtf(s4 / (float)a.K + a.a_eps);
                pc.r3 = a.a_poly[2] / sqrtf(s6 / (float)a.K + a.a_eps); pc.e = a.a_poly[3];
            } else sc = 1.0f / sqrtf(s2 / (float)a.K + a.a_eps);
        }
        for (uint32_t c = threadIdx.x; c < K4; c += kOneThreads) {          // a thread's own chunks
            float4 v = x[one_place<WT>(c)];
            if (nw) {
                const float si = EXT == 4 ? gsc[c * 4u / plen] : sc;
                const float4 g = __ldg(nw + c);
                v.x = v.x * si * g.x; v.y = v.y * si * g.y; v.z = v.z * si * g.z; v.w = v.w * si * g.w;
            }
            if (EXT == 2 && poly) { v.x = poly_of(v.x, pc); v.y = poly_of(v.y, pc); v.z = poly_of(v.z, pc); v.w = poly_of(v.w, pc); }
            x[one_place<WT>(c)] = a.round_a ? round4(v) : v;
        }
    }
    __syncthreads();
}

// what a column's epilogue reads from memory, asked for long before it is needed (tap, tail: lane j holds those of tap j)
struct OneEpi { float bias, mul, tap, tail, x, pw, pb, nw, nb; };

// Rows of a group past its first, where they are not the same: block bx's columns of them, the row from memory.  Such rows come from choices that tie at minus infinity,
// which no trained model makes: what counts is that other products pay nothing for it.  So only the instance for such rows (EXT 6, the second product of experts whose input is
// weighted by the choice; the plain one otherwise) has this, and everything is found anew here. (In the plain instance a
// token of two layers took 103.4 -> 105.6 us in 32 bits, 74.1 -> 74.5 in bf16: more code to fetch.)
template <typename WT>
__device__ __forceinline__ void one_more_rows(const GemmArgs &a, uint32_t bx, uint32_t nbx, uint32_t gy) {
    constexpr uint32_t VN = WVec<WT>::N;
    const GroupView gv = group_view(a, a.g_act ? a.g_act[gy] : gy);
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 1
    for (uint32_t i = 1; i < gv.rows; i++) {
        const float *row = a.A + (size_t)(gv.r0 + i) * a.lda + gv.a0;
#pragma unroll 1
        for (uint32_t n = bx * kOneWarps + (threadIdx.x >> 5); n < a.N; n += nbx * kOneWarps) {
            float v = 0.0f, w[VN];
#pragma unroll 1
            for (uint32_t k = lane * VN; k < a.K; k += 32u * VN) {
                WVec<WT>::load(static_cast<const WT *>(a.W) + gv.w0 + (size_t)n * a.ldw + k, w);
#pragma unroll
                for (uint32_t j = 0; j < VN; j++) v = fmaf(w[j], a.round_a ? round_bf16(row[k + j]) : row[k + j], v);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) store_c(a, a.C + (size_t)(gv.r0 + i) * a.ldc + gv.c0 + n, gated(a, epilogue(v, a, gv.bias, n), gv.r0 + i, gv.c0 + n));
        }
    }
}

// Block bx of nbx, place gy in the list of groups; a group has one row, or several of the same token.  The instances (EXT) are k_gemv's, and 6: the plain one whose groups may have rows that differ.
template <typename WT, int EXT>
__device__ __forceinline__ void gemv_one(const GemmArgs &a, uint32_t bx, uint32_t nbx, uint32_t gy) {
    constexpr uint32_t VN = WVec<WT>::N, STEP = one_step<WT>(), NW = EXT == 3 ? 2u : 1u, PRE = EXT == 3 ? 4u : 8u;
    extern __shared__ float4 one_x[];
    __shared__ float red[32];
    __shared__ float part_s[2][NW][kOneWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, steps = (a.K + STEP - 1u) / STEP;
    // a row is shared by 2^a.one_split warps, each with its share of the steps; a block has kOneWarps / that many rows at a time
    const uint32_t split = a.one_split, part = warp & ((1u << split) - 1u), rpb = kOneWarps >> split, share = (steps + (1u << split) - 1u) >> split;
    const uint32_t s_lo = min(steps, part * share), s_hi = min(steps, s_lo + share), nrows = nbx * rpb;
    const WT *W = static_cast<const WT *>(a.W);
    const bool fixed = !a.g_off;
    const uint32_t n0 = bx * rpb + (warp >> split);
    uint32_t n = n0;
    uint4 w[NW][PRE];
    const bool ragged = a.K % STEP != 0;          // the last step's lanes past the row: zeros
    auto fetch = [&](uint32_t row, uint32_t s0) {          // steps s0 .. of this warp's share (a row past the last: the last one, whose result nobody stores)
        const WT *p = W + (size_t)min(row, a.N - 1u) * a.ldw + s0 * STEP + lane * VN;
        const uint32_t left = a.K - s0 * STEP - lane * VN;
#pragma unroll
        for (uint32_t i = 0; i < PRE; i++) {
            if (s0 + i >= s_hi) break;
#pragma unroll
            for (uint32_t h = 0; h < NW; h++) {
                if (!ragged || (int32_t)(i * STEP) < (int32_t)left) w[h][i] = load_now(p + (size_t)(h * a.N) * a.ldw + i * STEP);
                else w[h][i] = make_uint4(0, 0, 0, 0);
            }
        }
    };
    if (fixed) {
        W += (uint64_t)gy * a.w_gstride;
        fetch(n, s_lo);
        if (share > PRE || n + nrows < a.N) prefetch_weight_rows(W, sizeof(WT), a.ldw, a.K, a.N, n, nrows, 2u);          // the rest of the first row, the second
        if (a.a_norm_w) for (uint32_t k = threadIdx.x * 32u; k < a.K; k += kOneThreads * 32u) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.a_norm_w + k));
    }
    // arguments that are read after the wait: a launch's arguments lie in memory that no cache near the SM holds yet
    uint32_t group = gy, r0 = 0, rows = 1;          // (several rows of one expert: choices that tie at -infinity, the same row but for EXT 6)
    const float *bias = a.bias, *row = a.A;
    float *C = a.C;
    auto place = [&]() {          // of the group
        if (bias) bias += (size_t)group * a.b_gstride;
        if (a.a_gmod > 1u) row += (size_t)(group % a.a_gmod) * a.a_gcols;
        C += (size_t)group * a.c_gcols;
    };
    OneEpi e{};
    if (fixed) {
        place();
        if (bias && n < a.N) e.bias = load_now_f(bias + n);
    }
    pdl_wait();
    if (!fixed) {
        group = a.g_act ? a.g_act[gy] : gy;
        if (group == 0xffffffffu) return;
        W += (uint64_t)group * a.w_gstride;
        fetch(n, s_lo);
        r0 = a.g_off[group];
        rows = a.g_off[group + 1u] - r0;
        if (rows == 0) return;
        place();
        if (bias && n < a.N) e.bias = __ldg(bias + n);
        C += (size_t)r0 * a.ldc;
        row += (size_t)(a.a_rows ? a.a_rows[r0] : r0) * a.lda;
    } else if (a.a_rows) row += (size_t)a.a_rows[0] * a.lda;
    const uint32_t c0 = group * a.c_gcols;
    // the convolution that column n is a channel of, if any
    auto conv_of = [&](uint32_t col, GemmArgs::ConvRange &r) -> bool {
        if (EXT == 0 && a.epi == EPI_GELU_CONV && col >= a.split) { r = GemmArgs::ConvRange{a.split, a.N, a.cv_taps, a.cv_bias, a.cv_state, a.cv_out, a.cv_K, 0u}; return true; }
        if (EXT == 1 && a.epi == EPI_CONV_RANGES) {
            if (col >= a.cr[0].n0 && col < a.cr[0].n1) { r = a.cr[0]; return true; }
            if (col >= a.cr[1].n0 && col < a.cr[1].n1) { r = a.cr[1]; return true; }
        }
        return false;
    };
    auto early = [&](uint32_t col) {
        if (col >= a.N) return;
        if (col != n0 && bias) e.bias = __ldg(bias + col);
        if (a.mul) e.mul = a.mul[(size_t)r0 * a.ldm + c0 + col];
        GemmArgs::ConvRange r;
        if ((EXT == 0 || EXT == 1) && conv_of(col, r)) {
            const uint32_t c = col - r.n0, C = r.n1 - r.n0;
            if (lane < r.K) e.tap = __ldg(r.taps + (size_t)c * r.K + lane);
            if (lane + 1u < r.K) e.tail = r.state[(size_t)lane * C + c];
            e.pb = r.bias ? __ldg(r.bias + c) : 0.0f;
        }
        if ((EXT == 4 || EXT == 5) && a.res_x) {
            e.x = a.res_x[(size_t)r0 * a.N + col]; e.pw = __ldg(a.res_pw + col); e.pb = __ldg(a.res_pb + col);
            if (a.res_out) { e.nw = __ldg(a.res_nw + col); e.nb = __ldg(a.res_nb + col); }
        }
    };
    if (!part) early(n);
    const float scale = EXT == 3 && a.row_scale ? a.row_scale[r0] : 1.0f;
    one_stage<WT, EXT>(a, row, one_x, red);

    for (uint32_t base = bx * rpb, turn = 0; base < a.N; base += nrows, n += nrows, turn ^= 1u) {          // the same turns for all of the block's warps
        float acc[NW];
#pragma unroll
        for (uint32_t h = 0; h < NW; h++) acc[h] = 0.0f;
        for (uint32_t s0 = s_lo;;) {
#pragma unroll
            for (uint32_t i = 0; i < PRE; i++) {
                if (s0 + i >= s_hi) break;
#pragma unroll
                for (uint32_t h = 0; h < NW; h++) one_fma<WT>(w[h][i], one_x, s0 + i, lane, acc[h]);
            }
            s0 += PRE;
            if (s0 >= s_hi) break;
            fetch(n, s0);
        }
        const OneEpi now = e;
        if (n + nrows < a.N) { fetch(n + nrows, s_lo); if (!part) early(n + nrows); }          // on their way during the sum and the epilogue
        float v = acc[0], up = NW == 2 ? acc[NW - 1u] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_xor_sync(0xffffffffu, v, o);
            if (NW == 2) up += __shfl_xor_sync(0xffffffffu, up, o);
        }
        if (split) {
            if (lane == 0) { part_s[turn][0][warp] = v; if (NW == 2) part_s[turn][NW - 1u][warp] = up; }
            __syncthreads();
            if (part) continue;
            for (uint32_t p = 1; p < 1u << split; p++) { v += part_s[turn][0][warp + p]; if (NW == 2) up += part_s[turn][NW - 1u][warp + p]; }
        }
        if (n >= a.N) continue;
        float *dst = C + n;
        GemmArgs::ConvRange r;
        if ((EXT == 0 || EXT == 1) && conv_of(n, r)) {          // one new input: lane j holds input j of the window, the last one is new
            const float in = lane + 1u == r.K ? (EXT == 0 ? v + now.bias : v) : now.tail;
            float s = now.pb;
            for (uint32_t j = 0; j < r.K; j++) s = fmaf(__shfl_sync(0xffffffffu, now.tap, j), __shfl_sync(0xffffffffu, in, j), s);
            const float next = __shfl_down_sync(0xffffffffu, in, 1);
            const uint32_t c = n - r.n0, C = r.n1 - r.n0;
            if (lane + 1u < r.K) r.state[(size_t)lane * C + c] = next;
            if (r.act) s = s / (1.0f + expf(-s));
            if (lane == 0) r.out[(size_t)r0 * C + c] = s;
            continue;
        }
        if (lane != 0) continue;
        if (EXT == 3) {          // the gated pair
            for (uint32_t i = 0; i < rows; i++) {
                const float f = i && a.row_scale ? a.row_scale[r0 + i] : scale, g = v * f, u = up * f;
                store_c(a, dst + (size_t)i * a.ldc, (a.glu == 3u ? clamped_glu(g, u, a.glu_limit) : (a.glu == 2u ? g / (1.0f + expf(-g)) : gelu_tanh(g)) * u));
            }
            continue;
        }
        v = epilogue(v + now.bias, a, nullptr, n);
        if ((EXT == 4 || EXT == 5) && a.res_x) {
            const size_t at = (size_t)r0 * a.N + n;
            const float xv = now.x + fmaf(tanhf(a.res_pa * v), now.pw, now.pb);
            a.res_x[at] = xv;
            if (a.res_keep) a.res_keep[at] = xv;
            if (a.res_out) a.res_out[at] = fmaf(tanhf(a.res_na * xv), now.nw, now.nb);
        } else for (uint32_t i = 0; i < (EXT == 6 ? 1u : rows); i++) store_c(a, dst + (size_t)i * a.ldc, a.mul ? v * now.mul : v);
    }
    if (EXT == 6 && rows > 1u) one_more_rows<WT>(a, bx, nbx, gy);
}

template <typename WT, int EXT>
__global__ void __launch_bounds__(kOneThreads, 4) k_gemv_one(const GemmArgs a) {
    pdl_launch_next();
    gemv_one<WT, EXT>(a, blockIdx.x, gridDim.x, blockIdx.y);
}
// the products that also norm (and turn) the token's latent into the cache: one more block does that beside them
template <typename WT>
__global__ void __launch_bounds__(kOneThreads, 4) k_gemv_one_latent(const GemvLatentArgs a) {
    pdl_launch_next();
    if (blockIdx.x + 1u == gridDim.x) {
        __shared__ float red[32];
        pdl_wait();
        latent_kv_row(a.n, 0, red);
        return;
    }
    gemv_one<WT, 0>(a.g, blockIdx.x, gridDim.x - 1u, 0u);
}
template <typename WT>
__global__ void __launch_bounds__(kOneThreads, 4) k_gemv_one_latent_rope(const GemvLatentRopeArgs a) {
    pdl_launch_next();
    if (blockIdx.y + 1u == gridDim.y) {
        __shared__ float red[32];
        pdl_wait();
        if (blockIdx.x == 0) latent_rope_row(a.n, 0, red);
        return;
    }
    gemv_one<WT, 0>(a.g, blockIdx.x, gridDim.x, blockIdx.y);
}

// k_rglru_gates_scan for one token: a warp per channel, both gate rows and the channel's constants in registers before the wait (blocks of at most
// 2 steps of columns, a multiple of a 16-byte load)
template <typename WT>
__global__ void __launch_bounds__(kOneThreads) k_rglru_gates_one(const GatesScanArgs a) {
    constexpr uint32_t VN = WVec<WT>::N, STEP = one_step<WT>();
    pdl_launch_next();
    const uint32_t lane = threadIdx.x & 31u, c = blockIdx.x * kOneWarps + (threadIdx.x >> 5);
    if (c >= a.C) return;
    const WT *wr = static_cast<const WT *>(a.W) + (size_t)c * a.bs, *wi = static_cast<const WT *>(a.W) + (size_t)(a.C + c) * a.bs;
    float r[2][VN], g[2][VN];
#pragma unroll
    for (uint32_t i = 0; i < 2u; i++) {
        const uint32_t k = i * STEP + lane * VN;
        if (k < a.bs) { WVec<WT>::load(wr + k, r[i]); WVec<WT>::load(wi + k, g[i]); }
        else
#pragma unroll
            for (uint32_t j = 0; j < VN; j++) r[i][j] = g[i][j] = 0.0f;
    }
    const float sp = softplusf_(__ldg(a.lam + c)), br = __ldg(a.bias + c), bi = __ldg(a.bias + a.C + c);
    pdl_wait();
    const float *u = a.u + (size_t)(c / a.bs) * a.bs;
    const float S0 = a.S[c], uc = a.u[c], y = a.y[c];
    float sr = 0.0f, si = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < 2u; i++) {
        const uint32_t k = i * STEP + lane * VN;
        if (k < a.bs) {
#pragma unroll
            for (uint32_t j = 0; j < VN; j += 4u) {
                float4 x = *reinterpret_cast<const float4 *>(u + k + j);
                if (a.round_a) x = round4(x);
                sr = fmaf(r[i][j], x.x, sr); sr = fmaf(r[i][j + 1], x.y, sr); sr = fmaf(r[i][j + 2], x.z, sr); sr = fmaf(r[i][j + 3], x.w, sr);
                si = fmaf(g[i][j], x.x, si); si = fmaf(g[i][j + 1], x.y, si); si = fmaf(g[i][j + 2], x.z, si); si = fmaf(g[i][j + 3], x.w, si);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { sr += __shfl_xor_sync(0xffffffffu, sr, o); si += __shfl_xor_sync(0xffffffffu, si, o); }
    if (lane) return;
    const float gr = sigmoidf_(sr + br), gi = sigmoidf_(si + bi), av = expf(-a.c_decay * gr * sp);
    const float S = av * S0 + sqrtf(1.0f - av * av) * (gi * uc);
    a.out[c] = S * y;
    a.S[c] = S;
}

// k_norm_shift for one token of at most 256 NK columns: the row in registers, one trip to memory and one sum (in the same order), weights before the wait.  What the
// combined kernel below shares with it: x[k], prev[k] are columns threadIdx.x + 256 k.
// A lone block passes its code once, and fetching it is what it waits for (some 8 cycles an instruction): so there is an instance for rows of up to 1024, 2048 and 4096, and a row's
// columns are one pointer with constant offsets.  Update and norm of 1024 columns with one instance of 4096: 669 instructions a warp and 5.4 us a link, now 3.5; 2048: 8.7 and 4.6.
template <int NK> struct NormOne { float mu[NK]; float g1, g2; bool on[NK]; };
template <int NK> __device__ __forceinline__ void norm_one_weights(const NormShiftArgs &a, NormOne<NK> &w) {
    const float *mu = a.mu + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++) { w.on[k] = threadIdx.x + k * kOneThreads < a.E; w.mu[k] = a.mu && w.on[k] ? load_now_f(mu + k * kOneThreads) : 0.0f; }
    w.g1 = load_now_f(a.g1); w.g2 = a.g2 ? load_now_f(a.g2) : 0.0f;
}
template <int NK> __device__ __forceinline__ void norm_one_row(const NormShiftArgs &a, const NormOne<NK> &w, const float (&x)[NK], const float (&prev)[NK], float *red) {
    float s = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++) s = fmaf(x[k], x[k], s);
    s = block_sum(s, red);
    const float rinv = 1.0f / sqrtf(s / (float)a.E + a.eps);
    float *hm = a.hm + threadIdx.x, *h2 = a.h2 + threadIdx.x, *state = a.state + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++)
        if (w.on[k]) {
            const float u = x[k] * rinv, n1 = u * w.g1;
            hm[k * kOneThreads] = a.mu ? n1 + (prev[k] - n1) * w.mu[k] : n1;
            if (a.h2) h2[k * kOneThreads] = u * w.g2;
            state[k * kOneThreads] = n1;
        }
}
template <int NK>
__global__ void __launch_bounds__(kOneThreads) k_norm_shift_one(const NormShiftArgs a) {
    pdl_launch_next();
    __shared__ float red[32];
    NormOne<NK> w;
    norm_one_weights(a, w);
    pdl_wait();
    float x[NK], p[NK];
    const float *xt = a.x + threadIdx.x, *st = a.state + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++) { x[k] = w.on[k] ? xt[k * kOneThreads] : 0.0f; p[k] = w.on[k] ? st[k * kOneThreads] : 0.0f; }
    norm_one_row(a, w, x, p, red);
}

// k_combine of one token and k_norm_shift_one of the run that follows, in one link: the updated row stays in the registers of the block that norms it
struct CombineNormArgs { CombineArgs c; NormShiftArgs n; };
template <int NK>
__global__ void __launch_bounds__(kOneThreads) k_combine_norm_one(const CombineNormArgs a) {
    pdl_launch_next();
    __shared__ float red[32];
    const CombineArgs &c = a.c;
    NormOne<NK> w;
    norm_one_weights(a.n, w);
    pdl_wait();
    uint32_t slot[2]; float wt[2];
    const bool routed = c.eo != nullptr;
#pragma unroll
    for (uint32_t j = 0; j < 2u; j++) { const bool in = routed && j < c.top; slot[j] = in ? c.slot[j] : 0u; wt[j] = in ? c.wt[j] : 0.0f; }
    float x[NK], p[NK], d[NK], sh[NK], f[NK];
    const bool shared = routed && c.shared;
    const float *xt = c.x + threadIdx.x, *st = a.n.state + threadIdx.x, *dt = c.d + threadIdx.x, *sht = c.shared + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++) {
        x[k] = p[k] = d[k] = sh[k] = f[k] = 0.0f;
        if (w.on[k]) { x[k] = xt[k * kOneThreads]; d[k] = dt[k * kOneThreads]; p[k] = st[k * kOneThreads]; if (shared) sh[k] = sht[k * kOneThreads]; }
    }
    if (routed) {          // the chosen experts' rows, two at a time (both rows' columns in flight), in their order
#pragma unroll 1
        for (uint32_t j = 0;;) {
            const float *e0 = c.eo + (size_t)slot[0] * c.E + threadIdx.x, *e1 = c.eo + (size_t)slot[1] * c.E + threadIdx.x;
            float v0[NK], v1[NK];
            const bool two = j + 1u < c.top;
#pragma unroll
            for (uint32_t k = 0; k < NK; k++) { v0[k] = w.on[k] ? e0[k * kOneThreads] : 0.0f; v1[k] = w.on[k] && two ? e1[k * kOneThreads] : 0.0f; }
#pragma unroll
            for (uint32_t k = 0; k < NK; k++) { f[k] = fmaf(wt[0], v0[k], f[k]); if (two) f[k] = fmaf(wt[1], v1[k], f[k]); }
            j += 2u;
            if (j >= c.top) break;
#pragma unroll
            for (uint32_t q = 0; q < 2u; q++) { const bool in = j + q < c.top; slot[q] = in ? c.slot[j + q] : 0u; wt[q] = in ? c.wt[j + q] : 0.0f; }
        }
    }
    float *xo = c.x + threadIdx.x, *kp = c.keep + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < NK; k++) {
        if (shared) f[k] += sh[k];
        x[k] += routed ? d[k] + f[k] : d[k];
        if (w.on[k]) { xo[k * kOneThreads] = x[k]; if (c.keep) kp[k * kOneThreads] = x[k]; }
    }
    norm_one_row(a.n, w, x, p, red);
}

// k_route_small for one token and at most 32 rows of the router: the same choice, weights and places (RouteArgs, route_pick), in registers.  A cluster of blocks
// shares the logits, with the router's rows in registers before the wait; the first block's first warp then holds an expert per lane, and everything it leaves is written
// once, by the lane that has it.  (k_route_small keeps the choice in memory and reads it back: 27 us of the chain of a step with eight routed layers; 6 here
// with 256 threads. 512 give each thread the share of a row that it has there, and so its sums: close calls between experts fall the same way.)
constexpr uint32_t kRouteOneThreads = 512;          // as k_route_small: the same shares of a row, the same sums
__global__ void __launch_bounds__(kRouteOneThreads) k_route_one(const RouteArgs a) {
    pdl_launch_next();
    cluster_arrive();                          // waited for before the first access to another block's shared memory
    __shared__ float z_s[32], zp[kRouteOneThreads / 32];
    constexpr uint32_t NW = kRouteOneThreads / 32, PRE = 8;
    const uint32_t NL = a.NE + a.extra, rank = blockIdx.x, nb = gridDim.x, nloc = (NL - rank + nb - 1u) / nb, ns = NW / nloc;      // this block's rows: rank, rank + nb, ...
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, per = ((a.E + ns - 1u) / ns + 3u) & ~3u;
    const uint32_t k0 = min(a.E, warp % ns * per), k1 = warp < nloc * ns ? min(a.E, k0 + per) : k0;
    const float *w = a.router + (size_t)(rank + min(warp / ns, nloc - 1u) * nb) * a.E;
    uint4 wv[PRE];
#pragma unroll
    for (uint32_t i = 0; i < PRE; i++) { const uint32_t k = k0 + i * 128u + lane * 4u; wv[i] = make_uint4(0, 0, 0, 0); if (k < k1) wv[i] = load_now(w + k); }
    pdl_wait();
    float acc = 0.0f;
    float4 h[PRE];
#pragma unroll
    for (uint32_t i = 0; i < PRE; i++) { const uint32_t k = k0 + i * 128u + lane * 4u; h[i] = make_float4(0, 0, 0, 0); if (k < k1) h[i] = *reinterpret_cast<const float4 *>(a.h + k); }
#pragma unroll
    for (uint32_t i = 0; i < PRE; i++)
        acc = fmaf(h[i].w, __uint_as_float(wv[i].w), fmaf(h[i].z, __uint_as_float(wv[i].z), fmaf(h[i].y, __uint_as_float(wv[i].y), fmaf(h[i].x, __uint_as_float(wv[i].x), acc))));
    for (uint32_t k = k0 + PRE * 128u + lane * 4u; k < k1; k += 128u) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(w + k)), x = *reinterpret_cast<const float4 *>(a.h + k);
        acc = fmaf(x.w, v.w, fmaf(x.z, v.z, fmaf(x.y, v.y, fmaf(x.x, v.x, acc))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) zp[warp] = acc;
    __syncthreads();
    cluster_wait();                            // every block of the cluster runs
    if (tid < nloc) {
        const uint32_t e = rank + tid * nb;
        float v = 0.0f;
        for (uint32_t sl = 0; sl < ns; sl++) v += zp[tid * ns + sl];
        st_cluster(z_s + e, 0u, a.mode == 3u && e < a.NE ? sigmoidf_(v) : v);
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (rank || warp) return;
    const bool expert = lane < a.NE;
    float z = lane < NL ? z_s[lane] : -INFINITY;
    if (lane >= a.NE && lane < NL) a.extra_out[lane - a.NE] = z;
    // the largest of `v` over the lanes below n (ties: the lower lane).  A score that is no number compares with nothing, so the lanes may end with different answers:
    // the first lane's counts, as in route_pick
    const bool odd = __any_sync(0xffffffffu, z != z);
    auto argmax = [&](float v, uint32_t n, float *value) {
        float best = lane < n ? v : -INFINITY; uint32_t bi = lane < n ? lane : 0xffffffffu;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o); const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (oi != 0xffffffffu && (bi == 0xffffffffu || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
        }
        if (odd) { best = __shfl_sync(0xffffffffu, best, 0); bi = __shfl_sync(0xffffffffu, bi, 0); }
        *value = best;
        return bi;
    };
    float zmax = expert ? z : -INFINITY, zden = 0.0f;
    if (a.mode == 2u) {                        // softmax over ALL experts
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
        zden = expert ? expf(z - zmax) : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) zden += __shfl_xor_sync(0xffffffffu, zden, o);
    }
    if (a.mode == 3u && a.keep < a.groups) {   // lane g: group g's score; then the experts of the groups that are not kept leave the choice
        const uint32_t size = a.NE / a.groups, g0 = min(lane, a.groups - 1u) * size;
        float b1 = -INFINITY, b2 = -INFINITY, v;
        for (uint32_t i = 0; i < size; i++) { const float x = __shfl_sync(0xffffffffu, z, g0 + i); b2 = fmaxf(b2, fminf(b1, x)); b1 = fmaxf(b1, x); }
        float zg = size > 1u ? b1 + b2 : b1;
        for (uint32_t j = 0; j < a.keep; j++) {
            const uint32_t g = argmax(zg, a.groups, &v);
            if (lane == g) zg = -INFINITY;
        }
        // a kept group's score is -infinity by now (one that was so from the start stays in the choice as well)
        const uint32_t open = __ballot_sync(0xffffffffu, lane < a.groups && zg == -INFINITY);
        if (expert && !(open >> (lane / size) & 1u)) z = -INFINITY;
    }
    uint32_t mine = 0xffffffffu;               // lane j: choice j and its weight
    float wt = 0.0f;
    for (uint32_t j = 0; j < a.top; j++) {
        float best;
        const uint32_t bi = argmax(z, a.NE, &best);
        if (lane == j) { mine = bi; wt = best; }
        if (lane == bi) z = -INFINITY;
    }
    const bool chose = lane < a.top;
    if (a.mode == 1u) wt = sigmoidf_(wt);
    else if (a.mode == 3u) wt *= a.wscale;
    else {
        const float first = __shfl_sync(0xffffffffu, wt, 0);
        wt = a.mode == 2u ? expf(wt - zmax) / zden : expf(wt - first);
        float s = 0.0f;
        for (uint32_t j = 0; j < a.top; j++) s += __shfl_sync(0xffffffffu, wt, j);
        wt /= a.mode == 2u ? s + 1e-20f : s;
    }
    // rows sorted by expert; choices of the same expert (-infinities only) follow in their order
    uint32_t before = 0, place = 0, below = 0, all = 0;
    bool first_of = chose;
    for (uint32_t j = 0; j < a.top; j++) {
        const uint32_t other = __shfl_sync(0xffffffffu, mine, j);
        if (other < mine || (other == mine && j < lane)) before++;
        if (other == mine && j < lane) first_of = false;
        if (other < lane) below++;
        if (other < 32u) all++;
    }
    const uint32_t heads = __ballot_sync(0xffffffffu, first_of);
    for (uint32_t j = 0; j < a.top; j++) {
        const uint32_t other = __shfl_sync(0xffffffffu, mine, j);
        if ((heads >> j & 1u) && other < mine) place++;
    }
    if (lane <= a.NE) a.off[lane] = below;     // rows of experts below
    if (a.NE == 32u && lane == 0) a.off[32] = all;
    if (chose) {
        a.idx[lane] = mine; a.wt[lane] = wt; a.slot[lane] = before; a.rows[before] = 0u;
        if (a.wrow) a.wrow[before] = wt;
        if (a.act && first_of) a.act[place] = mine;
        if (a.act && lane >= (uint32_t)__popc(heads)) a.act[lane] = 0xffffffffu;
    }
}

}  // namespace lm
}  // namespace nb
