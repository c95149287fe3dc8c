// stream.cuh -- the grid-wide persistent decode kernel (fast mode, one GPU): every SM keeps HBM streaming across
// phase, layer and token boundaries, and no phase boundary costs a fence or a barrier.
//
// One CTA per SM (cooperative launch).  Warp 15 of every CTA is a PRODUCER: it walks the static per-token schedule
//   for l in layers: QKV tiles | K/V tiles of this CTA's attention item | O tiles | W1|W3 tiles | W2 tiles ; classifier tiles
// and issues cp.async.bulk (TMA bulk copies, mbarrier complete_tx) into a shared-memory ring, as far ahead as the ring
// allows -- it never waits for a phase to end.  Weights come from a per-CTA, tile-ordered copy of the model (built once
// at load: a tile = [rows x (row bytes + 16)] [rows x aux] in exactly the order the CTA consumes it, so a tile is ONE
// bulk copy); K/V tiles come straight from the head-major KV cache.
//
// Activations between phases (x, q/k/v of the position, attention output, SwiGLU output) travel through small
// L2-resident vectors of 64-bit words {fp32 value, 32-bit epoch}: a producing warp publishes a finished element with
// ONE 8-byte store, a consuming CTA polls the words it needs until they carry the epoch of the exchange it is waiting
// for.  Value and epoch arrive together (single-copy atomic), so there is no fence, no counter and no grid barrier on
// the per-phase path (measured on B200: release fence ~1.1-1.7 k cycles, counter barrier ~1.6 k, against ~0.3-0.6 k
// from one word's store to its poll; a whole exchange, which is over when the last of 148 CTAs has published and a CTA has read all of a vector, takes 1.5 to 2 k).  Vectors that every CTA reads are written to kStRep replicas (different L2 slices;
// one hot copy read by 148 SMs at once costs ~600 cycles of slice bandwidth).
//   Why a word is never overwritten before its readers are done: a CTA reads an entire vector before it produces
//   anything of the next exchange, so "all of exchange k has arrived" implies every producer of exchange k has finished
//   reading exchange k-1; the writer of a later exchange into the same buffer has (transitively) seen all of k.
// One true grid barrier per token (release/acquire, at the classifier) orders the plain stores -- KV-cache rows, logits,
// ids, repetition-penalty flags -- against the next token's reads (TMA reads of the cache included).
//
// What bounds it at batch 1 is a chain: 5 exchanges a layer, and between two of them what every SM does with what arrived (norm and quantise, barrier, row dots,
// epilogue; attention in the CTAs that have an item).  A phase issues little work over 15 warps (4 a scheduler), so its time goes with the number of dependent
// steps and of instructions that every warp issues, not with bytes: no per-lane trip counts, one epilogue per block of rows, polls that ask for everything again instead of one
// word after the other, little state kept across phases.  Attention item without barriers between scores, softmax and values; one copy of each loop (197 KB of code before,
// 110 now).  Measured per token in the device loop, before -> now: Nano-168M Q80 at 16..40 positions 603 -> 366 us, Qwen3-0.6B Q80 at 260 961 -> 591, two layers of
// Qwen3-4B's width at 1500 143 -> 107, four of Nano's in F32 117 -> 88.
//
// Arithmetic (fast mode only; the bit-exact mode never runs this kernel): exact integer group dots; the fp32 combine of a
// quantised row (infer.c:668-674, tensor.c:425-430) as one partial per lane + a warp tree; tree reductions for rmsnorm / attention, expf and the division by sqrt(head_dim) as
// the reference.  Reference: llm_forward infer/infer.c:971-1018, transformer_block_forward :713-966.
#pragma once
#include "kernels.cuh"
#include "stream_args.h"

namespace nb {

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void *dst_smem, const void *src_gmem, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst_smem)), "l"(src_gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// A spin that cannot hang the GPU: after ~2 s the kernel records a code and traps (the host sees a launch failure).
static __device__ __noinline__ void st_give_up(uint32_t *err, uint32_t code) {
    if (err) *err = code;
    __threadfence_system();
    __trap();
}
// A polling warp must not monopolise the SM's MIO pipe (mbarrier, shared-memory and shuffle instructions share it): measured with
// the producer busy-polling a full ring, a 5-step warp shuffle reduction in a consumer warp took ~1000 cycles instead of ~150.
// `sleep_ns` > 0: back off between polls (the producer runs ahead of the consumers and is never latency-critical).
static __device__ __noinline__ void mbar_wait_slow(uint64_t *bar, uint32_t parity, uint32_t *err, uint32_t code, uint32_t sleep_ns) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (sleep_ns) __nanosleep(sleep_ns);
        if (clock64() - t0 > 4000000000ll) st_give_up(err, code);
    }
}
__device__ __forceinline__ void mbar_wait(uint64_t *bar, uint32_t parity, uint32_t *err, uint32_t code, uint32_t sleep_ns = 20) {
    if (!mbar_try_wait(bar, parity)) mbar_wait_slow(bar, parity, err, code, sleep_ns);
}
// barrier among the 15 consumer warps only (the producer warp never takes part)
__device__ __forceinline__ void cbar() { asm volatile("bar.sync 1, %0;" ::"n"(kConsThreads) : "memory"); }

// ---------------------------------------------------------------- exchange words {value, epoch}
__device__ __forceinline__ void xw_ld2(const unsigned long long *p, unsigned long long &a, unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long xw_ld1(const unsigned long long *p) {
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return a;
}
__device__ __forceinline__ void xw_st(unsigned long long *p, float v, uint32_t epoch) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)epoch << 32) | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ bool xw_ok(unsigned long long w, uint32_t need) { return (uint32_t)(w >> 32) == need; }
__device__ __forceinline__ float xw_val(unsigned long long w) { return __uint_as_float((uint32_t)w); }
// now and then inside a polling loop: start the clock, or give up after ~2 s
static __device__ __noinline__ long long st_still_waiting(long long t0, uint32_t *err, uint32_t code) {
    const long long now = clock64();
    if (t0 && now - t0 > 4000000000ll) st_give_up(err, code);
    return t0 ? t0 : now;
}
// 4 consecutive words (32-byte aligned) -> float4 once all of them carry `need`
static __device__ __noinline__ float4 xw_poll4_slow(const unsigned long long *p, uint32_t need, uint32_t *err) {
    unsigned long long a, b, c, d;
    long long t0 = 0;
    for (uint32_t it = 1;; it++) {
        xw_ld2(p, a, b); xw_ld2(p + 2, c, d);
        if (xw_ok(a, need) && xw_ok(b, need) && xw_ok(c, need) && xw_ok(d, need)) break;
        if ((it & 255u) == 0) {                      // the clock is read rarely: the loop stays a pair of loads and four compares
            if (t0 == 0) t0 = clock64();
            else if (clock64() - t0 > 4000000000ll) st_give_up(err, 0x50u);
        }
    }
    return make_float4(xw_val(a), xw_val(b), xw_val(c), xw_val(d));
}
__device__ __forceinline__ float4 xw_poll4(const unsigned long long *p, uint32_t need, uint32_t *err) {
    unsigned long long a, b, c, d;
    xw_ld2(p, a, b); xw_ld2(p + 2, c, d);
    if (xw_ok(a, need) && xw_ok(b, need) && xw_ok(c, need) && xw_ok(d, need)) return make_float4(xw_val(a), xw_val(b), xw_val(c), xw_val(d));
    return xw_poll4_slow(p, need, err);
}
// ---------------------------------------------------------------- schedule helpers shared by producer and consumers
// split of the attention range over CTAs: as few (kv head, split) items as keep an item under ~chunk_target rows
__device__ __forceinline__ void st_attn_plan(uint32_t range, uint32_t nsplit_max, uint32_t chunk_target, uint32_t &nsplit, uint32_t &chunk) {
    uint32_t ns = (range + chunk_target - 1) / chunk_target;
    if (ns < 1) ns = 1;
    if (ns > nsplit_max) ns = nsplit_max;
    uint32_t c = (range + ns - 1) / ns;
    c = (c + 7u) & ~7u;
    chunk = c;
    nsplit = (range + c - 1) / c;
}

struct StPlan { uint32_t nsplit, grp, sp, t0, t1; };          // this CTA's attention item of the token (grp >= groups: none)
struct StSmem { float red[2][16]; float best_v[kConsWarps]; uint32_t best_i[kConsWarps]; DevState st; uint32_t target, ti, tj; StPlan plan; };

struct StRing {
    uint64_t *full, *empty;
    volatile uint32_t *tile_id;   // [nstages] running index of the tile that owns the stage (written by the producer before the copy).
                                  // Warp-owned tiles are consumed out of step, and mbarrier parity is only unambiguous one phase
                                  // apart: a consumer first waits for ITS tile to own the stage, then for the bytes.
    unsigned char *buf;
    uint32_t nstages, stage_bytes;
};
__device__ __forceinline__ void mbar_arrive_n(uint64_t *bar, uint32_t n) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(n) : "memory");
}
struct StCursor { uint32_t s, par; };     // stage and parity of the next tile (producer: empty parity; consumer: full parity)
__device__ __forceinline__ void st_advance(StCursor &c, uint32_t nstages) { if (++c.s == nstages) { c.s = 0; c.par ^= 1u; } }
__device__ __forceinline__ void st_skip(StCursor &c, uint32_t n, uint32_t nstages) { c.s += n; while (c.s >= nstages) { c.s -= nstages; c.par ^= 1u; } }
// What a consumer needs of a phase kind, gathered once per launch in shared memory: two 16-byte loads at a phase's start.  (Kept in registers across the
// layer, these spilled, and one reload of a spilled register from local memory takes 1000 to 2700 cycles here: most of L1 is shared memory, and the polls keep L2 busy.)
struct __align__(16) StPhase {
    uint32_t n, row_stride, aux_stride, tile_rows;
    uint32_t rows, tiles, row0, mode;         // the rows and tiles this CTA owns; mode: owned | rb << 8 | tb << 16, shared tiles: rb = rows of a warp's pass, tb = blocks of rb rows in a full tile (mod 15)
    const unsigned long long *src; const float *gain;      // the replica this CTA reads (null gain: no norm before this product)
    uint32_t need, out, epi; float rn;        // epochs read and published, counted from the layer's first; rn = 1 / n
};

// ---------------------------------------------------------------- producer (warp 15, lane 0)
__device__ __forceinline__ void st_issue_kind(const StreamArgs &g, const StRing &r, StCursor &c, uint32_t &issued, const StKind &k, const uint8_t *base, uint32_t rows) {
    const uint8_t *src = base + k.off;
    for (uint32_t done = 0; done < rows; done += k.tile_rows) {
        const uint32_t tr = min(k.tile_rows, rows - done);
        const uint32_t bytes = (tr * (k.row_stride + k.aux_stride) + 15u) & ~15u;
        mbar_wait(&r.empty[c.s], c.par, g.err, 0x10u, 200);
        r.tile_id[c.s] = issued++;
        mbar_expect_tx(&r.full[c.s], bytes);
        bulk_g2s(r.buf + (size_t)c.s * r.stage_bytes, src, bytes, &r.full[c.s]);
        st_advance(c, r.nstages);
        src += k.tile_stride;
    }
}

static __device__ void st_producer(const StreamArgs &g, const StRing &r, const StPhase *own, uint32_t cta, volatile uint32_t *progress,
                                   uint32_t pos0, uint32_t causal, uint32_t advance) {
    const Dims &d = g.d;
    StCursor c{0u, 1u};                       // parity 1 passes at once on a stage's first use
    uint32_t issued = 0;                      // running tile index
    const uint8_t *base = g.stream + (uint64_t)cta * g.cta_stride;
    const size_t kvl = (size_t)d.KV * d.max_seq * d.hd;
    for (uint32_t step = 0; step < g.n_steps; step++) {
        const uint32_t pos = pos0 + (advance ? step : 0u);
        const uint32_t range = causal ? pos + 1u : d.max_seq;
        uint32_t nsplit, chunk;
        st_attn_plan(range, g.nsplit_max, g.chunk_target, nsplit, chunk);
        for (uint32_t l = 0; l < d.L; l++) {
            const uint8_t *lb = base + (uint64_t)l * g.layer_stride;
            st_issue_kind(g, r, c, issued, g.kind[SK_QKV], lb, own[SK_QKV].rows);
            if (cta < g.groups * nsplit) {
                const uint32_t kvh = cta / nsplit / g.group_div, sp = cta % nsplit;
                const uint32_t t0 = min(range, sp * chunk), t1 = min(range, t0 + chunk);
                const float *kb = g.kc + l * kvl + (size_t)kvh * d.max_seq * d.hd;
                const float *vb = g.vc + l * kvl + (size_t)kvh * d.max_seq * d.hd;
                for (uint32_t t = t0; t < t1; t += g.kv_tile_rows) {
                    const uint32_t tr = min(g.kv_tile_rows, t1 - t), bytes = tr * d.hd * 4u;
                    // The previous token's row was written with plain stores during this launch: it may be fetched once this
                    // CTA's consumers have passed that token's grid barrier (older rows: at least one barrier or launch ago).
                    if (step > 0 && pos > 0 && pos - 1u >= t && pos - 1u < t + tr) {
                        if (*progress < step) {
                            const long long c0 = clock64();
                            while (*progress < step) { __nanosleep(200); if (clock64() - c0 > 4000000000ll) st_give_up(g.err, 0x11u); }
                        }
                        asm volatile("fence.proxy.async.global;" ::: "memory");     // generic-proxy stores of this launch -> async-proxy (TMA) read
                    }
                    mbar_wait(&r.empty[c.s], c.par, g.err, 0x12u, 200);
                    r.tile_id[c.s] = issued++;
                    mbar_expect_tx(&r.full[c.s], 2u * bytes);
                    unsigned char *dst = r.buf + (size_t)c.s * r.stage_bytes;
                    bulk_g2s(dst, kb + (size_t)t * d.hd, bytes, &r.full[c.s]);
                    bulk_g2s(dst + (size_t)g.kv_tile_rows * d.hd * 4u, vb + (size_t)t * d.hd, bytes, &r.full[c.s]);
                    st_advance(c, r.nstages);
                }
            }
            st_issue_kind(g, r, c, issued, g.kind[SK_O], lb, own[SK_O].rows);
            st_issue_kind(g, r, c, issued, g.kind[SK_W13], lb, own[SK_W13].rows);
            st_issue_kind(g, r, c, issued, g.kind[SK_W2], lb, own[SK_W2].rows);
        }
        st_issue_kind(g, r, c, issued, g.kind[SK_CLS], base + g.cls_off, own[SK_CLS].rows);
    }
}

// ---------------------------------------------------------------- activation prologue (consumer threads)
// Source vector (exchange words of epoch `need`, or the embedding row in shared memory) -> (rmsnorm) -> activation
// operand of the matvec in shared memory:
//   Q80 (tensor.c:21-46): one quantisation group per 16 or 32 lanes, 4 elements per lane; F32: floats;
//   Q4K (tensor.c:144-242): one 256-element block per warp, 8 elements per lane.
// act layouts as in kernels.cuh (act_region_bytes).
template <int QUANT, int LPG>
__device__ __forceinline__ void st_prep(const StreamArgs &g, const unsigned long long *xsrc, const float *ssrc, uint32_t need, const float *__restrict__ gain,
                                        uint32_t n, float rn, unsigned char *act, float *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto sq = [](float4 v, float ss) -> float { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss)))); };
    auto nrm = [&](float4 v, float4 gn, float inv) -> float4 {      // infer.c:611: weight * (ss * x)
        return make_float4(__fmul_rn(gn.x, __fmul_rn(inv, v.x)), __fmul_rn(gn.y, __fmul_rn(inv, v.y)),
                           __fmul_rn(gn.z, __fmul_rn(inv, v.z)), __fmul_rn(gn.w, __fmul_rn(inv, v.w)));
    };
    auto inverse = [&](float ss) -> float {                         // infer.c:601-609, tree sum in a fixed order
        ss = warp_sum(ss);
        if (lane == 0) red[warp] = ss;
        cbar();
        const float4 *r4 = reinterpret_cast<const float4 *>(red);   // red[15] stays 0
        const float4 a = r4[0], b = r4[1], c = r4[2], e = r4[3];
        const float tot = (((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w))) + (((c.x + c.y) + (c.z + c.w)) + ((e.x + e.y) + (e.z + e.w)));
        // tot / n, rounded: the product by the rounded reciprocal with its remainder added back (Markstein's final step of a quotient, IBM J. Res. Dev. 34, 1990).  An
        // infinite sum has no remainder (inf - inf): it stays, and the row norms to zeros as on every other path
        const float q = tot * rn, mean = tot < INFINITY ? fmaf(fmaf(-q, (float)n, tot), rn, q) : tot;
        return __frcp_rn(__fsqrt_rn(__fadd_rn(mean, 1e-5f)));
    };
    if constexpr (QUANT == 0x42) {
        uint32_t *xe = reinterpret_cast<uint32_t *>(act);
        uint32_t *xo = reinterpret_cast<uint32_t *>(act + n / 2);
        float4 *gp = reinterpret_cast<float4 *>(act + n);
        const uint32_t NB = n / 256u;
        float4 v[kStKmaxQ4K][2];
        float ss = 0.0f;
#pragma unroll
        for (int j = 0; j < kStKmaxQ4K; j++) {
            const uint32_t b = warp + kConsWarps * j, base = b * 256u + lane * 8u;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                v[j][h] = make_float4(0, 0, 0, 0);
                if (b < NB) {
                    v[j][h] = ssrc ? *reinterpret_cast<const float4 *>(ssrc + base + 4 * h) : xw_poll4(xsrc + base + 4 * h, need, g.err);
                    ss = sq(v[j][h], ss);
                }
            }
        }
        float inv = 1.0f;
        if (gain) inv = inverse(ss);
#pragma unroll
        for (int j = 0; j < kStKmaxQ4K; j++) {
            const uint32_t b = warp + kConsWarps * j;
            if (b < NB) {                                            // warp-uniform
                float4 a0 = v[j][0], a1 = v[j][1];
                if (gain) {
                    const float4 *gp4 = reinterpret_cast<const float4 *>(gain + b * 256u + lane * 8u);
                    a0 = nrm(a0, __ldg(gp4), inv); a1 = nrm(a1, __ldg(gp4 + 1), inv);
                }
                const float vv[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                uint32_t c[8]; int csum, s6, b6; float sc, sbias;
                q4k_quantize_block(vv, c, csum, sc, sbias, s6, b6);
                xe[b * 32 + lane] = c[0] | (c[2] << 8) | (c[4] << 16) | (c[6] << 24);
                xo[b * 32 + lane] = c[1] | (c[3] << 8) | (c[5] << 16) | (c[7] << 24);
                if ((lane & 3) == 0) gp[b * 8 + (lane >> 2)] = make_float4(__fmul_rn((float)s6, sc), __fmul_rn((float)b6, sbias), (float)csum, 0.0f);
            }
        }
    } else {
        constexpr uint32_t gs = (QUANT == 0x80) ? LPG * 16u : 128u;      // Q80: elements of a group; F32: no grouping
        constexpr uint32_t LG = gs / 4u;                                 // lanes per group
        static_assert(LG == 16 || LG == 32, "stream kernel: Q80 group size 64 or 128");
        auto put = [&](float4 v, uint32_t i, bool on) {
            if constexpr (QUANT == 0x00) {
                if (on) *reinterpret_cast<float4 *>(act + (size_t)i * 4u) = v;
            } else {
                // tensor.c:21-46.  amax over the group with one REDUX (the values are non-negative: uint order == float order);
                // the exact scale amax/127 is off the codes' critical path; codes come from q = v * (127/amax) rounded by adding 1.5 * 2^23 (the integer is
                // then in the low bits), and any q within 1e-4 of a .5 boundary goes through the exact division + round().  (q and the quotient by sc are at most 4.2e-7 |q| apart:
                // two ulp of the approximate division, half an ulp each for the product, for sc and for the exact division.  A window of 1e-3 sent a warp's 128 values
                // there one time in four, so that of the warps of a row one nearly always went.)
                float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
                const uint32_t gmask = (LG == 32u) ? 0xffffffffu : ((lane & 16) ? 0xffff0000u : 0xffffu);
                amax = __uint_as_float(__reduce_max_sync(gmask, __float_as_uint(amax)));
                const float sc = __fdiv_rn(amax, 127.0f), rinv = __fdividef(127.0f, amax);
                const float q0 = v.x * rinv, q1 = v.y * rinv, q2 = v.z * rinv, q3 = v.w * rinv, magic = 12582912.0f;
                const float r0 = q0 + magic, r1 = q1 + magic, r2 = q2 + magic, r3 = q3 + magic;
                uint32_t c0 = __float_as_uint(r0), c1 = __float_as_uint(r1), c2 = __float_as_uint(r2), c3 = __float_as_uint(r3);
                const float off = fmaxf(fmaxf(fabsf(q0 - (r0 - magic)), fabsf(q1 - (r1 - magic))), fmaxf(fabsf(q2 - (r2 - magic)), fabsf(q3 - (r3 - magic))));
                if (sc == 0.0f) c0 = c1 = c2 = c3 = 0u;
                else if (off > 0.4999f) { c0 = q80_code_slow(v.x, sc); c1 = q80_code_slow(v.y, sc); c2 = q80_code_slow(v.z, sc); c3 = q80_code_slow(v.w, sc); }
                if (on) {
                    *reinterpret_cast<uint32_t *>(act + i) = __byte_perm(__byte_perm(c0, c1, 0x0040), __byte_perm(c2, c3, 0x0040), 0x5410);
                    if ((lane & (LG - 1u)) == 0) reinterpret_cast<float *>(act + ((n + 15u) & ~15u))[i / gs] = sc;
                }
            }
        };
        // Two slots of 128 elements per warp and turn: all their loads are in flight before the first epoch is looked at.  With a gain the
        // source is walked twice (sum of squares, then the operand); one turn (n <= 3840) keeps it in registers, longer ones read it again.  One copy of the
        // loop serves both walks and a third of the slots that the longest row needs: the kernel's instructions do not fit the caches near the SM, and what is
        // unrolled but skipped is fetched all the same (six slots unrolled: 197 KB of code, now about half).
        constexpr uint32_t turn = 2u * kConsWarps * 128u;
        float ss = 0.0f, inv = 1.0f;
        float4 v0 = make_float4(0, 0, 0, 0), v1 = v0, g0 = v0, g1 = v0;
#pragma unroll 1
        for (uint32_t walk = gain ? 0u : 1u; walk < 2u; walk++) {
#pragma unroll 1
            for (uint32_t s = warp * 128u; s < n; s += turn) {
                const uint32_t i0 = s + lane * 4u, i1 = i0 + kConsWarps * 128u;
                const bool on0 = i0 < n, on1 = i1 < n;
                if (walk == 0u || !gain || n > turn) {
                    if (gain) {
                        if (on0) g0 = __ldg(reinterpret_cast<const float4 *>(gain + i0));
                        if (on1) g1 = __ldg(reinterpret_cast<const float4 *>(gain + i1));
                    }
                    if (ssrc) {
                        v0 = v1 = make_float4(0, 0, 0, 0);
                        if (on0) v0 = *reinterpret_cast<const float4 *>(ssrc + i0);
                        if (on1) v1 = *reinterpret_cast<const float4 *>(ssrc + i1);
                    } else {
                        // both slots are asked for again until both are there: one after the other, the second would cost another trip to L2
                        long long t0 = 0;
#pragma unroll 1
                        for (uint32_t it = 1;; it++) {
                            unsigned long long w0, w1, w2, w3, z0, z1, z2, z3;
                            w0 = w1 = w2 = w3 = z0 = z1 = z2 = z3 = (unsigned long long)need << 32;
                            if (on0) { xw_ld2(xsrc + i0, w0, w1); xw_ld2(xsrc + i0 + 2, w2, w3); }
                            if (on1) { xw_ld2(xsrc + i1, z0, z1); xw_ld2(xsrc + i1 + 2, z2, z3); }
                            if (xw_ok(w0, need) && xw_ok(w1, need) && xw_ok(w2, need) && xw_ok(w3, need) && xw_ok(z0, need) && xw_ok(z1, need) && xw_ok(z2, need) && xw_ok(z3, need)) {
                                v0 = make_float4(xw_val(w0), xw_val(w1), xw_val(w2), xw_val(w3));
                                v1 = make_float4(xw_val(z0), xw_val(z1), xw_val(z2), xw_val(z3));
                                break;
                            }
                            if ((it & 255u) == 0) t0 = st_still_waiting(t0, g.err, 0x50u);          // the clock is read rarely: the loop stays loads and compares
                        }
                        __syncwarp();
                    }
                }
                if (walk == 0u) { ss = sq(v1, sq(v0, ss)); continue; }
                put(gain ? nrm(v0, g0, inv) : v0, i0, on0);
                if (s + kConsWarps * 128u < n) put(gain ? nrm(v1, g1, inv) : v1, i1, on1);         // warp-uniform
            }
            if (walk == 0u) inv = inverse(ss);
        }
    }
    cbar();
}

// ---------------------------------------------------------------- row dots on a shared-memory tile
// A warp takes RB rows, its lanes split the row in 16-byte chunks (512 bytes per step, conflict-free).  Nothing crosses lanes inside the loop: every lane
// keeps one fp32 partial per row, the steps are independent of each other.  (Fast mode: the fp32 summation order differs from matmul_quant
// infer.c:654-679; the bit-exact mode never runs this kernel.)  Row r of the block is rr + r; past the tile's last row the last one is read again.
template <int QUANT, int LPG, int RB>
__device__ __forceinline__ void st_partials(const unsigned char *tile, uint32_t row_stride, const unsigned char *aux, uint32_t aux_stride,
                                            uint32_t rr, uint32_t tr, uint32_t n, const unsigned char *act, float (&acc)[RB]) {
    const int lane = threadIdx.x & 31;
    const unsigned char *w[RB], *ws[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) {
        const uint32_t row = min(rr + (uint32_t)r, tr - 1u);
        w[r] = tile + row * row_stride; ws[r] = aux + row * aux_stride; acc[r] = 0.0f;
    }
    if constexpr (QUANT == 0x80) {
        constexpr uint32_t gs = LPG * 16;
        const float *xs = reinterpret_cast<const float *>(act + ((n + 15u) & ~15u));
        // Uniform trips of two steps; a lane past the row's end reads its last chunk with scale 0 (a trip count of each lane's own made three serial paths of a 768-wide row: 650
        // cycles a row).  The dot starts from the bits of 1.5 * 2^23, so that its float is the sum's low bits (|sum| <= 16 * 127 * 127 < 2^22).
        for (uint32_t k0 = 0; k0 < n; k0 += 1024u) {
#pragma unroll
            for (uint32_t h = 0; h < 2u; h++) {
                const uint32_t k = k0 + h * 512u + lane * 16u, kc = min(k, n - 16u), gi = kc / gs;
                const int4 xq = *reinterpret_cast<const int4 *>(act + kc);
                const float xsc = k < n ? xs[gi] : 0.0f;
#pragma unroll
                for (int r = 0; r < RB; r++) {
                    const int4 q = *reinterpret_cast<const int4 *>(w[r] + kc);
                    const float wsc = reinterpret_cast<const float *>(ws[r])[gi];
                    const int s0 = __dp4a(q.y, xq.y, __dp4a(q.x, xq.x, 0x4b400000)), s1 = __dp4a(q.w, xq.w, __dp4a(q.z, xq.z, 0));
                    acc[r] = fmaf(__int_as_float(s0 + s1) - 12582912.0f, wsc * xsc, acc[r]);
                }
            }
        }
    } else if constexpr (QUANT == 0x00) {          // matmul infer.c:637-651
        const float *x = reinterpret_cast<const float *>(act);
        for (uint32_t k0 = 0; k0 < n; k0 += 256u) {
#pragma unroll
            for (uint32_t h = 0; h < 2u; h++) {
                const uint32_t k = k0 + h * 128u + lane * 4u, kc = min(k, n - 4u);
                float4 xv = *reinterpret_cast<const float4 *>(x + kc);
                if (k >= n) xv = make_float4(0, 0, 0, 0);
#pragma unroll
                for (int r = 0; r < RB; r++) {
                    const float4 q = *reinterpret_cast<const float4 *>(w[r] + (size_t)kc * 4u);
                    acc[r] = fmaf(q.x, xv.x, acc[r]); acc[r] = fmaf(q.y, xv.y, acc[r]); acc[r] = fmaf(q.z, xv.z, acc[r]); acc[r] = fmaf(q.w, xv.w, acc[r]);
                }
            }
        }
    } else {
        // matmul_q4k / dot_two_blocks_q4k tensor.c:359-471: one lane = one 32-element group per step; side: 20-byte records
        const uint32_t *xe = reinterpret_cast<const uint32_t *>(act);
        const uint32_t *xo = reinterpret_cast<const uint32_t *>(act + n / 2);
        const float4 *gp = reinterpret_cast<const float4 *>(act + n);
        for (uint32_t k = lane * 16u; k < n / 2u; k += 512u) {
            const uint32_t grp = k / 16u, blk = grp >> 3, gi = grp & 7u, j = gi & 3u;
            const int4 e4 = *reinterpret_cast<const int4 *>(xe + grp * 4), o4 = *reinterpret_cast<const int4 *>(xo + grp * 4);
            const float4 q = gp[grp];
#pragma unroll
            for (int r = 0; r < RB; r++) {
                const int4 wq = *reinterpret_cast<const int4 *>(w[r] + k);
                const uint32_t *rec = reinterpret_cast<const uint32_t *>(ws[r] + (size_t)blk * 20u);
                const float ssc = __uint_as_float(rec[0]), sbi = __uint_as_float(rec[1]);
                const uint32_t bs = (rec[2] >> (8 * j)) & 0xff, bb = (rec[3] >> (8 * j)) & 0xff, bh = (rec[4] >> (8 * j)) & 0xff;
                const uint32_t s6 = (gi < 4) ? (bs & 0x3f) : ((((bs >> 6) << 4) | (bh & 0x0f)) & 0x3f);
                const uint32_t b6 = (gi < 4) ? (bb & 0x3f) : ((((bb >> 6) << 4) | (bh >> 4)) & 0x3f);
                const float sp = __fmul_rn((float)s6, ssc), bp = __fmul_rn((float)b6, sbi);
                const int wv[4] = {wq.x, wq.y, wq.z, wq.w}, ev[4] = {e4.x, e4.y, e4.z, e4.w}, ov[4] = {o4.x, o4.y, o4.z, o4.w};
                int spq = 0, spp = 0;
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int lo = wv[t] & 0x0f0f0f0f, hi = (wv[t] >> 4) & 0x0f0f0f0f;
                    spq = __dp4a(lo, ev[t], spq); spq = __dp4a(hi, ov[t], spq);
                    spp = __dp4a(lo, 0x01010101, spp); spp = __dp4a(hi, 0x01010101, spp);
                }
                float term = __fmul_rn(__fmul_rn(sp, q.x), (float)spq);                       // tensor.c:425-428, left to right
                term = __fsub_rn(term, __fmul_rn(__fmul_rn(sp, q.y), (float)spp));
                term = __fsub_rn(term, __fmul_rn(__fmul_rn(q.x, bp), q.z));
                term = __fadd_rn(term, __fmul_rn(__fmul_rn(32.0f, bp), q.y));
                acc[r] = __fadd_rn(acc[r], term);             // lane-local partial (fast mode: the order of the fp32 sum differs from tensor.c:425-471)
            }
        }
    }
}
// Row totals: lane l ends with the total of row rr + (l >> shift), the same number in all of that row's lanes, so that a row's epilogue and its stores into
// the replicas run once for the whole block (RB rows x 8 replicas = 8, 16 or 32 lanes).  The first steps trade rows for lanes: 6 shuffles for 4 rows, not 20.
template <int QUANT, int LPG, int RB>
__device__ __forceinline__ float st_rows(const unsigned char *tile, uint32_t row_stride, const unsigned char *aux, uint32_t aux_stride,
                                         uint32_t rr, uint32_t tr, uint32_t n, const unsigned char *act) {
    const int lane = threadIdx.x & 31;
    float acc[RB];
    st_partials<QUANT, LPG, RB>(tile, row_stride, aux, aux_stride, rr, tr, n, act, acc);
    float v;
    if constexpr (RB == 4) {
        const bool hi = lane & 16, od = lane & 8;
        const float k0 = hi ? acc[2] : acc[0], k1 = hi ? acc[3] : acc[1], s0 = hi ? acc[0] : acc[2], s1 = hi ? acc[1] : acc[3];
        const float a = k0 + __shfl_xor_sync(0xffffffffu, s0, 16), b = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
        v = od ? b : a;
        v += __shfl_xor_sync(0xffffffffu, od ? a : b, 8);
    } else if constexpr (RB == 2) {
        const bool hi = lane & 16;
        v = hi ? acc[1] : acc[0];
        v += __shfl_xor_sync(0xffffffffu, hi ? acc[0] : acc[1], 16);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
    } else {
        v = acc[0];
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// ---------------------------------------------------------------- one matvec phase: tiles from the ring -> epilogue
// The epilogue is selected at run time so that the kernel holds ONE copy of the row loops.
// Every finished element is published at once (st.relaxed {value, epoch}); nothing else marks the end of a phase.
// Two ways to share the tiles of a phase among the 15 consumer warps:
//   shared tiles (few rows per CTA: latency matters): every warp takes `rb` rows of every tile, the fewest that cover a tile in one pass;
//   owned tiles  (many rows per CTA: throughput matters): tile j belongs to warp j % 15, which walks its rows alone
//                while the other warps do the same on their tiles.
template <int QUANT, int LPG>
__device__ __forceinline__ void st_consume(const StreamArgs &g, const StRing &r, StCursor &c, uint32_t &tcount, const StPhase &ph, uint32_t layer,
                                           uint32_t epoch, const unsigned char *act, uint32_t pos, float *xown, StSmem &ms) {
    const Dims &d = g.d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4 pa = *reinterpret_cast<const uint4 *>(&ph), pb = *(reinterpret_cast<const uint4 *>(&ph) + 1);
    const uint32_t n = pa.x, row_stride = pa.y, aux_stride = pa.z, tile_rows = pa.w, rows = pb.x, nt = pb.y, row0 = pb.z, epi = ph.epi;
    const bool owned = pb.w & 1u;
    const uint32_t rb = owned ? (QUANT == 0x42 ? 2u : 4u) : (pb.w >> 8) & 255u, step = owned ? rb : rb * kConsWarps, tb = pb.w >> 16;
    float bestv = -FLT_MAX, kept = 0.0f; uint32_t besti = 0xffffffffu;
    const uint32_t jstep = owned ? (uint32_t)kConsWarps : 1u;
    uint32_t turn = (uint32_t)warp;                         // shared tiles: which block of rows of the tile is this warp's first
    StCursor cc = c;
    if (owned) st_skip(cc, (uint32_t)warp, r.nstages);
#pragma unroll 1
    for (uint32_t j = owned ? (uint32_t)warp : 0u; j < nt; j += jstep) {
        const uint32_t done = j * tile_rows, tr = min(tile_rows, rows - done);
        if (owned && r.tile_id[cc.s] != tcount + j) {
            const long long t0 = clock64();
            while (r.tile_id[cc.s] != tcount + j) { __nanosleep(20); if (clock64() - t0 > 4000000000ll) st_give_up(g.err, 0x28u); }
        }
        mbar_wait(&r.full[cc.s], cc.par, g.err, 0x20u + epi);
        const unsigned char *tile = r.buf + (size_t)cc.s * r.stage_bytes;
        const unsigned char *aux = tile + tr * row_stride;
#pragma unroll 1
        for (uint32_t rr = owned ? 0u : rb * turn; rr < tr; rr += step) {
            const uint32_t cnt = min(rb, tr - rr);
            uint32_t sh = 5u;                                   // lanes of a row: 2^sh
            float v;
            if (QUANT != 0x42 && cnt > 2u) { v = st_rows<QUANT, LPG, (QUANT == 0x42 ? 2 : 4)>(tile, row_stride, aux, aux_stride, rr, tr, n, act); sh = 3u; }
            else if (cnt == 2u) { v = st_rows<QUANT, LPG, 2>(tile, row_stride, aux, aux_stride, rr, tr, n, act); sh = 4u; }
            else v = st_rows<QUANT, LPG, 1>(tile, row_stride, aux, aux_stride, rr, tr, n, act);
            // ---- epilogue: lane = (row u of the block, replica) ----
            const uint32_t u = (uint32_t)lane >> sh, rep = lane & 7u, ri = done + rr + u, row = row0 + ri;
            const bool on = u < cnt && (lane & ((1u << sh) - 1u)) < (uint32_t)kStRep;
            if (epi == EPI_SWIGLU) {
                // rows (2i, 2i+1) = (w1 row i, w3 row i); infer.c:937-944
                const float v3 = __shfl_down_sync(0xffffffffu, v, 1u << (sh & 31u));
                if (on && !(u & 1u)) {
                    const float sg = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-v)));
                    xw_st(g.xv[2] + rep * g.rs[2] + (row >> 1), __fmul_rn(__fmul_rn(v, sg), v3), epoch);
                }
            } else if (epi == EPI_RESID) {
                float xn = 0.0f;
                if (on) { xn = __fadd_rn(xown[ri], v); xw_st(g.xv[0] + rep * g.rs[0] + row, xn, epoch); }      // infer.c:906, :963
                __syncwarp();
                if (on && rep == 0) xown[ri] = xn;
            } else if (epi == EPI_QKV) {
                if (on && rep == 0) {
                    xw_st(g.xq + row, v, epoch);
                    if (row >= d.q_dim + d.kv_dim) {                         // V rows also go to the cache for later positions
                        const uint32_t vc = row - d.q_dim - d.kv_dim, h = vc / d.hd, i = vc % d.hd;
                        g.vc[(size_t)layer * d.KV * d.max_seq * d.hd + ((size_t)h * d.max_seq + pos) * d.hd + i] = v;
                    }
                }
            } else {
                // classifier: up to 32 rows of an owned tile are gathered, lane by lane, so that they leave in one store (to the host as well, across PCIe, when a call returns logits)
                const uint32_t q = (uint32_t)lane - (owned ? rr & 31u : 0u);
                const float got = __shfl_sync(0xffffffffu, v, (q << (sh & 31u)) & 31u);
                if (q < cnt) kept = got;
                if (!owned || ((rr + step) & 31u) == 0u || rr + step >= tr) {
                    const uint32_t crow = row0 + done + (owned ? rr & ~31u : rr) + lane;
                    if ((uint32_t)lane < (owned ? (rr & 31u) + cnt : cnt)) {
                        // infer.c:1156-1167 penalty (division, any sign), then first-max argmax :1026-1037 (rows ascend per lane)
                        float w = kept;
                        const float pen = ms.st.penalty;
                        if (pen != 1.0f && __ldcg(g.seen + crow)) w = __fdiv_rn(w, pen);
                        g.logits[crow] = w;
                        if (g.logits_host) g.logits_host[crow] = w;
                        if (w > bestv) { bestv = w; besti = crow; }
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_n(&r.empty[cc.s], owned ? (uint32_t)kConsWarps : 1u);      // an owned tile has this one consumer
        if (!owned) { turn += kConsWarps - tb; if (turn >= (uint32_t)kConsWarps) turn -= kConsWarps; }      // long rows: few to a tile, the next tile's go to the next warps
        st_skip(cc, jstep, r.nstages);
    }
    st_skip(c, nt, r.nstages);
    tcount += nt;
    if (epi == EPI_CLS) {
#pragma unroll
        for (uint32_t o = 1u; o < 32u; o <<= 1) {                          // first max over the lanes of the warp
            const float ov = __shfl_xor_sync(0xffffffffu, bestv, o); const uint32_t oi = __shfl_xor_sync(0xffffffffu, besti, o);
            if (oi != 0xffffffffu && (besti == 0xffffffffu || ov > bestv || (ov == bestv && oi < besti))) { bestv = ov; besti = oi; }
        }
        if (lane == 0) { ms.best_v[warp] = bestv; ms.best_i[warp] = besti; }
    }
}

// ---------------------------------------------------------------- attention item (infer.c:814-879) on K/V tiles from the ring
// One CTA = one (group of KVM query heads of a key/value head, split).  The item's rows are processed in segments of up to kStSegTiles ring tiles that are resident at the same time.  A cache
// row belongs to LPR lanes of a warp, each with NC of its 16-byte chunks for all KVM query heads: a score is log2(LPR) shuffles, and the weighted value row stays
// in the lanes that have the weight, so there is no barrier and no shared memory between scores, softmax and values.  Every row slot keeps a running maximum, sum and
// accumulators of its own (KVM * NC = 4 or 8 float4).  LPR is the least that fits them: what bounds an item of this size is the instructions that its
// 15 warps issue (4 warps a scheduler), and those go with the number of passes.
// The slots are merged within the warp, the warps through shared memory, under the item's second and last barrier.
// q (and the position's k) are normalised + RoPE'd in registers (norm_rope_apply) by one warp each; the position's own K / V
// rows (this step's QKV outputs) are read from where those warps put them, not from the tile.
// A range held by one item is normalised and published at once; otherwise every item publishes its partial and the items of the kv head share the merge:
// a warp per 32 elements of a head, in split order.
template <int KVM, int HDC>
static __device__ void st_attention(const StreamArgs &g, const StRing &r, StCursor &c, uint32_t &tcount, uint32_t layer, uint32_t cta, uint32_t pos, const StPlan &plan,
                                    uint32_t e_in, uint32_t e_out, float *sm) {
    constexpr uint32_t LPR = KVM * HDC / 32 < HDC / 16 ? HDC / 16 : KVM * HDC / 32, NC = HDC / 4 / LPR, RP = 32 / LPR;          // lanes of a row, chunks of a lane, rows of a warp's pass
    const Dims &d = g.d;
    const uint32_t nsplit = plan.nsplit, grp = plan.grp, sp = plan.sp, t0 = plan.t0, t1 = plan.t1;
    if (grp >= g.groups) return;
    const uint32_t kvh = grp / g.group_div;
    const uint32_t hd = d.hd;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t kvr = g.kv_tile_rows, seg_max = (uint32_t)kStSegTiles * kvr;

    // shared-memory carve-up (floats)
    float *q_s = sm;                                   // [KVM][hd]   normalised + RoPE'd query heads
    float *krow = q_s + KVM * hd;                      // [hd] the position's k (post-RoPE), [hd] the position's v
    float *part_s = krow + 2 * hd;                     // [15][KVM][hd] the warps' weighted sums
    float *pm = part_s + kConsWarps * KVM * hd;        // [KVM][16] their maxima
    float *pl = pm + KVM * 16;                         // [KVM][16] their sums of weights

    // ---- this step's q / k / v: warp m < KVM prepares query head m, warp KVM the k row, warp KVM + 1 the v row ----
    if (warp < KVM + ((pos >= t0 && pos < t1) ? 2u : 0u)) {
        uint32_t lpr = 1; while (lpr * 4 < hd) lpr <<= 1;
        const uint32_t col = (lane & (lpr - 1u)) * 4;
        const bool colon = col < hd;
        const float *gains = warp < KVM ? g.qnorm : g.knorm;
        RopeTab rt; rt.c = rt.sn = make_float4(0, 0, 0, 0);
        float4 gn = make_float4(0, 0, 0, 0), v4 = gn;
        if (warp <= KVM) {
            rt = rope_tab_load(g.rope_cos + (size_t)pos * (hd / 2), g.rope_sin + (size_t)pos * (hd / 2), d, col, colon);
            if (d.arch == 3u && colon) gn = __ldg(reinterpret_cast<const float4 *>(gains + (size_t)layer * hd + col));
        }
        const uint32_t at = warp < KVM ? (grp * KVM + warp) * hd : d.q_dim + (warp == KVM ? 0u : d.kv_dim) + kvh * hd;
        if (colon) v4 = xw_poll4(g.xq + at + col, e_in, g.err);
        __syncwarp();
        if (warp <= KVM) v4 = norm_rope_apply(v4, gn, rt, d, lpr, col, colon);
        if (colon && lane < lpr) {
            *reinterpret_cast<float4 *>(q_s + warp * hd + col) = v4;               // krow follows q_s: row KVM is k, row KVM + 1 is v
            if (warp == KVM && grp == kvh * g.group_div)                           // K rows are cached post-RoPE, once
                *reinterpret_cast<float4 *>(g.kc + ((size_t)(layer * d.KV + kvh) * d.max_seq + pos) * hd + col) = v4;
        }
    }
    const uint32_t slot = lane / LPR, part = lane % LPR;
    const uint32_t rot = LPR == 4u ? (slot & 1u) : 0u;          // four lanes a row: neighbouring rows of a load read chunk groups of different banks
    uint32_t col[NC];
#pragma unroll
    for (uint32_t i = 0; i < NC; i++) col[i] = (part + LPR * ((i + rot) & (NC - 1u))) * 4u;
    float m_run[KVM], l_run[KVM]; float4 acc[KVM][NC];
#pragma unroll
    for (int m = 0; m < KVM; m++) {
        m_run[m] = -FLT_MAX; l_run[m] = 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < NC; i++) acc[m][i] = make_float4(0, 0, 0, 0);
    }
    const float dv = sqrtf((float)hd), rdv = 1.0f / dv;
    cbar();

#pragma unroll 1
    for (uint32_t s0 = t0; s0 < t1; s0 += seg_max) {
        const uint32_t rows_seg = min(seg_max, t1 - s0), nt = (rows_seg + kvr - 1u) / kvr;
        // stage of tile i of the segment (at most one turn of the ring away); lane i waits for tile i
        uint32_t my_s = c.s + lane, my_par = c.par;
        if (my_s >= r.nstages) { my_s -= r.nstages; my_par ^= 1u; }
        if (lane < nt) mbar_wait(&r.full[my_s], my_par, g.err, 0x30u);
        __syncwarp();
#pragma unroll 1
        for (uint32_t base = RP * warp; base < rows_seg; base += RP * kConsWarps) {          // warp-uniform
            const bool on = base + slot < rows_seg;
            const uint32_t idx = on ? base + slot : base;
            const uint32_t ti = __umulhi(idx, g.kv_tile_magic);
            uint32_t st = c.s + ti;
            if (st >= r.nstages) st -= r.nstages;
            const float *kr = reinterpret_cast<const float *>(r.buf + (size_t)st * r.stage_bytes) + (idx - ti * kvr) * hd, *vr = kr + kvr * hd;
            if (s0 + idx == pos) { kr = krow; vr = krow + hd; }
            float s[KVM];
#pragma unroll
            for (int m = 0; m < KVM; m++) s[m] = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < NC; i++)
                if (col[i] < hd) {
                    const float4 k4 = *reinterpret_cast<const float4 *>(kr + col[i]);
#pragma unroll
                    for (int m = 0; m < KVM; m++) {
                        const float4 q = *reinterpret_cast<const float4 *>(q_s + m * hd + col[i]);
                        s[m] = fmaf(k4.x, q.x, fmaf(k4.y, q.y, fmaf(k4.z, q.z, fmaf(k4.w, q.w, s[m]))));
                    }
                }
#pragma unroll
            for (uint32_t o = 1; o < LPR; o <<= 1)
#pragma unroll
                for (int m = 0; m < KVM; m++) s[m] += __shfl_xor_sync(0xffffffffu, s[m], o);
            bool up = false;
#pragma unroll
            for (int m = 0; m < KVM; m++) {          // infer.c:858: s / sqrt(head dim), as the product by the reciprocal with the remainder added back
                const float y = s[m] * rdv, e = fmaf(-y, dv, s[m]);
                s[m] = on ? (fabsf(y) < 3.0e38f ? fmaf(e, rdv, y) : y) : -INFINITY;
                up = up || s[m] > m_run[m];
            }
            if (__any_sync(0xffffffffu, up)) {       // some slot has a new maximum (the first rows, then rarely)
#pragma unroll
                for (int m = 0; m < KVM; m++) {
                    const float mn = fmaxf(m_run[m], s[m]), sc = expf(m_run[m] - mn);
                    m_run[m] = mn; l_run[m] *= sc;
#pragma unroll
                    for (uint32_t i = 0; i < NC; i++) { acc[m][i].x *= sc; acc[m][i].y *= sc; acc[m][i].z *= sc; acc[m][i].w *= sc; }
                }
            }
#pragma unroll
            for (int m = 0; m < KVM; m++) { s[m] = expf(s[m] - m_run[m]); l_run[m] += s[m]; }
#pragma unroll
            for (uint32_t i = 0; i < NC; i++)
                if (col[i] < hd) {
                    const float4 v4 = *reinterpret_cast<const float4 *>(vr + col[i]);
#pragma unroll
                    for (int m = 0; m < KVM; m++) {
                        acc[m][i].x = fmaf(s[m], v4.x, acc[m][i].x); acc[m][i].y = fmaf(s[m], v4.y, acc[m][i].y);
                        acc[m][i].z = fmaf(s[m], v4.z, acc[m][i].z); acc[m][i].w = fmaf(s[m], v4.w, acc[m][i].w);
                    }
                }
        }
        __syncwarp();
        if (lane < nt) mbar_arrive(&r.empty[my_s]);          // this warp is done with the segment's tiles
        st_skip(c, nt, r.nstages);
        tcount += nt;
    }
    // ---- the row slots of a warp (trading elements for lanes: the lane ends with KVM * HDC / 32 of them), then the warps that had rows ----
    const uint32_t nact = min((uint32_t)kConsWarps, (min(seg_max, t1 - t0) + RP - 1u) / RP);          // (t0 < t1: every split of the plan holds rows)
    if (warp < nact) {
        constexpr uint32_t NV = KVM * NC * 4;
        float f[NV];
#pragma unroll
        for (int m = 0; m < KVM; m++) {
            float mn = m_run[m];
#pragma unroll
            for (uint32_t o = LPR; o < 32; o <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            const float sc = expf(m_run[m] - mn);
            float l = l_run[m] * sc;
#pragma unroll
            for (uint32_t o = LPR; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0) { pm[m * 16 + warp] = mn; pl[m * 16 + warp] = l; }
#pragma unroll
            for (uint32_t i = 0; i < NC; i++) {
                const float4 e = acc[m][i], w = acc[m][(i + NC - 1u) & (NC - 1u)];          // rotated lanes hold chunk i one place earlier
                f[(m * NC + i) * 4] = sc * (rot ? w.x : e.x); f[(m * NC + i) * 4 + 1] = sc * (rot ? w.y : e.y);
                f[(m * NC + i) * 4 + 2] = sc * (rot ? w.z : e.z); f[(m * NC + i) * 4 + 3] = sc * (rot ? w.w : e.w);
            }
        }
        uint32_t f0 = 0;
#pragma unroll
        for (uint32_t o = 16, n = NV / 2; o >= LPR; o >>= 1, n >>= 1) {
            const bool hi = lane & o;
#pragma unroll
            for (uint32_t j = 0; j < n; j++) {
                const float keep = hi ? f[j + n] : f[j], give = hi ? f[j] : f[j + n];
                f[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
            f0 += hi ? n : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < NV / RP; j += 2) {
            const uint32_t e = f0 + j, at = (part + LPR * (e / 4u % NC)) * 4u + (e & 3u);
            if (at < hd) *reinterpret_cast<float2 *>(part_s + (warp * KVM + e / (NC * 4u)) * hd + at) = make_float2(f[j], f[j + 1]);
        }
    }
    cbar();
    const uint32_t pw = KVM * (hd + 2u);                               // words of one partial
    unsigned long long *part_x = g.xws + (size_t)grp * g.nsplit_max * pw;
    const uint32_t slabs = (hd + 31u) / 32u, units = KVM * slabs;
    auto publish = [&](uint32_t m, uint32_t i, float v) {
        unsigned long long *dst = g.xv[1] + (grp * KVM + m) * hd + i;
        const uint32_t rs = g.rs[1];
#pragma unroll
        for (uint32_t rep = 0; rep < (uint32_t)kStRep; rep++) xw_st(dst + rep * rs, v, e_out);
    };
#pragma unroll 1
    for (uint32_t u = warp; u < units; u += kConsWarps) {
        const uint32_t m = u / slabs, i = (u - m * slabs) * 32u + lane, src = lane & 15u;
        const float pmv = src < nact ? pm[m * 16 + src] : -FLT_MAX, plv = src < nact ? pl[m * 16 + src] : 0.0f;
        float M = pmv;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        const float w = src < nact ? expf(pmv - M) : 0.0f;
        float L = w * plv, o = 0.0f;
#pragma unroll
        for (int b = 1; b < 16; b <<= 1) L += __shfl_xor_sync(0xffffffffu, L, b);
        const float *ps = part_s + m * hd + i;
#pragma unroll 4
        for (uint32_t q = 0; q < nact; q++) {
            const float wq = __shfl_sync(0xffffffffu, w, q);
            if (i < hd) o = fmaf(wq, ps[q * KVM * hd], o);
        }
        if (nsplit == 1) { if (i < hd) publish(m, i, __fdiv_rn(o, L)); continue; }
        unsigned long long *dst = part_x + (size_t)sp * pw + m * (hd + 2u);
        if (i < hd) xw_st(dst + i, o, e_out);
        if (i == 0) { xw_st(dst + hd, M, e_out); xw_st(dst + hd + 1u, L, e_out); }
    }
    if (nsplit == 1) return;
    // ---- merge: 32 elements of a head per warp, dealt out over the items of the kv head ----
#pragma unroll 1
    for (uint32_t u = sp + nsplit * warp; u < units; u += nsplit * kConsWarps) {
        const uint32_t m = u / slabs, i = (u - m * slabs) * 32u + lane;
        const unsigned long long *src = part_x + m * (hd + 2u), *el = src + (i < hd ? i : 0u);
        // Eight splits' elements and (with the first eight) all statistics are asked for together, again until all are there: nothing is polled one by one.
        // nsplit_max <= 64: two splits' statistics per lane.
        const unsigned long long there = (unsigned long long)e_out << 32;
        unsigned long long w8[8], a0, a1, b0, b1;
        auto ask = [&](uint32_t s2, bool stats) {
            long long t0 = 0;
#pragma unroll 1
            for (uint32_t it = 1;; it++) {
                bool ok = true;
                if (stats) {
                    a0 = a1 = b0 = b1 = there;
                    if (lane < nsplit) xw_ld2(src + (size_t)lane * pw + hd, a0, a1);
                    if (lane + 32u < nsplit) xw_ld2(src + (size_t)(lane + 32u) * pw + hd, b0, b1);
                }
#pragma unroll
                for (uint32_t q = 0; q < 8u; q++) w8[q] = s2 + q < nsplit ? xw_ld1(el + (size_t)(s2 + q) * pw) : there;
#pragma unroll
                for (uint32_t q = 0; q < 8u; q++) ok = ok && xw_ok(w8[q], e_out);
                if (stats) ok = ok && xw_ok(a0, e_out) && xw_ok(a1, e_out) && xw_ok(b0, e_out) && xw_ok(b1, e_out);
                if (__all_sync(0xffffffffu, ok)) return;
                if ((it & 255u) == 0) t0 = st_still_waiting(t0, g.err, 0x51u);
            }
        };
        ask(0, true);
        const float m0 = lane < nsplit ? xw_val(a0) : -FLT_MAX, m1 = lane + 32u < nsplit ? xw_val(b0) : -FLT_MAX;
        const float M = warp_max(fmaxf(m0, m1));
        const float w0 = lane < nsplit ? expf(m0 - M) : 0.0f, w1 = lane + 32u < nsplit ? expf(m1 - M) : 0.0f;
        const float L = warp_sum(fmaf(lane < nsplit ? xw_val(a1) : 0.0f, w0, (lane + 32u < nsplit ? xw_val(b1) : 0.0f) * w1));
        float o = 0.0f;
#pragma unroll 1
        for (uint32_t s2 = 0; s2 < nsplit; s2 += 8u) {
            if (s2) ask(s2, false);
#pragma unroll
            for (uint32_t q = 0; q < 8u; q++) {
                const float wq = __shfl_sync(0xffffffffu, s2 < 32u ? w0 : w1, (s2 + q) & 31u);
                if (s2 + q < nsplit) o = fmaf(xw_val(w8[q]), wq, o);
            }
        }
        if (i < hd) publish(m, i, __fdiv_rn(o, L));
    }
}

// ---------------------------------------------------------------- grid barrier, once per token (consumer warps; the producer keeps streaming)
__device__ __forceinline__ void st_grid_barrier(const StreamArgs &g, unsigned int &target_smem, volatile uint32_t *progress, uint32_t ncta) {
    cbar();
    if (threadIdx.x == 0) {
        const unsigned int target = target_smem + ncta;
        target_smem = target;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(g.bar) : "memory");       // release: this CTA's plain stores of the token
        if ((int32_t)(ld_acquire_u32(g.bar) - target) < 0) {
            const long long t0 = clock64();
            while ((int32_t)(ld_acquire_u32(g.bar) - target) < 0) { if (clock64() - t0 > 4000000000ll) st_give_up(g.err, 0x40u); }
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");      // the token's plain K/V stores are TMA-read by later tokens
        *progress = *progress + 1u;
    }
    cbar();
}

// ---------------------------------------------------------------- the kernel
template <int QUANT, int LPG, int KVM, int HDC>
__global__ void __launch_bounds__(kThreads, 1) k_decode_stream(const __grid_constant__ StreamArgs gparam) {
    extern __shared__ __align__(128) unsigned char ssm[];
    // The argument block is read from shared memory: kernel parameters live in the constant bank, whose cache shares the
    // L1.5 with the instruction stream of this large kernel -- a parameter touched once per phase misses it every time.
    __shared__ __align__(16) StreamArgs sg;
    for (uint32_t i = threadIdx.x; i < sizeof(StreamArgs) / 4; i += kThreads) reinterpret_cast<uint32_t *>(&sg)[i] = reinterpret_cast<const uint32_t *>(&gparam)[i];
    __syncthreads();
    const StreamArgs &g = sg;
    __shared__ uint64_t full_bar[kStMaxStages], empty_bar[kStMaxStages];
    __shared__ volatile uint32_t stage_tile[kStMaxStages];
    __shared__ __align__(16) StSmem ms;
    __shared__ StPhase phase[5];
    __shared__ float xown[kStOwnMax];
    __shared__ volatile uint32_t s_progress;
    const Dims &d = g.d;
    const uint32_t cta = blockIdx.x, ncta = gridDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    const StRing ring{full_bar, empty_bar, stage_tile, ssm + g.off_ring, g.nstages, g.stage_bytes};
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < g.nstages; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], kConsWarps); stage_tile[s] = 0xffffffffu; }
        s_progress = 0; ms.target = g.bar_base; ms.ti = ms.tj = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 5) {          // (64-bit divisions: once, not once per phase)
        const uint32_t kid = threadIdx.x;
        const StKind &k = g.kind[kid];
        const uint32_t u0 = (uint32_t)(((uint64_t)cta * k.units) / ncta), u1 = (uint32_t)(((uint64_t)(cta + 1) * k.units) / ncta);
        const uint32_t rows = (u1 - u0) * k.unit_rows, xi = kid == SK_O ? 1u : kid == SK_W2 ? 2u : 0u;
        uint32_t rb = k.unit_rows;
        while (rb < (QUANT == 0x42 ? 2u : 4u) && rb * kConsWarps < min(rows, k.tile_rows)) rb *= 2u;
        StPhase &ph = phase[kid];
        ph.n = k.n; ph.row_stride = k.row_stride; ph.aux_stride = k.aux_stride; ph.tile_rows = k.tile_rows;
        ph.rows = rows; ph.tiles = (rows + k.tile_rows - 1u) / k.tile_rows; ph.row0 = u0 * k.unit_rows;
        ph.mode = (k.owned ? 1u : 0u) | rb << 8 | (((k.tile_rows + rb - 1u) / rb) % kConsWarps) << 16;
        ph.src = g.xv[xi] + (size_t)(cta % (uint32_t)kStRep) * g.rs[xi];
        ph.gain = kid == SK_QKV ? g.g_attn : kid == SK_W13 ? g.g_ffn : kid == SK_CLS ? g.g_final : nullptr;
        // layer l publishes e0 + 5l + {1: q/k/v, 2: attention output, 3: x after O, 4: SwiGLU output, 5: x after W2}; x before a layer carries the epoch e0 + 5l
        ph.need = kid == SK_O ? 2u : kid == SK_W13 ? 3u : kid == SK_W2 ? 4u : 0u;
        ph.out = kid == SK_QKV ? 1u : ph.need + 1u;
        ph.epi = kid == SK_QKV ? EPI_QKV : kid == SK_W13 ? EPI_SWIGLU : kid == SK_CLS ? EPI_CLS : EPI_RESID;
        ph.rn = 1.0f / (float)k.n;
    }
    if (threadIdx.x < 32) reinterpret_cast<float *>(ms.red)[threadIdx.x] = 0.0f;
    if (threadIdx.x < sizeof(DevState) / 4)        // the call's state: with the launch, or left on the device by the launch before
        reinterpret_cast<uint32_t *>(&ms.st)[threadIdx.x] = g.with_state ? reinterpret_cast<const uint32_t *>(&g.st0)[threadIdx.x] : __ldcg(reinterpret_cast<const uint32_t *>(g.st) + threadIdx.x);
    __syncthreads();

    // step state (identical in every CTA; advanced locally)
    uint32_t pos = ms.st.pos;
    uint32_t tok = ms.st.use_token ? ms.st.token : __ldcg(g.ids + pos);

    if (warp == kConsWarps) {
        if (lane == 0) st_producer(g, ring, phase, cta, &s_progress, pos, ms.st.is_causal, ms.st.advance);
        return;
    }

    StCursor cur{0u, 0u};
    uint32_t tcount = 0;                                                // tiles consumed so far (the producer counts the same way)
    uint32_t half = 0, el = g.epoch_base;                               // epochs: see StPhase
    // stamps (trace != nullptr: CTA 0 / thread 0, last step): [0..] after every phase; [1024..] inside layer L/2
#define ST_TRACE() do { if (g.trace && cta == 0 && threadIdx.x == 0 && step + 1 == g.n_steps && ms.ti < 1000) g.trace[ms.ti++] = clock64(); } while (0)
#define ST_STAMP() do { if (g.trace && cta == 0 && threadIdx.x == 0 && step + 1 == g.n_steps && l == d.L / 2 && ms.tj < 60) g.trace[1024 + ms.tj++] = clock64(); } while (0)

#pragma unroll 1
    for (uint32_t step = 0; step < g.n_steps; step++) {
        ST_TRACE();
        float *x_s = reinterpret_cast<float *>(ssm + g.off_xs);
        if (threadIdx.x == 0) {
            const uint32_t range = ms.st.is_causal ? pos + 1u : d.max_seq;
            uint32_t nsplit, chunk;
            st_attn_plan(range, g.nsplit_max, g.chunk_target, nsplit, chunk);
            const uint32_t grp = cta / nsplit, sp = cta - grp * nsplit, t0 = min(range, sp * chunk);
            ms.plan = StPlan{nsplit, grp, sp, t0, min(range, t0 + chunk)};
        }
        // embedding row (infer.c:987-988) into shared memory; the rows this CTA owns in the residual phases start from it
        embed_row<kConsThreads>(g.emb_w, g.emb_aux, x_s, tok, d);
        cbar();
        for (uint32_t i = threadIdx.x; i < phase[SK_O].rows; i += kConsThreads) xown[i] = x_s[phase[SK_O].row0 + i];

        // ---- layers 0..L-1: QKV | attention | O | W1,W3 | W2 ; pseudo-layer L: the classifier.  One call site per function. ----
#pragma unroll 1
        for (uint32_t l = 0; l <= d.L; l++) {
            ST_STAMP();
#pragma unroll 1
            for (uint32_t p4 = 0; p4 < 4; p4++) {
                const bool cls = (l == d.L);
                const StPhase &ph = phase[cls ? (uint32_t)SK_CLS : p4];
                if (ph.rows) {                // CTA-uniform: a CTA without rows of this kind neither reads the source nor publishes
                    half ^= 1u;               // consecutive phases alternate between the two operands
                    unsigned char *act = ssm + (half ? g.off_act2 : g.off_act);
                    const float *gain = ph.gain;
                    if (gain && !cls) gain += (size_t)l * d.E;
                    st_prep<QUANT, LPG>(g, ph.src, l == 0 && p4 == SK_QKV && !cls ? x_s : nullptr, el + ph.need, gain, ph.n, ph.rn, act, ms.red[half]);
                    ST_STAMP();
                    st_consume<QUANT, LPG>(g, ring, cur, tcount, ph, l, el + ph.out, act, pos, xown, ms);
                } else {
                    ST_STAMP();
                    if (cls && lane == 0) { ms.best_v[warp] = -FLT_MAX; ms.best_i[warp] = 0xffffffffu; }
                }
                ST_STAMP();
                ST_TRACE();
                if (cls) break;
                if (p4 == SK_QKV) {
                    st_attention<KVM, HDC>(g, ring, cur, tcount, l, cta, pos, ms.plan, el + 1u, el + 2u, reinterpret_cast<float *>(ssm + g.off_attn));
                    ST_STAMP();
                    ST_TRACE();
                }
            }
            if (l < d.L) el += 5u;
        }
        cbar();
        if (threadIdx.x == 0) {
            float bv = ms.best_v[0]; uint32_t bi = ms.best_i[0];
            for (int w = 1; w < kConsWarps; w++)
                if (ms.best_i[w] != 0xffffffffu && (bi == 0xffffffffu || ms.best_v[w] > bv || (ms.best_v[w] == bv && ms.best_i[w] < bi))) { bv = ms.best_v[w]; bi = ms.best_i[w]; }
            g.cls_val[cta] = bv; g.cls_idx[cta] = bi;
        }
        st_grid_barrier(g, ms.target, &s_progress, ncta);
        ST_TRACE();
        // ---- every CTA picks the token from the per-CTA partials (no second barrier) and advances its copy of the state ----
        {
            float bv = -FLT_MAX; uint32_t bi = 0xffffffffu;
            for (uint32_t c2 = threadIdx.x; c2 < ncta; c2 += kConsThreads) {
                const float v = __ldcg(g.cls_val + c2); const uint32_t i = __ldcg(g.cls_idx + c2);
                if (i != 0xffffffffu && (bi == 0xffffffffu || v > bv || (v == bv && i < bi))) { bv = v; bi = i; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o); const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (oi != 0xffffffffu && (bi == 0xffffffffu || ov > bv || (ov == bv && oi < bi))) { bv = ov; bi = oi; }
            }
            if (lane == 0) { ms.best_v[warp] = bv; ms.best_i[warp] = bi; }
            cbar();
            bv = -FLT_MAX; bi = 0xffffffffu;
#pragma unroll 1
            for (int w = 0; w < kConsWarps; w++)
                if (ms.best_i[w] != 0xffffffffu && (bi == 0xffffffffu || ms.best_v[w] > bv || (ms.best_v[w] == bv && ms.best_i[w] < bi))) { bv = ms.best_v[w]; bi = ms.best_i[w]; }
            if (bi == 0xffffffffu) bi = 0;       // all-NaN row: the reference's argmax returns index 0
            uint32_t nxt = bi;
            if (ms.st.advance) {
                const bool forced = (pos + 1 < ms.st.n_prompt);            // infer.c:1250 is_prefilling
                if (forced) nxt = __ldcg(g.ids + pos + 1);
                if (cta == 0 && threadIdx.x == 0) {
                    g.seen[tok] = 1;                                 // ids[0..pos] are "seen" for step pos+1
                    if (!forced) g.ids[pos + 1] = bi;
                    g.st->pos = pos + 1;
                    g.st->next_token = nxt;
                }
                tok = nxt; pos = pos + 1;
            } else if (cta == 0 && threadIdx.x == 0) {
                g.st->next_token = bi;
                if (g.next_host) *g.next_host = bi;
            }
            cbar();
        }
    }
#undef ST_TRACE
#undef ST_STAMP
}

}  // namespace nb
