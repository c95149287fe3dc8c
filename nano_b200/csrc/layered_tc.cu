// layered_tc.cu -- matrix products of long portions on the fifth-generation tensor cores (layered.cu chooses them; layered_kernels.cuh has
// the tile products for shapes that this path does not take).
//
//   k_rows_bf16   the product's fp32 activation rows, rounded once to bfloat16 (what every product of this family does to its operand; short portions round them in k_gemm_tc) and
//                 gathered into expert order where a row list says so: a dense matrix that bulk copies can read
//   k_gemm_tc     C^T = W A^T in tiles of 128 weight rows x TN tokens: tcgen05.mma (one issuing thread), operands by cp.async.bulk.tensor into a ring of
//                 128-byte-swizzled stages, fp32 accumulators in tensor memory.  A tensor-memory lane is an output COLUMN of C, so a
//                 warp's stores of one token are 128 contiguous bytes and need no transposition.  1024 x 12288 x 2048 takes
//                 59 us (870 TFLOP/s, 52 % of the measured 1664) where the mma.sync tiles it replaces took 542; 1024 x 2048 x 2048 18.7 us (145).  Tensor pipe and
//                 L2 are each busy for 39 % of the large one and 17 % of the small one, whose single block per SM has three stages on the way: it waits
//                 for memory.  Two blocks per SM hide one's epilogue behind the other's products.
//
// Every wait is bounded: one that runs out records a code in a host-visible word, the kernel drains and leaves, and the step fails.
#include "layered_tc.h"

#include "family.h"
#include "tc_ptx.cuh"

namespace nb {
namespace lm {

constexpr uint32_t kTcRows = 128, kTcK = 64;       // weight rows of a tile; depth of a stage (64 bfloat16 = one 128-byte swizzle row)
__host__ __device__ constexpr uint32_t tc_stages(int tn) { return tn <= 32 ? 5u : tn <= 64 ? 4u : 3u; }      // 96..100 KB: two blocks per SM
__host__ __device__ constexpr uint32_t tc_stage_bytes(int tn) { return (kTcRows + (uint32_t)tn) * kTcK * 2u; }
inline size_t tc_smem(int tn) { return (size_t)tc_stages(tn) * tc_stage_bytes(tn) + 1024u; }

struct RowsArgs { const float *src; uint32_t ld; const uint32_t *rows; __nv_bfloat16 *dst; uint32_t ldd, M, width; };
// dst[r][c] = bf16(src[rows ? rows[r] : r][c]), c < width (a multiple of 8); a thread makes 8 columns, one 16-byte store
__global__ void __launch_bounds__(256) k_rows_bf16(const RowsArgs a) {
    pdl_enter();
    const uint32_t w8 = a.width >> 3;
    const bool vec = (a.ld & 3u) == 0 && (reinterpret_cast<uintptr_t>(a.src) & 15u) == 0;
    const size_t total = (size_t)a.M * w8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / w8), c = (uint32_t)(i % w8) * 8u;
        const float *s = a.src + (size_t)(a.rows ? a.rows[r] : r) * a.ld + c;
        float v[8];
        if (vec) {
            const float4 p = *reinterpret_cast<const float4 *>(s), q = *reinterpret_cast<const float4 *>(s + 4);
            v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = s[j];
        }
        uint4 o;
        __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
        for (int j = 0; j < 4; j++) ob[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        *reinterpret_cast<uint4 *>(a.dst + (size_t)r * a.ldd + c) = o;
    }
}

struct PlaneArgs { const float *cache; const uint32_t *table; uint32_t ld, first, rows, K, Kp; __nv_bfloat16 *dst; };
// dst[r] = [x3 | x2 | x1], x = x1 + x2 + x3 to 2^-26: the small parts first, so that the sum's large part is added last; each part padded to Kp with zeros
__global__ void __launch_bounds__(256) k_rows_split(const PlaneArgs a) {
    pdl_enter();
    const uint32_t k8 = a.Kp >> 3;
    const size_t total = (size_t)a.rows * k8;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t r = (uint32_t)(i / k8), c = (uint32_t)(i % k8) * 8u, j = a.first + r;
        const float *s = a.cache + ((size_t)a.table[j / 32u] * 32u + j % 32u) * a.ld + c;
        float v[8];
#pragma unroll
        for (uint32_t q = 0; q < 2; q++) {          // K is a multiple of 8
            const float4 p = c < a.K ? *reinterpret_cast<const float4 *>(s + 4u * q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            v[4 * q] = p.x; v[4 * q + 1] = p.y; v[4 * q + 2] = p.z; v[4 * q + 3] = p.w;
        }
#pragma unroll
        for (int part = 2; part >= 0; part--) {
            uint4 o;
            __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                ob[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                const float2 b = __bfloat1622float2(ob[q]);
                v[2 * q] -= b.x; v[2 * q + 1] -= b.y;
            }
            *reinterpret_cast<uint4 *>(a.dst + (size_t)r * 3u * a.Kp + part * a.Kp + c) = o;
        }
    }
}

// g: the product; wmap: [groups][N][K], in boxes of 128 weight rows x 64.  Where a rounded copy is read, amap is that: [rows][a_gmod][K], gathered, boxes of TN tokens x 64, and A and
// a_rows are unused; instances that read their rows themselves take them from A and a_rows, and amap is empty.  ks: blocks of a cluster that share one tile's depth (grid.z = groups * ks);
// wsteps: the stages after which W starts over (rows in several parts; the whole depth otherwise)
struct alignas(64) TcArgs { CUtensorMap wmap, amap; GemmArgs g; uint32_t ks, wsteps; uint32_t *err; };

// Epilogue of NJ tokens of one output column: every option is looked at once for the NJ values (inside the loop over tokens the switch alone made a
// tile's epilogue 44 instructions per value, most of them instruction-cache misses: 1024 x 2048 x 128 took 38 us, the same as at a depth of
// 2048; it takes 9).  live: how many of the tokens exist.  The long functions are inlined NJ times, so they come in fours.
__device__ __forceinline__ bool light_epilogue(uint32_t epi) { return epi == EPI_NONE || epi == EPI_BIAS || epi == EPI_GELU_SPLIT || epi == EPI_RELU2 || epi == EPI_SIGMOID || epi == EPI_SIGMOID_TAIL; }
template <int NJ>
__device__ __forceinline__ void finish(const GemmArgs &a, float (&v)[NJ], const float *bias, uint32_t n, uint32_t row, uint32_t col, uint32_t live) {
    const float b = bias ? bias[n] : 0.0f;
    if (bias) {
#pragma unroll
        for (int j = 0; j < NJ; j++) v[j] += b;
    }
    if (a.epi == EPI_RELU2) {
#pragma unroll
        for (int j = 0; j < NJ; j++) { const float r = fmaxf(v[j], 0.0f); v[j] = r * r; }
    } else if (a.epi == EPI_SIGMOID || (a.epi == EPI_SIGMOID_TAIL && n >= a.split)) {
#pragma unroll
        for (int j = 0; j < NJ; j++) v[j] = sigmoidf_(v[j]);
    } else if (a.epi == EPI_GELU_SPLIT) {
        if (n < a.split) {
#pragma unroll
            for (int j = 0; j < NJ; j++) v[j] = gelu_tanh(v[j]);
        }
    } else if (NJ <= 4 && !light_epilogue(a.epi)) {
#pragma unroll
        for (int j = 0; j < NJ; j++) v[j] = epilogue(v[j], a, nullptr, n);
    }
    if (a.mul) {
        const float *m = a.mul + (size_t)row * a.ldm + col;
#pragma unroll
        for (uint32_t j = 0; j < NJ; j++) if (j < live) v[j] *= m[(size_t)j * a.ldm];
    }
    float *c = a.C + (size_t)row * a.ldc + col;
    if (a.c_mode & C_SCALE) {
#pragma unroll
        for (int j = 0; j < NJ; j++) v[j] *= a.c_scale;
    }
    if (a.c_mode & C_ADD) {
#pragma unroll
        for (uint32_t j = 0; j < NJ; j++) if (j < live) v[j] += c[(size_t)j * a.ldc];
    }
    if (live >= (uint32_t)NJ) {
#pragma unroll
        for (uint32_t j = 0; j < NJ; j++) c[(size_t)j * a.ldc] = v[j];
    } else {
#pragma unroll
        for (uint32_t j = 0; j < NJ; j++) if (j < live) c[(size_t)j * a.ldc] = v[j];
    }
}
// the sums of the cluster's partial tiles for the tokens [j0, j1) of this thread's column, in the order of the depth, finished
template <int NJ>
__device__ __forceinline__ void gather(const TcArgs &ta, const GroupView &gv, uint32_t at, uint32_t j0, uint32_t j1, uint32_t m0, uint32_t n) {
    const GemmArgs &a = ta.g;
    for (uint32_t j = j0; j < j1; j += NJ) {
        float f[NJ];
#pragma unroll
        for (int i = 0; i < NJ; i++) f[i] = 0.0f;
#pragma unroll 2
        for (uint32_t p = 0; p < ta.ks; p++) {
            uint32_t peer;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at + j * kTcRows * 4u), "r"(p));
#pragma unroll
            for (uint32_t i = 0; i < NJ; i++) f[i] += ld_cluster_f32(peer + i * kTcRows * 4u);          // (a tile's buffer holds all TN tokens)
        }
        finish<NJ>(a, f, gv.bias, n, gv.r0 + m0 + j, gv.c0 + n, j1 - j);
    }
}

// A tile's activations, rounded to bfloat16 and swizzled as a bulk copy would leave them, by the four warps that finish the tile later: a thread has 16 columns of every 32nd row of a
// stage.  Short portions (TN 32 and 64), whose products are a chain of launches: a kernel of its own for the rows, and the wait for it, cost 2 to 4 us a product.
template <int TN>
__device__ __forceinline__ bool tc_rows(const GemmArgs &a, const GroupView &gv, uint32_t m0, uint32_t s0, uint32_t ns, uint32_t ring, uint32_t full, uint32_t empty) {
    constexpr uint32_t ST = tc_stages(TN), SB = tc_stage_bytes(TN), NR = TN / 32;
    const uint32_t t = threadIdx.x - 64u, r = t >> 2, c16 = (t & 3u) * 16u;
    const float *src[NR];
#pragma unroll
    for (uint32_t h = 0; h < NR; h++) {
        const uint32_t row = m0 + r + 32u * h;
        src[h] = row < gv.rows ? a.A + (size_t)(a.a_rows ? a.a_rows[gv.r0 + row] : gv.r0 + row) * a.lda + gv.a0 : nullptr;
    }
    float4 v[NR][4];
    auto load = [&](uint32_t i) {
        const uint32_t k = (s0 + i) * kTcK + c16;
#pragma unroll
        for (uint32_t h = 0; h < NR; h++)
#pragma unroll
            for (uint32_t q = 0; q < 4u; q++) v[h][q] = src[h] && k + 4u * q < a.K ? *reinterpret_cast<const float4 *>(src[h] + k + 4u * q) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    if (ns) load(0);
    for (uint32_t i = 0; i < ns; i++) {
        const uint32_t st = i % ST, rows = ring + st * SB + kTcRows * kTcK * 2u;
        uint4 o[NR][2];
#pragma unroll
        for (uint32_t h = 0; h < NR; h++)
#pragma unroll
            for (uint32_t q = 0; q < 4u; q++) {
                __nv_bfloat162 *ob = reinterpret_cast<__nv_bfloat162 *>(&o[h][q >> 1]) + (q & 1u) * 2u;
                ob[0] = __floats2bfloat162_rn(v[h][q].x, v[h][q].y); ob[1] = __floats2bfloat162_rn(v[h][q].z, v[h][q].w);
            }
        if (i + 1u < ns) load(i + 1u);
        if (i >= ST && !mbar_wait_warp(empty + st * 8u, ((i / ST) - 1u) & 1u)) return false;
#pragma unroll
        for (uint32_t h = 0; h < NR; h++)
#pragma unroll
            for (uint32_t q = 0; q < 2u; q++) {
                const uint32_t row = r + 32u * h, at = rows + row * 128u + ((((c16 >> 3) + q) ^ (row & 7u)) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(o[h][q].x), "r"(o[h][q].y), "r"(o[h][q].z), "r"(o[h][q].w) : "memory");
            }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");          // plain stores, read by the tensor core
        __syncwarp();
        if ((threadIdx.x & 31u) == 0) mbar_arrive(full + st * 8u);
    }
    return true;
}

// RAW: the activations are ta.g.A itself (fp32 rows of whole 16-byte pieces), not a rounded copy that bulk copies read
template <int TN, bool RAW>
__global__ void __launch_bounds__(192) k_gemm_tc(const __grid_constant__ TcArgs ta) {
    constexpr uint32_t ST = tc_stages(TN), SB = tc_stage_bytes(TN), COLS = TN < 32 ? 32 : TN, LOADED = RAW ? kTcRows * kTcK * 2u : SB;          // bytes of a stage that bulk copies bring
    extern __shared__ uint8_t tc_raw[];
    __shared__ __align__(8) uint64_t bars[2 * ST + 1];
    __shared__ uint32_t tmem_s, bad_s;
    const GemmArgs &a = ta.g;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ring = (smem_u32(tc_raw) + 1023u) & ~1023u;
    const uint32_t group = blockIdx.z / ta.ks, part = blockIdx.z % ta.ks;
    const uint32_t m0 = blockIdx.y * TN, n0 = blockIdx.x * kTcRows;
    const uint32_t full = smem_u32(bars), empty = full + ST * 8u, done = full + 2u * ST * 8u;
    const uint32_t steps = (a.K + kTcK - 1u) / kTcK, per = (steps + ta.ks - 1u) / ta.ks, s0 = min(steps, part * per), ns = min(steps, s0 + per) - s0;
    if (a.g_off) {          // a group's rows are known on the device only; all blocks of a cluster leave together
        pdl_wait();
        if (m0 >= a.g_off[group + 1] - a.g_off[group]) return;
    }
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < ST; i++) { mbar_init(full + i * 8u, RAW ? 5 : 1); mbar_init(empty + i * 8u, 1); }
        mbar_init(done, 1);
        bad_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) { tc_alloc(smem_u32(&tmem_s), COLS); tc_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Only now may the next kernels' blocks come: one that waits for this grid while it holds tensor memory must not be in the way of an allocation here
    pdl_launch_next();
    const uint32_t tmem = tmem_s, npre = a.g_off ? 0u : min(ST, ns);
    if (warp == 0 && lane == 0)          // weights do not depend on the kernel before: their first tiles are on the way while it ends
        for (uint32_t i = 0; i < npre; i++) { mbar_expect(full + i * 8u, LOADED); tma_3d(ring + i * SB, &ta.wmap, (s0 + i) % ta.wsteps * kTcK, n0, group, full + i * 8u); }
    pdl_wait();
    const GroupView gv = group_view(a, group);
    if (warp == 0 && lane == 0) {
        for (uint32_t i = 0; i < ns; i++) {
            const uint32_t st = i % ST, bar = full + st * 8u, dst = ring + st * SB;
            if (i >= ST && !mbar_wait(empty + st * 8u, ((i / ST) - 1u) & 1u)) { bad_s = 1; break; }
            if (i >= npre) { mbar_expect(bar, LOADED); tma_3d(dst, &ta.wmap, (s0 + i) % ta.wsteps * kTcK, n0, group, bar); }
            if (!RAW) tma_3d(dst + kTcRows * kTcK * 2u, &ta.amap, (s0 + i) * kTcK, group % a.a_gmod, gv.r0 + m0, bar);
        }
    } else if (warp == 1 && lane == 0) {
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((kTcRows >> 4) << 24);      // fp32 += bf16 x bf16, both K-major
        bool ok = true;
        for (uint32_t i = 0; i < ns && ok; i++) {
            const uint32_t st = i % ST;
            ok = mbar_wait(full + st * 8u, (i / ST) & 1u);
            if (!ok) break;
            tc_fence_after();
            const uint64_t wd = tc_desc(ring + st * SB), ad = tc_desc(ring + st * SB + kTcRows * kTcK * 2u);
#pragma unroll
            for (uint32_t k = 0; k < kTcK / 16u; k++) tc_mma_ss(tmem, wd + 2u * k, ad + 2u * k, idesc, i > 0 || k > 0);
            tc_commit(empty + st * 8u);
        }
        if (!ok) bad_s = 2;
        tc_commit(done);
    }
    __syncwarp();
    bool live = true;
    const uint32_t quad = warp & 3u, n = n0 + quad * 32u + lane, rows = gv.rows;
    if (warp >= 2) {
        if constexpr (RAW) { if (!tc_rows<TN>(a, gv, m0, s0, ns, ring, full, empty)) bad_s = 4; }
        live = mbar_wait_warp(done, 0);
        if (!live) bad_s = 3;
        tc_fence_after();
    }
    // partial tiles and long epilogues pass through this block's shared memory (the ring is free: all its products are done): [TN][128]
    float *mine = reinterpret_cast<float *>(tc_raw + (ring - smem_u32(tc_raw))) + quad * 32u + lane;
    const bool light = light_epilogue(a.epi), stage = ta.ks > 1 || !light;
    if (warp >= 2 && live) {
#pragma unroll 1
        for (uint32_t c = 0; c < TN; c += 32u) {
            if (m0 + c >= rows) break;
            uint32_t v[32];
            if (ns) tc_ld32(tmem + ((quad * 32u) << 16) + c, v);
            float f[32];
#pragma unroll
            for (uint32_t j = 0; j < 32; j++) f[j] = ns ? __uint_as_float(v[j]) : 0.0f;
            if (stage) {
#pragma unroll
                for (uint32_t j = 0; j < 32; j++) mine[(c + j) * kTcRows] = f[j];
            } else if (n < a.N) finish<32>(a, f, gv.bias, n, gv.r0 + m0 + c, gv.c0 + n, rows - m0 - c);
        }
    }
    if (ta.ks == 1) {
        if (!light && warp >= 2 && live && n < a.N)          // a thread reads what it wrote itself
            for (uint32_t j = 0; j < min((uint32_t)TN, rows - m0); j += 4u) {
                float f[4];
#pragma unroll
                for (uint32_t i = 0; i < 4; i++) f[i] = mine[(j + i) * kTcRows];
                finish<4>(a, f, gv.bias, n, gv.r0 + m0 + j, gv.c0 + n, rows - m0 - j);
            }
    } else {
        // every block of the cluster finishes TN / ks tokens (4 .. 64): a result does not depend on which block was first
        cluster_sync_all();
        if (warp >= 2 && live && n < a.N) {
            const uint32_t span = TN / ta.ks, j0 = part * span, j1 = min(j0 + span, rows - m0), at = smem_u32(mine);
            if (span >= 32u && light) gather<32>(ta, gv, at, j0, j1, m0, n);
            else gather<4>(ta, gv, at, j0, j1, m0, n);
        }
        cluster_sync_all();          // no block leaves while another reads its partials
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (bad_s && threadIdx.x == 0) {
        *ta.err = 0x100u + bad_s;
        __threadfence_system();
        const long long t0 = clock64();
        while (clock64() - t0 < 20000000ll) __nanosleep(1000);          // copies still in flight land in this block's shared memory before it is given back
    }
    __syncthreads();
    if (warp == 1) tc_dealloc(tmem, COLS);
}

// ---- host side ----
namespace {
bool tensor_map(const TcState *t, CUtensorMap *m, const void *base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1, uint64_t s2, uint32_t b0, uint32_t b1, uint32_t b2) {
    const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {s1, s2};
    const cuuint32_t box[3] = {b0, b1, b2}, step[3] = {1, 1, 1};
    return t->encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
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
    if (cluster_z > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 1; attr[cfg.numAttrs].val.clusterDim.y = 1; attr[cfg.numAttrs++].val.clusterDim.z = cluster_z;
    }
    NB_CK(cudaLaunchKernelEx(&cfg, k, args));
    return 0;
}
template <int TN, bool RAW>
int optin() { NB_CK(nb::smem_at_least((const void *)k_gemm_tc<TN, RAW>, (int)tc_smem(TN))); return 0; }
}  // namespace

int tc_setup(TcState *t, size_t elems, uint32_t sms) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult got;
    NB_CK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &got));
    if (got != cudaDriverEntryPointSuccess || !fn) return fail(NB200_ECUDA, "the driver has no cuTensorMapEncodeTiled");
    t->encode = reinterpret_cast<decltype(t->encode)>(fn);
    t->sms = sms;
    for (auto &p : t->rows) if (cudaMalloc(&p, elems * 2) != cudaSuccess) { p = nullptr; return fail(NB200_ENOMEM, "cudaMalloc(%zu) failed", elems * 2); }
    t->elems = elems;
    NB_CK(cudaHostAlloc(&t->err_host, 64, cudaHostAllocMapped));
    *t->err_host = 0;
    NB_CK(cudaHostGetDevicePointer(&t->err_dev, t->err_host, 0));
    int r;
    if ((r = optin<32, true>()) || (r = optin<64, true>()) || (r = optin<32, false>()) || (r = optin<64, false>()) || (r = optin<128, false>())) return r;
    return 0;
}
void tc_free(TcState *t) {
    for (auto &p : t->rows) { if (p) cudaFree(p); p = nullptr; }
    tc_split_free(t);
    if (t->err_host) cudaFreeHost(t->err_host);
    t->err_host = t->err_dev = nullptr; t->encode = nullptr; t->elems = 0;
}
void tc_split_free(TcState *t) {
    if (t->planes) cudaFree(t->planes);
    t->planes = nullptr; t->plane_elems = 0;
}
int tc_check(TcState *t) {
    if (!t->err_host || !*static_cast<volatile uint32_t *>(t->err_host)) return 0;
    const uint32_t code = *t->err_host;
    *t->err_host = 0;
    return fail(NB200_ECUDA, "a wait inside a kernel ran out (code 0x%x): the results of this call are not valid", code);
}
// bulk copies need 16-byte aligned bases and strides: every row of W, every group's weights and every group's columns of A start on a multiple of 8
bool tc_fits(const TcState *t, const GemmArgs &a, uint32_t rows) {
    const size_t width = (size_t)(a.a_gmod - 1) * a.a_gcols + a.K;
    return t->encode && a.K % 8u == 0 && a.ldw % 8u == 0 && a.w_gstride % 8u == 0 && (a.a_gmod == 1 || a.a_gcols % 8u == 0) && (reinterpret_cast<uintptr_t>(a.W) & 15u) == 0 && rows * width <= t->elems;
}
int tc_gemm(TcState *t, GemmArgs a, uint32_t groups, uint32_t maxM, uint32_t rows, uint32_t each, uint32_t buf, cudaStream_t stream, bool pdl) {
    const uint32_t width = (a.a_gmod - 1) * a.a_gcols + a.K, tn = tc_tile_tokens(each);
    const bool raw = tc_raw_rows(a, groups, each);
    __nv_bfloat16 *dst = t->rows[buf];
    int r;
    TcArgs ta{};
    if (!raw) {
        const RowsArgs ra{a.A, a.lda, a.a_rows, dst, width, rows, width};
        const size_t threads = (size_t)rows * width / 8u;
        if ((r = launch<RowsArgs>(k_rows_bf16, dim3((uint32_t)((threads + 255u) / 256u < t->sms * 16u ? (threads + 255u) / 256u : t->sms * 16u)), dim3(256), 0, stream, pdl, ra))) return r;
        a.A = nullptr; a.a_rows = nullptr;
        if (!tensor_map(t, &ta.amap, dst, a.K, a.a_gmod, rows, (uint64_t)(a.a_gmod > 1 ? a.a_gcols : width) * 2u, (uint64_t)width * 2u, kTcK, 1, tn))
            return fail(NB200_ECUDA, "cuTensorMapEncodeTiled refused the rows of a product of %u x %u x %u", rows, a.N, a.K);
    }
    ta.g = a; ta.err = t->err_dev;
    if (!tensor_map(t, &ta.wmap, a.W, a.K, a.N, groups, (uint64_t)a.ldw * 2u, groups > 1 ? a.w_gstride * 2u : (uint64_t)a.ldw * 2u * a.N, kTcK, kTcRows, 1))
        return fail(NB200_ECUDA, "cuTensorMapEncodeTiled refused a product of %u x %u x %u", rows, a.N, a.K);
    // Blocks of a cluster share a tile's depth while fewer than 7 of 10 SMs have one, down to two stages each (two layers of width 2048: 200 tokens 644 us
    // before, 443 with it; up to two blocks per SM, ks = 2 for 128 tiles, was the same within the noise at 1024 tokens)
    const uint32_t tiles = (a.N + kTcRows - 1u) / kTcRows * ((each + tn - 1u) / tn) * groups, steps = (a.K + kTcK - 1u) / kTcK;
    uint32_t ks = 1;
    while (ks < 8u && tiles * ks * 10u <= t->sms * 7u && steps >= ks * 4u) ks *= 2u;
    ta.ks = ks; ta.wsteps = steps;
    const dim3 grid((a.N + kTcRows - 1u) / kTcRows, (maxM + tn - 1u) / tn, groups * ks), block(192);
    if (tn == 32) return launch<TcArgs>(raw ? k_gemm_tc<32, true> : k_gemm_tc<32, false>, grid, block, tc_smem(32), stream, pdl, ta, ks);
    if (tn == 64) return launch<TcArgs>(raw ? k_gemm_tc<64, true> : k_gemm_tc<64, false>, grid, block, tc_smem(64), stream, pdl, ta, ks);
    return launch<TcArgs>(k_gemm_tc<128, false>, grid, block, tc_smem(128), stream, pdl, ta, ks);
}

int tc_split_setup(TcState *t, size_t elems) {
    if (cudaMalloc(&t->planes, elems * 2) != cudaSuccess) { t->planes = nullptr; return fail(NB200_ENOMEM, "cudaMalloc(%zu) failed", elems * 2); }
    t->plane_elems = elems;
    return 0;
}
bool tc_split_fits(const TcState *t, uint32_t N, uint32_t K, uint32_t rows, const void *W, const float *cache, uint32_t ld) {
    return t->encode && t->planes && N && K % 8u == 0 && ld % 4u == 0 && ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(cache)) & 15u) == 0 && (size_t)rows * tc_split_width(K) <= t->plane_elems;
}
int tc_gemm_split(TcState *t, const float *cache, const uint32_t *table, uint32_t ld, uint32_t first, uint32_t rows, const void *W, uint32_t N, uint32_t K, float *C, uint32_t ldc, cudaStream_t stream, bool pdl) {
    const uint32_t width = tc_split_width(K);
    int r;
    const PlaneArgs pa{cache, table, ld, first, rows, K, width / 3u, t->planes};
    const size_t threads = (size_t)rows * (width / 24u);
    if ((r = launch<PlaneArgs>(k_rows_split, dim3((uint32_t)((threads + 255u) / 256u < t->sms * 16u ? (threads + 255u) / 256u : t->sms * 16u)), dim3(256), 0, stream, pdl, pa))) return r;
    TcArgs ta{};
    ta.g.C = C; ta.g.ldc = ldc; ta.g.M = rows; ta.g.N = N; ta.g.K = width; ta.g.a_gmod = 1;
    ta.err = t->err_dev; ta.ks = 1; ta.wsteps = width / 3u / kTcK;
    if (!tensor_map(t, &ta.wmap, W, K, N, 1, (uint64_t)K * 2u, (uint64_t)K * 2u * N, kTcK, kTcRows, 1) || !tensor_map(t, &ta.amap, t->planes, width, 1, rows, (uint64_t)width * 2u, (uint64_t)width * 2u, kTcK, 1, 128))
        return fail(NB200_ECUDA, "cuTensorMapEncodeTiled refused a product of %u x %u x %u", rows, N, width);
    return launch<TcArgs>(k_gemm_tc<128, false>, dim3((N + kTcRows - 1u) / kTcRows, (rows + 127u) / 128u, 1), dim3(192), tc_smem(128), stream, pdl, ta);
}

}  // namespace lm
}  // namespace nb
