// layered_common.cuh -- what the translation units of the layered runtime share: the argument block of a matrix product, its epilogues, the
// programmatic-launch helpers.  Device functions and types only.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace nb {
namespace lm {

constexpr uint32_t kPage = 32;            // tokens per cache page == keys per attention tile
constexpr uint32_t kAttnWarps = 8;        // heads per attention block
constexpr uint32_t kGemvMaxM = 4;         // rows a k_gemv launch handles per group

enum CMode : uint32_t { C_ADD = 1, C_SCALE = 2 };
enum Epi : uint32_t { EPI_NONE = 0, EPI_BIAS = 1, EPI_GELU_SPLIT = 2, EPI_SIGMOID = 3, EPI_RELU2 = 4, EPI_GELU_CONV = 5, EPI_SOFTPLUS = 6, EPI_CONV_RANGES = 7, EPI_SIGMOID_TAIL = 8, EPI_GELU_ERF = 9, EPI_SOFTCAP = 10 };

// C[r, c0 + n] = epi( sum_k A[arow(r), a0 + k] * W[g][n, k] + bias[g][n] )   for the rows r of group g
//   rows of group g : [g_off[g], g_off[g+1])  when g_off is given (sizes known on the device only), else [0, M)
//   arow(r)         : a_rows[r] when given (gather), else r
//   a0 = (g % a_gmod) * a_gcols,  c0 = g * c_gcols,  W[g] = W + g * w_gstride,  bias[g] = bias + g * b_gstride
struct GemmArgs {
    const float *A; const void *W; float *C; const float *bias;
    const uint32_t *g_off; const uint32_t *a_rows;
    const uint32_t *g_act;    // k_gemv with g_off: blockIdx.y is a place in this list of the groups that have rows (0xffffffff past its end)
    uint32_t M, N, K, lda, ldw, ldc;
    uint32_t a_gmod, a_gcols, c_gcols, b_gstride;
    uint64_t w_gstride;
    uint32_t epi, split;      // EPI_GELU_SPLIT: gelu_tanh on columns n < split, bias only on the others; EPI_SIGMOID_TAIL: sigmoid on columns n >= split
    uint32_t round_a;         // k_gemv: round A to bf16 first (what the tensor-core kernel does to its operand)
    // k_gemv only.  Prologue: when a_norm_w is given, row r of A is used as A[r, k] / rms(A[r, 0..K)) * a_norm_w[k] (eps inside the root).
    const float *a_norm_w; float a_eps;
    // k_gemv only.  Epilogue EPI_GELU_CONV: columns n < split get gelu_tanh and go to C; a column n >= split is channel c = n - split of a
    // causal convolution over the rows in order (taps cv_taps[c][cv_K], bias cv_bias, tail cv_state [cv_K - 1][N - split]) whose
    // outputs go to cv_out [rows][N - split]; the tail moves on.  One warp owns a channel, so the tail has one reader and one writer.
    const float *cv_taps, *cv_bias; float *cv_state, *cv_out; uint32_t cv_K;
    // After the epilogue: with c_mode & C_SCALE the value is multiplied by c_scale, with c_mode & C_ADD it is added to what C holds,
    // so two products can be summed with fixed weights into one output (C = s1 A1 W1^T, then C += s2 A2 W2^T).
    float c_scale; uint32_t c_mode;
    // k_gemv only.  Prologue: when a_poly is given (4 numbers a, b, c, e), row r of A is used as a N(z) + b N(z^2) + c N(z^3) + e with
    // z = A[r, 0..K), powers element by element and N(u) = u / sqrt(mean(u^2) + a_eps).
    const float *a_poly;
    // k_gemv only.  Epilogue EPI_CONV_RANGES: a column n inside [cr[i].n0, cr[i].n1) is channel n - n0 of causal convolution i over the
    // rows in order (no epilogue before it); every other column is stored as usual.
    struct ConvRange { uint32_t n0, n1; const float *taps, *bias; float *state, *out; uint32_t K, act; } cr[2];
    // k_gemv only.  Gated pair (glu 1: gelu_tanh, 2: silu, 3: the clamped unit below): W holds 2 N rows per group, [gate rows | up rows]; column n of C receives
    // act(s g_n) (s u_n) with g_n, u_n the products of rows n and N + n and s = row_scale[row] (1 when null): a routed expert whose
    // input is weighted by the router's score, without a pass over the input.
    uint32_t glu; const float *row_scale;
    // k_gemv only.  Prologue (with a_norm_w): a_parts > 1 norms row r of A in a_parts equal parts, each by its own root mean square
    // (K / a_parts columns each, a multiple of 8; at most 32 parts).
    uint32_t a_parts;
    // k_gemv only (instances EXT 4 and 5).  Residual epilogue of a sublayer's last product, for designs whose norms are elementwise
    // (Dynamic Tanh, tanh(alpha u) w + b): instead of storing C, column n of row r updates the residual stream in place,
    // x[r][n] += tanh(res_pa v) res_pw[n] + res_pb[n], keeps a copy (res_keep, optional) and writes the next sublayer's input
    // res_out[r][n] = tanh(res_na x[r][n]) res_nw[n] + res_nb[n] (res_out optional).  Rows of x, res_out and res_keep are N long.
    float *res_x, *res_out, *res_keep; const float *res_pw, *res_pb, *res_nw, *res_nb; float res_pa, res_na;
    // After the epilogue: with mul given, the value of row r (of the output) and column c0 + n is multiplied by mul[r * ldm + c0 + n]
    // (an output gate computed by an earlier product).
    const float *mul; uint32_t ldm;
    // Gated pair, glu 3: the clamped unit  g' = min(g, glu_limit), u' = clamp(u, -glu_limit, glu_limit),  g' sigmoid(1.702 g') (u' + 1).
    float glu_limit;
    // EPI_SOFTCAP: cap tanh(v / cap)
    float cap;
    // k_gemv_one only: 2^one_split warps share a row; own_rows: rows of one group may differ though they are of one token
    uint32_t one_split; bool own_rows;
};

// Programmatic dependent launch: every kernel first lets the NEXT kernel of its stream be scheduled (its blocks then sit in their own
// pdl_enter until this grid has finished and its writes are visible), then waits for the kernels before it.  Launch latency and block
// scheduling of a chain of short kernels overlap with the tail of the kernel before; no kernel reads or writes what another kernel
// produces before the wait (weights may be prefetched: nothing writes them).
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() { pdl_launch_next(); pdl_wait(); }
// Weights do not depend on the kernel before: a matrix-vector kernel asks for its weight rows (L2 prefetch, no register, no wait)
// BETWEEN the two halves of pdl_enter, so their trip from HBM overlaps the tail of the kernel it waits for.  One 128-byte line per
// lane and step; at most `cols` rows per warp.
__device__ __forceinline__ void prefetch_weight_rows(const void *W, size_t elem, uint32_t ldw, uint32_t K, uint32_t N, uint32_t warp0, uint32_t nwarps, uint32_t cols) {
    const uint32_t lane = threadIdx.x & 31u, row_bytes = K * (uint32_t)elem;
    for (uint32_t n = warp0, c = 0; n < N && c < cols; n += nwarps, c++) {
        const char *p = static_cast<const char *>(W) + (size_t)n * ldw * elem;
        for (uint32_t off = lane * 128u; off < row_bytes; off += 32u * 128u) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + off));
    }
}

__device__ __forceinline__ float gelu_tanh(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplusf_(float z) { return log1pf(expf(-fabsf(z))) + fmaxf(z, 0.0f); }
// the clamped gated unit: the gate is capped from above, the linear branch on both sides and shifted by one
__device__ __forceinline__ float clamped_glu(float g, float u, float limit) {
    g = fminf(g, limit); u = fminf(fmaxf(u, -limit), limit);
    return g * sigmoidf_(1.702f * g) * (u + 1.0f);
}

__device__ __forceinline__ float epilogue(float v, const GemmArgs &a, const float *bias, uint32_t n) {
    if (bias) v += bias[n];
    switch (a.epi) {
        case EPI_GELU_SPLIT: case EPI_GELU_CONV: return n < a.split ? gelu_tanh(v) : v;
        case EPI_SIGMOID: return sigmoidf_(v);
        case EPI_RELU2: { const float r = fmaxf(v, 0.0f); return r * r; }
        case EPI_SOFTPLUS: return softplusf_(v);
        case EPI_SIGMOID_TAIL: return n >= a.split ? sigmoidf_(v) : v;
        case EPI_SOFTCAP: return a.cap * tanhf(v / a.cap);
        case EPI_GELU_ERF: return 0.5f * v * (1.0f + erff(v * 0.70710678118654752f));
        default: return v;
    }
}
__device__ __forceinline__ float gated(const GemmArgs &a, float v, uint32_t row, uint32_t col) { return a.mul ? v * a.mul[(size_t)row * a.ldm + col] : v; }
__device__ __forceinline__ void store_c(const GemmArgs &a, float *dst, float v) {
    if (a.c_mode & C_SCALE) v *= a.c_scale;
    *dst = (a.c_mode & C_ADD) ? *dst + v : v;
}

struct GroupView { uint32_t r0, rows, a0, c0; const float *bias; uint64_t w0; };
__device__ __forceinline__ GroupView group_view(const GemmArgs &a, uint32_t g) {
    GroupView v;
    v.r0 = a.g_off ? a.g_off[g] : 0u;
    v.rows = a.g_off ? a.g_off[g + 1] - v.r0 : a.M;
    v.a0 = (g % a.a_gmod) * a.a_gcols; v.c0 = g * a.c_gcols;
    v.bias = a.bias ? a.bias + (size_t)g * a.b_gstride : nullptr;
    v.w0 = (uint64_t)g * a.w_gstride;
    return v;
}

__device__ __forceinline__ float wval(const float *w) { return *w; }
__device__ __forceinline__ float wval(const __nv_bfloat16 *w) { return __bfloat162float(*w); }

}  // namespace lm
}  // namespace nb
