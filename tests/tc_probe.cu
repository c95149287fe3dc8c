// Calls the tensor-core attention and the 32-bit product of the latents (csrc/attn_tc.h, csrc/layered_tc.h) on device arrays of the caller's; built by
// tests/test_gpu_tc_precision.py
#include "attn_tc.h"
#include "layered_tc.h"

namespace {
struct Err {
    uint32_t *host = nullptr, *dev = nullptr;
    Err() { cudaHostAlloc(&host, 64, cudaHostAllocMapped); *host = 0; cudaHostGetDevicePointer(&dev, host, 0); }
    ~Err() { cudaFreeHost(host); }
};
}  // namespace

// n: T, H, G, D, VD, pos0, block, window, ldq, q_head, ldk, ldv, k_head, v_head, ldg, ldm
extern "C" int probe_attention(const float *q, const float *k, const float *v, const uint32_t *table, float *out, const uint32_t *n, float scale, float softcap, const float *sink, const float *gate,
                               const float *mul) {
    nb::TcAttn a{};
    a.q = q; a.k = k; a.v = v; a.table = table; a.out = out; a.scale = scale; a.softcap = softcap; a.sink = sink; a.gate = gate; a.mul = mul;
    a.T = n[0]; a.H = n[1]; a.G = n[2]; a.D = n[3]; a.VD = n[4]; a.pos0 = n[5]; a.block = n[6]; a.window = n[7]; a.ldq = n[8]; a.q_head = n[9]; a.ldk = n[10]; a.ldv = n[11]; a.k_head = n[12];
    a.v_head = n[13]; a.ldg = n[14]; a.ldm = n[15];
    Err err;
    nb::TcAttnState s;
    const uint32_t keys = a.pos0 + a.T;
    int r = nb::attn_tc_setup(&s, nb::attn_tc_bytes(keys, a.G, a.D, a.VD), nb::attn_tc_tiles(keys, a.G), err.dev);
    if (!r) r = nb::attn_tc_fits(&s, a) ? nb::attn_tc_launch(&s, a, nullptr, false) : 1;
    if (!r) r = (int)cudaDeviceSynchronize();
    if (!r) r = (int)*err.host;
    nb::attn_tc_free(&s);
    return r;
}

extern "C" int probe_split(const float *cache, const uint32_t *table, uint32_t ld, uint32_t first, uint32_t rows, const void *W, uint32_t N, uint32_t K, float *C, uint32_t ldc) {
    nb::lm::TcState t;
    int r = nb::lm::tc_setup(&t, 1024, 148);
    if (!r) r = nb::lm::tc_split_setup(&t, (size_t)rows * nb::lm::tc_split_width(K));
    if (!r) r = nb::lm::tc_split_fits(&t, N, K, rows, W, cache, ld) ? nb::lm::tc_gemm_split(&t, cache, table, ld, first, rows, W, N, K, C, ldc, nullptr, false) : 1;
    if (!r) r = (int)cudaDeviceSynchronize();
    if (!r) r = nb::lm::tc_check(&t);
    nb::lm::tc_free(&t);
    return r;
}
