// prefill.h -- prompts of model files in whole portions (prefill.cu): the K and V rows of many positions at once instead of one decode step each
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

#include "attn_tc.h"

namespace nb {

struct PrefillMat { const void *w, *aux; uint32_t rows, n; };      // the fused matrices of the multi-kernel path (engine.cu "HBM layout")
struct PrefillModel {
    uint32_t arch, quant, gs, V, L, E, H, KV, F, hd, q_dim, kv_dim, max_seq;
    PrefillMat emb; std::vector<PrefillMat> qkv, wo, w13, w2;
    const float *norm_attn, *norm_ffn, *qnorm, *knorm, *rope_cos, *rope_sin;
    float *kc, *vc;
};
struct PrefillState;
// *out stays null (and 0 is returned) when the model's shapes have no portion kernels
int prefill_create(PrefillState **out, const PrefillModel &m, uint32_t sms);
void prefill_destroy(PrefillState *p);
// K and V rows of the positions [0, n) of the tokens ids[0..n) on the device; n <= max_seq.  pdl: with programmatic dependent launch; launches: how many kernels were put on the stream
int prefill_run(PrefillState *p, const uint32_t *ids, uint32_t n, cudaStream_t stream, bool pdl, uint64_t *launches);
bool prefill_fits(const PrefillState *p, uint32_t n);      // whether the attention has room for that many positions
// after a synchronisation: did a bounded wait of a kernel run out
int prefill_check(PrefillState *p);

}  // namespace nb
