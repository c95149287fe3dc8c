// attn_tc.h -- softmax attention of long portions on the tensor cores, in 32-bit precision (attn_tc.cu)
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace nb {

// out[t][h][:] = softmax over the keys that query t sees of (q[t][h] . k[j][g]) * scale, times v[j][g];  g = h / (H / G).
// Query t sits at position pos0 + t and sees key j of [0, pos0 + t] when j lies in the query's block of `block` positions (0: no blocks) and less than
// `window` positions back (0: no window).  softcap (0: none): cap tanh(s / cap) on the scaled score.  sink (optional): one number per
// head that joins the softmax denominator as exp(sink_h).  gate (optional): the output of (t, h) is multiplied by sigmoid(gate[t * ldg + h]).
// mul (optional): ... and by mul[t * ldm + h * VD + d].  Everything is fp32 in memory.  Key j of head g is the D floats at k + row(j) * ldk + g * k_head, its value the VD floats at
// v + row(j) * ldv + g * v_head; row(j) = table ? table[j / 32] * 32 + j % 32 : j - first_row.
struct TcAttn {
    const float *q; uint32_t ldq, q_head;      // query (t, h): D floats at q + t * ldq + h * q_head
    const float *k, *v; uint64_t ldk, ldv, k_head, v_head; const uint32_t *table; uint32_t first_row;
    float *out;                                // [T][H VD]
    uint32_t T, H, G, D, VD, pos0, block, window;
    float scale, softcap; const float *sink, *gate; uint32_t ldg;
    const float *mul; uint32_t ldm;
};
// what the kernels keep: the split keys and values of one portion's attention, the word a bounded wait reports to
struct TcAttnState { unsigned char *images = nullptr; float *scales = nullptr; size_t bytes = 0, tiles = 0; uint32_t *err_dev = nullptr; };
// images for `keys` keys of G heads; setup allocates room for the most that any layer asks
size_t attn_tc_bytes(uint32_t keys, uint32_t G, uint32_t D, uint32_t VD);
int attn_tc_setup(TcAttnState *s, size_t bytes, size_t tiles, uint32_t *err_dev);
void attn_tc_free(TcAttnState *s);
inline size_t attn_tc_tiles(uint32_t keys, uint32_t G) { return (size_t)((keys + 127u) / 128u) * G; }
// the first key of the first tile that any query sees
uint32_t attn_tc_first(const TcAttn &a);
// whether shapes, alignment and the room for the images allow it
bool attn_tc_fits(const TcAttnState *s, const TcAttn &a);
// two launches
int attn_tc_launch(TcAttnState *s, const TcAttn &a, cudaStream_t stream, bool pdl);

}  // namespace nb
