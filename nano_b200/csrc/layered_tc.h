// layered_tc.h -- host side of layered_tc.cu: matrix products of long portions on tcgen05
#pragma once
#include <cuda.h>
#include <stddef.h>

#include "layered_common.cuh"
#include "tc_tiles.h"

namespace nb {
namespace lm {

// what an engine keeps for these products: rounded activation rows (one buffer for each of its three streams), the driver's tensor-map encoder,
// the word a bounded wait reports to
struct TcState {
    __nv_bfloat16 *rows[3] = {nullptr, nullptr, nullptr}; size_t elems = 0;
    decltype(&cuTensorMapEncodeTiled) encode = nullptr;
    uint32_t *err_host = nullptr, *err_dev = nullptr, sms = 148;
    __nv_bfloat16 *planes = nullptr; size_t plane_elems = 0;      // tc_gemm_split's rows in three parts
};
int tc_setup(TcState *t, size_t elems, uint32_t sms);
void tc_free(TcState *t);
// after a synchronisation: did a bounded wait of a kernel run out
int tc_check(TcState *t);
// whether the product's layout allows it.  rows: all rows of A it reads (a routed product: tokens x choices)
bool tc_fits(const TcState *t, const GemmArgs &a, uint32_t rows);
// whether the product reads its fp32 rows itself (tc_tiles.h); they have to be whole 16-byte pieces
inline bool tc_raw_rows(const GemmArgs &a, uint32_t groups, uint32_t each) {
    return a.lda % 4u == 0 && (reinterpret_cast<uintptr_t>(a.A) & 15u) == 0 && tc_reads_rows(a.N, groups, each, a.K);
}
// one or two launches on `stream` (with programmatic serialization when pdl).  buf: which of the row buffers is the stream's; maxM: the most rows of a group, each:
// how many a group has on average
int tc_gemm(TcState *t, GemmArgs a, uint32_t groups, uint32_t maxM, uint32_t rows, uint32_t each, uint32_t buf, cudaStream_t stream, bool pdl);

// C[r] = W x_r in 32-bit precision for the rows r of a paged fp32 cache, x_r = cache + (table[j / 32] * 32 + j % 32) * ld, j = first + r: the fp32 operand
// goes in as three bfloat16 parts (W is bfloat16 anyway).  Room for keys * tc_split_width(K) numbers is asked from setup.
inline uint32_t tc_split_width(uint32_t K) { return 3u * ((K + 63u) & ~63u); }
int tc_split_setup(TcState *t, size_t elems);
void tc_split_free(TcState *t);
bool tc_split_fits(const TcState *t, uint32_t N, uint32_t K, uint32_t rows, const void *W, const float *cache, uint32_t ld);
int tc_gemm_split(TcState *t, const float *cache, const uint32_t *table, uint32_t ld, uint32_t first, uint32_t rows, const void *W, uint32_t N, uint32_t K, float *C, uint32_t ldc, cudaStream_t stream, bool pdl);

}  // namespace lm
}  // namespace nb
