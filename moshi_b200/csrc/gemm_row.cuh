// Linears of a few activation rows, whole output rows per CTA; see gemm_row.cu.
#pragma once

#include "gemm_sk.cuh"

namespace b200 {
namespace tc {

constexpr int ROW_MAX_M = 16;
bool row_wins(int M, int epi, int gate_rows, bool i8, int sms);
bool row_supported(int M, int K, bool i8, const void* x, long long ldx_bytes);
// x: bf16 rows, or int8 with the scales of its rows (sa) and of the weight rows (sw); w_tiles as packed for gemm_sk.cu
int row_linear(const void* x, long long ldx_bytes, const void* w_tiles, __nv_bfloat16* y, long long ldy, const __nv_bfloat16* res, long long ldr, int M, int N,
               int K, int epi, int gate_rows, const float* sa, const float* sw, int sms, int pdl, cudaStream_t stream);

}  // namespace tc
}  // namespace b200
