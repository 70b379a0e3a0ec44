// Linears of a few activation rows, weights through registers; see gemm_reg.cu.
#pragma once

#include <type_traits>

#include "gemm_sk.cuh"

namespace b200 {
namespace tc {

constexpr int REG_MAX_M = 32;                // half of it for gated pairs
bool reg_wins(int M, int N, int epi, int gate_rows, bool i8, int sms);
bool reg_supported(int M, int epi, const void* x, long long ldx_bytes);
// x: bf16, or int8 with the scales of its rows (sa) and of the weight rows (sw); w_tiles as packed for gemm_sk.cu; ws / counters: zeroed counters, left zeroed
int reg_linear(const void* x, long long ldx_bytes, const void* w_tiles, __nv_bfloat16* y, long long ldy, const __nv_bfloat16* res, long long ldr, int M, int N,
               int K, int epi, int gate_rows, const float* sa, const float* sw, float* ws, size_t ws_bytes, int* counters, int n_counters, int sms, int pdl,
               cudaStream_t stream);

}  // namespace tc
}  // namespace b200
