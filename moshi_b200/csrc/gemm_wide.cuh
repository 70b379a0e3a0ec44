// Tensor-core GEMM for many activation rows and for grouped (routed expert) products; see gemm_wide.cu.
#pragma once

#include "gemm_sk.cuh"

namespace b200 {
namespace tc {

enum { WIDE_STORE = 0, WIDE_RELU2 = 1, WIDE_CLAMPED_GLU = 2, WIDE_SILU_GLU = 3, WIDE_GELU = 4 };      // what happens to the sums; the GLUs halve the columns
constexpr int WIDE_ERR_WAIT = 2;             // bit raised in *err when a wait inside the kernel ran out
constexpr int WIDE_EXPERT_ROWS = 128;        // rows per tile of a grouped product's table

struct WideGemm {
  const __nv_bfloat16* x = nullptr; long long ldx = 0; long long x_rows = 0;      // [x_rows][K]
  const void* w = nullptr; bool packed = false; long long w_rows = 0;             // packed tiles (gemm_sk.cu) or row-major [w_rows][K]
  __nv_bfloat16* y = nullptr; long long ldy = 0;
  int M = 0, N = 0, K = 0;                   // N: weight rows (of one expert)
  int act = WIDE_STORE; float limit = 0.f;
  // columns [act_from, act_to), both multiples of 32, go through relu(.)^2 to y2 instead (act_to = 0: none; WIDE_STORE only)
  int act_from = 0, act_to = 0; __nv_bfloat16* y2 = nullptr; long long ldy2 = 0;
  // grouped product: tiles of up to WIDE_EXPERT_ROWS neighbouring rows of one expert, listed on the device; at most max_tiles of them
  const int *tile_e = nullptr, *tile_r0 = nullptr, *tile_n = nullptr, *n_tiles = nullptr, *y_rows = nullptr;
  int max_tiles = 0, e_rows = 0, max_rows = 0;      // max_rows: no expert has more (0: unknown)
  int* err = nullptr;
  // k cut into ranges whose partial sums meet in ws: 0 = where the tiles leave SMs idle; needs zeroed arrival counters, left zeroed
  int splits = 0;
  float* ws = nullptr; size_t ws_bytes = 0; int* counters = nullptr; int n_counters = 0;
};
bool wide_supported(const WideGemm& g);
int wide_gemm(const WideGemm& g, cudaStream_t st);

}  // namespace tc
}  // namespace b200
