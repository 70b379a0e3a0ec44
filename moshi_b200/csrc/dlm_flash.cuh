// Causal attention of a prompt portion on keys and values per head; see dlm_flash.cu.
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace b200 {
namespace dlm {

constexpr int FLASH_D = 128;                 // query / key and value size per head
struct FlashAttn {
  const __nv_bfloat16* q; long long ldq;     // [T][ldq], head h at h * FLASH_D
  const __nv_bfloat16* k; long long ldk;     // [pos0 + T][ldk], head h at h * FLASH_D
  const __nv_bfloat16* vt; long long ldv;    // [H * FLASH_D][ldv]: values transposed, a column per key
  const float* sink;                         // [H] logits that stand in the denominator beside the keys (null: none)
  __nv_bfloat16* out; long long ldo;         // [T][ldo], head h at h * FLASH_D
  int T, pos0, H;                            // query t sits at position pos0 + t and sees keys 0 .. pos0 + t
  float scale;
  int* err;                                  // gets FLASH_ERR_WAIT when a wait inside the kernel ran out (may be null)
};
constexpr int FLASH_ERR_WAIT = 2;
bool flash_supported(const FlashAttn& a);
int flash_attention(const FlashAttn& a, cudaStream_t st);

}  // namespace dlm
}  // namespace b200
