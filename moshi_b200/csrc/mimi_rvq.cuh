// Residual VQ of a frame's latents, one launch per level (vq.py:269-287, core_vq.py:270-276, 507-519): codebooks of 256 dimensions, latents token-major.
//
// A level's search depends on the level before it only through one subtraction, so every CTA repeats the choice of the previous level for
// its eight queries (128 partial minima each) instead of waiting for a launch of its own, and a level's codebook rows, which depend on
// nothing, are requested before the wait on that launch.  A warp owns four codes, lanes own the dimensions, the 4 x 8 dot products
// meet in a transposing butterfly that leaves one per lane.  One query: 7 levels 160 us -> 35 us against a search that walked 256
// dimensions per thread on 16 CTAs and a choosing kernel after each.
#pragma once

#include "mimi_lin.cuh"

namespace b200 {
namespace mimi {

constexpr int RVL_CODES = 16, RVL_Q = 8, RVL_D = 256;

struct RvqStep {
  const float* res_in[2]; long long res_in_ld;   // [Q][res_in_ld]
  float* res_out[2];                             // [Q][RVL_D]: the residuals after the previous level
  const float *cb[2], *cnorm[2];                 // this level
  const float* cb_prev[2];
  float* best[2]; int* idx[2];                   // this level's minima [Q][n_chunks]
  const float* prev_best[2]; const int* prev_idx[2];
  int active[2], prev_active[2], prev_code[2];   // quantizer has this / the previous level; output codebook of the latter
  long long* codes; long long cs_b, cs_k;
  int n_query, bins, n_chunks;
};

// grid (n_chunks, queries / RVL_Q, 2), 128 threads
static __global__ void __launch_bounds__(128) rvq_level_kernel(const RvqStep a) {
  __shared__ float s_res[RVL_Q][RVL_D];
  __shared__ float s_best[4][RVL_Q];
  __shared__ int s_idx[4][RVL_Q];
  const int which = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q0 = blockIdx.y * RVL_Q;
  const bool active = a.active[which], chosen = a.prev_active[which];
  const int code0 = blockIdx.x * RVL_CODES + warp * 4;
  float4 c[4][2];
  if (active) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) c[j][e] = __ldg(reinterpret_cast<const float4*>(a.cb[which] + (long long)(code0 + j) * RVL_D + e * 128) + lane);
  }
  tcp::pdl_trigger();
  tcp::pdl_wait();
  if (!active && !(chosen && blockIdx.x == 0)) return;
  for (int r = warp; r < RVL_Q; r += 4) {
    const int q = q0 + r;
    float4 v[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
    if (q < a.n_query) {
      const float4* in = reinterpret_cast<const float4*>(a.res_in[which] + (long long)q * a.res_in_ld) + lane;
      v[0] = in[0]; v[1] = in[32];
      if (chosen) {
        float best = INFINITY;
        int bi = 0x7fffffff;
        for (int k = lane; k < a.n_chunks; k += 32) {
          const float ob = a.prev_best[which][(long long)q * a.n_chunks + k];
          const int oi = a.prev_idx[which][(long long)q * a.n_chunks + k];
          if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
          if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (bi >= a.bins) bi = 0;                // no minimum among the scores of a latent that is not a number
        const float4* p = reinterpret_cast<const float4*>(a.cb_prev[which] + (long long)bi * RVL_D) + lane;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float4 w = __ldg(p + 32 * e);
          v[e].x -= w.x; v[e].y -= w.y; v[e].z -= w.z; v[e].w -= w.w;
        }
        if (blockIdx.x == 0) {
          float4* out = reinterpret_cast<float4*>(a.res_out[which] + (long long)q * RVL_D) + lane;
          out[0] = v[0]; out[32] = v[1];
          if (lane == 0) a.codes[(long long)q * a.cs_b + a.prev_code[which] * a.cs_k] = bi;
        }
      }
    }
    reinterpret_cast<float4*>(s_res[r])[lane] = v[0];
    reinterpret_cast<float4*>(s_res[r])[lane + 32] = v[1];
  }
  __syncthreads();
  if (!active) return;
  float acc[4 * RVL_Q];
#pragma unroll
  for (int q = 0; q < RVL_Q; ++q) {
    const float4 x0 = reinterpret_cast<const float4*>(s_res[q])[lane], x1 = reinterpret_cast<const float4*>(s_res[q])[lane + 32];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float s = c[j][0].x * x0.x;
      s = fmaf(c[j][0].y, x0.y, s); s = fmaf(c[j][0].z, x0.z, s); s = fmaf(c[j][0].w, x0.w, s);
      s = fmaf(c[j][1].x, x1.x, s); s = fmaf(c[j][1].y, x1.y, s); s = fmaf(c[j][1].z, x1.z, s); s = fmaf(c[j][1].w, x1.w, s);
      acc[j * RVL_Q + q] = s;
    }
  }
  butterfly<4 * RVL_Q>(acc);                     // lane = (code, query)
  const int q = lane & 7;
  int bi = code0 + (lane >> 3);
  float best = a.cnorm[which][bi] - 2.f * acc[0];          // |c|^2 - 2 x.c  (core_vq.py:270-276 without the constant |x|^2)
  if (!(best == best)) { best = INFINITY; bi = 0x7fffffff; }
#pragma unroll
  for (int o = 8; o <= 16; o <<= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
  }
  if (lane < RVL_Q) { s_best[warp][q] = best; s_idx[warp][q] = bi; }
  __syncthreads();
  if (threadIdx.x < RVL_Q && q0 + (int)threadIdx.x < a.n_query) {
    best = s_best[0][threadIdx.x]; bi = s_idx[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < 4; ++w) {
      const float ob = s_best[w][threadIdx.x];
      const int oi = s_idx[w][threadIdx.x];
      if (ob < best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    a.best[which][(long long)(q0 + threadIdx.x) * a.n_chunks + blockIdx.x] = best;
    a.idx[which][(long long)(q0 + threadIdx.x) * a.n_chunks + blockIdx.x] = bi;
  }
}

// codes [B][K] -> the summed code vectors of both quantizers side by side, [B][2][RVL_D]; one CTA of 128 threads per session.  A code outside
// [0, bins) counts as the zero vector and raises the codec's error flag.
struct RvqGather {
  const long long* codes; long long cs_b, cs_k;
  const float* cb[2]; int levels[2], level_offset[2];
  float* out; int bins; int* err;
};
static __global__ void __launch_bounds__(128) rvq_gather_kernel(const RvqGather a) {
  tcp::pdl_trigger();
  tcp::pdl_wait();
  const int which = threadIdx.x >> 6, e = threadIdx.x & 63;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int l = 0; l < a.levels[which]; ++l) {
    const long long code = a.codes[blockIdx.x * a.cs_b + (a.level_offset[which] + l) * a.cs_k];
    if (code < 0 || code >= a.bins) {
      if (e == 0) atomicOr(a.err, B200_FLAG_CODE_RANGE);
      continue;
    }
    const float4 v = __ldg(reinterpret_cast<const float4*>(a.cb[which] + ((long long)l * a.bins + code) * RVL_D) + e);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  reinterpret_cast<float4*>(a.out)[(long long)blockIdx.x * 128 + threadIdx.x] = s;
}

}  // namespace mimi
}  // namespace b200
