// Linears of more than a few tokens in fp32 on the CUDA cores: mimi_lin_kernel's contract, for K = 512 n.
//
// mimi_lin_kernel keeps a warp's weights in registers and reads every token past them: 16 tokens of 4 outputs per warp cost 64 reads of shared memory and a
// butterfly of 64 sums, and 80 tokens of 512 -> 1536 took 12.4 us where the products are 1.7.  Here a CTA owns 8 RO outputs of 4 RT tokens, its 16 warps
// share k, and a lane owns RO x RT of them: a step of 4 k is RO + RT reads of 16 bytes for 2 RO RT packed FMAs (fma.rn.f32x2: even and odd k apart).
//   * weights and tokens lie in shared memory in rows of 512 + 4 floats, so that the eight rows (four tokens) of a read fall into different banks;
//   * the weights are asked for before the wait on the preceding kernel; for K > 512 the next 512 are under way while these are multiplied;
//   * the layer norm is done on the way into shared memory, one warp per token;
//   * the warps' sums meet in shared memory, in pairs, always the same: a result depends on no other token.
// Bound by latency: load, norm, products and exchange of a CTA follow one another; 64 tokens are 1.4 us of FMAs at their rate and 6.7 us here.  (mma.sync with tf32 parts
// is slower than the FMAs on this chip: 80 tokens of 512 -> 1536 with its three products 11.6 us.  With tokens' rows on tcgen05 a linear is two launches: mimi_tc.cu.)
// Encode + decode of a frame, before / with these tiles: 4 sessions (8 tokens) 903 / 824 us, 8 1127 / 874, 16 1262 / 1014, 32 1587 / 1259.
#pragma once

#include "mimi_lin.cuh"
#include "row_stream.cuh"

namespace b200 {
namespace mimi {

constexpr int TILE_K = 512, TILE_LD = TILE_K + 4, TILE_WARPS = 16;

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void lds_pairs(uint32_t at, uint64_t (&v)[2]) {
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(at));
}

// grid (N / (8 RO), tokens / (4 RT)); warp w has k in [32 w, 32 w + 32) of every 512
template <int RO, int RT>
__global__ void __launch_bounds__(32 * TILE_WARPS, 2) mimi_tile_kernel(const LinP p) {
  constexpr int NR = 8 * RO, NK = 4 * RT, STAGE = (NR + NK) * TILE_LD;
  extern __shared__ __align__(16) float sm[];    // per stage [NR][TILE_LD] weights, [NK][TILE_LD] tokens; at the end the warps' sums
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row0 = tid >> 7, piece = tid & 127;
  const int n0 = blockIdx.x * NR, tok0 = blockIdx.y * NK, chunks = p.K / TILE_K;
  const uint32_t base = tcp::smem_u32(sm);
  // a thread brings 16-byte piece `piece` of every fourth row
  auto ask_w = [&](int c) {
    const uint32_t to = base + ((c & 1) * STAGE + row0 * TILE_LD + piece * 4) * 4;
#pragma unroll
    for (int i = 0; i < NR / 4; ++i) rows::copy16(to + i * 4 * TILE_LD * 4, p.w + (long long)(n0 + i * 4 + row0) * p.K + c * TILE_K + piece * 4);
  };
  auto ask_x = [&](int c) {                      // tokens beyond the last repeat it; their results are not stored
    const uint32_t to = base + ((c & 1) * STAGE + (NR + row0) * TILE_LD + piece * 4) * 4;
#pragma unroll
    for (int i = 0; i < NK / 4; ++i) rows::copy16(to + i * 4 * TILE_LD * 4, p.x + (long long)min(tok0 + i * 4 + row0, p.n_tok - 1) * p.K + c * TILE_K + piece * 4);
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
  ask_w(0);
  if (chunks > 1) ask_w(1);
  commit();
  tcp::pdl_trigger();
  tcp::pdl_wait();
  if (p.gamma) {                                 // K == TILE_K (host)
    for (int t = warp; t < NK; t += TILE_WARPS) {
      const float* xr = p.x + (long long)min(tok0 + t, p.n_tok - 1) * TILE_K + lane * 4;
      float4 v[4];
      float s = 0.f, q = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = *reinterpret_cast<const float4*>(xr + c * 128);
#pragma unroll
      for (int c = 0; c < 4; ++c) s += (v[c].x + v[c].y) + (v[c].z + v[c].w);
      const float mean = warp_sum(s) / TILE_K;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        v[c].x -= mean; v[c].y -= mean; v[c].z -= mean; v[c].w -= mean;
        q += (v[c].x * v[c].x + v[c].y * v[c].y) + (v[c].z * v[c].z + v[c].w * v[c].w);
      }
      const float r = rsqrtf(warp_sum(q) / TILE_K + p.eps);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 g = __ldg(reinterpret_cast<const float4*>(p.gamma + c * 128 + lane * 4)), b = __ldg(reinterpret_cast<const float4*>(p.beta + c * 128 + lane * 4));
        *reinterpret_cast<float4*>(sm + (NR + t) * TILE_LD + c * 128 + lane * 4) =
            make_float4(v[c].x * r * g.x + b.x, v[c].y * r * g.y + b.y, v[c].z * r * g.z + b.z, v[c].w * r * g.w + b.w);
      }
    }
  } else {
    ask_x(0);
  }
  commit();
  if (chunks > 1) ask_x(1);
  commit();
  uint64_t acc[RO][RT];                          // sums over even k | over odd k
#pragma unroll
  for (int i = 0; i < RO; ++i)
#pragma unroll
    for (int j = 0; j < RT; ++j) acc[i][j] = 0ull;
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // all but the newest group: stage c is here
    __syncthreads();
    const uint32_t st = base + (c & 1) * STAGE * 4, wp = st + ((lane >> 2) * TILE_LD + warp * 32) * 4, xp = st + ((NR + (lane & 3)) * TILE_LD + warp * 32) * 4;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      uint64_t x[RT][2];
#pragma unroll
      for (int j = 0; j < RT; ++j) lds_pairs(xp + (j * 4 * TILE_LD + s * 4) * 4, x[j]);
#pragma unroll
      for (int i = 0; i < RO; ++i) {
        uint64_t w[2];
        lds_pairs(wp + (i * 8 * TILE_LD + s * 4) * 4, w);
#pragma unroll
        for (int j = 0; j < RT; ++j) { fma2(acc[i][j], w[0], x[j][0]); fma2(acc[i][j], w[1], x[j][1]); }
      }
    }
    __syncthreads();
    if (c + 2 < chunks) { ask_x(c + 2); ask_w(c + 2); }
    commit();
  }
  float* red = sm;                               // [warp][i][j][lane]
#pragma unroll
  for (int i = 0; i < RO; ++i)
#pragma unroll
    for (int j = 0; j < RT; ++j)
      red[((warp * RO + i) * RT + j) * 32 + lane] = __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
  __syncthreads();
  for (int o = tid; o < 32 * RO * RT; o += 32 * TILE_WARPS) {
    const int l = o & 31, i = (o >> 5) / RT, j = (o >> 5) - i * RT, n = n0 + i * 8 + (l >> 2), tok = tok0 + j * 4 + (l & 3);
    if (tok >= p.n_tok) continue;
    float s[TILE_WARPS];
#pragma unroll
    for (int w = 0; w < TILE_WARPS; ++w) s[w] = red[w * (32 * RO * RT) + o];
#pragma unroll
    for (int d = TILE_WARPS / 2; d > 0; d >>= 1)
#pragma unroll
      for (int w = 0; w < d; ++w) s[w] += s[w + d];
    lin_result(p, tok, n, s[0]);
  }
}

template <int RO, int RT>
int tile_launch_one(const LinP& p, cudaStream_t st, bool early) {
  constexpr int STAGE_BYTES = (8 * RO + 4 * RT) * TILE_LD * 4;
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, 2 * STAGE_BYTES, mimi_tile_kernel<RO, RT>));
  return launch_early_if(early, mimi_tile_kernel<RO, RT>, dim3((unsigned)(p.N / (8 * RO)), (unsigned)ceil_div(p.n_tok, 4 * RT)), dim3(32 * TILE_WARPS),
                         p.K > TILE_K ? 2 * STAGE_BYTES : STAGE_BYTES, st, p);
}

// Times in us, one launch behind the other with cold weights, mimi_lin_kernel / this kernel (its token tile):
//   512 -> 1536 (norm): 2 tokens 2.82 / 2.87 (4), 4 3.36 / 2.67 (4), 8 4.35 / 3.09 (4), 16 6.2 / 4.2 (4), 32 6.6 / 5.0 (8), 64 12.1 / 6.7 (12)
//   512 -> 2048 (norm): 2 tokens 2.75 / 3.07, 4 3.70 / 3.06, 8 4.44 / 3.44, 16 6.2 / 4.5, 32 6.6 / 5.8, 64 12.4 / 7.7
//   512 -> 512: 4 tokens 1.7 / 2.2, 8 2.1 / 2.4, 16 3.3 / 2.6, 32 3.3 / 3.1, 64 4.2 / 3.9
//   2048 -> 512, mimi_lin_kernel with 512 k at a time and 8 or 16 tokens per CTA as it was / as many k as fit / this kernel: 8 tokens 6.3 / 4.6 / 6.4,
//   16 9.8 / 4.9 / 6.5, 32 13.0 / 5.7 / 7.4, 48 13.2 / - / 9.1, 64 13.4 / 10.8 / 9.4
// Here the smallest token tile is the best one with which the CTAs fit the chip together, two to an SM (one with two stages).
// early: the launch may begin under the preceding kernel, which does not write the weights
inline int lin_launch(const LinP& p, int sms, cudaStream_t st, bool early = mtc::tc_pdl()) {
  if (p.K % 2048 == 0 && !p.gamma) {
    if (p.n_tok <= 2) return lin_launch_one<1, 2, 16>(p, st, early);
    if (p.n_tok <= 4) return lin_launch_one<1, 4, 16>(p, st, early);
    if (p.n_tok <= 16) return lin_launch_one<1, 8, 16>(p, st, early);
    if (p.n_tok <= 32) return lin_launch_one<2, 8, 8>(p, st, early);
  } else if (p.n_tok <= 2) {
    return lin_launch_one<1, 2, 4>(p, st, early);
  } else if (p.n_tok <= 8 && p.N <= 4 * sms) {   // one output per warp, one CTA per SM
    return p.n_tok <= 4 ? lin_launch_one<1, 4, 4>(p, st, early) : lin_launch_one<2, 8, 4>(p, st, early);
  }
  const int wide = p.N / 32, room = p.K > TILE_K ? sms : 2 * sms;
  if (p.N % 32) return tile_launch_one<2, 4>(p, st, early);
  if (p.n_tok <= 4) return tile_launch_one<2, 1>(p, st, early);
  if (wide * ceil_div(p.n_tok, 4) <= room) return tile_launch_one<4, 1>(p, st, early);
  if (wide * ceil_div(p.n_tok, 8) <= room) return tile_launch_one<4, 2>(p, st, early);
  if (wide * ceil_div(p.n_tok, 12) <= room) return tile_launch_one<4, 3>(p, st, early);
  return tile_launch_one<4, 4>(p, st, early);
}

}  // namespace mimi
}  // namespace b200
