// The linears and the attention of Mimi's bottleneck transformers in fp32 on the CUDA cores (transformer.py:752-777, 557-597).
//
// A frame brings two tokens per session and layer: what a layer costs is the chain of its launches, not its products.  A launch
// of mimi_tc_kernel takes about 6 us whether there are 2 tokens or 80, a layer is four of them, two layer norms and an attention.  Here a
// layer is five launches of 2 to 3:
//   mimi_lin_kernel: a warp owns NO outputs for TOK tokens.  Its weights (fp32, row-major) are requested before the wait on the
//     preceding kernel (programmatic dependent launch), up to 2048 elements per output at a time; every CTA brings the tokens' rows into
//     shared memory, normed in front of in_proj and linear1; lanes own k, their sums meet in a transposing butterfly that leaves each
//     lane one output; epilogues as in mimi_tc.cu (GELU, residual + layer scale, hi / lo parts for a convolution behind).  Up to two tokens everywhere;
//     with more of them most linears take mimi_tile.cuh.
//   mimi_attn_kernel: a half-warp per key, keys and values of four keys in flight, running maximum; the eight half-warps meet in
//     shared memory.
#pragma once

#include "common.cuh"
#include "mimi_tc.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace mimi {

enum { LIN_STORE = 0, LIN_GELU = 1, LIN_RESIDUAL = 2 };

struct LinP {
  const float* x;                                // rows [n_tok][K]
  const float *gamma, *beta;                     // layer norm of the rows (null: none)
  const float* w;                                // [N][K]
  int n_tok, N, K, T, epi;                       // T: tokens per session
  float* y;                                      // [n_tok][N] (null: not stored)
  const float *res, *scale;                      // LIN_RESIDUAL: y = res + scale * .
  float *a_hi, *a_lo; long long a_sb, a_row; int a_elu;      // hi / lo parts of the result at session * a_sb + step * a_row + n (null: none)
  float eps;
};

__device__ __forceinline__ void lin_result(const LinP& p, int tok, int n, float v) {
  if (p.epi == LIN_GELU) v = gelu_erf(v);
  else if (p.epi == LIN_RESIDUAL) v = p.res[(long long)tok * p.N + n] + p.scale[n] * v;
  if (p.y) p.y[(long long)tok * p.N + n] = v;
  if (p.a_hi) {
    float hi, lo;
    mtc::split_tf32(p.a_elu ? elu1(v) : v, hi, lo);
    const int b = tok / p.T;
    const long long at = (long long)b * p.a_sb + (long long)(tok - b * p.T) * p.a_row + n;
    p.a_hi[at] = hi;
    p.a_lo[at] = lo;
  }
}

// lanes hold V partial sums each; afterwards a lane holds the totals of R = max(1, V / 32) of them: values index * R .. index * R + R - 1, with
// index made of the leading lane bits
template <int V>
__device__ __forceinline__ int butterfly(float (&v)[V]) {
  const int lane = threadIdx.x & 31;
  int n = V, index = 0;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    if (n > 1) {
      const bool upper = lane & m;
      n >>= 1;
      index = index * 2 + (upper ? 1 : 0);
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (i < n) {
          const float send = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
    }
  }
  return index;
}

// 4 warps; KC = K / 128 of a chunk (all of K where it fits); grid (N / (4 NO), tokens / TOK)
template <int NO, int TOK, int KC>
__global__ void __launch_bounds__(128) mimi_lin_kernel(const LinP p) {
  constexpr int CH = KC * 128;
  extern __shared__ __align__(16) float xs[];    // [TOK][CH]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 4 + warp) * NO, tok0 = blockIdx.y * TOK, nt = min(TOK, p.n_tok - tok0);
  const float* wr = p.w + (long long)n0 * p.K + lane * 4;
  float4 w[NO][KC];
#pragma unroll
  for (int o = 0; o < NO; ++o)
#pragma unroll
    for (int c = 0; c < KC; ++c) w[o][c] = __ldg(reinterpret_cast<const float4*>(wr + (long long)o * p.K + c * 128));
  tcp::pdl_trigger();
  tcp::pdl_wait();
  float acc[NO * TOK];
#pragma unroll
  for (int i = 0; i < NO * TOK; ++i) acc[i] = 0.f;
  for (int k0 = 0; k0 < p.K; k0 += CH) {
    if (k0 > 0) __syncthreads();
    for (int t = warp; t < TOK; t += 4) {
      float4 v[KC];
      const float* xr = p.x + (long long)(tok0 + t) * p.K + k0 + lane * 4;
#pragma unroll
      for (int c = 0; c < KC; ++c) {
        v[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < nt) {
          v[c] = *reinterpret_cast<const float4*>(xr + c * 128);
        }
      }
      if (p.gamma) {                             // the whole row is here (host: K == CH)
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int c = 0; c < KC; ++c) s += (v[c].x + v[c].y) + (v[c].z + v[c].w);
        const float mean = warp_sum(s) / CH;
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          v[c].x -= mean; v[c].y -= mean; v[c].z -= mean; v[c].w -= mean;
          q += (v[c].x * v[c].x + v[c].y * v[c].y) + (v[c].z * v[c].z + v[c].w * v[c].w);
        }
        const float r = rsqrtf(warp_sum(q) / CH + p.eps);
#pragma unroll
        for (int c = 0; c < KC; ++c) {
          const float4 g = __ldg(reinterpret_cast<const float4*>(p.gamma + c * 128 + lane * 4)), b = __ldg(reinterpret_cast<const float4*>(p.beta + c * 128 + lane * 4));
          v[c] = make_float4(v[c].x * r * g.x + b.x, v[c].y * r * g.y + b.y, v[c].z * r * g.z + b.z, v[c].w * r * g.w + b.w);
        }
      }
#pragma unroll
      for (int c = 0; c < KC; ++c) *reinterpret_cast<float4*>(xs + t * CH + c * 128 + lane * 4) = v[c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < KC; ++c) {
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + t * CH + c * 128 + lane * 4);
#pragma unroll
        for (int o = 0; o < NO; ++o) {
          float& a = acc[t * NO + o];
          a = fmaf(w[o][c].x, xv.x, a); a = fmaf(w[o][c].y, xv.y, a); a = fmaf(w[o][c].z, xv.z, a); a = fmaf(w[o][c].w, xv.w, a);
        }
      }
      if (k0 + CH < p.K) {
#pragma unroll
        for (int o = 0; o < NO; ++o) w[o][c] = __ldg(reinterpret_cast<const float4*>(wr + (long long)o * p.K + k0 + CH + c * 128));
      }
    }
  }
  constexpr int V = NO * TOK, R = V > 32 ? V / 32 : 1, COPIES = V >= 32 ? 1 : 32 / V;
  const int index = butterfly<V>(acc);
  if (COPIES > 1 && (lane & (COPIES - 1))) return;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = index * R + r, t = i / NO, n = n0 + i - t * NO;
    if (t < nt) lin_result(p, tok0 + t, n, acc[r]);
  }
}

inline bool lin_takes(int N, int K) { return K % 512 == 0 && N % 16 == 0; }

// The row-major weights are held only while a batch small enough for mimi_lin_kernel streams: 201 MB that a full server has no use for, an
// eighth of a session's rings.  They come back from the packed hi / lo tiles (mimi_tc.cu) bit for bit: hi is the weight rounded to 11
// significant bits, so the remainder r = w - hi is exact and has at most 12, and lo is r rounded away from zero at the 11th; all that is
// lost is whether the 12th was set.  In the encoding of a float that rounding adds bit 12 to r where r has it; that bit is kept, one
// per weight (6.3 MB), and taken off again.  Only the sign of a zero, and weights below 2^-100, where r is no normal number, may differ.
static __global__ void __launch_bounds__(256) lin_lost_bits_kernel(const float* w, uint32_t* bits) {      // grid N * K / 256
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const float v = w[i];
  float hi, lo;
  mtc::split_tf32(v, hi, lo);
  const uint32_t word = __ballot_sync(0xffffffffu, (__float_as_uint(v - hi) >> 12) & 1u);
  if ((threadIdx.x & 31) == 0) bits[i >> 5] = word;
}
static __global__ void __launch_bounds__(256) lin_rows_kernel(const float* tiles, const uint32_t* bits, float* rows, int K, int NT) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const int n = (int)(i / K), k = (int)(i - (long long)n * K), r = n % NT;
  // 16-byte piece c of a tile row lies at position c ^ (row & 7); the lo tile follows the hi tile of its k-block
  const long long o = (((long long)(n / NT) * (K / mtc::TC_KB) + k / mtc::TC_KB) * 2 * NT + r) * mtc::TC_KB + ((((k & 31) >> 2) ^ (r & 7)) << 2) + (k & 3);
  const uint32_t lost = (bits[i >> 5] >> (i & 31)) & 1u;
  rows[i] = tiles[o] + __uint_as_float(__float_as_uint(tiles[o + (long long)NT * mtc::TC_KB]) - (lost << 12));
}
inline size_t lin_lost_words(int N, int K) { return (size_t)N * K / 32; }
inline int lin_lost_bits(const float* w, uint32_t* bits, int N, int K, cudaStream_t st) {
  B200_LAUNCH(lin_lost_bits_kernel, (unsigned)((long long)N * K / 256), 256, 0, st, w, bits);
  return check_launch("lin_lost_bits");
}
inline int lin_rows(const uint8_t* tiles, const uint32_t* bits, float* rows, int N, int K, int NT, cudaStream_t st) {
  B200_LAUNCH(lin_rows_kernel, (unsigned)((long long)N * K / 256), 256, 0, st, reinterpret_cast<const float*>(tiles), bits, rows, K, NT);
  return check_launch("lin_rows");
}

template <int NO, int TOK, int KC>
int lin_launch_one(const LinP& p, cudaStream_t st, bool early) {
  constexpr int SMEM = TOK * KC * 128 * 4;
  if constexpr (SMEM > 48 * 1024) {
    static std::atomic<uint64_t> limits{0};
    B200_TRY(allow_smem(limits, SMEM, mimi_lin_kernel<NO, TOK, KC>));
  }
  return launch_early_if(early, mimi_lin_kernel<NO, TOK, KC>, dim3((unsigned)(p.N / (4 * NO)), (unsigned)ceil_div(p.n_tok, TOK)), dim3(128), SMEM, st, p);
}

// One attention step of T <= 4 tokens per session: RoPE (rope.py:45-82), ring append for executing sessions, attention over the ring under
// the causal / context mask (transformer.py:247-286, 557-597) -> [n_tok][C].  Head size 64, one CTA per (session, head).
struct MimiAttn {
  const float* qkv; float *kc, *vc, *out, *out_lo;      // out_lo: the result as a hi / lo pair (null: out alone, in full)
  const long long* offset; const uint8_t* exec_mask;
  int H, cap, context; float neg_log_period_2_over_d;
};
template <int T>
__global__ void __launch_bounds__(128) mimi_attn_kernel(const MimiAttn p) {
  constexpr int D = 64, U = 4;                   // U keys per half-warp in flight
  __shared__ float sq[T][D];
  __shared__ float sm[8][T], sl[8][T], so[8][T][D];
  tcp::pdl_trigger();
  tcp::pdl_wait();
  const int b = blockIdx.x / p.H, h = blockIdx.x - b * p.H, C = p.H * D, tid = threadIdx.x;
  const long long off = p.offset[b];
  const bool exec = p.exec_mask[b] != 0;
  float* kb = p.kc + ((long long)b * p.H + h) * p.cap * D;
  float* vb = p.vc + ((long long)b * p.H + h) * p.cap * D;
  for (int i = tid; i < T * (D / 2); i += 128) {
    const int t = i / (D / 2), pr = i - t * (D / 2);
    float sn, cs;
    sincosf(expf((float)pr * p.neg_log_period_2_over_d) * ((float)off + (float)t), &sn, &cs);
    const float* base = p.qkv + ((long long)b * T + t) * 3 * C + h * D + 2 * pr;
    const float2 q = *reinterpret_cast<const float2*>(base), k = *reinterpret_cast<const float2*>(base + C), v = *reinterpret_cast<const float2*>(base + 2 * C);
    sq[t][2 * pr] = q.x * cs - q.y * sn;
    sq[t][2 * pr + 1] = q.x * sn + q.y * cs;
    if (exec) {
      const int slot = (int)((off + t) % p.cap);
      const float2 kr = make_float2(k.x * cs - k.y * sn, k.x * sn + k.y * cs);
      *reinterpret_cast<float2*>(kb + (long long)slot * D + 2 * pr) = kr;
      *reinterpret_cast<float2*>(vb + (long long)slot * D + 2 * pr) = v;
    }
  }
  __syncthreads();
  const long long end_after = exec ? off + T : off, last = off + T - 1;
  const int end_index = (int)(last % p.cap), n_keys = (int)min((long long)p.cap, end_after);
  const int hw = tid >> 4, l = tid & 15;
  const float scale = rsqrtf((float)D);
  float4 q[T], o[T];
  float m[T], sum[T];
#pragma unroll
  for (int t = 0; t < T; ++t) {
    q[t] = *reinterpret_cast<const float4*>(&sq[t][4 * l]);
    o[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    m[t] = -INFINITY; sum[t] = 0.f;
  }
  for (int base = 0; base < n_keys; base += 8 * U) {      // the same count for both halves of a warp
    const int s0 = base + hw;
    float4 k[U], v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = min(s0 + 8 * u, n_keys - 1);
      k[u] = *reinterpret_cast<const float4*>(kb + (long long)s * D + 4 * l);
      v[u] = *reinterpret_cast<const float4*>(vb + (long long)s * D + 4 * l);
    }
    float sc[U][T];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int t = 0; t < T; ++t) sc[u][t] = q[t].x * k[u].x + q[t].y * k[u].y + q[t].z * k[u].z + q[t].w * k[u].w;
#pragma unroll
    for (int d = 8; d > 0; d >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int t = 0; t < T; ++t) sc[u][t] += __shfl_xor_sync(0xffffffffu, sc[u][t], d);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      float mx = m[t];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int s = s0 + 8 * u, delta = s - end_index;
        const long long pos = delta <= 0 ? last + delta : last + delta - p.cap, back = off + t - pos;
        sc[u][t] = s < n_keys && pos >= 0 && back >= 0 && back < p.context ? sc[u][t] * scale : -INFINITY;      // transformer.py:576-580
        mx = fmaxf(mx, sc[u][t]);
      }
      if (mx == -INFINITY) continue;
      const float f = expf(m[t] - mx);
      m[t] = mx;
      sum[t] *= f; o[t].x *= f; o[t].y *= f; o[t].z *= f; o[t].w *= f;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float e = expf(sc[u][t] - mx);
        sum[t] += e;
        o[t].x = fmaf(e, v[u].x, o[t].x); o[t].y = fmaf(e, v[u].y, o[t].y); o[t].z = fmaf(e, v[u].z, o[t].z); o[t].w = fmaf(e, v[u].w, o[t].w);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < T; ++t) {
    if (l == 0) { sm[hw][t] = m[t]; sl[hw][t] = sum[t]; }
    *reinterpret_cast<float4*>(&so[hw][t][4 * l]) = o[t];
  }
  __syncthreads();
  for (int i = tid; i < T * D; i += 128) {
    const int t = i / D, d = i - t * D;
    float mx = -INFINITY, den = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = fmaxf(mx, sm[w][t]);
    if (mx > -INFINITY) {
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float f = expf(sm[w][t] - mx);
        den += f * sl[w][t];
        a = fmaf(f, so[w][t][d], a);
      }
    }
    const long long o = ((long long)b * T + t) * C + h * D + d;
    const float v = den > 0.f ? a / den : 0.f;
    if (p.out_lo) mtc::split_tf32(v, p.out[o], p.out_lo[o]);
    else p.out[o] = v;
  }
}

template <int T>
int attn_launch_one(const MimiAttn& p, int B, cudaStream_t st) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(B * p.H)); cfg.blockDim = dim3(128); cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = mtc::tc_pdl() ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, mimi_attn_kernel<T>, p);
  if (e != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "mimi_attn launch failed: %s", cudaGetErrorString(e));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200_OK;
}

inline int attn_launch(const MimiAttn& p, int B, int T, cudaStream_t st) {
  switch (T) {
    case 1: return attn_launch_one<1>(p, B, st);
    case 2: return attn_launch_one<2>(p, B, st);
    case 3: return attn_launch_one<3>(p, B, st);
    default: return attn_launch_one<4>(p, B, st);
  }
}

}  // namespace mimi
}  // namespace b200
