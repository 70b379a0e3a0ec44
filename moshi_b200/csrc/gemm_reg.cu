// Linears of up to 32 activation rows with the weights going through registers:  y[M][N] = epi(x[M][K] . w[N][K]^T), same packed tiles, epilogues and
// cast points as gemm_sk.cu; bf16, and int8 with int32 sums.
//
// With so few rows a linear is a stream of its weights, and what counts is how many bytes of them are under way.  The bulk-copy engine that
// feeds tcgen05 tops out near 36 GB/s per SM (5.3 TB/s); plain 16-byte loads do not (the attention kernel reads 7 TB/s with them).  So a
// thread loads 16-byte pieces of the tiles straight into the A fragments of mma.sync (m16n8k16; int8 m16n8k32): which k a fragment slot holds
// does not matter as long as the activations' fragment agrees, so the thread (g, t) of a warp takes piece t and piece t + 4 of rows g and
// g + 8, every piece serving two products, and the same pieces of row g of x are the B fragments.  A warp owns 16 rows of a tile (of both
// tiles of a gated pair), eight warps a tile; DEPTH k-blocks of weights are in flight per thread and the first ones are requested before
// the wait on the preceding kernel.  Where tiles are few, k is cut; the CTA that arrives last adds the ranges in order.
//
// Against the tcgen05 stream-K kernel of gemm_sk.cu: gated 4096 -> 11264, 6 rows 44.8 -> 33.3 us (185 MB of weights, 28 us at the measured copy rate); a width-2048 decoder
// layer's linears at 8 rows 26 -> 18.6 us each.  From 17 rows on gemm_ns.cu has k of 4096 and more (24 rows: 4096 -> 12288 28.0 us here,
// 19.9 there) but for few tiles of long k, whose ranges are more here, and results off a 16-byte border; shorter k stays here.
#include <algorithm>

#include "gemm_reg.cuh"
#include "row_stream.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace tc {

namespace {

using namespace tcp;
using namespace rows;

constexpr int EPI_STORE = 0, EPI_RESADD = 1, EPI_GATE = 2;
constexpr int THREADS = 256, ROWS = 128, TILE16 = 1024;      // 16-byte pieces of a tile (128 rows x 128 bytes)

struct RegP {
  int M, N, out_rows, n_tiles, num_kb, S, kbps;
  long long row_bytes;                    // bytes of x per row that exist (K elements)
  const uint4* wt;
  const uint8_t* x; long long ldx;        // bytes
  __nv_bfloat16* y; long long ldy;
  const __nv_bfloat16* res; long long ldr;
  const float *sa, *sw;                   // int8: scales of activation and weight rows
  int late;                               // nothing is read before the wait on the preceding kernel
  float* ws; int* counters;               // partial sums [tile][split][A][8 NT][128], arrivals per tile
};

__device__ __forceinline__ float rbf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// Not ld.global.nc: that promises weights that nobody writes while the kernel runs, and one that was launched early runs beside the kernel in front, which
// may be writing them; such a load may move above the wait.
__device__ __forceinline__ uint4 ldg_stream(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int EPI, bool I8>
__device__ __forceinline__ void finish(const RegP& p, int m, int n, float a, float b) {
  if constexpr (I8) {                     // the sums are whole numbers in 32 bits
    const float s = p.sa[m];
    a = (float)__float_as_int(a) * (s * p.sw[n] * (1.f / 16129.f));
    if (EPI == EPI_GATE) b = (float)__float_as_int(b) * (s * p.sw[n + p.out_rows] * (1.f / 16129.f));
  }
  float v;
  if (EPI == EPI_STORE) v = a;
  else if (EPI == EPI_RESADD) v = __bfloat162float(p.res[(long long)m * p.ldr + n]) + rbf16(a);
  else { const float g = rbf16(a), u = rbf16(b); v = rbf16(g / (1.f + expf(-g))) * u; }
  p.y[(long long)m * p.ldy + n] = __float2bfloat16_rn(v);
}

constexpr int CTAS_PER_SM = 2;             // 128 registers per thread

template <int EPI, int NT, bool I8>
__global__ void __launch_bounds__(THREADS, CTAS_PER_SM) gemm_reg_kernel(const RegP p) {
  using Acc = typename std::conditional<I8, int, float>::type;
  constexpr int A = EPI == EPI_GATE ? 2 : 1, DEPTH = A == 2 ? 2 : NT == 4 ? 3 : 4;
  __shared__ int arrived;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tile = blockIdx.x / p.S, sp = blockIdx.x - tile * p.S;
  const int kb0 = sp * p.kbps, n_kb = min(p.num_kb, kb0 + p.kbps) - kb0;
  // piece c of row r lies at position c ^ (r & 7) of the row; rows g and g + 8 of the warp's 16 share r & 7 = g
  const uint4* wrow = p.wt + ((size_t)tile * p.num_kb + kb0) * (A * TILE16) + (warp * 16 + g) * 8;
  const int c0 = t ^ g, c1 = (t + 4) ^ g;
  if (p.late) pdl_wait();
  uint4 w[DEPTH][A][4];
  auto load_w = [&](int i, uint4 (&d)[A][4]) {
    const uint4* s = wrow + (size_t)i * (A * TILE16);
#pragma unroll
    for (int a = 0; a < A; ++a) {
      d[a][0] = ldg_stream(s + a * TILE16 + c0);
      d[a][1] = ldg_stream(s + a * TILE16 + 64 + c0);
      d[a][2] = ldg_stream(s + a * TILE16 + c1);
      d[a][3] = ldg_stream(s + a * TILE16 + 64 + c1);
    }
  };
#pragma unroll
  for (int i = 0; i < DEPTH; ++i)
    if (i < n_kb) load_w(i, w[i]);
  pdl_trigger();
  pdl_wait();
  // rows of x: token 8 j + g (the last row again where there is none: its sums are dropped)
  const uint8_t* xr[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) xr[j] = p.x + (long long)min(8 * j + g, p.M - 1) * p.ldx;
  uint4 xb[2][NT];                        // pieces t, then pieces t + 4 of a k-block
  auto load_x = [&](int i, int h, uint4 (&d)[NT]) {
    const long long k = (long long)(kb0 + i) * 128 + h * 64 + t * 16;
#pragma unroll
    for (int j = 0; j < NT; ++j) d[j] = k < p.row_bytes ? *reinterpret_cast<const uint4*>(xr[j] + k) : make_uint4(0u, 0u, 0u, 0u);
  };
  Acc acc[A][NT][4];
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[a][j][0] = acc[a][j][1] = acc[a][j][2] = acc[a][j][3] = 0;
  if (n_kb > 0) { load_x(0, 0, xb[0]); load_x(0, 1, xb[1]); }
  for (int i0 = 0; i0 < n_kb; i0 += DEPTH) {
#pragma unroll
    for (int r = 0; r < DEPTH; ++r) {
      const int i = i0 + r;
      if (i < n_kb) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int a = 0; a < A; ++a) {
            const uint4 lo = w[r][a][2 * h], hi = w[r][a][2 * h + 1];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              mma_step(acc[a][j], lo.x, hi.x, lo.y, hi.y, xb[h][j].x, xb[h][j].y);
              mma_step(acc[a][j], lo.z, hi.z, lo.w, hi.w, xb[h][j].z, xb[h][j].w);
            }
          }
          if (i + 1 < n_kb) load_x(i + 1, h, xb[h]);
        }
        if (i + DEPTH < n_kb) load_w(i + DEPTH, w[r]);
      }
    }
  }
  const int row = warp * 16 + g;          // and row + 8
  auto bits = [](Acc v) { if constexpr (I8) return __int_as_float(v); else return v; };
  if (p.S == 1) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 8 * j + 2 * t + (e & 1), n = tile * ROWS + row + (e >> 1) * 8;
        if (m < p.M && n < p.out_rows) finish<EPI, I8>(p, m, n, bits(acc[0][j][e]), bits(acc[A - 1][j][e]));
      }
    return;
  }
  constexpr int SLOT = A * 8 * NT * ROWS;
  float* slot = p.ws + ((size_t)tile * p.S + sp) * SLOT;
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 8 * j + 2 * t + (e & 1);
        if (m < p.M) __stcg(slot + (a * 8 * NT + m) * ROWS + row + (e >> 1) * 8, bits(acc[a][j][e]));
      }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    arrived = atomicAdd(p.counters + tile, 1);
    if (arrived == p.S - 1) p.counters[tile] = 0;
    __threadfence();
  }
  __syncthreads();
  if (arrived != p.S - 1) return;
  // four neighbouring rows of one token per thread, eight ranges' loads in flight
  const float4* part = reinterpret_cast<const float4*>(p.ws + (size_t)tile * p.S * SLOT);
  for (int i = threadIdx.x; i < p.M * (ROWS / 4); i += THREADS) {
    const int m = i / (ROWS / 4), r4 = i - m * (ROWS / 4);
    Acc v[2][4];
#pragma unroll
    for (int a = 0; a < A; ++a) {
      v[a][0] = v[a][1] = v[a][2] = v[a][3] = 0;
      const float4* q = part + (a * 8 * NT + m) * (ROWS / 4) + r4;
      for (int s0 = 0; s0 < p.S; s0 += 8) {
        float4 f[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (s0 + u < p.S) f[u] = __ldcg(q + (size_t)(s0 + u) * (SLOT / 4));
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (s0 + u >= p.S) break;
          if constexpr (I8) {
            v[a][0] += __float_as_int(f[u].x); v[a][1] += __float_as_int(f[u].y); v[a][2] += __float_as_int(f[u].z); v[a][3] += __float_as_int(f[u].w);
          } else {
            v[a][0] += f[u].x; v[a][1] += f[u].y; v[a][2] += f[u].z; v[a][3] += f[u].w;
          }
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int n = tile * ROWS + r4 * 4 + e;
      if (n < p.out_rows) finish<EPI, I8>(p, m, n, bits(v[0][e]), bits(v[A - 1][e]));
    }
  }
}

template <int EPI, bool I8>
cudaError_t launch_nt(const cudaLaunchConfig_t& cfg, const RegP& p) {
  if (p.M <= 8) return cudaLaunchKernelEx(&cfg, gemm_reg_kernel<EPI, 1, I8>, p);
  if (p.M <= 16) return cudaLaunchKernelEx(&cfg, gemm_reg_kernel<EPI, 2, I8>, p);
  if constexpr (EPI == EPI_GATE) return cudaErrorInvalidValue;      // not supported (reg_supported)
  else return cudaLaunchKernelEx(&cfg, gemm_reg_kernel<EPI, 4, I8>, p);
}

}  // namespace

// Where the kernel is ahead of gemm_sk.cu, asked where gemm_row.cu does not take the shape: 17 to 32 rows, and 16-bit gated pairs of up to 16 rows that it leaves (fewer
// rows come here through b200_op_linear_reg and B200_ROW_MAX_M only).  7B shapes, bf16, us: up to 32 rows of as many tiles as SMs (4096 -> 4096 41.0 -> 17.0, -> 12288
// 35.7 -> 29.8), and any width up to 8 rows, but not gated pairs beyond 16 rows, whose fragments left one CTA per SM (52 -> 64; not built), nor 16-bit weights of
// more tiles than SMs beyond 8 rows, where whole tiles per CTA leave the second CTA of an SM idle (250 tiles, 32 rows 55.6 -> 67.9; int8 39.4 -> 38.1).
bool reg_wins(int M, int N, int epi, int gate_rows, bool i8, int sms) {
  const int tiles = ((epi == EPI_GATE ? gate_rows : N) + ROWS - 1) / ROWS;
  return i8 || M <= 8 || tiles <= sms;
}

bool reg_supported(int M, int epi, const void* x, long long ldx_bytes) {
  return M >= 1 && M <= (epi == EPI_GATE ? REG_MAX_M / 2 : REG_MAX_M) && ldx_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
}

int reg_linear(const void* x, long long ldx_bytes, const void* w_tiles, __nv_bfloat16* y, long long ldy, const __nv_bfloat16* res, long long ldr, int M, int N,
               int K, int epi, int gate_rows, const float* sa, const float* sw, float* ws, size_t ws_bytes, int* counters, int n_counters, int sms, int pdl,
               cudaStream_t stream) {
  if (!reg_supported(M, epi, x, ldx_bytes)) B200_FAIL(B200_ERR_SHAPE, "register GEMM: unsupported shape M=%d", M);
  const bool i8 = sa != nullptr;
  RegP p;
  p.M = M; p.N = N; p.out_rows = epi == EPI_GATE ? gate_rows : N;
  p.n_tiles = (p.out_rows + ROWS - 1) / ROWS;
  p.row_bytes = (long long)K * (i8 ? 1 : 2);
  p.num_kb = (int)((p.row_bytes + 127) / 128);
  const size_t slot = (size_t)(epi == EPI_GATE ? 2 : 1) * (M <= 8 ? 8 : M <= 16 ? 16 : 32) * ROWS * 4;
  const int slots = sms * CTAS_PER_SM;
  // one wave where possible; a range of k costs about six blocks of start-up and exchange on top of its own
  int best = 1;
  long long cost = -1;
  for (int s = 1; s <= 32 && (s == 1 || p.num_kb / s >= 4); ++s) {
    if (s > 1 && ((size_t)p.n_tiles * s * slot > ws_bytes || p.n_tiles > n_counters)) break;
    const long long waves = (p.n_tiles * s + slots - 1) / slots;
    const long long c = waves * ((p.num_kb + s - 1) / s + 6) + (s > 1 ? 2 : 0);
    if (cost < 0 || c < cost) { cost = c; best = s; }
  }
  p.kbps = (p.num_kb + best - 1) / best;
  p.S = (p.num_kb + p.kbps - 1) / p.kbps;
  p.late = pdl != PDL_WEIGHTS_FIRST;
  p.wt = static_cast<const uint4*>(w_tiles); p.x = static_cast<const uint8_t*>(x); p.ldx = ldx_bytes;
  p.y = y; p.ldy = ldy; p.res = res; p.ldr = ldr; p.sa = sa; p.sw = sw; p.ws = ws; p.counters = counters;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(p.n_tiles * p.S)); cfg.blockDim = dim3(THREADS); cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  cudaError_t e;
  if (i8) e = epi == EPI_STORE ? launch_nt<EPI_STORE, true>(cfg, p) : epi == EPI_RESADD ? launch_nt<EPI_RESADD, true>(cfg, p) : launch_nt<EPI_GATE, true>(cfg, p);
  else e = epi == EPI_STORE ? launch_nt<EPI_STORE, false>(cfg, p) : epi == EPI_RESADD ? launch_nt<EPI_RESADD, false>(cfg, p) : launch_nt<EPI_GATE, false>(cfg, p);
  if (e != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_reg launch failed: %s", cudaGetErrorString(e));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("gemm_reg");
}

}  // namespace tc
}  // namespace b200
