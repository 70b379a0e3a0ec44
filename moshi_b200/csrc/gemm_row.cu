// Linears of 1..16 activation rows:  y[M][N] = epi(x[M][K] . w[N][K]^T), same packed tiles, epilogues and cast points as gemm_sk.cu; bf16, and int8 with int32 sums.
//
// A linear of so few rows is a stream of its weights with a start and an end.  A kernel that cuts K over CTAs (gemm_reg.cu) pays for the cut
// at the end: partial sums written, a fence, an arrival counter, and the last CTA's read of all of them.  Here a CTA owns whole output rows, so
// nothing leaves an SM but results:
//   * one CTA of 16 warps per SM; the output rows are dealt in units of 8 (4096 -> 12288: 10.4 a CTA, the fullest has 11), the warps share the k-blocks;
//   * a warp asks for its weights with cp.async, SLOTS pairs of units x 64 k (2 KB) ahead of the one it multiplies, from before the wait on the preceding
//     kernel to the last block.  64 KB under way per SM are the full rate of HBM (7 TB/s for a plain stream), 96 KB are slower: the activations' reads queue
//     behind them.  No registers are held for what is under way;
//   * a pair of units, or the gate and value rows of one, is the A fragment of mma.sync m16n8k16 (int8 m16n8k32); which k a slot holds does not matter as
//     long as the activations' fragment agrees, so every thread takes whole 16-byte pieces of the tiles;
//   * activations of KC k-blocks are in registers; the warps' sums meet in shared memory, as many units at a time as fit;
//   * one CTA fits an SM (512 threads of 98 to 109 registers): with two, early launches would put both of the next linear's on whichever SM is done first.
//
// Bound by HBM, start and end.  7B shapes, cold weights, behind one another through the entry points (early launches that wait), us, gemm_reg.cu (K cut over CTAs) /
// this kernel / weights at 6.55 TB/s:
//   1 row: 4096 -> 12288 22.4 / 18.0 / 15.4, 4096 -> 4096 11.0 / 7.6 / 5.1, gated -> 11264 31.8 / 29.5 / 28.2, 11264 -> 4096 21.2 / 16.5 / 14.1, -> 32000 51.2 / 40.9 / 40.0;
//   8 rows: 22.9 / 19.1, 11.2 / 8.1, 32.2 / 31.4, 21.5 / 17.1, 51.4 / 43.6; 16 rows: 24.8 / 20.6, 13.1 / 9.8, -, 24.2 / 20.1, 53.2 / 48.0;
//   1024 -> 3072 5.6 / 3.9, 2816 -> 1024 6.3 / 4.2; int8 4096 -> 12288 13.5 / 10.2, 11264 -> 4096 13.0 / 9.9.
// Launched alone (clean caches, with about 5 us of launch and events): 1 row 26.6 / 22.5, 16.4 / 12.3, 36.8 / 34.0, 26.5 / 20.5, 55.3 / 45.1; gated 8 rows 36.9 / 36.4.
// Counters (1 row of 4096 -> 12288): DRAM 60 % over the whole launch, L2 hits 0.6 %, warps wait for their weights (6.3 of 11.4 cycles an instruction).
// Error of the sums alone (terms whose exact sum is 0, over the rms of a random sum of them), 4096 -> 12288: 1 row 6.9e-8 (fp32 FMAs 7.4e-8; chains of 16 instructions
// 1.27e-7), 12 rows 8.4e-8 (gemm_reg.cu 6.7e-7); 11264 -> 4096: 1 row 7.7e-8 (8.5e-8; 1.31e-7).
// Steps of the 7B, before this kernel and the weight streams of dep_reg.cuh / with this kernel alone / now: 1 session 4482 / 4014 / 3657 us, 3: 4605 / 4223 / 3857, 8: 4761 / 4397 /
// 4053, 16 with full rings 6960 / 6560 / 6017.
#include "gemm_row.cuh"

#include <algorithm>
#include <type_traits>

#include "row_stream.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace tc {

namespace {

using namespace tcp;
using namespace rows;

constexpr int EPI_STORE = 0, EPI_RESADD = 1, EPI_GATE = 2;
constexpr int THREADS = 512, WARPS = 16, UNIT = 8;
constexpr int TILE = 16384, UNIT_BYTES = 1024;   // a tile: 128 rows x 128 bytes of k
constexpr int SLOTS = 2;                         // pairs of units under way per warp: 64 KB per SM
constexpr int RING_BYTES = SLOTS * WARPS * 2 * UNIT_BYTES;
constexpr int RED_BYTES = 128 * 1024;            // the warps' sums of one pass

struct RowP {
  int M, out_rows, units, num_kb, subs_pass;     // subs_pass: 8-row pieces (gate and value rows apart) of a pass, even
  int row_bytes;                                 // bytes of x per row that exist (K elements)
  int late;                                      // nothing is read before the wait on the preceding kernel
  const uint8_t* wt;
  const uint8_t* x; long long ldx;               // bytes
  __nv_bfloat16* y; long long ldy;
  const __nv_bfloat16* res; long long ldr;
  const float *sa, *sw;                          // int8: scales of activation and weight rows
};

__device__ __forceinline__ float rbf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <int EPI, int NT, bool I8>
__global__ void __launch_bounds__(THREADS, 1) gemm_row_kernel(const RowP p) {
  using Acc = typename std::conditional<I8, int, float>::type;
  constexpr int G = EPI == EPI_GATE ? 1 : 0;     // gated: the tiles of gate and value rows lie behind each other
  constexpr int KC = NT == 1 ? 4 : 2;            // k-blocks of a warp whose activations are in registers together
  // The tensor core cuts its fp32 sums off where an FMA rounds, and the error grows with the chain: up to 8 rows two instructions (32 k) at a time, added in fp32,
  // are as exact as fp32 FMAs throughout, at no cost in time (above 8 rows they cost 2 % of 11264 -> 4096; there the kernels that cut K chain far more).
  constexpr bool SHORT_CHAINS = NT == 1 && !I8;
  extern __shared__ __align__(16) uint8_t smem[];
  Acc* red = reinterpret_cast<Acc*>(smem + RING_BYTES);      // [warp][sub][row of x][8]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, M = p.M;
  const int u0 = (int)((unsigned)p.units * blockIdx.x / gridDim.x), subs = ((int)((unsigned)p.units * (blockIdx.x + 1) / gridDim.x) - u0) << G;
  const uint32_t ring = smem_u32(smem) + warp * 2 * UNIT_BYTES, tile_bytes = (uint32_t)p.num_kb << (14 + G), step = (uint32_t)(WARPS * TILE) << G;
  constexpr uint32_t SLOT = WARPS * 2 * UNIT_BYTES;

  // the stream of this warp: per pass, KC of its k-blocks at a time, and for these every pair of subs, k-block by k-block
  const int my_kb = (p.num_kb - warp + WARPS - 1) / WARPS;
  const uint8_t* const w0 = p.wt + (size_t)(u0 >> 4) * tile_bytes + ((uint32_t)(warp * TILE) << G) + lane * 16;
  const uint8_t* base = my_kb > 0 && subs > 0 ? w0 : nullptr;      // the next k-block asked for (null: none left)
  int a_pass = 0, a_end = min(p.subs_pass, subs), a_sub = 0, a_j = 0, a_nj = min(KC, my_kb), a_left = my_kb;
  auto ask = [&](uint32_t at) {
    if (base) {
      const uint32_t to = ring + at + lane * 16;
      const int ua = (u0 & 15) + (a_sub >> G), ub = ua + 1;
      const uint8_t* s = base + ((ua >> 4) * tile_bytes + (ua & 15) * UNIT_BYTES);
      copy16(to, s);
      copy16(to + 512, s + 512);
      if (a_sub + 1 < a_end) {
        s = G ? s + TILE : base + ((ub >> 4) * tile_bytes + (ub & 15) * UNIT_BYTES);
        copy16(to + 1024, s);
        copy16(to + 1536, s + 512);
      }
      base += step;
      if (++a_j == a_nj) {
        a_j = 0;
        a_sub += 2;
        if (a_sub < a_end) base -= a_nj * step;
        else {
          a_left -= a_nj;
          if (a_left == 0) {                     // the next pass
            a_pass = a_end;
            a_end = min(a_end + p.subs_pass, subs);
            a_left = my_kb;
            base = a_pass < subs ? w0 : nullptr;
          }
          a_nj = min(KC, a_left);
          a_sub = a_pass;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (p.late) pdl_wait();
#pragma unroll 1
  for (int s = 0; s < SLOTS; ++s) ask((uint32_t)s * SLOT);
  uint32_t slot = 0;
  pdl_trigger();
  pdl_wait();

  for (int pass = 0; pass < subs; pass += p.subs_pass) {
    const int n = min(p.subs_pass, subs - pass);
    Acc* mine = red + (warp * n * M + 2 * t) * 8 + row_of(g);
#pragma unroll 1
    for (int kb0 = warp; kb0 == warp || kb0 < p.num_kb; kb0 += WARPS * KC) {      // once at least: a warp without a k-block stores zeros
      uint4 xb[KC][NT][2];
#pragma unroll
      for (int i = 0; i < KC; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int k = (kb0 + i * WARPS) * 128 + h * 64 + t * 16;
            xb[i][j][h] = 8 * j + g < M && k < p.row_bytes ? __ldcg(reinterpret_cast<const uint4*>(p.x + (8 * j + g) * p.ldx + k)) : make_uint4(0u, 0u, 0u, 0u);
          }
#pragma unroll 1
      for (int sub = 0; sub < n; sub += 2) {
        Acc acc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0;
#pragma unroll
        for (int i = 0; i < KC; ++i) {
          if (kb0 + i * WARPS >= p.num_kb) break;
          const uint32_t row = ring + slot + row_of(g) * 128, c = (uint32_t)(t ^ row_of(g)) << 4;
          asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
          __syncwarp();
          const uint4 a[2] = {lds16(row + c), lds16(row + (c ^ 64))}, b[2] = {lds16(row + 1024 + c), lds16(row + 1024 + (c ^ 64))};
          __syncwarp();
          ask(slot);
          slot = slot + SLOT == SLOTS * SLOT ? 0u : slot + SLOT;
          if constexpr (SHORT_CHAINS) {
            Acc part[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              mma_step(part[h], a[h].x, b[h].x, a[h].y, b[h].y, xb[i][0][h].x, xb[i][0][h].y);
              mma_step(part[h], a[h].z, b[h].z, a[h].w, b[h].w, xb[i][0][h].z, xb[i][0][h].w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[0][e] += part[0][e] + part[1][e];
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int j = 0; j < NT; ++j) {
                mma_step(acc[j], a[h].x, b[h].x, a[h].y, b[h].y, xb[i][j][h].x, xb[i][j][h].y);
                mma_step(acc[j], a[h].z, b[h].z, a[h].w, b[h].w, xb[i][j][h].z, xb[i][j][h].w);
              }
          }
        }
        // rows g of either sub; the second of a last odd pair is whatever its slot held before, and is not stored
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (8 * j + 2 * t + (e & 1) < M && sub + (e >> 1) < n) {
              Acc* o = mine + ((sub + (e >> 1)) * M + 8 * j + (e & 1)) * 8;
              *o = kb0 == warp ? acc[j][e] : *o + acc[j][e];
            }
      }
    }
    __syncthreads();
    // results of the pass: the warps' sums in pairs, always the same
    const int rows = (n >> G) * UNIT, first = (u0 + (pass >> G)) * UNIT;
    for (int i = tid; i < rows * M; i += THREADS) {
      const int m = i / rows, r = i - m * rows, o = first + r;
      if (o >= p.out_rows) continue;
      Acc v[2];
#pragma unroll
      for (int a = 0; a <= G; ++a) {
        Acc s[WARPS];
#pragma unroll
        for (int w = 0; w < WARPS; ++w) s[w] = red[((w * n + ((r >> 3) << G) + a) * M + m) * 8 + (r & 7)];
#pragma unroll
        for (int d = WARPS / 2; d > 0; d >>= 1)
#pragma unroll
          for (int w = 0; w < d; ++w) s[w] += s[w + d];
        v[a] = s[0];
      }
      float f[2] = {(float)v[0], (float)v[G]};
      if (I8) {                                  // the sums are whole numbers in 32 bits
        const float s = p.sa[m];
        f[0] *= s * p.sw[o] * (1.f / 16129.f);
        if (G) f[1] *= s * p.sw[o + p.out_rows] * (1.f / 16129.f);
      }
      float out;
      if (EPI == EPI_STORE) out = f[0];
      else if (EPI == EPI_RESADD) out = __bfloat162float(p.res[(long long)m * p.ldr + o]) + rbf16(f[0]);
      else { const float gt = rbf16(f[0]), u = rbf16(f[1]); out = rbf16(gt / (1.f + expf(-gt))) * u; }
      p.y[(long long)m * p.ldy + o] = __float2bfloat16_rn(out);
    }
    if (pass + p.subs_pass < subs) __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// 8-row pieces of the fullest CTA, and how many of them a pass takes: as few equal passes as the warps' sums fit, an even number of pieces each
int subs_at_most(int out_rows, int epi, int sms) {
  const int units = (out_rows + UNIT - 1) / UNIT, grid = std::min(sms, units);
  return ((units + grid - 1) / grid) << (epi == EPI_GATE ? 1 : 0);
}
int pass_of(int M, int most) {
  const int fit = RED_BYTES / (WARPS * M * UNIT * 4) / 2 * 2, passes = (most + fit - 1) / fit;
  return ((most + passes - 1) / passes + 1) / 2 * 2;
}

template <int EPI, bool I8>
cudaError_t launch_nt(const cudaLaunchConfig_t& cfg, const RowP& p) {
  if (p.M <= 8) return cudaLaunchKernelEx(&cfg, gemm_row_kernel<EPI, 1, I8>, p);
  return cudaLaunchKernelEx(&cfg, gemm_row_kernel<EPI, 2, I8>, p);
}

}  // namespace

// Everything but 16-bit gated pairs of so many rows that their sums need a second pass, which reads the activations again.  Behind one another, us, register kernel /
// this one: 4096 -> 11264, one pass, 3 rows 32.0 / 29.9, 6 rows 32.1 / 30.7, 8 rows 32.2 / 31.4, 12 rows 35.2 / 32.4; two passes, 16 rows 35.4 / 34.9 (alone the same); but
// 4096 -> 28672, two passes, 6 rows 72.6 / 74.4, four, 16 rows 78.8 / 84.4 (there gemm_sk.cu's kernel).
bool row_wins(int M, int epi, int gate_rows, bool i8, int sms) {
  if (M > ROW_MAX_M) return false;
  if (epi != EPI_GATE || i8) return true;
  const int most = subs_at_most(gate_rows, epi, sms);
  return pass_of(M, most) >= most;
}

bool row_supported(int M, int K, bool i8, const void* x, long long ldx_bytes) {
  return M >= 1 && M <= ROW_MAX_M && K % (i8 ? 16 : 8) == 0 && ldx_bytes % 16 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
}

int row_linear(const void* x, long long ldx_bytes, const void* w_tiles, __nv_bfloat16* y, long long ldy, const __nv_bfloat16* res, long long ldr, int M, int N,
               int K, int epi, int gate_rows, const float* sa, const float* sw, int sms, int pdl, cudaStream_t stream) {
  const bool i8 = sa != nullptr;
  if (!row_supported(M, K, i8, x, ldx_bytes)) B200_FAIL(B200_ERR_SHAPE, "row GEMM: unsupported shape M=%d K=%d", M, K);
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, RING_BYTES + RED_BYTES, gemm_row_kernel<EPI_STORE, 1, false>, gemm_row_kernel<EPI_STORE, 2, false>, gemm_row_kernel<EPI_RESADD, 1, false>,
                      gemm_row_kernel<EPI_RESADD, 2, false>, gemm_row_kernel<EPI_GATE, 1, false>, gemm_row_kernel<EPI_GATE, 2, false>, gemm_row_kernel<EPI_STORE, 1, true>,
                      gemm_row_kernel<EPI_STORE, 2, true>, gemm_row_kernel<EPI_RESADD, 1, true>, gemm_row_kernel<EPI_RESADD, 2, true>, gemm_row_kernel<EPI_GATE, 1, true>,
                      gemm_row_kernel<EPI_GATE, 2, true>));
  RowP p;
  p.M = M; p.out_rows = epi == EPI_GATE ? gate_rows : N;
  p.units = (p.out_rows + UNIT - 1) / UNIT;
  p.row_bytes = K * (i8 ? 1 : 2);
  p.late = pdl != PDL_WEIGHTS_FIRST;
  p.num_kb = (p.row_bytes + 127) / 128;
  p.wt = static_cast<const uint8_t*>(w_tiles); p.x = static_cast<const uint8_t*>(x); p.ldx = ldx_bytes;
  p.y = y; p.ldy = ldy; p.res = res; p.ldr = ldr; p.sa = sa; p.sw = sw;
  const int grid = std::min(sms, p.units), most = subs_at_most(p.out_rows, epi, sms);
  p.subs_pass = pass_of(M, most);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(THREADS); cfg.stream = stream;
  cfg.dynamicSmemBytes = RING_BYTES + (size_t)WARPS * std::min(p.subs_pass, most) * M * UNIT * 4;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  cudaError_t e;
  if (i8) e = epi == EPI_STORE ? launch_nt<EPI_STORE, true>(cfg, p) : epi == EPI_RESADD ? launch_nt<EPI_RESADD, true>(cfg, p) : launch_nt<EPI_GATE, true>(cfg, p);
  else e = epi == EPI_STORE ? launch_nt<EPI_STORE, false>(cfg, p) : epi == EPI_RESADD ? launch_nt<EPI_RESADD, false>(cfg, p) : launch_nt<EPI_GATE, false>(cfg, p);
  if (e != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_row launch failed: %s", cudaGetErrorString(e));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("gemm_row");
}

}  // namespace tc
}  // namespace b200
