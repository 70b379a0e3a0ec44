// tcgen05 GEMM for many activation rows (prompt portions, scoring, routed experts):  y[M][N] = epi(x[M][K] . w[N][K]^T), bf16 in, fp32 in
// TMEM, bf16 out.  gemm_ns.cu streams weights past at most 256 rows; here the rows are many and both operands are tiled:
//
//   * CG = 2: a pair of CTAs owns a tile of 256 rows x BN columns (tcgen05.mma.cta_group::2, M = 256): every CTA stages its own 128 rows
//     of x and half of the BN weight rows, so an SM takes in 32 KB per 256 x 256 x 64 step instead of the 48 KB that a 128 x 256 tile of
//     its own needs.  CG = 1: one CTA, 128 rows x BN columns: routed experts, whose row counts rarely fill 256.  (A tile of 256 x 128 takes as
//     long as one of 256 x 256: 2048 x 8192 -> 2048 columns 92 us against 52; so few tiles are cut along k instead.)
//   * persistent, one CTA per SM: tiles in the order "all row tiles of a column block", so that the weights of a block are read from HBM
//     once and the rows stay in L2; two accumulators in TMEM, the epilogue of a tile runs under the products of the next.
//   * weights either as the packed SWIZZLE_128B tiles of gemm_sk.cu (fetched as they are by an unswizzled box) or row-major (swizzled
//     by the TMA unit): the packed form serves the decoding kernels too, and nothing is held twice.
//   * grouped products: the row tiles come from a table on the device (expert, first row, rows), rows of one expert being neighbours; few
//     rows per expert make it a stream of the experts' weights, up to 192 KB of them in flight per SM.  16 experts of width 2048 and
//     hidden size 4096, both products: 2000 rows 450 -> 170 us, 16 rows 191 -> 114 us (the mma.sync kernel before had two stages of 64 k).
//
// Bound by the tensor pipe: 2048 x 2048 -> 14848 columns 94 us (1321 TFLOP/s, 0.79 of the measured cuBLAS rate; cuBLAS itself 90 us), 2048 x
// 8192 -> 2048 52 us (1325); with one launch of gemm_ns.cu per 256 rows, 58 of 148 SMs busy at a time, the four linears of such a layer took
// 680 us instead of 200.  Below about 1000 rows the last wave is what is lost (300 rows: 560-700 TFLOP/s).
//
// A wait that lasts longer than ten seconds raises the caller's error flag and the kernel winds down.
#include "gemm_wide.cuh"

#include <algorithm>
#include <cmath>

#include "tc_prims.cuh"

namespace b200 {
namespace tc {

namespace {

using namespace tcp;

constexpr int BK = 64;                       // 128 bytes of K per row and stage
constexpr int THREADS = 192;                 // warp 0 producer, warp 1 MMA, warps 2-5 epilogue
constexpr int MAX_ST = 8;

struct WideP {
  int M, N, num_kb, stages, mt, nt, packed, act;      // mt x nt tiles (mt: of the table with a grouped product)
  int splits, kb_per;                                 // k cut into `splits` ranges of kb_per blocks
  float* ws; int* counters;                           // splits > 1: partial sums [split][tile][CTA of the pair][BN / 4][128 rows][4], arrivals per tile and CTA
  float limit;
  __nv_bfloat16* y; long long ldy;
  const int *tile_e, *tile_r0, *tile_n, *n_tiles;     // grouped: row tiles on the device
  const int* y_rows;                                  // grouped: result row of every row (null: the row itself)
  int e_rows;                                         // grouped: weight rows per expert
  int vec;                                            // results in 16-byte stores
  int act_from, act_to; __nv_bfloat16* y2; long long ldy2;
  uint32_t stage_bytes;
  uint32_t a_bytes, bars_at;                          // bytes of a box of x rows (128 rows; fewer where no tile has more); mbarriers of gemm_expert_kernel
  int* err;
};

// false: ten seconds have passed, or another role of this CTA has given up
__device__ __forceinline__ bool wait_or_quit(uint32_t bar, uint32_t parity, volatile int* quit) {
  uint32_t done, spins = 0;
  uint64_t t0 = 0;
  for (;;) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if ((++spins & 1023u) == 0u) {
      if (*quit) return false;
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) { *quit = 1; return false; }
    }
  }
}

// the same for a whole warp: all of it goes on, or all of it gives up
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* quit) { return __all_sync(0xffffffffu, wait_or_quit(bar, parity, quit)); }

template <int CG>
__device__ __forceinline__ uint32_t leader_addr(uint32_t local) {      // the same address in the first CTA of the pair
  if (CG == 1) return local;
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(local));
  return r;
}
template <int CG>
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if constexpr (CG == 2)
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
  else
    tma_load_2d(dst, map, bar, c0, c1);
}
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar) {                 // signals the barrier in both CTAs of a pair
  if constexpr (CG == 2) {
    const uint16_t both = 3;
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"(both) : "memory");
  } else {
    commit_elected(bar);
  }
}
template <int CG>
__device__ __forceinline__ void arrive_leader(uint32_t bar) {
  if constexpr (CG == 2) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr<2>(bar)) : "memory");
  else mbar_arrive(bar);
}
template <int CG>
__device__ __forceinline__ void alloc_tmem(uint32_t dst, uint32_t cols) {
  if constexpr (CG == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  } else {
    tmem_alloc(dst, cols);
  }
}
template <int CG>
__device__ __forceinline__ void dealloc_tmem(uint32_t addr, uint32_t cols) {
  if constexpr (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
  else tmem_dealloc(addr, cols);
}
template <int CG>
__device__ __forceinline__ void pair_sync() {
  if constexpr (CG == 2) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

// `n` results of one row to y[col ..): 16-byte stores where the whole run fits and is aligned
template <int NV>
__device__ __forceinline__ void store_run(__nv_bfloat16* row, int col, int cols, const float* v, bool vec) {
  if (vec && col + NV <= cols) {
#pragma unroll
    for (int j = 0; j < NV; j += 8) {
      __nv_bfloat162 o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = __floats2bfloat162_rn(v[j + 2 * i], v[j + 2 * i + 1]);
      *reinterpret_cast<uint4*>(row + col + j) = *reinterpret_cast<const uint4*>(o);
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (col + j < cols) row[col + j] = __float2bfloat16_rn(v[j]);
  }
}

// NV (16 or 32) neighbouring sums of one row through the epilogue
template <int NV>
__device__ __forceinline__ void finish_run(const WideP& p, __nv_bfloat16* y, long long yr, int n, float* v) {
  if (p.act == WIDE_CLAMPED_GLU || p.act == WIDE_SILU_GLU) {      // weight rows interleave gate and value
    float o[NV / 2];
#pragma unroll
    for (int j = 0; j < NV / 2; ++j) {
      const float g = v[2 * j], w = v[2 * j + 1];
      if (p.act == WIDE_SILU_GLU) {
        o[j] = g / (1.f + expf(-g)) * w;
      } else {
        const float gc = fminf(g, p.limit), wc = fminf(fmaxf(w, -p.limit), p.limit);
        o[j] = gc / (1.f + expf(-1.702f * gc)) * (wc + 1.f);
      }
    }
    store_run<NV / 2>(y, n >> 1, p.N >> 1, o, p.vec);
    return;
  }
  const bool aside = n >= p.act_from && n < p.act_to;
  if (p.act == WIDE_RELU2 || aside) {
#pragma unroll
    for (int j = 0; j < NV; ++j) { v[j] = fmaxf(v[j], 0.f); v[j] *= v[j]; }
  } else if (p.act == WIDE_GELU) {
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = 0.5f * v[j] * (1.f + erff(v[j] * 0.7071067811865476f));
  }
  if (aside) store_run<NV>(p.y2 + yr * p.ldy2, n - p.act_from, p.act_to - p.act_from, v, p.vec);
  else store_run<NV>(y, n, p.N, v, p.vec);
}

// whether all 128 epilogue threads say so (a barrier of theirs)
__device__ __forceinline__ bool epilogue_all(bool ok) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "bar.red.and.pred p, 1, 128, q;\n\t"
      "selp.s32 %0, 1, 0, p;\n\t}"
      : "=r"(r) : "r"((int)ok) : "memory");
  return r != 0;
}

template <int CG, int BN>
__global__ void __launch_bounds__(THREADS, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const WideP p) {
  constexpr int WROWS = BN / CG;                       // weight rows that this CTA stages
  constexpr int BOX = WROWS < 128 ? WROWS : 128;       // rows per weight box
  constexpr uint32_t B_STAGE = WROWS * BK * 2;
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int quit;
  __shared__ int arrived;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t stage_bytes = p.stage_bytes, a_stage = stage_bytes - B_STAGE;      // x rows first (at least the box), then weight rows
  const uint32_t bars = base + (uint32_t)p.stages * stage_bytes;
  const uint32_t full0 = bars, empty0 = bars + 8 * MAX_ST, tfull0 = bars + 16 * MAX_ST, tempty0 = tfull0 + 16, tptr = tempty0 + 16;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0;
  const int first = blockIdx.x / CG, step = gridDim.x / CG;
  const bool grouped = p.tile_e != nullptr;

  if (threadIdx.x == 0) {
    quit = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 4 * CG);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) alloc_tmem<CG>(tptr, 2 * BN);
  tc_fence_before();
  __syncthreads();
  pair_sync<CG>();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<const uint32_t*>(smem_raw + (tptr - raw));
  pdl_trigger();
  pdl_wait();                                           // set-up ran under the preceding kernel; rows, tile table and results are its business too
  const int mt = grouped ? p.n_tiles[0] : p.mt;
  const int tiles = mt * p.nt, units = tiles * p.splits;      // unit: a tile's sums over one range of k

  // Both loops are walked by their whole warps, so that what the copies and products take is in uniform registers, and one thread issues.  (One thread alone: a prompt
  // of 2048 tokens 1181 us, so 1131; 895 tokens scored 1271 and 1243.)
  if (warp == 0) {
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    for (int u = first; ok && u < units; u += step) {
      const int t = u % tiles, m = t % mt, n = t / mt;
      const int kb0 = u / tiles * p.kb_per, kb1 = min(p.num_kb, kb0 + p.kb_per);
      const int row0 = (grouped ? p.tile_r0[m] : m * 128 * CG) + rank * 128;
      const int w0 = n * BN + rank * WROWS;             // first weight row (of the expert) of this CTA
      const int wbase = grouped ? p.tile_e[m] * p.e_rows : 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!warp_wait(empty0 + 8 * s, ph ^ 1u, &quit)) { ok = false; break; }
        const uint32_t sa = base + (uint32_t)s * stage_bytes, bar = leader_addr<CG>(full0 + 8 * s);
        if (elected()) {
          if (rank == 0) mbar_expect_tx(full0 + 8 * s, CG * (p.a_bytes + B_STAGE));
          load_box<CG>(sa, &map_x, bar, kb * BK, row0);
#pragma unroll
          for (int j = 0; j < WROWS / BOX; ++j) {
            const int w = w0 + j * BOX;
            // a packed tile holds 128 rows x 64 k; tiles of one row block follow one another along k
            if (p.packed) load_box<CG>(sa + a_stage + j * BOX * BK * 2, &map_w, bar, 0, ((w >> 7) * p.num_kb + kb) * 128 + (w & 127));
            else load_box<CG>(sa + a_stage + j * BOX * BK * 2, &map_w, bar, kb * BK, wbase + w);
          }
        }
        __syncwarp();
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
    }
    if (!ok) {                                          // let copies in flight land before the block ends
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = make_idesc(128 * CG, BN);
      int s = 0; uint32_t ph = 0;
      bool ok = true;
      for (int u = first, it = 0; ok && u < units; u += step, ++it) {
        const uint32_t a = it & 1, d = tmem + a * BN;
        const int kb0 = u / tiles * p.kb_per, kb1 = min(p.num_kb, kb0 + p.kb_per);
        if (!warp_wait(tempty0 + 8 * a, ((it >> 1) & 1) ^ 1u, &quit)) break;
        tc_fence_after();
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!warp_wait(full0 + 8 * s, ph, &quit)) { ok = false; break; }
          tc_fence_after();
          umma_block<CG>(d, desc_low(base + (uint32_t)s * stage_bytes), a_stage >> 4, idesc, kb > kb0 ? 1u : 0u);
          commit<CG>(empty0 + 8 * s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        if (ok) commit<CG>(tfull0 + 8 * a);
      }
    }
    __syncwarp();
  } else {
    const int q4 = warp & 3;
    for (int u = first, it = 0; u < units; u += step, ++it) {
      const uint32_t a = it & 1;
      if (!epilogue_all(wait_or_quit(tfull0 + 8 * a, (it >> 1) & 1, &quit))) break;
      tc_fence_after();
      const int t = u % tiles, m = t % mt, n0 = (t / mt) * BN;
      const int r = rank * 128 + q4 * 32 + lane;        // row of the tile
      const int row0 = grouped ? p.tile_r0[m] : m * 128 * CG, rows = grouped ? p.tile_n[m] : p.M - row0;
      const bool row_ok = r < rows;
      const long long yr = row_ok && p.y_rows ? p.y_rows[row0 + r] : row0 + r;
      __nv_bfloat16* y = p.y + yr * p.ldy;
      const uint32_t src = tmem + ((uint32_t)(q4 * 32) << 16) + a * BN;
      const bool whole = p.splits == 1;
      bool finish = whole;
      float4* part = nullptr;
      if (!whole) {
        // partial sums go to L2; the CTA whose range arrives last adds the ranges in order, so that the result does not depend on who that is
        part = reinterpret_cast<float4*>(p.ws) + ((size_t)u * CG + rank) * (BN / 4) * 128 + (q4 * 32 + lane);
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t v[32];
          __syncwarp();
          tmem_ld32(src + (uint32_t)c, v);
          tmem_ld_wait();
          if (row_ok && n0 + c < p.N) {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              __stcg(part + (size_t)((c + j) >> 2) * 128, make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3])));
          }
        }
        tc_fence_before();
        __threadfence();
        if (epilogue_all(true) && threadIdx.x == 64) {
          arrived = atomicAdd(p.counters + t * CG + rank, 1);
          if (arrived == p.splits - 1) p.counters[t * CG + rank] = 0;
          __threadfence();
        }
        epilogue_all(true);
        finish = arrived == p.splits - 1;
        if (lane == 0) arrive_leader<CG>(tempty0 + 8 * a);
        epilogue_all(true);                             // `arrived` has been read by everyone
        part = reinterpret_cast<float4*>(p.ws) + ((size_t)t * CG + rank) * (BN / 4) * 128 + (q4 * 32 + lane);
      }
      if (finish) {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          float v[32];
          const int n = n0 + c;
          if (whole) {
            uint32_t r32[32];
            __syncwarp();                               // the load is one instruction of the whole warp
            tmem_ld32(src + (uint32_t)c, r32);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r32[j]);
          } else if (row_ok && n < p.N) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.f;
            for (int s = 0; s < p.splits; ++s) {
              const float4* q = part + ((size_t)s * tiles * CG * (BN / 4) + (c >> 2)) * 128;
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                const float4 f = __ldcg(q + (size_t)(j >> 2) * 128);
                v[j] += f.x; v[j + 1] += f.y; v[j + 2] += f.z; v[j + 3] += f.w;
              }
            }
          }
          if (row_ok && n < p.N) finish_run<32>(p, y, yr, n, v);
        }
      }
      if (whole) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_leader<CG>(tempty0 + 8 * a);
      }
    }
  }
  __syncthreads();
  pair_sync<CG>();                                      // both CTAs are done with their accumulators and barriers
  if (warp == 1) dealloc_tmem<CG>(tmem, 2 * BN);
  if (threadIdx.x == 0 && quit && p.err) atomicOr(p.err, WIDE_ERR_WAIT);
  pair_sync<CG>();
}

// Grouped product of few rows per expert (one tile each): a stream of the experts' weights.  Their rows, laid end to end, are dealt to the CTAs in units of 16, so that
// every SM streams the same number of them to within one unit; a CTA takes its share in tiles of up to 128 rows of one expert.  With whole tiles of 256 columns dealt over
// 148 SMs the last of few waves was mostly empty: 10 experts of 8192 x 2048 are 320 tiles in three waves, and of 2048 x 4096 80 tiles for 148 SMs.
// us, tiles of 256 columns / here / the weights at 6.55 TB/s: 8192 x 2048, 2 experts 33.1 / 16.5 / 10.2, 10 81.4 / 62.2 / 51.2, 16 with 4 rows each 126.3 / 100.6 / 81.9, with
// 16 rows 157.1 / 118.1; 2048 x 4096, 2 experts 25.9 / 11.1 / 5.1, 10 34.3 / 31.0 / 25.6, 16 with 16 rows 48.6 / 49.8 / 41.0.
// What bounded it on the way is how fast a thread asks and issues: a copy per unit and products from one thread 90 us for 10 experts of 8192 x 2048, both loops
// walked by whole warps 60.8 (2048 x 4096: 60 and 37.3), one copy and two k-blocks per stage 62.2 and 31.0.
constexpr int EXPERT_SMEM = 216 * 1024;
constexpr int UNIT = 16, TILE_UNITS = 8, EXPERT_ST = 6, STAGE_KB = 2;      // STAGE_KB: k-blocks per stage
struct alignas(64) ExpertMaps { CUtensorMap x, w[TILE_UNITS]; };             // w[n - 1]: boxes of n units, so that a tile's rows come in one copy per k-block
struct ExpertTile { int m, row, units; };      // tile of the table, first weight row of the expert, units of 16
__device__ __forceinline__ ExpertTile expert_tile(int u, int end, int per_expert) {
  ExpertTile t;
  t.m = u / per_expert;
  const int left = min(end, (t.m + 1) * per_expert) - u, tiles = (left + TILE_UNITS - 1) / TILE_UNITS;
  t.row = (u - t.m * per_expert) * UNIT;
  t.units = (left + tiles - 1) / tiles;        // tiles of equal length
  return t;
}

__global__ void __launch_bounds__(THREADS, 1)
gemm_expert_kernel(const __grid_constant__ ExpertMaps maps, const WideP p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int quit;
  constexpr int COLS = TILE_UNITS * UNIT;
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t stage_bytes = p.stage_bytes, x_bytes = (p.a_bytes + 1023u) / 1024u * 1024u, w_at = STAGE_KB * x_bytes;      // x rows of the k-blocks first, then weight rows
  const uint32_t bars = base + p.bars_at;
  const uint32_t full0 = bars, empty0 = bars + 8 * EXPERT_ST, tfull0 = bars + 16 * EXPERT_ST, tempty0 = tfull0 + 16, tptr = tempty0 + 16;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    quit = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.x) : "memory");
  }
  if (warp == 1) tmem_alloc(tptr, 2 * COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<const uint32_t*>(smem_raw + (tptr - raw));
  pdl_trigger();
  pdl_wait();                                           // rows, table and results are the preceding kernels' business
  const int per_expert = (p.N + UNIT - 1) / UNIT;
  const unsigned units = (unsigned)(p.n_tiles[0] * per_expert);
  const int u0 = (int)((unsigned long long)units * blockIdx.x / gridDim.x), u1 = (int)((unsigned long long)units * (blockIdx.x + 1) / gridDim.x);

  // both loops are walked by their whole warps, so that what the copies and products take is in uniform registers, and one thread issues
  if (warp == 0) {
    int s = 0; uint32_t ph = 0;
    bool ok = true;
    for (int u = u0; ok && u < u1;) {
      const ExpertTile t = expert_tile(u, u1, per_expert);
      const int row0 = p.tile_r0[t.m], w0 = p.tile_e[t.m] * p.e_rows + t.row;
      const uint32_t bytes = STAGE_KB * (p.a_bytes + (uint32_t)t.units * UNIT * BK * 2);
      const CUtensorMap* map_w = &maps.w[t.units - 1];
      for (int kb = 0; kb < p.num_kb; kb += STAGE_KB) {      // blocks beyond the last are zeroes
        const uint32_t bar = full0 + 8 * s, sa = base + (uint32_t)s * stage_bytes;
        if (!warp_wait(empty0 + 8 * s, ph ^ 1u, &quit)) { ok = false; break; }
        if (elected()) {
          mbar_expect_tx(bar, bytes);
#pragma unroll
          for (int j = 0; j < STAGE_KB; ++j) {
            tma_load_2d(sa + w_at + j * COLS * BK * 2, map_w, bar, (kb + j) * BK, w0);
            tma_load_2d(sa + j * x_bytes, &maps.x, bar, (kb + j) * BK, row0);
          }
        }
        __syncwarp();
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
      u += t.units;
    }
    if (!ok) {                                          // let copies in flight land before the block ends
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
    __syncwarp();
  } else if (warp == 1) {
    int s = 0, it = 0; uint32_t ph = 0;
    bool ok = true;
    for (int u = u0; ok && u < u1; ++it) {
      const ExpertTile t = expert_tile(u, u1, per_expert);
      const uint32_t a = it & 1, d = tmem + a * COLS, idesc = make_idesc(128, t.units * UNIT);
      if (!warp_wait(tempty0 + 8 * a, ((it >> 1) & 1) ^ 1u, &quit)) break;
      tc_fence_after();
      for (int kb = 0; kb < p.num_kb; kb += STAGE_KB) {
        if (!warp_wait(full0 + 8 * s, ph, &quit)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sa = desc_low(base + (uint32_t)s * stage_bytes);
#pragma unroll
        for (int j = 0; j < STAGE_KB; ++j) umma_block<1>(d, sa + j * (x_bytes >> 4), (w_at + j * (COLS * BK * 2 - x_bytes)) >> 4, idesc, kb + j > 0 ? 1u : 0u);
        commit<1>(empty0 + 8 * s);
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
      if (ok) commit<1>(tfull0 + 8 * a);
      u += t.units;
    }
    __syncwarp();
  } else {
    const int q4 = warp & 3, r = q4 * 32 + lane;        // row of the tile
    int it = 0;
    for (int u = u0; u < u1; ++it) {
      const ExpertTile t = expert_tile(u, u1, per_expert);
      const int rows = p.tile_n[t.m], row0 = p.tile_r0[t.m];
      const bool row_ok = r < rows;
      const long long yr = row_ok && p.y_rows ? p.y_rows[row0 + r] : row0 + r;
      __nv_bfloat16* y = p.y + yr * p.ldy;
      const uint32_t a = it & 1;
      if (!epilogue_all(wait_or_quit(tfull0 + 8 * a, (it >> 1) & 1, &quit))) break;
      tc_fence_after();
      if (q4 * 32 < rows) {
#pragma unroll 1
        for (int c = 0; c < t.units * UNIT; c += UNIT) {
          uint32_t v[16];
          __syncwarp();
          tmem_ld16(tmem + ((uint32_t)(q4 * 32) << 16) + a * COLS + (uint32_t)c, v);
          tmem_ld_wait();
          float f[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(v[j]);
          if (row_ok && t.row + c < p.N) finish_run<16>(p, y, yr, t.row + c, f);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * a);
      u += t.units;
    }
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 2 * COLS);
  if (threadIdx.x == 0 && quit && p.err) atomicOr(p.err, WIDE_ERR_WAIT);
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_fn(EncodeFn* out) {
  static const EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  if (!fn) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
  *out = fn;
  return B200_OK;
}

// rows x cols bf16, row stride ld elements; boxes of box_rows x 64
int make_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, long long ld, int box_rows, bool swizzle) {
  EncodeFn fn = nullptr;
  B200_TRY(encode_fn(&fn));
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows}, est[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, est, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) B200_FAIL(B200_ERR_CUDA, "wide GEMM: tensor map of %lld x %lld (ld %lld) refused (%d)", rows, cols, ld, (int)r);
  return B200_OK;
}

template <int CG, int BN>
int launch(const WideGemm& g, WideP p, int clusters, cudaStream_t st) {
  constexpr int WROWS = BN / CG, BOX = WROWS < 128 ? WROWS : 128;
  CUtensorMap mx, mw;
  // no expert has more rows than the step has tokens: with fewer than 128 a smaller box saves the traffic, and the accumulator rows
  // beyond it, products of whatever the stage held before, are not stored
  const int box_rows = g.tile_e && g.max_rows > 0 ? std::min(128, ceil_div(g.max_rows, 8) * 8) : 128;
  p.a_bytes = (uint32_t)box_rows * BK * 2;
  B200_TRY(make_map(&mx, g.x, g.x_rows, g.K, g.ldx, box_rows, true));
  if (g.packed) B200_TRY(make_map(&mw, g.w, (long long)ceil_div(g.N, 128) * p.num_kb * 128, BK, BK, BOX, false));
  else B200_TRY(make_map(&mw, g.w, (long long)g.w_rows, g.K, g.K, BOX, true));
  // the products read 128 rows of x from a stage: where the box is smaller they run into the weight rows behind it
  p.stage_bytes = (p.a_bytes + 1023) / 1024 * 1024 + WROWS * BK * 2;
  p.stages = std::min(MAX_ST, 200 * 1024 / (int)p.stage_bytes);
  const size_t smem = (size_t)p.stages * p.stage_bytes + 1024 + 16 * MAX_ST + 64;
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, 220 * 1024, gemm_wide_kernel<CG, BN>));
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(std::min(clusters, p.mt * p.nt * p.splits) * CG)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CG; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = CG > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_wide_kernel<CG, BN>, mx, mw, p);
  if (e != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_wide launch failed: %s", cudaGetErrorString(e));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("gemm_wide");
}

int launch_experts(const WideGemm& g, WideP p, int sms, cudaStream_t st) {
  ExpertMaps maps;
  const int box_rows = ceil_div(g.max_rows, 8) * 8;
  p.a_bytes = (uint32_t)box_rows * BK * 2;
  B200_TRY(make_map(&maps.x, g.x, g.x_rows, g.K, g.ldx, box_rows, true));
  for (int n = 1; n <= TILE_UNITS; ++n) B200_TRY(make_map(&maps.w[n - 1], g.w, (long long)g.w_rows, g.K, g.K, n * UNIT, true));
  p.stage_bytes = STAGE_KB * ((p.a_bytes + 1023) / 1024 * 1024 + TILE_UNITS * UNIT * BK * 2);
  p.stages = std::min(EXPERT_ST, EXPERT_SMEM / (int)p.stage_bytes);
  // the products read 128 rows of x from a stage, which run into what lies behind a smaller box: a tile's accumulator rows beyond it are not stored
  p.bars_at = (uint32_t)p.stages * p.stage_bytes;
  const size_t smem = p.bars_at + 1024 + 16 * EXPERT_ST + 64;
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, EXPERT_SMEM + 1024 + 16 * EXPERT_ST + 64, gemm_expert_kernel));
  B200_TRY(launch_early(gemm_expert_kernel, dim3((unsigned)sms), dim3(THREADS), smem, st, maps, p));
  return check_launch("gemm_expert");
}

// Few rows per expert: units of rows dealt over the SMs (gemm_expert_kernel) or tiles of 256 columns, a wave of them after the other?  The tiles lose what the last wave leaves idle
// and have the longer way through a gated unit's epilogue; the units bring every CTA's rows of x once per 128 weight rows instead of 256.  How many experts have rows is the router's
// business; as many as an even one would choose are reckoned with.  us, tiles / units, rows of x per box after the @:
//   one wave, 2048 x 4096: 2 experts 26 / 14, 10 34 / 31, 14 of 16 (0.76 of a wave) 52.8 / 55.5 @32, 16 (0.86) 59.9 / 61.5 @8, 62.1 / 70.5 @128; 4096 x 8192, 7 (0.76) 89.8 / 99.2 @8, 6 83.7 / 79.0;
//   more, 4096 x 4096: 15 experts (1.6 waves) 94.7 / 96.4, 60 (6.4) 304 / 308, 128 (13.8) 648 / 674;
//   gated, 8192 x 2048: 16 experts 126 / 101 @4, 173 / 130 @128, 48 (10.8) 276 / 297 @16, 64 (13.8) 473 / 416 @128, 108 (22) 576 / 599 @32; 4096 x 1024: 58 experts 152 / 113.
bool experts_win(const WideGemm& g, int sms) {
  const double E = (double)g.w_rows / g.e_rows, used = E * (1. - pow(1. - 1. / E, (double)g.M)), waves = used * ceil_div(g.N, 256) / sms;
  if (g.act == WIDE_CLAMPED_GLU || g.act == WIDE_SILU_GLU) return waves < 9. || (waves < 16. && g.max_rows >= 64);
  return ceil(waves) * sms * 256. > used * g.N * (waves <= 1. ? 1.45 : 1.25);
}

}  // namespace

bool wide_supported(const WideGemm& g) {
  return g.M >= 1 && g.N >= 1 && g.K >= 8 && g.K % 8 == 0 && g.ldx % 8 == 0 && g.ldx >= g.K &&
         ((reinterpret_cast<uintptr_t>(g.x) | reinterpret_cast<uintptr_t>(g.w)) & 15) == 0;
}

int wide_gemm(const WideGemm& g, cudaStream_t st) {
  if (!wide_supported(g)) B200_FAIL(B200_ERR_SHAPE, "wide GEMM: unsupported shape M=%d N=%d K=%d ld=%lld", g.M, g.N, g.K, g.ldx);
  int dev = 0, sms = 0;
  B200_CUDA(cudaGetDevice(&dev));
  B200_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  WideP p;
  memset(&p, 0, sizeof(p));
  p.M = g.M; p.N = g.N; p.num_kb = ceil_div(g.K, BK); p.packed = g.packed ? 1 : 0; p.act = g.act; p.limit = g.limit;
  p.y = g.y; p.ldy = g.ldy; p.err = g.err;
  p.vec = g.ldy % 8 == 0 && (reinterpret_cast<uintptr_t>(g.y) & 15) == 0;
  if (g.act_to > 0) {
    if (g.tile_e || g.act != WIDE_STORE || !g.y2 || (g.act_from | g.act_to) % 32 || g.act_to > g.N) B200_FAIL(B200_ERR_SHAPE, "wide GEMM: bad range of activated columns");
    p.act_from = g.act_from; p.act_to = g.act_to; p.y2 = g.y2; p.ldy2 = g.ldy2;
    p.vec = p.vec && g.ldy2 % 8 == 0 && (reinterpret_cast<uintptr_t>(g.y2) & 15) == 0;
  }
  if (g.tile_e) {
    p.tile_e = g.tile_e; p.tile_r0 = g.tile_r0; p.tile_n = g.tile_n; p.n_tiles = g.n_tiles; p.y_rows = g.y_rows; p.e_rows = g.e_rows;
    p.mt = g.max_tiles; p.nt = ceil_div(g.N, 256); p.splits = 1; p.kb_per = p.num_kb;
    if (g.max_rows > 0 && g.max_rows <= WIDE_EXPERT_ROWS && experts_win(g, sms)) return launch_experts(g, p, sms, st);      // one tile per expert
    return launch<1, 256>(g, p, sms, st);
  }
  p.mt = ceil_div(g.M, 256);
  p.nt = ceil_div(g.N, 256);
  const int pairs = sms / 2, tiles = p.mt * p.nt;
  // few tiles: k is cut while the pairs of SMs stay in one wave and a range keeps 32 blocks of k.  Writing and adding the partial sums costs
  // about as much as 16 blocks: 1009 x 8192 -> 2048 51.4 us whole, 40.8 in two ranges, 47.8 in four; 300 x 8192 -> 2048 49.1, 37.4, 31.7;
  // 1009 x 2048 -> 2048 18.3, 21.9, 28.5
  int splits = g.splits > 0 ? g.splits : std::min(std::min(pairs / tiles, p.num_kb / 32), 8);
  while (splits > 1 && (!g.ws || (size_t)splits * tiles * 2 * 128 * 256 * 4 > g.ws_bytes || tiles * 2 > g.n_counters)) --splits;
  splits = std::max(1, std::min(splits, p.num_kb));
  p.kb_per = ceil_div(p.num_kb, splits);
  p.splits = ceil_div(p.num_kb, p.kb_per);
  p.ws = g.ws; p.counters = g.counters;
  return launch<2, 256>(g, p, pairs, st);
}

}  // namespace tc
}  // namespace b200

using namespace b200;

extern "C" {

int b200_op_linear_wide(const void* x_dev, const void* w_dev, void* y_dev, int M, int N, int K, int ldy, int packed, int splits, void* stream) {
  if (!x_dev || !w_dev || !y_dev) B200_FAIL(B200_ERR_INVALID, "op_linear_wide: null pointer");
  if (M < 1 || N < 1 || ldy < N || splits < 0 || splits > 64) B200_FAIL(B200_ERR_SHAPE, "op_linear_wide: bad shape");
  tc::WideGemm g;
  g.x = static_cast<const __nv_bfloat16*>(x_dev); g.ldx = K; g.x_rows = M; g.w = w_dev; g.packed = packed != 0; g.w_rows = N;
  g.y = static_cast<__nv_bfloat16*>(y_dev); g.ldy = ldy; g.M = M; g.N = N; g.K = K; g.splits = splits;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t counters = 4096;
  g.ws_bytes = (size_t)ceil_div(M, 256) * ceil_div(N, 256) * 256 * 256 * 4 * (splits > 0 ? splits : 8);
  if (splits == 1 || g.ws_bytes > ((size_t)1 << 30)) return tc::wide_gemm(g, st);
  void* buf = nullptr;
  B200_CUDA(cudaMalloc(&buf, counters * 4 + g.ws_bytes));
  cudaError_t e = cudaMemsetAsync(buf, 0, counters * 4, st);
  g.counters = static_cast<int*>(buf); g.n_counters = (int)counters; g.ws = static_cast<float*>(buf) + counters;
  int rc = e == cudaSuccess ? tc::wide_gemm(g, st) : B200_ERR_CUDA;
  e = cudaStreamSynchronize(st);
  cudaFree(buf);
  if (rc == B200_OK && e != cudaSuccess) { set_error("op_linear_wide: %s", cudaGetErrorString(e)); rc = B200_ERR_CUDA; }
  return rc;
}

int b200_op_grouped_wide(const void* x_dev, const void* w_dev, void* y_dev, const int32_t* counts_host, int E, int M, int N, int K, int ldy,
                         int act, float limit, void* stream) {
  if (!x_dev || !w_dev || !y_dev || !counts_host) B200_FAIL(B200_ERR_INVALID, "op_grouped_wide: null pointer");
  const bool glu = act == tc::WIDE_CLAMPED_GLU || act == tc::WIDE_SILU_GLU;
  if (E < 1 || M < 1 || N < 1 || act < 0 || act > 4 || (glu && N % 2) || ldy < (glu ? N / 2 : N)) B200_FAIL(B200_ERR_SHAPE, "op_grouped_wide: bad shape");
  std::vector<int> te, tr, tn;
  int row = 0, most = 0;
  for (int e = 0; e < E; ++e) {
    if (counts_host[e] < 0 || counts_host[e] > M - row) B200_FAIL(B200_ERR_SHAPE, "op_grouped_wide: the counts do not add up to M");
    for (int r = 0; r < counts_host[e]; r += tc::WIDE_EXPERT_ROWS) {
      te.push_back(e); tr.push_back(row + r); tn.push_back(std::min(tc::WIDE_EXPERT_ROWS, counts_host[e] - r));
    }
    row += counts_host[e];
    most = std::max(most, (int)counts_host[e]);
  }
  if (row != M) B200_FAIL(B200_ERR_SHAPE, "op_grouped_wide: the counts do not add up to M");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int nt = (int)te.size();
  int* table = nullptr;
  B200_CUDA(cudaMalloc(&table, (size_t)(3 * nt + 1) * sizeof(int)));
  std::vector<int> all(te);
  all.insert(all.end(), tr.begin(), tr.end());
  all.insert(all.end(), tn.begin(), tn.end());
  all.push_back(nt);
  cudaError_t e = cudaMemcpyAsync(table, all.data(), all.size() * sizeof(int), cudaMemcpyHostToDevice, st);
  tc::WideGemm g;
  g.x = static_cast<const __nv_bfloat16*>(x_dev); g.ldx = K; g.x_rows = M; g.w = w_dev; g.w_rows = (long long)E * N;
  g.y = static_cast<__nv_bfloat16*>(y_dev); g.ldy = ldy; g.M = M; g.N = N; g.K = K; g.act = act; g.limit = limit;
  g.tile_e = table; g.tile_r0 = table + nt; g.tile_n = table + 2 * nt; g.n_tiles = table + 3 * nt; g.max_tiles = nt; g.e_rows = N; g.max_rows = most;
  int rc = e == cudaSuccess ? tc::wide_gemm(g, st) : B200_ERR_CUDA;
  const cudaError_t e2 = cudaStreamSynchronize(st);
  cudaFree(table);
  if (rc == B200_OK && e2 != cudaSuccess) { set_error("op_grouped_wide: %s", cudaGetErrorString(e2)); rc = B200_ERR_CUDA; }
  return rc;
}

}  // extern "C"
