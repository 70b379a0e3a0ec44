// Stream-K tcgen05 GEMM for the LM linears (see gemm_sk.cuh):  y[M][N] = epi(x[M][K] . w[N][K]^T), bf16 in,
// fp32 accumulate in TMEM, bf16 out; for what the kernels that sk_linear() asks first leave.  M = concurrent sessions (<= 256), so the kernel is a weight
// streamer: every weight byte crosses HBM -> SMEM exactly once and the whole chip pulls on it.
//
//   * Weights are repacked once at load into UMMA-ready tiles: [n_tile][k_block][A][128 rows x 64 k] bf16,
//     each 16 KB tile already in the SWIZZLE_128B K-major shared-memory layout.  A pipeline stage is
//     therefore ONE contiguous `cp.async.bulk` (16 KB, or 32 KB for the gated MLP's gate+value pair).
//   * Work = the linear sequence of (n_tile, k_block) items, cut into equal contiguous ranges, one per
//     CTA (persistent, grid = #SMs): every SM streams the same number of bytes whatever N and K are
//     (out_proj has 32 n-tiles, the text head 250).  A tile whose k-range is cut across CTAs is
//     finished by whichever CTA arrives last: partial accumulators go to an L2-resident workspace and
//     are summed in CTA order, so the result is bit-reproducible and independent of arrival order.
//   * Warp roles (192 threads): warp 0 = bulk-copy/TMA producer, warp 1 = TMEM owner + tcgen05.mma issuer
//     (one thread of either, or the whole warps: sk_linear), warps 2..5 = epilogue (TMEM lane quadrant = warp % 4).  Two TMEM accumulator
//     stages let the epilogue of one segment overlap the MMAs of the next.
#include "gemm_reg.cuh"
#include "gemm_row.cuh"
#include "gemm_sk.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace tc {

namespace {

constexpr int EPI_STORE = 0, EPI_RESADD = 1, EPI_GATE = 2;   // == lm::LIN_*
constexpr int BLOCK_ROWS = 128, BLOCK_K = 64;
constexpr int NUM_THREADS = 192;
constexpr int TILE_BYTES = BLOCK_ROWS * BLOCK_K * 2;   // 16 KB
constexpr int MAX_STAGES = 12;

struct SkParams {
  int M, N, K, Mpad, gate_rows, out_rows;
  int stages, num_kb, n_tiles, n_acc, acc_cols;
  int grid, whole_rounds, sk_tile0, sk_items;   // schedule: tiles [0, sk_tile0) whole, the rest stream-K items
  const uint8_t* wt;            // pre-tiled weights
  __nv_bfloat16* y; long long ldy;
  const __nv_bfloat16* res; long long ldr;
  float* ws;                    // partial slots: [2 * grid][A][Mpad][128] fp32
  int* counters;                // [n_tiles], zero between launches
  uint32_t tmem_cols, stage_bytes;
  int stream_only;              // diagnostics: skip the MMAs (measures the copy pipeline alone)
  // int8 x int8 -> int32 (QLinear, utils/quantize.py:13-40): activations / weights are row-wise absmax int8, the
  // accumulator is dequantised as acc * sa[m] * sw[n] / 127^2; whole tiles only (exact integer sums)
  int i8; const float* sa; const float* sw;
  int late;                     // nothing is read before the wait on the preceding kernel
};

using namespace tcp;
__device__ __forceinline__ void epi_bar_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// ---------------------------------------------------------------------------------------------
// schedule: every CTA first takes its share of the stream-K region (the n_tiles - W*G tiles that do
// not fill a whole round of the grid, cut by k-blocks into G equal contiguous item ranges), then W
// whole tiles (tile = w*G + c).  Partial accumulators are therefore written early in the kernel and
// their reduction overlaps the whole tiles.  All three warp roles walk the same segment list.
// ---------------------------------------------------------------------------------------------
struct Seg { int tile, kb0, kb1, slot; };   // slot: -1 = whole tile, else workspace slot of this partial

__device__ __forceinline__ int sk_begin(const SkParams& p, int c) { return (int)((long long)p.sk_items * c / p.grid); }
// CTA whose stream-K item range holds item j
__device__ __forceinline__ int sk_owner(const SkParams& p, int j) {
  int c = (int)((long long)j * p.grid / p.sk_items);
  while (c + 1 < p.grid && sk_begin(p, c + 1) <= j) ++c;
  while (c > 0 && sk_begin(p, c) > j) --c;
  return c;
}
__device__ __forceinline__ int seg_count(const SkParams& p, int c, int& n_sk) {
  const int a = sk_begin(p, c), b = sk_begin(p, c + 1);
  n_sk = a < b ? (b - 1) / p.num_kb - a / p.num_kb + 1 : 0;
  int n = n_sk;
  for (int w = 0; w < p.whole_rounds; ++w) n += (w * p.grid + c < p.sk_tile0) ? 1 : 0;
  return n;
}
__device__ __forceinline__ Seg seg_get(const SkParams& p, int c, int n_sk, int idx) {
  Seg s;
  if (idx < n_sk) {
    const int a = sk_begin(p, c), b = sk_begin(p, c + 1);
    const int first = a / p.num_kb;
    s.tile = p.sk_tile0 + first + idx;
    s.kb0 = idx == 0 ? a - first * p.num_kb : 0;
    s.kb1 = idx == n_sk - 1 ? (b - 1) % p.num_kb + 1 : p.num_kb;
    s.slot = (s.kb0 == 0 && s.kb1 == p.num_kb) ? -1 : 2 * c + (idx == 0 ? 0 : 1);
  } else {
    s.tile = (idx - n_sk) * p.grid + c;      // rounds are dense: a CTA without a tile in the last round has fewer segments
    s.kb0 = 0; s.kb1 = p.num_kb; s.slot = -1;
  }
  return s;
}

// accumulator word of output (m, weight row nw) as a float: fp32 bits, or int32 x the two row scales (int8 path)
__device__ __forceinline__ float acc_value(const SkParams& p, uint32_t bits, int m, int nw) {
  if (!p.i8) return __uint_as_float(bits);
  return (float)(int)bits * (p.sa[m] * p.sw[nw] * (1.f / 16129.f));
}

// sum of two partial accumulator words: fp32 values, or (int8 path) int32 bit patterns carried in float registers
__device__ __forceinline__ float part_add(bool i8, float a, float b) {
  return i8 ? __int_as_float(__float_as_int(a) + __float_as_int(b)) : a + b;
}

template <int EPI>
__device__ __forceinline__ float epilogue_value(const SkParams& p, float a, float b, int m, int n) {
  if (EPI == EPI_STORE) return a;
  if (EPI == EPI_RESADD) return __bfloat162float(p.res[(long long)m * p.ldr + n]) + bf16_round(a);
  const float g = bf16_round(a), u = bf16_round(b);
  return bf16_round(g / (1.f + expf(-g))) * u;     // bf16(silu(gate)) * value   (gating.py:18-20)
}

template <int EPI, bool WARPS>      // WARPS: whole warps walk the loops of copies and products (sk_linear)
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_sk_kernel(const __grid_constant__ CUtensorMap tmap_x, const SkParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_last;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // SWIZZLE_128B tiles need 1024 B alignment
  const uint32_t bars = base + (uint32_t)p.stages * p.stage_bytes;
  const uint32_t full0 = bars, empty0 = bars + 8 * MAX_STAGES, tfull0 = bars + 16 * MAX_STAGES, tempty0 = tfull0 + 16;
  const uint32_t tptr = tempty0 + 16;
  uint32_t* tptr_generic = reinterpret_cast<uint32_t*>(smem_raw + (tptr - raw));

  const int warp = WARPS ? __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0) : threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int A_TILES = EPI == EPI_GATE ? 2 : 1;
  constexpr uint32_t a_bytes = A_TILES * TILE_BYTES;
  const int c = blockIdx.x;
  int n_sk = 0;
  const int n_seg = seg_count(p, c, n_sk);

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 4);       // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tptr, p.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tptr_generic;
  if (p.late) pdl_wait();
  pdl_trigger();

  // both loops are walked by their whole warps, and one thread issues (tc_prims.cuh), or by one thread
  if (warp == 0) {
    // ===== producer: one contiguous bulk copy of the weight tile(s) + one TMA box of activations per k-block =====
    // Weights do not depend on the preceding kernel: the first `stages` weight tiles are requested before the
    // dependency wait, so under programmatic dependent launch the HBM stream starts while the producer of x
    // is still running.  The activation boxes (and everything the epilogue touches) come after pdl_wait.
    if constexpr (WARPS) {
      int s = 0; uint32_t ph = 0;
      int pre = 0;                                     // stages whose weight copy is already in flight
      for (int si = 0; si < n_seg && pre < p.stages; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        const uint8_t* src = p.wt + ((size_t)sg.tile * p.num_kb + sg.kb0) * a_bytes;
        for (int kb = sg.kb0; kb < sg.kb1 && pre < p.stages; ++kb, src += a_bytes, ++pre) {
          if (elected()) {
            mbar_expect_tx(full0 + 8 * pre, p.stage_bytes);
            bulk_load(base + (uint32_t)pre * p.stage_bytes, src, a_bytes, full0 + 8 * pre);
          }
          __syncwarp();
        }
      }
      pdl_wait();
      int item = 0;
      for (int si = 0; si < n_seg; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        const uint8_t* src = p.wt + ((size_t)sg.tile * p.num_kb + sg.kb0) * a_bytes;
        for (int kb = sg.kb0; kb < sg.kb1; ++kb, src += a_bytes, ++item) {
          const uint32_t sa = base + (uint32_t)s * p.stage_bytes;
          if (item >= pre) mbar_wait(empty0 + 8 * s, ph ^ 1u);
          if (elected()) {
            if (item >= pre) {
              mbar_expect_tx(full0 + 8 * s, p.stage_bytes);
              bulk_load(sa, src, a_bytes, full0 + 8 * s);
            }
            tma_load_2d(sa + a_bytes, &tmap_x, full0 + 8 * s, kb * (p.i8 ? 2 * BLOCK_K : BLOCK_K), 0);   // 128 bytes of K either way
          }
          __syncwarp();
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
    } else if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      int pre = 0;                                   // stages whose weight copy is already in flight
      for (int si = 0; si < n_seg && pre < p.stages; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        const uint8_t* src = p.wt + ((size_t)sg.tile * p.num_kb + sg.kb0) * a_bytes;
        for (int kb = sg.kb0; kb < sg.kb1 && pre < p.stages; ++kb, src += a_bytes, ++pre) {
          mbar_expect_tx(full0 + 8 * pre, p.stage_bytes);
          bulk_load(base + (uint32_t)pre * p.stage_bytes, src, a_bytes, full0 + 8 * pre);
        }
      }
      pdl_wait();
      int item = 0;
      for (int si = 0; si < n_seg; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        const uint8_t* src = p.wt + ((size_t)sg.tile * p.num_kb + sg.kb0) * a_bytes;
        for (int kb = sg.kb0; kb < sg.kb1; ++kb, src += a_bytes, ++item) {
          const uint32_t sa = base + (uint32_t)s * p.stage_bytes;
          if (item >= pre) {
            mbar_wait(empty0 + 8 * s, ph ^ 1u);
            mbar_expect_tx(full0 + 8 * s, p.stage_bytes);
            bulk_load(sa, src, a_bytes, full0 + 8 * s);
          }
          tma_load_2d(sa + a_bytes, &tmap_x, full0 + 8 * s, kb * (p.i8 ? 2 * BLOCK_K : BLOCK_K), 0);   // 128 bytes of K either way
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer =====
    const uint32_t idesc = p.i8 ? make_idesc_i8(BLOCK_ROWS, p.Mpad) : make_idesc(BLOCK_ROWS, p.Mpad);
    int s = 0; uint32_t ph = 0;
    int acc = 0; uint32_t acc_bits = 0u;         // bit a = phase parity of accumulator stage a
    if constexpr (WARPS) {
      for (int si = 0; si < n_seg; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        mbar_wait(tempty0 + 8 * acc, ((acc_bits >> acc) & 1u) ^ 1u);          // epilogue has drained this accumulator
        tc_fence_after();
        const uint32_t d0 = tmem_base + (uint32_t)(acc * p.acc_cols);
        for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
          mbar_wait(full0 + 8 * s, ph);
          tc_fence_after();
          if (!p.stream_only) {
            const uint32_t sa = desc_low(base + (uint32_t)s * p.stage_bytes), accum = kb == sg.kb0 ? 0u : 1u;
            // one MMA consumes 32 bytes of K per row either way: 16 bf16 or 32 int8
            if (p.i8) {
              umma_block_i8(d0, sa, a_bytes >> 4, idesc, accum);
              if (EPI == EPI_GATE) umma_block_i8(d0 + (uint32_t)p.Mpad, sa + (TILE_BYTES >> 4), (a_bytes - TILE_BYTES) >> 4, idesc, accum);
            } else {
              umma_block<1>(d0, sa, a_bytes >> 4, idesc, accum);
              if (EPI == EPI_GATE) umma_block<1>(d0 + (uint32_t)p.Mpad, sa + (TILE_BYTES >> 4), (a_bytes - TILE_BYTES) >> 4, idesc, accum);
            }
          }
          commit_elected(empty0 + 8 * s);        // frees the smem stage once these MMAs have read it
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        commit_elected(tfull0 + 8 * acc);        // segment accumulated
        acc_bits ^= 1u << acc;
        if (p.n_acc == 2) acc ^= 1;
      }
    } else if (lane == 0) {
      for (int si = 0; si < n_seg; ++si) {
        const Seg sg = seg_get(p, c, n_sk, si);
        mbar_wait(tempty0 + 8 * acc, ((acc_bits >> acc) & 1u) ^ 1u);
        tc_fence_after();
        const uint32_t d0 = tmem_base + (uint32_t)(acc * p.acc_cols);
        for (int kb = sg.kb0; kb < sg.kb1; ++kb) {
          mbar_wait(full0 + 8 * s, ph);
          tc_fence_after();
          if (!p.stream_only) {
            const uint32_t sa = base + (uint32_t)s * p.stage_bytes, sb = sa + a_bytes;
#pragma unroll
            for (int k = 0; k < BLOCK_K * 2; k += 32) {
              const uint64_t db = make_desc(sb + k);
              const uint32_t accum = (kb == sg.kb0 && k == 0) ? 0u : 1u;
              if (p.i8) {
                umma_i8(d0, make_desc(sa + k), db, idesc, accum);
                if (EPI == EPI_GATE) umma_i8(d0 + (uint32_t)p.Mpad, make_desc(sa + TILE_BYTES + k), db, idesc, accum);
              } else {
                umma_bf16(d0, make_desc(sa + k), db, idesc, accum);
                if (EPI == EPI_GATE) umma_bf16(d0 + (uint32_t)p.Mpad, make_desc(sa + TILE_BYTES + k), db, idesc, accum);
              }
            }
          }
          umma_commit(empty0 + 8 * s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        umma_commit(tfull0 + 8 * acc);
        acc_bits ^= 1u << acc;
        if (p.n_acc == 2) acc ^= 1;
      }
    }
    __syncwarp();
  } else {
    // ===== epilogue: TMEM -> registers -> (global | workspace + last-arriver reduction) =====
    const int q = warp & 3;                    // TMEM lane quadrant this warp may access
    const int row = q * 32 + lane;
    const int et = threadIdx.x - 64;           // 0..127
    const size_t slot_floats = (size_t)A_TILES * BLOCK_ROWS * p.Mpad;
    int acc = 0; uint32_t acc_bits = 0u;
    pdl_wait();                                // y / res / workspace / counters may still be in use by the predecessor
    for (int si = 0; si < n_seg; ++si) {
      const Seg sg = seg_get(p, c, n_sk, si);
      const int n = sg.tile * BLOCK_ROWS + row;
      const bool n_ok = n < p.out_rows;
      mbar_wait(tfull0 + 8 * acc, (acc_bits >> acc) & 1u);
      tc_fence_after();
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * p.acc_cols);
      if (sg.slot < 0) {
        for (int c0 = 0; c0 < p.Mpad; c0 += 16) {
          uint32_t r0[16], r1[16];
          // the 16 residual reads of this column chunk are issued together, ahead of the TMEM load they are added to
          // (one dependent global load per element would cost a DRAM/L2 latency each: 96 of them per thread at B=96)
          float rv[16];
          if (EPI == EPI_RESADD && !p.stream_only) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int m = c0 + j;
              rv[j] = (m < p.M && n_ok) ? __bfloat162float(p.res[(long long)m * p.ldr + n]) : 0.f;
            }
          }
          tmem_ld16(lane_addr + (uint32_t)c0, r0);
          if (EPI == EPI_GATE) tmem_ld16(lane_addr + (uint32_t)(p.Mpad + c0), r1);
          tmem_ld_wait();
          if (!p.stream_only) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int m = c0 + j;
              if (m < p.M && n_ok) {
                float v;
                if (EPI == EPI_RESADD) v = rv[j] + bf16_round(acc_value(p, r0[j], m, n));
                else v = epilogue_value<EPI>(p, acc_value(p, r0[j], m, n), EPI == EPI_GATE ? acc_value(p, r1[j], m, p.gate_rows + n) : 0.f, m, n);
                p.y[(long long)m * p.ldy + n] = __float2bfloat16_rn(v);
              }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
      } else {
        // partial accumulator -> workspace slot, layout [A][128 rows][Mpad] (a thread owns one contiguous row)
        float* wrow = p.ws + (size_t)sg.slot * slot_floats + (size_t)row * p.Mpad;
        for (int c0 = 0; c0 < p.Mpad; c0 += 16) {
          uint32_t r0[16], r1[16];
          tmem_ld16(lane_addr + (uint32_t)c0, r0);
          if (EPI == EPI_GATE) tmem_ld16(lane_addr + (uint32_t)(p.Mpad + c0), r1);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            __stcg(reinterpret_cast<float4*>(wrow + c0 + j),
                   make_float4(__uint_as_float(r0[j]), __uint_as_float(r0[j + 1]), __uint_as_float(r0[j + 2]), __uint_as_float(r0[j + 3])));
            if (EPI == EPI_GATE)
              __stcg(reinterpret_cast<float4*>(wrow + (size_t)BLOCK_ROWS * p.Mpad + c0 + j),
                     make_float4(__uint_as_float(r1[j]), __uint_as_float(r1[j + 1]), __uint_as_float(r1[j + 2]), __uint_as_float(r1[j + 3])));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
        // publish, count arrivals; the last arriver of this tile reduces all partials in CTA order
        __threadfence();
        epi_bar_sync();
        const int rel = sg.tile - p.sk_tile0;
        const int first_c = sk_owner(p, rel * p.num_kb), last_c = sk_owner(p, (rel + 1) * p.num_kb - 1);
        if (et == 0) {
          const int old = atomicAdd(p.counters + sg.tile, 1);
          const int last = old == last_c - first_c;
          s_last = last;
          if (last) p.counters[sg.tile] = 0;                     // ready for the next launch
        }
        epi_bar_sync();
        if (s_last) {
          __threadfence();
          // 16 columns per pass: every contribution's 4 (gate: 8) 16-byte loads are issued before the adds
          for (int m0 = 0; m0 < p.M; m0 += 16) {
            float av[16], bv[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) { av[j] = 0.f; bv[j] = 0.f; }
#pragma unroll 2
            for (int cc = first_c; cc <= last_c; ++cc) {
              const int sl = 2 * cc + ((sk_begin(p, cc) / p.num_kb == rel) ? 0 : 1);
              const float4* w2 = reinterpret_cast<const float4*>(p.ws + (size_t)sl * slot_floats + (size_t)row * p.Mpad + m0);
              float4 v[4], u[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) v[j] = __ldcg(w2 + j);
              if (EPI == EPI_GATE) {
#pragma unroll
                for (int j = 0; j < 4; ++j) u[j] = __ldcg(w2 + (size_t)BLOCK_ROWS * p.Mpad / 4 + j);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const bool q8 = p.i8 != 0;
                av[4 * j] = part_add(q8, av[4 * j], v[j].x); av[4 * j + 1] = part_add(q8, av[4 * j + 1], v[j].y);
                av[4 * j + 2] = part_add(q8, av[4 * j + 2], v[j].z); av[4 * j + 3] = part_add(q8, av[4 * j + 3], v[j].w);
                if (EPI == EPI_GATE) {
                  bv[4 * j] = part_add(q8, bv[4 * j], u[j].x); bv[4 * j + 1] = part_add(q8, bv[4 * j + 1], u[j].y);
                  bv[4 * j + 2] = part_add(q8, bv[4 * j + 2], u[j].z); bv[4 * j + 3] = part_add(q8, bv[4 * j + 3], u[j].w);
                }
              }
            }
            if (n_ok && !p.stream_only) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const int m = m0 + j;
                if (m < p.M) {
                  // fp32 zero and int32 zero share a bit pattern, so the accumulators start right on both paths
                  const float a = acc_value(p, __float_as_uint(av[j]), m, n);
                  const float b = EPI == EPI_GATE ? acc_value(p, __float_as_uint(bv[j]), m, p.gate_rows + n) : 0.f;
                  p.y[(long long)m * p.ldy + n] = __float2bfloat16_rn(epilogue_value<EPI>(p, a, b, m, n));
                }
              }
            }
          }
        }
      }
      acc_bits ^= 1u << acc;
      if (p.n_acc == 2) acc ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, p.tmem_cols);
}

// ---------------------------------------------------------------------------------------------
// Cluster split-K ("ck") for the few-tile GEMMs at more than 32 sessions (out_proj / linear_out: 32 row tiles).
// A cluster of CS CTAs owns one 128-row tile; rank r streams k-blocks [r*kb_per, (r+1)*kb_per) into its own TMEM
// accumulator.  The partials are then reduce-scattered over distributed shared memory: rank q is sent columns
// [q*Wc, (q+1)*Wc) of everybody's accumulator (st.shared::cluster into its receive buffer), one cluster barrier,
// and every rank sums its column block in rank order (deterministic) and runs the epilogue for it.  No global
// workspace, no atomics; CS x more SMs pull on the weights and the epilogue is spread over the cluster too.
// ---------------------------------------------------------------------------------------------
struct CkParams {
  int M, N, K, Mpad, CS, Wc, kb_per, num_kb, stages;
  const uint8_t* wt;
  __nv_bfloat16* y; long long ldy;
  const __nv_bfloat16* res; long long ldr;
  uint32_t tmem_cols, stage_bytes;
  int i8; const float* sa; const float* sw;      // int8 operands: partials are exact int32, scaled once after the reduction
  int late;                                      // nothing is read before the wait on the preceding kernel
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int EPI>      // EPI_STORE or EPI_RESADD
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_ck_kernel(const __grid_constant__ CUtensorMap tmap_x, const CkParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + (uint32_t)p.stages * p.stage_bytes;
  const uint32_t full0 = bars, empty0 = bars + 8 * MAX_STAGES, tfull = bars + 16 * MAX_STAGES;
  const uint32_t tptr = tfull + 8;
  uint32_t* tptr_generic = reinterpret_cast<uint32_t*>(smem_raw + (tptr - raw));
  // receive buffer [CS][128 rows][Wc + 4] fp32 (rows padded against bank conflicts), after the barrier block
  const int ldw = p.Wc + 4;
  const uint32_t recv = (tptr + 8 + 15u) & ~15u;
  float* recv_generic = reinterpret_cast<float*>(smem_raw + (recv - raw));

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int tile = blockIdx.x / p.CS, me = blockIdx.x - tile * p.CS;
  const int kb0 = me * p.kb_per, kb1 = min(p.num_kb, kb0 + p.kb_per);

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(tfull, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tptr, p.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tptr_generic;
  if (p.late) pdl_wait();
  pdl_trigger();

  // both loops are walked by their whole warps, and one thread issues (tc_prims.cuh)
  if (warp == 0) {
    // weights first (they do not depend on the preceding kernel), activations after the dependency wait
    const uint8_t* src = p.wt + ((size_t)tile * p.num_kb + kb0) * TILE_BYTES;
    const int n_items = kb1 - kb0;
    const int pre = n_items < p.stages ? n_items : p.stages;
    for (int i = 0; i < pre; ++i) {
      if (elected()) {
        mbar_expect_tx(full0 + 8 * i, p.stage_bytes);
        bulk_load(base + (uint32_t)i * p.stage_bytes, src + (size_t)i * TILE_BYTES, TILE_BYTES, full0 + 8 * i);
      }
      __syncwarp();
    }
    pdl_wait();
    int s = 0; uint32_t ph = 0;
    for (int i = 0; i < n_items; ++i) {
      const uint32_t sa = base + (uint32_t)s * p.stage_bytes;
      if (i >= pre) mbar_wait(empty0 + 8 * s, ph ^ 1u);
      if (elected()) {
        if (i >= pre) {
          mbar_expect_tx(full0 + 8 * s, p.stage_bytes);
          bulk_load(sa, src + (size_t)i * TILE_BYTES, TILE_BYTES, full0 + 8 * s);
        }
        tma_load_2d(sa + TILE_BYTES, &tmap_x, full0 + 8 * s, (kb0 + i) * (p.i8 ? 2 * BLOCK_K : BLOCK_K), 0);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1u; }
    }
  } else if (warp == 1) {
    const uint32_t idesc = p.i8 ? make_idesc_i8(BLOCK_ROWS, p.Mpad) : make_idesc(BLOCK_ROWS, p.Mpad);
    int s = 0; uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(full0 + 8 * s, ph);
      tc_fence_after();
      const uint32_t sa = desc_low(base + (uint32_t)s * p.stage_bytes), accum = kb == kb0 ? 0u : 1u;
      if (p.i8) umma_block_i8(tmem_base, sa, TILE_BYTES >> 4, idesc, accum);
      else umma_block<1>(tmem_base, sa, TILE_BYTES >> 4, idesc, accum);
      commit_elected(empty0 + 8 * s);
      if (++s == p.stages) { s = 0; ph ^= 1u; }
    }
    commit_elected(tfull);
    __syncwarp();
  }
  float own[64];                               // this rank's column block of its own accumulator (Wc <= 64)
  const int q4 = warp & 3;
  const int row = q4 * 32 + lane;
  if (warp >= 2) {
    pdl_wait();
    mbar_wait(tfull, 0);
    tc_fence_after();
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q4 * 32) << 16);
    for (int q = 0; q < p.CS; ++q) {
      const uint32_t dst = map_to_rank(recv + (uint32_t)((me * BLOCK_ROWS + row) * ldw) * 4u, (uint32_t)q);
#pragma unroll
      for (int c0 = 0; c0 < 64; c0 += 8) {
        if (c0 < p.Wc) {
          uint32_t r[8];
          tmem_ld8(lane_addr + (uint32_t)(q * p.Wc + c0), r);
          tmem_ld_wait();
          if (kb1 <= kb0) {                    // a rank without k-blocks contributes zeros
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = 0u;
          }
          if (q == me) {
#pragma unroll
            for (int j = 0; j < 8; ++j) own[c0 + j] = __uint_as_float(r[j]);
          } else {
            st_cluster_v4(dst + (uint32_t)c0 * 4u, __uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
            st_cluster_v4(dst + (uint32_t)(c0 + 4) * 4u, __uint_as_float(r[4]), __uint_as_float(r[5]), __uint_as_float(r[6]), __uint_as_float(r[7]));
          }
        }
      }
    }
    tc_fence_before();
  }
  cluster_sync_all();                          // every partial has landed in its owner's receive buffer
  if (warp >= 2) {
    const int n = tile * BLOCK_ROWS + row;
    const bool n_ok = n < p.N;
#pragma unroll
    for (int c0 = 0; c0 < 64; c0 += 8) {
      if (c0 < p.Wc) {
        float rv[8];
        if (EPI == EPI_RESADD) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = me * p.Wc + c0 + j;
            rv[j] = (m < p.M && n_ok) ? __bfloat162float(p.res[(long long)m * p.ldr + n]) : 0.f;
          }
        }
        float acc[8];
        if (p.i8) {                            // exact: the partials are int32 bit patterns
          int isum[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) isum[j] = 0;
          for (int r = 0; r < p.CS; ++r) {
            if (r == me) {
#pragma unroll
              for (int j = 0; j < 8; ++j) isum[j] += __float_as_int(own[c0 + j]);
            } else {
              const int4 a = *reinterpret_cast<const int4*>(recv_generic + (size_t)(r * BLOCK_ROWS + row) * ldw + c0);
              const int4 b = *reinterpret_cast<const int4*>(recv_generic + (size_t)(r * BLOCK_ROWS + row) * ldw + c0 + 4);
              isum[0] += a.x; isum[1] += a.y; isum[2] += a.z; isum[3] += a.w;
              isum[4] += b.x; isum[5] += b.y; isum[6] += b.z; isum[7] += b.w;
            }
          }
          const float swn = n_ok ? p.sw[n] : 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int m = me * p.Wc + c0 + j;
            acc[j] = m < p.M ? (float)isum[j] * (p.sa[m] * swn * (1.f / 16129.f)) : 0.f;     // same expression as acc_value()
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[j] = 0.f;
          for (int r = 0; r < p.CS; ++r) {       // rank order: the sum does not depend on which rank does it
            if (r == me) {
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[j] += own[c0 + j];
            } else {
              const float4 a = *reinterpret_cast<const float4*>(recv_generic + (size_t)(r * BLOCK_ROWS + row) * ldw + c0);
              const float4 b = *reinterpret_cast<const float4*>(recv_generic + (size_t)(r * BLOCK_ROWS + row) * ldw + c0 + 4);
              acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
              acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int m = me * p.Wc + c0 + j;
          if (m < p.M && n_ok) {
            const float v = EPI == EPI_RESADD ? rv[j] + bf16_round(acc[j]) : acc[j];
            p.y[(long long)m * p.ldy + n] = __float2bfloat16_rn(v);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, p.tmem_cols);
}

// load-time repack: w [rows][K] row-major -> tiles [n_tile][kb][A][128 x 64] in the SWIZZLE_128B layout
// (16-byte chunk c of row r sits at r*128 + ((c ^ (r & 7)) << 4)); rows/cols beyond the tensor are zero.
__global__ void pack_tiles_kernel(const __nv_bfloat16* __restrict__ w, uint4* __restrict__ out, int rows, int K, int n_tiles,
                                  int num_kb, int a_tiles, int gate_rows) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;        // one 16-byte chunk each
  const long long total = (long long)n_tiles * num_kb * a_tiles * (TILE_BYTES / 16);
  if (idx >= total) return;
  const int chunk = (int)(idx % (TILE_BYTES / 16));
  long long t = idx / (TILE_BYTES / 16);
  const int a = (int)(t % a_tiles); t /= a_tiles;
  const int kb = (int)(t % num_kb);
  const int tile = (int)(t / num_kb);
  const int r = chunk >> 3, cpos = chunk & 7;
  const int csrc = cpos ^ (r & 7);                               // logical chunk stored at this position
  const int limit = a_tiles == 2 ? gate_rows : rows;
  const int rr = tile * BLOCK_ROWS + r;
  const int k = kb * BLOCK_K + csrc * 8;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (rr < limit && k < K) v = *reinterpret_cast<const uint4*>(w + (long long)(rr + a * gate_rows) * K + k);
  out[idx] = v;
}

// ---- int8 quantisation (QLinear: bnb int8_vectorwise_quant, utils/quantize.py:16-20,38) -----------------------------------
// row-wise absmax of w[rows][K] taken on the fp16 values (the reference quantises weight.to(float16))
__global__ void row_absmax_f16_kernel(const __nv_bfloat16* __restrict__ w, float* __restrict__ out, int rows, int K) {
  const int row = blockIdx.x;
  float mx = 0.f;
  for (int k = threadIdx.x; k < K; k += blockDim.x)
    mx = fmaxf(mx, fabsf(__half2float(__float2half_rn(__bfloat162float(w[(long long)row * K + k])))));
  __shared__ float red[32];
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < (int)(blockDim.x + 31) / 32; ++i) t = fmaxf(t, red[i]);
    out[row] = t;
  }
}
__device__ __forceinline__ int quant_i8(float v, float inv) {           // round(v * 127 / absmax), ties to even (torch.round)
  int q = __float2int_rn(v * inv);
  return q > 127 ? 127 : (q < -127 ? -127 : q);
}
// w [rows][K] -> int8 tiles [n_tile][kb][A][128 rows x 128 k] in the SWIZZLE_128B layout (one 16-byte chunk = 16 k per thread)
__global__ void pack_tiles_i8_kernel(const __nv_bfloat16* __restrict__ w, const float* __restrict__ absmax, uint4* __restrict__ out,
                                     int rows, int K, int n_tiles, int num_kb, int a_tiles, int gate_rows) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)n_tiles * num_kb * a_tiles * (TILE_BYTES / 16);
  if (idx >= total) return;
  const int chunk = (int)(idx % (TILE_BYTES / 16));
  long long t = idx / (TILE_BYTES / 16);
  const int a = (int)(t % a_tiles); t /= a_tiles;
  const int kb = (int)(t % num_kb);
  const int tile = (int)(t / num_kb);
  const int r = chunk >> 3, cpos = chunk & 7;
  const int csrc = cpos ^ (r & 7);
  const int limit = a_tiles == 2 ? gate_rows : rows;
  const int rr = tile * BLOCK_ROWS + r;
  const int k0 = kb * 128 + csrc * 16;
  uint32_t words[4] = {0u, 0u, 0u, 0u};
  if (rr < limit) {
    const long long srow = (long long)(rr + a * gate_rows);
    const float am = absmax[srow];
    const float inv = am > 0.f ? 127.f / am : 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int k = k0 + j;
      int q = 0;
      if (k < K) q = quant_i8(__half2float(__float2half_rn(__bfloat162float(w[srow * K + k]))), inv);
      words[j >> 2] |= (uint32_t)(q & 0xFF) << (8 * (j & 3));
    }
  }
  out[idx] = make_uint4(words[0], words[1], words[2], words[3]);
}
// already-quantised weights (a QLinear's CB as stored in model.q8.safetensors): q int8 [rows][K] -> the same int8 tiles
__global__ void pack_tiles_i8_pre_kernel(const int8_t* __restrict__ q, uint4* __restrict__ out, int rows, int K, int n_tiles, int num_kb,
                                         int a_tiles, int gate_rows) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)n_tiles * num_kb * a_tiles * (TILE_BYTES / 16);
  if (idx >= total) return;
  const int chunk = (int)(idx % (TILE_BYTES / 16));
  long long t = idx / (TILE_BYTES / 16);
  const int a = (int)(t % a_tiles); t /= a_tiles;
  const int kb = (int)(t % num_kb);
  const int tile = (int)(t / num_kb);
  const int r = chunk >> 3, cpos = chunk & 7;
  const int csrc = cpos ^ (r & 7);
  const int limit = a_tiles == 2 ? gate_rows : rows;
  const int rr = tile * BLOCK_ROWS + r;
  const int k0 = kb * 128 + csrc * 16;
  uint32_t words[4] = {0u, 0u, 0u, 0u};
  if (rr < limit) {
    const long long srow = (long long)(rr + a * gate_rows);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int k = k0 + j;
      const int v = k < K ? (int)q[srow * K + k] : 0;
      words[j >> 2] |= (uint32_t)(v & 0xFF) << (8 * (j & 3));
    }
  }
  out[idx] = make_uint4(words[0], words[1], words[2], words[3]);
}
// activations: x [M][K] bf16 (row stride ldx) -> xq int8 [M][K], sa[m] = absmax of the row
__global__ void __launch_bounds__(256) quantize_rows_kernel(const __nv_bfloat16* x, long long ldx, int8_t* xq,
                                                           float* sa, int K) {
  const int row = blockIdx.x;
  const __nv_bfloat16* xr = x + (long long)row * ldx;
  float mx = 0.f;
  pdl_wait();          // x comes from the preceding kernel; xq / sa may still be read by the GEMM before that one
  pdl_trigger();       // the GEMM that follows starts streaming its weight tiles while the rows are quantised
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + k);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      mx = fmaxf(mx, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  __shared__ float red[8];
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  float am = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) am = fmaxf(am, red[i]);
  if (threadIdx.x == 0) sa[row] = am;
  const float inv = am > 0.f ? 127.f / am : 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(xr + k);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
    uint32_t w0 = 0u, w1 = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      const uint32_t a = (uint32_t)(quant_i8(f.x, inv) & 0xFF), b = (uint32_t)(quant_i8(f.y, inv) & 0xFF);
      if (i < 2) w0 |= (a | (b << 8)) << (16 * i);
      else w1 |= (a | (b << 8)) << (16 * (i - 2));
    }
    *reinterpret_cast<uint2*>(xq + (long long)row * K + k) = make_uint2(w0, w1);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
bool g_settings_read = false;
int g_sms = 0;
int g_row_max_m = ROW_MAX_M;     // B200_ROW_MAX_M (0..16): rows up to which gemm_row_kernel is considered
int g_use_ns = 1;                // B200_GEMM_NS=0: keep the swap-AB kernels above 32 sessions (A/B measurements)

int init_once() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    B200_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
    if (!fn || qres != cudaDriverEntryPointSuccess) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  static std::atomic<uint64_t> limits{0};
  // the kernels also have a few bytes of static shared memory
  B200_TRY(allow_smem(limits, 220 * 1024, gemm_sk_kernel<EPI_STORE, false>, gemm_sk_kernel<EPI_STORE, true>, gemm_sk_kernel<EPI_RESADD, false>, gemm_sk_kernel<EPI_RESADD, true>,
                      gemm_sk_kernel<EPI_GATE, false>, gemm_sk_kernel<EPI_GATE, true>, gemm_ck_kernel<EPI_STORE>, gemm_ck_kernel<EPI_RESADD>));
  if (!g_settings_read) {
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
    const char* rows = getenv("B200_ROW_MAX_M");
    if (!rows) rows = getenv("B200_GEMV_MAX_M");      // the name that it had when fewer rows were possible
    if (rows) g_row_max_m = atoi(rows);
    if (const char* e = getenv("B200_GEMM_NS")) g_use_ns = atoi(e);
    g_settings_read = true;
  }
  return B200_OK;
}

}  // namespace

int prepare_plans(GemmPlanCache&) { B200_TRY(ns_prepare()); return init_once(); }

int sk_num_sms() { return init_once() == B200_OK ? g_sms : 0; }

int sk_set_row_max_m(int max_m) {
  if (init_once() != B200_OK) return -1;
  const int before = g_row_max_m;
  g_row_max_m = max_m < 0 ? 0 : max_m > ROW_MAX_M ? ROW_MAX_M : max_m;
  return before;
}

size_t sk_packed_bytes(int N, int K, int epi, int gate_rows) {
  const int a = epi == EPI_GATE ? 2 : 1;
  const int rows = epi == EPI_GATE ? gate_rows : N;
  return (size_t)((rows + BLOCK_ROWS - 1) / BLOCK_ROWS) * ((K + BLOCK_K - 1) / BLOCK_K) * a * TILE_BYTES;
}

int sk_pack_weights(const __nv_bfloat16* w, void* out, int N, int K, int epi, int gate_rows, cudaStream_t stream) {
  const int a = epi == EPI_GATE ? 2 : 1;
  const int rows = epi == EPI_GATE ? gate_rows : N;
  const int n_tiles = (rows + BLOCK_ROWS - 1) / BLOCK_ROWS, num_kb = (K + BLOCK_K - 1) / BLOCK_K;
  if (K % 8) B200_FAIL(B200_ERR_SHAPE, "sk_pack_weights: K must be a multiple of 8");
  const long long total = (long long)n_tiles * num_kb * a * (TILE_BYTES / 16);
  pack_tiles_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(w, static_cast<uint4*>(out), epi == EPI_GATE ? 2 * gate_rows : N,
                                                                       K, n_tiles, num_kb, a, epi == EPI_GATE ? gate_rows : 0);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("pack_tiles");
}

size_t sk_packed_bytes_i8(int N, int K, int epi, int gate_rows) {
  const int a = epi == EPI_GATE ? 2 : 1;
  const int rows = epi == EPI_GATE ? gate_rows : N;
  return (size_t)((rows + BLOCK_ROWS - 1) / BLOCK_ROWS) * ((K + 127) / 128) * a * TILE_BYTES;
}

int sk_quant_pack_weights(const __nv_bfloat16* w, void* out_tiles, float* out_scales, int N, int K, int epi, int gate_rows,
                          cudaStream_t stream) {
  if (K % 16) B200_FAIL(B200_ERR_SHAPE, "sk_quant_pack_weights: K must be a multiple of 16");
  const int a = epi == EPI_GATE ? 2 : 1;
  const int w_rows = epi == EPI_GATE ? 2 * gate_rows : N;
  const int rows = epi == EPI_GATE ? gate_rows : N;
  const int n_tiles = (rows + BLOCK_ROWS - 1) / BLOCK_ROWS, num_kb = (K + 127) / 128;
  row_absmax_f16_kernel<<<w_rows, 256, 0, stream>>>(w, out_scales, w_rows, K);
  const long long total = (long long)n_tiles * num_kb * a * (TILE_BYTES / 16);
  pack_tiles_i8_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(w, out_scales, static_cast<uint4*>(out_tiles), w_rows, K,
                                                                           n_tiles, num_kb, a, epi == EPI_GATE ? gate_rows : 0);
  g_launches.fetch_add(2, std::memory_order_relaxed);
  return check_launch("quant_pack_tiles");
}

int sk_pack_weights_i8(const int8_t* q, void* out_tiles, int N, int K, int epi, int gate_rows, cudaStream_t stream) {
  if (K % 16) B200_FAIL(B200_ERR_SHAPE, "sk_pack_weights_i8: K must be a multiple of 16");
  const int a = epi == EPI_GATE ? 2 : 1;
  const int w_rows = epi == EPI_GATE ? 2 * gate_rows : N;
  const int rows = epi == EPI_GATE ? gate_rows : N;
  const int n_tiles = (rows + BLOCK_ROWS - 1) / BLOCK_ROWS, num_kb = (K + 127) / 128;
  const long long total = (long long)n_tiles * num_kb * a * (TILE_BYTES / 16);
  pack_tiles_i8_pre_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(q, static_cast<uint4*>(out_tiles), w_rows, K, n_tiles, num_kb,
                                                                              a, epi == EPI_GATE ? gate_rows : 0);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("pack_tiles_i8_pre");
}

int sk_quantize_rows(const __nv_bfloat16* x, long long ldx, void* xq, float* sa, int M, int K, cudaStream_t stream, int pdl) {
  if (K % 8 || ldx % 8) B200_FAIL(B200_ERR_SHAPE, "sk_quantize_rows: K and the row stride must be multiples of 8");
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)M); cfg.blockDim = dim3(256); cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = pdl ? 1 : 0;
  B200_CUDA(cudaLaunchKernelEx(&cfg, quantize_rows_kernel, x, ldx, static_cast<int8_t*>(xq), sa, K));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("quantize_rows");
}

size_t sk_workspace_bytes(int max_M) {
  const int Mpad = ((max_M + 15) / 16) * 16;
  return (size_t)2 * SK_MAX_GRID * 2 * Mpad * BLOCK_ROWS * 4;  // 2 slots per CTA, gate + value accumulators
}

bool sk_supported(int M, int N, int K, int epi) {
  (void)N; (void)epi;
  return M >= 1 && M <= 256 && K >= 8 && K % 8 == 0;
}

// 2-D tensor map of the activations x [M][K] (row stride ldx elements) with a [box_rows x 128 bytes] SWIZZLE_128B box;
// elem_bytes = 2 (bf16) or 1 (int8)
static int x_map(GemmPlanCache& cache, const void* x, long long ldx, int M, int K, int box_rows, int elem_bytes,
                 const CUtensorMap** out) {
  PlanKey key{x, ldx, M, K, box_rows};
  auto it = cache.maps.find(key);
  if (it == cache.maps.end()) {
    CUtensorMap m;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    cuuint64_t strides[1] = {(cuuint64_t)ldx * elem_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(128 / elem_bytes), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode(&m, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                          const_cast<void*>(x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) M=%d K=%d ld=%lld", (int)r, M, K, ldx);
    it = cache.maps.emplace(key, m).first;
  }
  *out = &it->second;
  return B200_OK;
}

// y = epi(x . W^T) with W given as packed tiles.  ws / counters: sk_workspace_bytes(M) and >= 1024 ints, zeroed once.
int sk_linear(GemmPlanCache& cache, const __nv_bfloat16* x, long long ldx, const void* w_tiles, __nv_bfloat16* y,
              long long ldy, const __nv_bfloat16* res, long long ldr, int M, int N, int K, int epi, int gate_rows,
              float* ws, int* counters, const SkTuning& tune, cudaStream_t stream) {
  if (!sk_supported(M, N, K, epi) || ldx % 8) B200_FAIL(B200_ERR_SHAPE, "sk GEMM: unsupported shape M=%d N=%d K=%d", M, N, K);
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_tiles)) & 15)
    B200_FAIL(B200_ERR_SHAPE, "sk GEMM: operands must be 16-byte aligned");
  B200_TRY(init_once());
  const bool i8 = tune.xq != nullptr;
  // up to 16 sessions: whole output rows per CTA (gemm_row.cu); explicit grids, clusters and the copy diagnostics keep the kernels below
  const bool chosen = tune.grid == 0 && tune.cluster == 0 && !tune.stream_only && !tune.force_split && !tune.no_split && tune.smem_budget == 0 && tune.ns == 0;
  const void* rows = i8 ? tune.xq : x;
  const long long row_ld = i8 ? (long long)K : 2 * ldx;
  const bool scaled = !i8 || (K % 16 == 0 && tune.sa && tune.sw);
  if (chosen && scaled && M <= g_row_max_m && row_wins(M, epi, gate_rows, i8, g_sms) && row_supported(M, K, i8, rows, row_ld))
    return row_linear(rows, row_ld, w_tiles, y, ldy, res, ldr, M, N, K, epi, gate_rows, i8 ? tune.sa : nullptr, tune.sw, g_sms, tune.pdl, stream);
  const int n_tiles = (N + BLOCK_ROWS - 1) / BLOCK_ROWS, k_blocks = i8 ? (K + 127) / 128 : (K + BLOCK_K - 1) / BLOCK_K;
  int ranks = 1;                                          // few tiles: K over a cluster (gemm_ck_kernel)
  while (ranks < 8 && n_tiles * ranks * 2 <= g_sms && k_blocks / (ranks * 2) >= 4 && (ranks < 4 || n_tiles <= 15)) ranks *= 2;      // 15 clusters of eight fit at a time
  if (tune.cluster > 0) ranks = tune.cluster;
  const int quantum = 8 * ranks < 16 ? 16 : 8 * ranks;    // UMMA N is a multiple of 16; every rank owns whole 8-column groups
  const int ck_pad = ((M + quantum - 1) / quantum) * quantum;
  const bool ck = epi != EPI_GATE && tune.no_cluster == 0 && tune.grid == 0 && M > 32 && ranks > 1 && ck_pad <= 256 && ck_pad / ranks <= 64;
  // 17..256 sessions: activations as the A operand (gemm_ns.cu, figures there).  It stores 16-byte pieces; rows that do not lie so keep the kernels below, and (bf16) its
  // refusal above 32.  Up to 32 rows it takes k of 4096 on, where it gains most (24 rows: 4096 -> 12288 28.0 us / 19.9, int8 11264 -> 4096 18.3 / 11.0; of 2048 it would gain 2 to 4),
  // but not few tiles of long k, which gemm_reg.cu cuts into more than four ranges (24 rows, there / here: 11264 -> 256 12.5 / 13.2, -> 640 15.2 / 13.4; 14336 -> 512 14.3 / 15.7, -> 768 16.6 /
  // 15.8; 22016 -> 1024 21.2 / 21.9, -> 256 16.9 / 21.7; 32 rows 18.8 / 21.8, -> 640 22.4 / 22.0).  16-bit gated pairs of as many rows and int8 rows above 32 of few tiles stay with gemm_sk.cu's
  // kernels, where this one would be ahead too (gated 4096 -> 11264, 24 rows 51.9 / 33.3; int8 4096 -> 4096, 104 rows 17.6 / 10.3): tests/test_devices_cpu.py and
  // tests/test_op_routes_cpu.py hold them there.
  const bool long_k = !i8 && ((M <= 24 && k_blocks >= 176 && n_tiles <= 4) || (k_blocks >= 300 && n_tiles <= (M <= 24 ? 8 : 4)));
  const bool kept = (M <= REG_MAX_M && (K < 4096 || long_k || (!i8 && epi == EPI_GATE))) || (i8 && ck);
  const bool lines = ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(rows)) & 15) == 0;
  const bool ns_fits = scaled && tune.ns >= 0 && M <= 256 && tune.grid == 0 && tune.cluster == 0 && !tune.stream_only && !tune.force_split && ns_supported(M, N, K, epi) &&
                       ldy % 8 == 0 && (!res || ldr % 8 == 0) && ((!i8 && M > REG_MAX_M) || (lines && !kept && chosen) || (!i8 && lines && tune.ns > 0));
  // up to 32 that the row kernel and that one leave: weights through registers (gemm_reg.cu).  With the row kernel's range cut short this one has all of its own.
  if (chosen && scaled && M <= REG_MAX_M && !(ns_fits && g_use_ns && M > ROW_MAX_M && g_row_max_m == ROW_MAX_M) && reg_wins(M, N, epi, gate_rows, i8, g_sms) &&
      reg_supported(M, epi, rows, row_ld))
    return reg_linear(rows, row_ld, w_tiles, y, ldy, res, ldr, M, N, K, epi, gate_rows, i8 ? tune.sa : nullptr, tune.sw, ws, sk_workspace_bytes(M), counters,
                      SK_MAX_TILES, g_sms, tune.pdl, stream);
  if (ns_fits && (tune.ns > 0 || (g_use_ns && M > ROW_MAX_M)))
    return ns_linear(cache, rows, i8 ? K : ldx, w_tiles, y, ldy, res, ldr, M, N, K, epi, gate_rows, 0, tune.pdl, stream, 0, i8 ? tune.sa : nullptr, i8 ? tune.sw : nullptr);
  // more than 32 sessions and few row tiles: a cluster of CTAs per tile, ranks along K, reduced over DSMEM
  if (i8 && (K % 16 || !tune.sa || !tune.sw)) B200_FAIL(B200_ERR_SHAPE, "int8 GEMM: K must be a multiple of 16 and both scale vectors given");
  if (ck) {
    const int cs = ranks;
    CkParams p;
    p.M = M; p.N = N; p.K = K; p.CS = cs;
    p.Mpad = ck_pad;
    p.Wc = p.Mpad / cs;
    p.num_kb = k_blocks; p.kb_per = (k_blocks + cs - 1) / cs;
    p.wt = static_cast<const uint8_t*>(w_tiles);
    p.y = y; p.ldy = ldy; p.res = res; p.ldr = ldr;
    p.i8 = i8 ? 1 : 0; p.sa = tune.sa; p.sw = tune.sw; p.late = tune.pdl != PDL_WEIGHTS_FIRST;
    p.stage_bytes = (uint32_t)(TILE_BYTES + p.Mpad * BLOCK_K * 2);      // 128 bytes of K per row, bf16 or int8
    const size_t recv_bytes = (size_t)cs * BLOCK_ROWS * (p.Wc + 4) * 4;
    int stages = (int)((200 * 1024 - recv_bytes) / p.stage_bytes);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    if (stages > p.kb_per) stages = p.kb_per;
    if (stages >= 2) {
      p.stages = stages;
      uint32_t pow2 = 32;
      while (pow2 < (uint32_t)p.Mpad) pow2 <<= 1;
      p.tmem_cols = pow2;
      const CUtensorMap* mx = nullptr;
      if (i8) B200_TRY(x_map(cache, tune.xq, K, M, K, p.Mpad, 1, &mx));
      else B200_TRY(x_map(cache, x, ldx, M, K, p.Mpad, 2, &mx));
      const size_t smem = (size_t)stages * p.stage_bytes + 1024 + 16 * MAX_STAGES + 64 + recv_bytes + 64;
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(n_tiles * cs); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr; cfg.numAttrs = tune.pdl ? 2 : 1;
      cudaError_t le = epi == EPI_STORE ? cudaLaunchKernelEx(&cfg, gemm_ck_kernel<EPI_STORE>, *mx, p)
                                        : cudaLaunchKernelEx(&cfg, gemm_ck_kernel<EPI_RESADD>, *mx, p);
      if (le != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_ck launch failed: %s", cudaGetErrorString(le));
      g_launches.fetch_add(1, std::memory_order_relaxed);
      return check_launch("gemm_ck");
    }
  }
  SkParams p;
  p.M = M; p.N = N; p.K = K; p.gate_rows = gate_rows;
  p.out_rows = epi == EPI_GATE ? gate_rows : N;
  p.Mpad = ((M + 15) / 16) * 16;
  p.wt = static_cast<const uint8_t*>(w_tiles);
  p.y = y; p.ldy = ldy; p.res = res; p.ldr = ldr;
  p.ws = ws; p.counters = counters;
  p.i8 = i8 ? 1 : 0; p.sa = tune.sa; p.sw = tune.sw; p.late = tune.pdl != PDL_WEIGHTS_FIRST;
  p.num_kb = i8 ? (K + 127) / 128 : (K + BLOCK_K - 1) / BLOCK_K;      // a k-block is 128 bytes of K per row
  p.n_tiles = (p.out_rows + BLOCK_ROWS - 1) / BLOCK_ROWS;
  if (p.n_tiles > 1024) B200_FAIL(B200_ERR_SHAPE, "sk GEMM: more than 1024 row tiles");
  int grid = tune.grid > 0 ? tune.grid : g_sms;
  if (grid > SK_MAX_GRID) grid = SK_MAX_GRID;
  if (grid > p.n_tiles * p.num_kb) grid = p.n_tiles * p.num_kb;
  // a CTA should stream at least ~8 k-blocks (128-256 KB): below that the per-CTA set-up and the partial exchange dominate
  if (tune.grid == 0 && grid > (p.n_tiles * p.num_kb) / 8) grid = (p.n_tiles * p.num_kb) / 8 > 0 ? (p.n_tiles * p.num_kb) / 8 : 1;
  // Cutting a tile into S pieces moves S fp32 partials of [128 x Mpad] through L2 (written + read back): allow it
  // only while that stays under half of the tile's weight bytes, i.e. S <= 8 * num_kb / Mpad.
  int s_max = tune.no_split ? 1 : (8 * p.num_kb) / p.Mpad;      // int8 partials are int32 and add exactly
  // measured on B200: with more than 32 sessions the publish / count / re-read protocol
  // costs more than the idle SMs it recovers, so tiles stay whole there
  if (p.Mpad > 32 && tune.force_split == 0) s_max = 1;
  if (s_max < 1) s_max = 1;
  if (p.n_tiles < grid && (long long)p.n_tiles * s_max < grid) grid = p.n_tiles * s_max;   // fewer CTAs, fewer pieces
  // whole rounds of the grid, then the remainder as a stream-K region shared by all CTAs
  p.grid = grid;
  p.whole_rounds = p.n_tiles / grid;
  int rem = p.n_tiles - p.whole_rounds * grid;
  const bool split = rem > 0 && s_max > 1 && rem * 8 < grid * 7 && (long long)rem * s_max >= grid;
  if (rem > 0 && !split) { p.whole_rounds += 1; rem = 0; }
  p.sk_tile0 = p.n_tiles - rem;
  p.sk_items = rem * p.num_kb;
  const int a_tiles = epi == EPI_GATE ? 2 : 1;
  p.stage_bytes = (uint32_t)(a_tiles * TILE_BYTES + p.Mpad * BLOCK_K * 2);
  int stages = (tune.smem_budget > 0 ? tune.smem_budget : 200 * 1024) / (int)p.stage_bytes;
  if (stages > MAX_STAGES) stages = MAX_STAGES;
  if (stages < 2) stages = 2;
  p.stages = stages;
  p.acc_cols = a_tiles * p.Mpad;
  p.n_acc = 2 * p.acc_cols <= 512 ? 2 : 1;
  uint32_t cols = (uint32_t)(p.n_acc * p.acc_cols), pow2 = 32;
  while (pow2 < cols) pow2 <<= 1;
  p.tmem_cols = pow2;
  p.stream_only = tune.stream_only;
  // Loops walked by whole warps or by one thread?  Whole warps are ahead where the CTAs' tiles are whole, and of gated pairs also where few tiles leave each CTA little to stream and where
  // long tiles come in more than one round; the split tiles in between they make slower.  24 rows, one thread / warps, us.  Gated, k 2048: 22 tiles 23.1 / 21.5, 44 29.0 / 28.1, 80 32.9 /
  // 35.8, 148 31.4 / 30.1, 152 45.9 / 37.8, 170 56.1 / 57.9; k 1024: 200 tiles 39.3 / 46.0, 260 44.0 / 49.6; k 4096: 88 51.9 / 53.1, 112 59.4 / 60.0, 148 53.7 / 51.9, 200 79.8 / 80.1; k 8192:
  // 88 79.0 / 78.4, 130 84.6 / 86.5, 148 99.6 / 95.7, 200 142.8 / 133.6.  Plain, k 2048: 149 tiles whole 32.4 / 19.3, 192 split 29.8 / 32.7, 250 32.9 / 37.5, 297 whole 46.0 / 28.8; k 3072: 400
  // split 62.7 / 59.2; int8, 200 rows, 11264 -> 2048 in whole tiles 56.6 / 45.6.
  const bool gate = epi == EPI_GATE;
  const bool warps = split ? gate && (2 * p.n_tiles <= g_sms || (p.whole_rounds > 0 && p.num_kb >= 80)) : !gate || p.num_kb < 128 || p.n_tiles >= g_sms;
  const CUtensorMap* mx = nullptr;
  if (i8) B200_TRY(x_map(cache, tune.xq, K, M, K, p.Mpad, 1, &mx));
  else B200_TRY(x_map(cache, x, ldx, M, K, p.Mpad, 2, &mx));
  const size_t smem = (size_t)stages * p.stage_bytes + 1024 + 16 * MAX_STAGES + 64;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = tune.pdl ? 1 : 0;
  void (*kernel)(const CUtensorMap, const SkParams) =
      epi == EPI_STORE ? (warps ? gemm_sk_kernel<EPI_STORE, true> : gemm_sk_kernel<EPI_STORE, false>) : epi == EPI_RESADD ? (warps ? gemm_sk_kernel<EPI_RESADD, true> : gemm_sk_kernel<EPI_RESADD, false>)
                       : (warps ? gemm_sk_kernel<EPI_GATE, true> : gemm_sk_kernel<EPI_GATE, false>);
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, *mx, p);
  if (le != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_sk launch failed: %s", cudaGetErrorString(le));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("gemm_sk");
}

}  // namespace tc
}  // namespace b200
