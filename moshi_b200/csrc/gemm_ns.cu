// tcgen05 GEMM for the LM linears at 17..256 sessions (which of them: sk_linear):  y[M][N] = epi(x[M][K] . w[N][K]^T), bf16 in, fp32 in TMEM, bf16 out; int8 in, exact int32 sums, scaled, bf16 out.
//
// gemm_sk.cu feeds the 128-row weight tile as the UMMA *A* operand and the sessions as N ("swap-AB").  Here the operands keep their textbook roles:
//
//   * A = the activations, one SWIZZLE_128B box of 128 bytes of k per k-block (2-D TMA; two blocks of rows above 128 sessions).  The box has as many rows as there are
//     sessions, to whole eights: a row-wise copy costs about 2.7 ns per row and SM, zeroes too.  The instruction reads 128 rows all the same: what lies behind the box (the
//     next stage's weights, free space behind the last) goes into rows of the accumulator that nobody reads.  The stages that this leaves room for are in flight instead;
//   * B = the weight rows of a unit, 16 to 256 of them in one instruction; gated: as many of the gate and behind them those of the value, so that the accumulator holds gate
//     and value of an output in the SAME thread and silu(g) * u needs no exchange.  Eight rows of a packed tile are 1024 bytes on end, so a unit need not be whole tiles:
//     where K is whole every SM gets the same share of the rows (ns_default_plan);
//   * D = [128 sessions (TMEM lanes) x 128 or 256 weight rows (columns)] fp32.  k-blocks go to the accumulators that fit into TMEM in turn (4 up to 128 columns, 2 beyond or gated;
//     half above 128 sessions), which are added in fp32: the tensor cores cut off what a long chain's additions leave over.  Error of the sums alone (terms whose exact sum is 0, over
//     the rms of a random sum of them), 24 rows, one accumulator / these / what took 17..32 rows before: 4096 -> 12288 2.0e-6 / 4.8e-7 / 6.6e-7, 4096 -> 4096 4.8e-7 / 1.3e-7
//     / 2.4e-7, 11264 -> 4096 1.5e-6 / 3.4e-7 / 6.2e-7, 4096 -> 32000 2.0e-6 / 1.0e-6 / 1.7e-6.  The epilogue keeps its registers without a stack for it: a stack
//     frame of a few words costs a launch 2 to 3 us.  int8 sums are exact: one accumulator;
//   * results go through shared memory (the stage ring, empty by then), so that a warp stores and reads whole lines: 3 us less per launch than 32 bytes per session and
//     instruction;
//   * shapes with few units are cut along K over a cluster of 2..4 CTAs; every CTA adds the sums of all of them over distributed shared memory for its share of the
//     sessions, in rank order (deterministic): no workspace, no atomics.  ns_default_plan() holds the measured choice per shape;
//   * copies and products are issued from uniform registers (tc_prims.cuh).
// us, launches behind one another in a graph, cold weights (launched one by one 2 us more), before these / now.  104 sessions: 4096 -> 12288 27.9 / 20.6, 4096 -> 4096 16.1 / 13.3, 11264 -> 4096
// 26.4 / 22.1, 4096 -> 32000 50.9 / 44.0, gated -> 11264 37.9 / 33.5 (37.6 in whole tiles), gated 1024 -> 2816 12.8 / 9.0 (12.2).  48: 25.3 / 20.0, 13.5 / 10.7, 23.6 / 19.3, 48.5 /
// 42.7, 37.1 / 33.2, 12.2 / 8.2.  256: 44.3 / 32.2, 27.5 / 21.8, 42.3 / 34.6, 70.8 / 61.2, 54.6 / 45.2, 20.5 / 12.0.  24 sessions (gemm_reg.cu, gemm_sk.cu / now): 28.0 / 19.9, 15.0 /
// 10.0, 28.0 / 18.4, 53.5 / 42.7; gated pairs of up to 32 rows stay with those two (50.3, this kernel 33.3).  int8 (gemm_reg.cu, gemm_sk.cu / this kernel, which has not all of them): 24 17.6 / 11.8, 11.3 / 7.4, 18.3 / 11.0, 34.2 / 24.1, 34.5 / 20.9, 11.6 / 6.5 (k below 4096 stays); more than 32 of few tiles stay with gemm_sk.cu; 104
// 26.5 / 12.2, 17.6 / 10.3, 23.2 / 14.4, 41.0 / 25.6, 40.5 / 22.1, 25.3 / 7.2; 256 40.4 / 17.2, 57.3 / 18.0, 88.6 / 23.2, 68.5 / 37.1, 69.8 / 32.4, 51.5 / 10.1.  A step of the 7B with 40
// sessions 6.81 -> 6.31 ms, with 72 7.56 -> 7.11.
//
// Same packed weights, same epilogues and cast points as gemm_sk.cu (residual add bf16(res + bf16(acc)), gated SiLU
// bf16(bf16(silu(g)) * u), gating.py:18-20); same PDL protocol (weights requested before griddepcontrol.wait).
#include <algorithm>

#include "gemm_sk.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace tc {

namespace {

using namespace tcp;

constexpr int EPI_STORE = 0, EPI_RESADD = 1, EPI_GATE = 2;
constexpr int BLOCK_ROWS = 128, BLOCK_K = 64;
// warp 0 producer, warp 1 MMA, warps 2-17 epilogue: four per TMEM quadrant, every fourth run of 16 columns each.  The epilogue is a chain
// of latencies per run (TMEM load, silu, store) that nothing hides.  One warp per quadrant: the gated product 22528 x 4096 took 57.5 us at
// 104 sessions and 92.4 at 200, of which 29 did not depend on K (half the K: 43.3); four: 41.8 and 60.2.  Plain products gain 0-1 us.
constexpr int NUM_THREADS = 576;
constexpr int EPI_STEP = 64;                 // columns between the runs of one epilogue warp
constexpr int TILE_BYTES = BLOCK_ROWS * BLOCK_K * 2;
constexpr int A_BYTES = 128 * BLOCK_K * 2;   // a block of 128 session rows x 128 bytes of k
constexpr int MAX_STAGES = 12;
constexpr int MAX_CS = 8;
// All of it: one CTA per SM.  A CTA that asks for columns beside this one waits until it ends, in nobody's way, for this kernel needs nothing of the other.  None gets that far: registers
// (576 threads of up to 96) or shared memory (200 KB) keep the CTAs of the other tensor-core kernels off the SM.
constexpr int TMEM_COLS = 512;

struct NsParams {
  int M, N, K, out_rows, gate_rows, CS, num_kb, kb_per, stages, n_tiles, unit_rows, acc_cols, mblocks, n_acc, box_rows;
  const uint8_t* wt;
  __nv_bfloat16* y; long long ldy;
  const __nv_bfloat16* res; long long ldr;
  const float *sa, *sw;                          // int8: scales of activation and weight rows
  uint32_t block_step;                           // bytes between two blocks' sums in a cluster's shared memory (0: in the same place)
  int late;                                      // nothing is read before the wait on the preceding kernel
};

__device__ __forceinline__ float4 ns_lds_of(uint32_t at, int rank) {      // the same shared address in CTA `rank` of the cluster
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ns_lds(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ float4 ns_lds_f4(uint32_t at) {
  const uint4 v = ns_lds(at);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ void ns_sts(uint32_t at, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void ns_cluster_meet() {      // orders nothing
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void ns_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ns_bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ uint32_t ns_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Results and partial sums lie in shared memory as rows of 16-byte pieces, piece c of row r at position c ^ (r & 7): lanes write a row each, and read neighbouring pieces.
__device__ __forceinline__ uint32_t ns_piece(uint32_t base, int row, int c, int per_row_log2) { return base + (uint32_t)(((row << per_row_log2) + (c ^ (row & 7))) << 4); }

// sixteen columns' sums over the accumulators, which lie `cols` columns apart (whole warps); int8: one accumulator of whole numbers
template <int MOST>
__device__ __forceinline__ void ns_sums(uint32_t at, uint32_t cols, int n_acc, float (&v)[16]) {
  uint32_t g[16], h[16];
  tmem_ld16(at, g);
  if (MOST > 1 && n_acc > 1) tmem_ld16(at + cols, h);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = MOST > 1 && n_acc > 1 ? __uint_as_float(g[j]) + __uint_as_float(h[j]) : __uint_as_float(g[j]);
  if (MOST > 2 && n_acc > 2) {
    tmem_ld16(at + 2 * cols, g);
    if (n_acc > 3) tmem_ld16(at + 3 * cols, h);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] += n_acc > 3 ? __uint_as_float(g[j]) + __uint_as_float(h[j]) : __uint_as_float(g[j]);
  }
}
// int8: the value of a sum, scaled as everywhere else (gemm_sk.cu)
__device__ __forceinline__ float ns_scaled(float bits, float sa, float sw) { return (float)__float_as_int(bits) * (sa * sw * (1.f / 16129.f)); }
__device__ __forceinline__ float ns_lds1(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void ns_sts1(uint32_t at, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory"); }
// one more rank's partial sums
template <bool I8>
__device__ __forceinline__ void ns_add(float4& f, const float4& x) {
  if (I8) {
    f.x = __int_as_float(__float_as_int(f.x) + __float_as_int(x.x)); f.y = __int_as_float(__float_as_int(f.y) + __float_as_int(x.y));
    f.z = __int_as_float(__float_as_int(f.z) + __float_as_int(x.z)); f.w = __int_as_float(__float_as_int(f.w) + __float_as_int(x.w));
  } else {
    f.x += x.x; f.y += x.y; f.z += x.z; f.w += x.w;
  }
}

// eight neighbouring residuals of session m from output column o on (valid: how many exist)
__device__ __forceinline__ uint4 ns_residual(const NsParams& p, int m, int o, int valid) {
  const __nv_bfloat16* src = p.res + (long long)m * p.ldr + o;
  if (valid >= 8) return *reinterpret_cast<const uint4*>(src);
  uint32_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < valid) v[j >> 1] |= (uint32_t)__bfloat16_as_ushort(src[j]) << (16 * (j & 1));
  return make_uint4(v[0], v[1], v[2], v[3]);
}
// Session rows row, row + step, .. below end of a block (m0: its first session), a thread's eight columns from output column o on (piece c of a row).  The block's sums lie at
// `sums`: in fp32 in every CTA of a cluster, added in rank order, or (CS == 1) rounded to bf16, what the epilogues do anyway.
template <int EPI, bool I8>
__device__ __forceinline__ void ns_finish(const NsParams& p, uint32_t sums, uint32_t sa, uint32_t sw, int m0, int row, int end, int step, int c, int width_log2, int nb, int o_end, uint4 res) {
  const int o = nb + c * 8, valid = o_end - o;
  if (valid <= 0) return;
#pragma unroll 1
  for (; row < end; row += step) {
    const uint4 old = res;
    if (EPI == EPI_RESADD && row + step < end) res = ns_residual(p, m0 + row + step, o, valid);
    uint4 v;
    if (EPI == EPI_GATE || p.CS == 1) {
      v = ns_lds(ns_piece(sums, row, c, width_log2 - 3));
    } else {
      const uint32_t a0 = ns_piece(sums, row, 2 * c, width_log2 - 2), a1 = ns_piece(sums, row, 2 * c + 1, width_log2 - 2);
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f), g = f;
#pragma unroll 1
      for (int r0 = 0; r0 < p.CS; r0 += 4) {     // four ranks' sums under way: eight were more than the registers hold
        float4 x[4], y[4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r0 + r < p.CS) { x[r] = ns_lds_of(a0, r0 + r); y[r] = ns_lds_of(a1, r0 + r); }
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r0 + r < p.CS) { ns_add<I8>(f, x[r]); ns_add<I8>(g, y[r]); }
      }
      if (I8) {
        const float m = ns_lds1(sa + 4u * (uint32_t)(m0 + row));
        const float4 u = ns_lds_f4(sw + 32u * (uint32_t)c), w = ns_lds_f4(sw + 32u * (uint32_t)c + 16u);
        f = make_float4(ns_scaled(f.x, m, u.x), ns_scaled(f.y, m, u.y), ns_scaled(f.z, m, u.z), ns_scaled(f.w, m, u.w));
        g = make_float4(ns_scaled(g.x, m, w.x), ns_scaled(g.y, m, w.y), ns_scaled(g.z, m, w.z), ns_scaled(g.w, m, w.w));
      }
      v = make_uint4(ns_pack(f.x, f.y), ns_pack(f.z, f.w), ns_pack(g.x, g.y), ns_pack(g.z, g.w));
    }
    if (EPI == EPI_RESADD) {
      const __nv_bfloat162 *a = reinterpret_cast<const __nv_bfloat162*>(&v), *b = reinterpret_cast<const __nv_bfloat162*>(&old);
      uint4 w;
      uint32_t* u = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 s = __bfloat1622float2(a[j]), r = __bfloat1622float2(b[j]);
        u[j] = ns_pack(r.x + s.x, r.y + s.y);
      }
      v = w;
    }
    __nv_bfloat16* dst = p.y + (long long)(m0 + row) * p.ldy + o;
    if (valid >= 8) *reinterpret_cast<uint4*>(dst) = v;
    else {
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < valid) dst[j] = __ushort_as_bfloat16((unsigned short)(u[j >> 1] >> (16 * (j & 1))));
    }
  }
}

template <int EPI, bool I8>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_ns_kernel(const __grid_constant__ CUtensorMap tmap_x, const NsParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int R = p.unit_rows;                                              // output rows of a unit (gated: of the gate, and as many of the value)
  const uint32_t a_off = (uint32_t)(EPI == EPI_GATE ? 2 * R : R) * 128u;  // stage = B (the unit's weight rows) | A (activation box)
  const uint32_t a_bytes = (uint32_t)p.box_rows * 128u;                   // the rows that exist, to whole eights: what follows them is multiplied too, into rows that nobody reads
  const uint32_t stage_bytes = a_off + a_bytes;
  const uint32_t bars = base + (uint32_t)p.stages * stage_bytes + ((uint32_t)p.mblocks * A_BYTES - a_bytes);      // the last stage's products read as far
  const uint32_t full0 = bars, empty0 = bars + 8 * MAX_STAGES, tfull = bars + 16 * MAX_STAGES;
  const uint32_t tptr = tfull + 8;
  uint32_t* tptr_generic = reinterpret_cast<uint32_t*>(smem_raw + (tptr - raw));
  const uint32_t sa = bars + 16 * MAX_STAGES + 64, sw = sa + 4 * 256;      // int8: scales of the sessions and of the unit's weight rows

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int unit = blockIdx.x / p.CS, me = blockIdx.x - unit * p.CS;
  const int kb0 = me * p.kb_per, kb1 = min(p.num_kb, kb0 + p.kb_per);
  const int n_items = kb1 > kb0 ? kb1 - kb0 : 0;
  const int nb = unit * R, width = EPI == EPI_GATE ? 2 * R : R;           // first output row; accumulator columns in use
  const uint32_t acc_cols = (uint32_t)p.acc_cols;                         // and those that an accumulator is given: mblocks x n_acc x acc_cols = TMEM_COLS

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_x) : "memory");
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(tfull, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tptr, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tptr_generic;
  if (p.late) pdl_wait();
  pdl_trigger();

  // both loops are walked by their whole warps, and one thread issues (tc_prims.cuh)
  if (warp == 0) {
    const int there = min(R, p.n_tiles * BLOCK_ROWS - nb);                  // the last unit may reach beyond the last tile: its columns there are multiplied and not stored
    const uint32_t b_bytes = (uint32_t)(EPI == EPI_GATE ? 2 * there : there) * 128u;
    auto load_b = [&](int i, int s) {
      // eight rows of a tile are 1024 bytes on end: one copy per tile that the unit has rows of (gated: one of each of a pair's tiles)
      const uint32_t sb = base + (uint32_t)s * stage_bytes;
#pragma unroll 1
      for (int r = 0; r < there; ) {
        const int tile = (nb + r) >> 7, in = (nb + r) & 127, n = min(128 - in, there - r);
        const uint8_t* src = p.wt + ((size_t)tile * p.num_kb + (kb0 + i)) * (EPI == EPI_GATE ? 2 * TILE_BYTES : TILE_BYTES) + in * 128;
        bulk_load(sb + (uint32_t)r * 128u, src, (uint32_t)n * 128u, full0 + 8 * s);
        if (EPI == EPI_GATE) bulk_load(sb + (uint32_t)(R + r) * 128u, src + TILE_BYTES, (uint32_t)n * 128u, full0 + 8 * s);
        r += n;
      }
    };
    // weights first (they do not depend on the preceding kernel), activations after the dependency wait
    const int pre = n_items < p.stages ? n_items : p.stages;
    for (int i = 0; i < pre; ++i) {
      if (elected()) {
        mbar_expect_tx(full0 + 8 * i, b_bytes + a_bytes);
        load_b(i, i);
      }
      __syncwarp();
    }
    pdl_wait();
    int s = 0; uint32_t ph = 0;
    for (int i = 0; i < n_items; ++i) {
      if (i >= pre) mbar_wait(empty0 + 8 * s, ph ^ 1u);
      if (elected()) {
        if (i >= pre) {
          mbar_expect_tx(full0 + 8 * s, b_bytes + a_bytes);
          load_b(i, s);
        }
        tma_load_2d(base + (uint32_t)s * stage_bytes + a_off, &tmap_x, full0 + 8 * s, (kb0 + i) * (I8 ? 2 * BLOCK_K : BLOCK_K), 0);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1u; }
    }
  } else if (warp == 1) {
    const uint32_t idesc = I8 ? make_idesc_i8(128, width) : make_idesc(128, width);
    int s = 0, acc = 0; uint32_t ph = 0;
    for (int i = 0; i < n_items; ++i) {
      mbar_wait(full0 + 8 * s, ph);
      tc_fence_after();
      const uint32_t sb = desc_low(base + (uint32_t)s * stage_bytes);
      for (int mb = 0; mb < p.mblocks; ++mb) {
        const uint32_t d = tmem_base + (uint32_t)(mb * p.n_acc + acc) * acc_cols, sa = sb + ((a_off + (uint32_t)mb * A_BYTES) >> 4), first = i < p.n_acc ? 0u : 1u;
        if constexpr (I8) umma_block_i8(d, sa, sb - sa, idesc, first);
        else umma_block<1>(d, sa, sb - sa, idesc, first);
      }
      commit_elected(empty0 + 8 * s);
      if (++acc == p.n_acc) acc = 0;
      if (++s == p.stages) { s = 0; ph ^= 1u; }
    }
    commit_elected(tfull);
    __syncwarp();
  }

  // ===== epilogue: TMEM lane = session row.  Results go through the ring, which is empty by then, so that what is stored and read is whole lines =====
  const int q4 = warp & 3, sub = (warp - 2) >> 2, qt = sub * 32 + lane, tid = threadIdx.x - 64;      // TMEM quadrant, this warp's place among its four
  const int out_log2 = R <= 128 ? 7 : 8, pieces = 1 << (out_log2 - 3);      // a row of results in shared memory has 128 or 256 columns, R of which are in use
  // CS == 1: a quadrant's 128 threads finish its 32 rows; else every CTA of the cluster its share of the block's rows, 512 threads
  const int t = p.CS == 1 ? qt : tid, step = (p.CS == 1 ? 128 : 512) >> (out_log2 - 3), c = t & (pieces - 1), o_end = min(p.out_rows, nb + R);
  const int n_acc = min(p.n_acc, n_items);
  if (I8 && warp >= 2) {                        // scales: the weights' like the weights, the sessions' after the wait
    if (tid < width) {
      const bool value = EPI == EPI_GATE && tid >= R;
      const int n = nb + (value ? tid - R : tid);
      ns_sts1(sw + 4u * (uint32_t)tid, n < p.out_rows ? p.sw[value ? p.gate_rows + n : n] : 0.f);
    }
    pdl_wait();
    if (tid < p.M) ns_sts1(sa + 4u * (uint32_t)tid, p.sa[tid]);
    asm volatile("bar.sync 5, 512;" ::: "memory");
  }
  for (int mb = 0; mb < p.mblocks; ++mb) {      // blocks of 128 sessions
    const uint32_t sums = base + (uint32_t)mb * p.block_step;
    const int rows = min(128, p.M - mb * 128);
    const int row0 = (p.CS == 1 ? q4 * 32 : rows * me / p.CS) + (t >> (out_log2 - 3)), end = p.CS == 1 ? min(rows, q4 * 32 + 32) : rows * (me + 1) / p.CS;
    if (warp >= 2) {
      uint4 res = make_uint4(0u, 0u, 0u, 0u);
      if (mb == 0) pdl_wait();                  // y / res may still be in use by the predecessor
      if (EPI == EPI_RESADD && row0 < end && nb + c * 8 < o_end) res = ns_residual(p, mb * 128 + row0, nb + c * 8, o_end - nb - c * 8);
      if (mb == 0) {
        mbar_wait(tfull, 0);
        tc_fence_after();
      }
      const int row = q4 * 32 + lane;
      const bool m_ok = row < rows;
      const float m_scale = I8 && m_ok ? ns_lds1(sa + 4u * (uint32_t)(mb * 128 + row)) : 0.f;
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(mb * p.n_acc) * acc_cols;
#pragma unroll EPI == EPI_GATE ? 2 : 1
      for (int c0 = sub * 16; c0 < R; c0 += EPI_STEP) {
        float v[16];
        if (n_items > 0) {
          __syncwarp();
          ns_sums<I8 ? 1 : EPI == EPI_GATE ? 2 : 4>(lane_addr + (uint32_t)c0, acc_cols, n_acc, v);
          if (EPI == EPI_GATE) {
            // columns j (gate) and R + j (value) of the same output; K whole
            float u[16];
            ns_sums<I8 ? 1 : 2>(lane_addr + (uint32_t)(R + c0), acc_cols, n_acc, u);
            if (m_ok) {                         // not for rows of zeroes: a division of zero takes the long way (33 to 104 rows: 41 us instead of 35)
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if (I8) {
                  v[j] = ns_scaled(v[j], m_scale, ns_lds1(sw + 4u * (uint32_t)(c0 + j)));
                  u[j] = ns_scaled(u[j], m_scale, ns_lds1(sw + 4u * (uint32_t)(R + c0 + j)));
                }
                const float gt = ns_bf16_round(v[j]), ut = ns_bf16_round(u[j]);
                v[j] = ns_bf16_round(gt / (1.f + expf(-gt))) * ut;
              }
            }
          } else if (I8 && p.CS == 1) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = ns_scaled(v[j], m_scale, ns_lds1(sw + 4u * (uint32_t)(c0 + j)));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
        if (m_ok) {
          if (EPI == EPI_GATE || p.CS == 1) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              ns_sts(ns_piece(base, row, (c0 >> 3) + j, out_log2 - 3), make_uint4(ns_pack(v[8 * j], v[8 * j + 1]), ns_pack(v[8 * j + 2], v[8 * j + 3]), ns_pack(v[8 * j + 4], v[8 * j + 5]),
                                                                                   ns_pack(v[8 * j + 6], v[8 * j + 7])));
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              ns_sts(ns_piece(sums, row, (c0 >> 2) + j, out_log2 - 2),
                     make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3])));
          }
        }
      }
      if (EPI == EPI_GATE || p.CS == 1) {
        asm volatile("bar.sync %0, 128;" ::"r"(1 + q4) : "memory");
        ns_finish<EPI, I8>(p, base, sa, sw, mb * 128, row0, end, step, c, out_log2, nb, o_end, res);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + q4) : "memory");
      } else {
        __syncwarp();
        ns_cluster_sync();
        ns_finish<EPI, I8>(p, sums, sa, sw, mb * 128, row0, end, step, c, out_log2, nb, o_end, res);
      }
      tc_fence_before();
    } else if (p.CS > 1) {
      __syncwarp();
      ns_cluster_sync();
    }
    if (p.CS > 1 && mb + 1 < p.mblocks && p.block_step == 0) {
      __syncwarp();
      ns_cluster_sync();                        // the block's sums have been read everywhere, before the next block's take their place
    }
  }
  if (p.CS > 1) {
    __syncwarp();
    ns_cluster_meet();                          // nobody leaves while its sums are read
  }
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_ns_encode = nullptr;
int g_ns_sms = 0;

int ns_init() {
  if (!g_ns_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    B200_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
    if (!fn || qres != cudaDriverEntryPointSuccess) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
    g_ns_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, 220 * 1024, gemm_ns_kernel<EPI_STORE, false>, gemm_ns_kernel<EPI_RESADD, false>, gemm_ns_kernel<EPI_GATE, false>, gemm_ns_kernel<EPI_STORE, true>,
                      gemm_ns_kernel<EPI_RESADD, true>, gemm_ns_kernel<EPI_GATE, true>));
  if (!g_ns_sms) {
    int dev = 0;
    B200_CUDA(cudaGetDevice(&dev));
    B200_CUDA(cudaDeviceGetAttribute(&g_ns_sms, cudaDevAttrMultiProcessorCount, dev));
  }
  return B200_OK;
}

}  // namespace

bool ns_supported(int M, int N, int K, int epi) {
  (void)N; (void)epi;
  return M >= 1 && M <= 256 && K >= 8 && K % 8 == 0;
}

int ns_prepare() { return ns_init(); }

// The LM's choice of unit and K-split for a shape:
//   * gated, or more tiles than SMs: K whole, and as many output rows per CTA as put the same share (in sixteens; at most 128 pairs or 256) on every SM.  In whole tiles
//     the 88 pairs of the 7B leave 60 SMs without work;
//   * plain, tiles for more than half the SMs: tiles, K whole (equal shares of the 96 of 4096 -> 12288 gave 20.5 us for 19.7 at 64 sessions, 27.0 for 28.4 at 160);
//   * fewer (out_proj / linear_out: 32 tiles, depformer_in: 64): tiles, so that activations are not copied too often, K cut over the largest power of two <= 4
//     that keeps the grid resident (32 x 4, 64 x 2 = 128 CTAs).
static void ns_default_plan(int out_rows, int n_tiles, int num_kb, int epi, int* unit_rows, int* cs) {
  *cs = 1;
  if (epi == EPI_GATE || n_tiles > g_ns_sms) {
    const int most = epi == EPI_GATE ? 128 : 256, waves = (out_rows + g_ns_sms * most - 1) / (g_ns_sms * most), ctas = waves * g_ns_sms;
    *unit_rows = ((out_rows + ctas - 1) / ctas + 15) & ~15;
    return;
  }
  *unit_rows = BLOCK_ROWS;
  while (*cs < 4 && n_tiles * *cs * 2 <= g_ns_sms && num_kb / (*cs * 2) >= 4) *cs *= 2;
}

int ns_linear(GemmPlanCache& cache, const void* x, long long ldx, const void* w_tiles, __nv_bfloat16* y, long long ldy,
              const __nv_bfloat16* res, long long ldr, int M, int N, int K, int epi, int gate_rows, int cluster, int pdl,
              cudaStream_t stream, int unit_tiles, const float* sa, const float* sw) {
  const bool i8 = sa != nullptr;
  const int elem = i8 ? 1 : 2;
  if (!ns_supported(M, N, K, epi) || ldx * elem % 16 || (i8 && K % 16)) B200_FAIL(B200_ERR_SHAPE, "ns GEMM: unsupported shape M=%d N=%d K=%d", M, N, K);
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w_tiles) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(res)) & 15)
    B200_FAIL(B200_ERR_SHAPE, "ns GEMM: operands must be 16-byte aligned");
  if ((ldy % 8) || (res && ldr % 8)) B200_FAIL(B200_ERR_SHAPE, "ns GEMM: row strides must be multiples of 8");
  B200_TRY(ns_init());
  NsParams p;
  p.M = M; p.N = N; p.K = K; p.gate_rows = gate_rows;
  p.out_rows = epi == EPI_GATE ? gate_rows : N;
  p.n_tiles = (p.out_rows + BLOCK_ROWS - 1) / BLOCK_ROWS;
  p.num_kb = (K * elem + 127) / 128;
  int def_rows = 0, def_cs = 1;
  ns_default_plan(p.out_rows, p.n_tiles, p.num_kb, epi, &def_rows, &def_cs);
  p.unit_rows = unit_tiles == 0 && cluster <= 0 ? def_rows : (unit_tiles == 1 || epi == EPI_GATE) ? BLOCK_ROWS : 2 * BLOCK_ROWS;
  const int b_rows = epi == EPI_GATE ? 2 * p.unit_rows : p.unit_rows;
  p.acc_cols = b_rows <= 128 ? 128 : 256;
  p.mblocks = M > 128 ? 2 : 1;
  p.n_acc = i8 ? 1 : std::min(epi == EPI_GATE ? 2 : 4, TMEM_COLS / (p.mblocks * p.acc_cols));
  p.box_rows = (M + 7) & ~7;
  const uint32_t stage_bytes = (uint32_t)b_rows * 128u + (uint32_t)p.box_rows * 128u, beyond = (uint32_t)p.mblocks * A_BYTES - (uint32_t)p.box_rows * 128u;
  const int n_units = (p.out_rows + p.unit_rows - 1) / p.unit_rows;
  int cs = cluster > 0 ? cluster : def_cs;
  if (epi == EPI_GATE) cs = 1;
  if (cs > MAX_CS) cs = MAX_CS;
  if (cs > p.num_kb) cs = p.num_kb;
  p.CS = cs;
  p.kb_per = (p.num_kb + cs - 1) / cs;
  int stages = (int)((208 * 1024 - beyond) / stage_bytes);
  if (stages > MAX_STAGES) stages = MAX_STAGES;
  if (stages > p.kb_per && p.kb_per >= 2) stages = p.kb_per;
  if (stages < 2) stages = 2;
  const size_t sums = (size_t)128 * (p.unit_rows <= 128 ? 128 : 256) * (cs > 1 ? 4 : 2);      // a block's results or partial sums, in the ring
  while ((size_t)stages * stage_bytes < sums) ++stages;
  // a cluster's sums of two blocks lie side by side where there is room: in one place the second's have to wait until the first's have been read everywhere, and a barrier that orders this
  // waits for the first block's results to be stored as well (4096 -> 4096, 160 sessions 18.4 us, side by side 17.5)
  p.block_step = 0;
  if (cs > 1 && p.mblocks > 1) {
    int wide = stages;
    while ((size_t)wide * stage_bytes < 2 * sums) ++wide;
    if ((size_t)wide * stage_bytes + beyond <= 208 * 1024) { stages = wide; p.block_step = (uint32_t)sums; }
  }
  p.stages = stages;
  p.wt = static_cast<const uint8_t*>(w_tiles);
  p.y = y; p.ldy = ldy; p.res = res; p.ldr = ldr;
  // activations x [M][K]: boxes of [128 rows x 64 k]; rows >= M are zero-filled by the TMA unit
  PlanKey key{x, ldx, M, K, p.box_rows + (i8 ? 1024 : 0)};
  auto it = cache.maps.find(key);
  if (it == cache.maps.end()) {
    CUtensorMap mp;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    cuuint64_t strides[1] = {(cuuint64_t)ldx * elem};
    cuuint32_t box[2] = {(cuuint32_t)(128 / elem), (cuuint32_t)p.box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_ns_encode(&mp, i8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(x), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) M=%d K=%d ld=%lld", (int)r, M, K, ldx);
    it = cache.maps.emplace(key, mp).first;
  }
  p.late = pdl != PDL_WEIGHTS_FIRST;
  p.sa = sa; p.sw = sw;
  const size_t smem = (size_t)stages * stage_bytes + beyond + 1024 + 16 * MAX_STAGES + 64 + (i8 ? 2048 : 0);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(n_units * cs)); cfg.blockDim = dim3(NUM_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (cs > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = cs; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  void (*kernel)(const CUtensorMap, const NsParams) =
      i8 ? (epi == EPI_STORE ? gemm_ns_kernel<EPI_STORE, true> : epi == EPI_RESADD ? gemm_ns_kernel<EPI_RESADD, true> : gemm_ns_kernel<EPI_GATE, true>)
         : (epi == EPI_STORE ? gemm_ns_kernel<EPI_STORE, false> : epi == EPI_RESADD ? gemm_ns_kernel<EPI_RESADD, false> : gemm_ns_kernel<EPI_GATE, false>);
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, it->second, p);
  if (le != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "gemm_ns launch failed: %s", cudaGetErrorString(le));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("gemm_ns");
}

}  // namespace tc
}  // namespace b200
