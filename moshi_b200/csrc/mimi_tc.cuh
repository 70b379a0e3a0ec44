// Mimi's contractions on the 5th-generation tensor cores: every StreamingConv1d / StreamingConvTranspose1d of the SEANet
// (conv.py:245-274, 340-362; seanet.py:90-93) and every nn.Linear of the two bottleneck transformers (transformer.py:752-777)
// is one launch of mimi_tc_kernel, a persistent TMA + tcgen05 (kind::tf32) implicit GEMM with fp32-equivalent accuracy:
//
//     out[token][n] = epi( sum_{tap, ci} act[session][row0 + t * stride + tap * dil][ci] * w[n][tap][ci] )
//
//   * Activations are TOKEN-MAJOR: act[session][row][channel], channel fastest.  A layer's input lives in its own extended
//     buffer ext[b][carried rows | frame rows][Cin] (the producing layer's epilogue writes the consumer's activation, ELU
//     applied, straight behind the consumer's carried left context, so `cat(previous, x)` (conv.py:261) is an address).  A
//     tile of 128 GEMM rows = bb sessions x tt consecutive output steps, fetched per tap by ONE 3-D TMA box
//     (32 channels, tt rows with element stride = conv stride, bb sessions) into a K-major SWIZZLE_128B tile: the im2col
//     matrix never exists and strided convolutions cost no gather instructions.
//   * ConvTranspose1d with K = 2 S is the same kernel: out[b][t*S + r][co] = x[t] . W[:, co, r] + x[t-1] . W[:, co, S + r], i.e.
//     two taps over [x[t-1], x[t]], N = S * Cout ordered (r, co), whose row-major result IS the token-major output; the
//     overlap-add carry of conv.py:349-361 becomes one carried input row (x[-1] of the next frame).
//   * 3xTF32: a = a_hi + a_lo with a_hi = tf32(a) and a_lo = tf32(a - a_hi) (both round-to-nearest, written by the producing
//     epilogue), likewise for the weights at load; the product is a_hi*w_hi + a_hi*w_lo + a_lo*w_hi with fp32 accumulation
//     in TMEM (dropped terms <= 2^-22 relative).  The RVQ indices downstream stay exact up to the margin the parity tests
//     define (tests/util.py).
//   * Warp roles (576 threads): warp 0 = TMA producer (A hi + A lo boxes, one contiguous bulk copy of the pre-tiled weight
//     pair per k-block), warp 1 = TMEM owner + MMA issuer, warps 2-17 = epilogue: the sums go through shared memory, so that a
//     warp stores and reads whole lines (bias, residual, ELU / GELU / layer-scale, hi/lo split).  Persistent grid, two TMEM
//     accumulator stages: the epilogue of a tile overlaps the MMAs of the next.
//   * Few tiles: a cluster of 2 to 8 CTAs shares a tile's k, every CTA adds the sums of all of them over distributed shared
//     memory for its share of the rows, in order, and finishes those (one tile per CTA).
//   * Few rows against 128 features: the features are the tensor core's rows and the activation rows its 16..112 columns.
//   * A chain of more than TC_CHAIN k-blocks is summed up in fp32 registers piece by piece: the tensor core cuts off where an
//     addition rounds (2 x 8192 -> 1024: error 7.2e-6 in chains of 32 k-blocks, 9e-7 in chains of 4).
//
// What bounds a launch of a few tiles is a chain of latencies, 4 to 6 us behind the wait: load 1.1, products 0.35 a k-block, TMEM
// to shared memory 0.5, the cluster's barrier 0.3, exchange and epilogue 1.2.  Found on the way, encode + decode of a frame of 1 / 40
// sessions, us: partial sums through L2 and a second launch 695 / 1857; clusters and whole lines 645 / 1811; residual, bias and all
// index divisions (a tenth of a microsecond each) in front of the waits, layer norm and attention of many tokens launched early,
// 604 / 1498; the issuing warp walking along as a whole with its operands in uniform registers, 548 / 1378 (one thread issued
// an instruction every 90 to 100 clocks at any size).
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace b200 {
namespace mtc {

constexpr int TC_ROWS = 128;            // GEMM rows (tokens) per tile = UMMA M
constexpr int TC_KB = 32;               // fp32 elements per k-block row: 128 bytes = one SWIZZLE_128B row
constexpr int TC_MAX_NT = 128;          // output features per tile (64 KB per stage and 3 stages where all 128 rows exist)
constexpr int TC_EPI_WARPS = 16;         // four per TMEM quadrant: the epilogue is a chain of latencies per run of 16 features
                                        // (one per quadrant, before the sums went through shared memory: a frame of 40 sessions took 1982 us, of one session 739; four: 1850 and 690)
constexpr int TC_THREADS = 64 + 32 * TC_EPI_WARPS;
constexpr int TC_MAX_STAGES = 8;
constexpr int TC_MAX_SPLIT = 8;         // CTAs of a cluster that share a tile's k
constexpr int TC_CHAIN = 4;              // k-blocks that the tensor core sums up by itself: it cuts off where an fp32 addition rounds
constexpr int TC_SMEM = 225 * 1024;     // ring and sums

enum { TC_EPI_CONV = 0, TC_EPI_GELU = 1, TC_EPI_RES_SCALE = 2 };
enum { TC_ACT_NONE = 0, TC_ACT_SPLIT = 1, TC_ACT_FULL = 2 };      // how the consumer wants its input: hi/lo pair or plain fp32

struct TcParams {
  // ---- geometry of the A operand (tensor maps are kernel arguments)
  int tt, bb, tt_log2;        // tile = bb sessions x tt steps, tt * bb == 128
  int T;                      // output steps per session (tt divides T, or T < tt == 128 for the flat linear case)
  int n_sessions;             // B (rows beyond it are zero-filled by TMA and masked in the epilogue)
  int n_taps, dil, stride, row0, Cin, cb_per_tap, tiles_per_group;
  // ---- B operand: pre-tiled weights [n_tile][kb][hi | lo][NT rows][32] (SWIZZLE_128B), kb = tap * (Cin / 32) + ci_block
  const uint8_t* wt; int NT, n_tiles_n, num_kb, N;
  // ---- schedule
  int m_tiles, ksplit, kb_per_split;
  int swap;                   // 0, or: weights are the tensor core's rows, and this many (a multiple of 16) activation rows its columns
  // ---- epilogue
  int epi;
  const float* bias; int bias_mod;                 // bias[n % bias_mod] (conv: bias_mod = N; convtr: Cout)
  float* y; long long y_sb, y_row;                 // raw output: y[b * y_sb + t * y_row + n] (null = not stored)
  const float* res; long long r_sb, r_row;         // residual source (conv: same indexing; lin: res[token * r_row + n])
  const float* scale;                              // lin RES_SCALE: per-feature layer scale
  int act_mode, act_elu;
  float *a_hi, *a_lo; long long a_sb, a_row;       // activated copy for the consumer: a[b * a_sb + t * a_row + n]
  uint32_t stage_bytes, box_bytes, a_bytes, bars_at, tmem_cols; int stages;      // box: the rows of a tile that can exist; bars_at: mbarriers, behind the ring and the sums
};

// y = hi + lo with hi = tf32(y) and lo = tf32(y - hi), both round-to-nearest (cvt.rna): |y - hi - lo| <= 2^-23 |y|
__device__ __forceinline__ void split_tf32(float v, float& hi, float& lo) {
  uint32_t h, l;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
  hi = __uint_as_float(h);
  const float r = v - hi;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(r));
  lo = __uint_as_float(l);
}

// ---- host side ---------------------------------------------------------------------------------------------------------
struct TcLayer {
  // static description
  int kind = 0;               // 0 conv, 1 convtr, 2 linear
  int Cin = 0, N = 0, n_taps = 1, dil = 1, stride = 1;
  int bias_mod = 0;
  uint8_t* wt = nullptr;      // packed hi/lo tiles
  const float* bias = nullptr;
  int NT = 0, n_tiles_n = 0, num_kb = 0;
  // per-session-batch plan (streaming_begin)
  CUtensorMap map_hi, map_lo;
  TcParams p;
  int grid = 0; size_t smem = 0;
};

size_t tc_packed_bytes(int N, int Cin, int n_taps);
// w: fp32 [N][n_taps * Cin] (k = tap * Cin + ci) -> tiles
int tc_pack_weights(const float* w_dev, void* out_dev, int N, int Cin, int n_taps, cudaStream_t st);
bool tc_pdl();                           // the codec's kernels may start while their predecessor drains (B200_MIMI_PDL=0: off)
int tc_init();
// 3-D tensor map over a token-major activation buffer base[b][row][Cin] (session stride sb elements, row stride = Cin)
int tc_make_map(CUtensorMap* m, const float* base, int Cin, long long rows_per_session, long long sb_elems, int n_sessions, int tt,
                int bb, int stride);
int tc_plan(TcLayer& L, int n_sessions, int T, int sms);
int tc_launch(const TcLayer& L, cudaStream_t st);

}  // namespace mtc
}  // namespace b200
