// mimi_tc_kernel: TMA + tcgen05 kind::tf32 implicit GEMM with 3xTF32 split products (see mimi_tc.cuh).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "mimi_tc.cuh"
#include "tc_prims.cuh"

namespace b200 {
namespace mtc {

namespace {

using namespace tcp;

constexpr uint32_t A_TILE_BYTES = TC_ROWS * TC_KB * 4;      // 16 KB

struct Tile { int m, n, split, b0, t0, kb0, kb1; };

// An integer division is a chain of a tenth of a microsecond: none where the divisor is 1, and all of them before a wait where that can be.
__device__ __forceinline__ void divide(int a, int b, int& q, int& r) {
  q = b == 1 ? a : a / b;
  r = a - q * b;
}
__device__ __forceinline__ Tile tile_at(const TcParams& p, int id) {
  Tile t;
  int mn, group, j;
  divide(id, p.ksplit, mn, t.split);
  divide(mn, p.n_tiles_n, t.m, t.n);
  divide(t.m, p.tiles_per_group, group, j);                 // tiles along the steps of one session group
  t.b0 = group * p.bb;
  t.t0 = j << p.tt_log2;
  t.kb0 = t.split * p.kb_per_split;
  t.kb1 = min(p.num_kb, t.kb0 + p.kb_per_split);
  return t;
}

// rows of a tile that exist, from the first on
__device__ __forceinline__ int valid_rows(const TcParams& p, const Tile& tl) {
  return p.bb == 1 ? min(p.tt, p.T - tl.t0) : min(p.bb, p.n_sessions - tl.b0) * p.tt;
}

// What a thread's four output features n.. take from memory once per launch or tile: the bias, or the layer scale.
__device__ __forceinline__ float4 feature_terms(const TcParams& p, int n) {
  float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.epi == TC_EPI_RES_SCALE) {
    f = __ldg(reinterpret_cast<const float4*>(p.scale + n));
  } else if (p.epi == TC_EPI_CONV && p.bias != nullptr) {
    const int m = p.bias_mod;
    f = make_float4(__ldg(p.bias + n % m), __ldg(p.bias + (n + 1) % m), __ldg(p.bias + (n + 2) % m), __ldg(p.bias + (n + 3) % m));
  }
  return f;
}
// Epilogue of 4 consecutive output features n.. of GEMM row (b, t); rv: the residual's.
__device__ __forceinline__ void store_four(const TcParams& p, int b, int t, int n, float4 v, float4 f, float4 rv) {
  if (p.epi == TC_EPI_GELU) {
    v = make_float4(gelu_erf(v.x), gelu_erf(v.y), gelu_erf(v.z), gelu_erf(v.w));
  } else if (p.epi == TC_EPI_RES_SCALE) {                       // x + layer_scale * update (transformer.py:769,777)
    v = make_float4(rv.x + f.x * v.x, rv.y + f.y * v.y, rv.z + f.z * v.z, rv.w + f.w * v.w);
  } else {
    v.x += f.x; v.y += f.y; v.z += f.z; v.w += f.w;
    if (p.res != nullptr) { v.x += rv.x; v.y += rv.y; v.z += rv.z; v.w += rv.w; }      // SEANetResnetBlock: u + v (seanet.py:90-93)
  }
  if (p.y != nullptr) *reinterpret_cast<float4*>(p.y + (long long)b * p.y_sb + (long long)t * p.y_row + n) = v;
  if (p.act_mode != TC_ACT_NONE) {
    if (p.act_elu) v = make_float4(elu1(v.x), elu1(v.y), elu1(v.z), elu1(v.w));
    const long long o = (long long)b * p.a_sb + (long long)t * p.a_row + n;
    if (p.act_mode == TC_ACT_SPLIT) {
      float4 lo;
      split_tf32(v.x, v.x, lo.x); split_tf32(v.y, v.y, lo.y); split_tf32(v.z, v.z, lo.z); split_tf32(v.w, v.w, lo.w);
      *reinterpret_cast<float4*>(p.a_lo + o) = lo;
    }
    *reinterpret_cast<float4*>(p.a_hi + o) = v;
  }
}

// A step of 8 k with 3xTF32 parts, small terms first: lo * hi, hi * lo, hi * hi.  The whole warp calls, so that the operands are in uniform registers, and one
// thread issues.  A k-block of four steps takes 0.35 us so with few columns; 0.58 where one thread alone walks the loop, 0.64 where it also makes whole
// descriptors.
__device__ __forceinline__ void umma_tf32_split(uint32_t d, uint32_t m_hi, uint32_t m_lo, uint32_t n_hi, uint32_t n_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 mh, ml, nh, nl;\n\t"
      "mov.b64 mh, {%1, %7};\n\tmov.b64 ml, {%2, %7};\n\tmov.b64 nh, {%3, %7};\n\tmov.b64 nl, {%4, %7};\n\t"
      "setp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 t, %7, 0;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], ml, nh, %5, p;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], mh, nl, %5, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], mh, nh, %5, t;\n\t}"
      ::"r"(d), "r"(m_hi), "r"(m_lo), "r"(n_hi), "r"(n_lo), "r"(idesc), "r"(accumulate), "r"(DESC_HIGH) : "memory");
}

__device__ __forceinline__ float4 lds_four(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds_four_of(uint32_t at, int rank) {      // the same address in CTA `rank` of the cluster
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ void sts_four(uint32_t at, const float* r) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_meet() {      // orders nothing
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// Sums lie in shared memory as rows of `cols4` (a multiple of 4) runs of four, run c of row r at position c ^ (r & 7): lanes write a row each, and read neighbouring runs.
__device__ __forceinline__ uint32_t four_at(uint32_t base, int row, int c, int cols4) {
  return base + (uint32_t)(row * cols4 + (c ^ (row & (cols4 & 4 ? 3 : 7)))) * 16u;
}

// Rows r, r + step, .. below r1 of a tile: run c of four features (n: its first) of each; f: its feature_terms.  A thread keeps its run, so that bias and scale are
// loaded once and early, and asks for the residual of its next row while it finishes one (next: of the first).  cluster: the sums of a cluster's CTAs, in order.
__device__ __forceinline__ float4 residual_of(const TcParams& p, const Tile& tl, int r, int r1, int n) {
  if (p.res == nullptr || r >= r1) return make_float4(0.f, 0.f, 0.f, 0.f);
  const int bi = r >> p.tt_log2;
  return *reinterpret_cast<const float4*>(p.res + (long long)(tl.b0 + bi) * p.r_sb + (long long)(tl.t0 + r - (bi << p.tt_log2)) * p.r_row + n);
}
__device__ __forceinline__ void finish_rows(const TcParams& p, bool cluster, uint32_t sums, const Tile& tl, int r, int r1, int step, int c, int cols4, int n, float4 f, float4 next) {
#pragma unroll 1
  for (; r < r1; r += step) {
    const float4 rv = next;
    next = residual_of(p, tl, r + step, r1, n);
    const int bi = r >> p.tt_log2;
    const uint32_t at = four_at(sums, r, c, cols4);
    float4 v;
    if (!cluster) {
      v = lds_four(at);
    } else {
      float4 s[TC_MAX_SPLIT];
#pragma unroll
      for (int i = 0; i < TC_MAX_SPLIT; ++i) s[i] = i < p.ksplit ? lds_four_of(at, i) : make_float4(0.f, 0.f, 0.f, 0.f);
      v = s[0];
#pragma unroll
      for (int i = 1; i < TC_MAX_SPLIT; ++i) { v.x += s[i].x; v.y += s[i].y; v.z += s[i].z; v.w += s[i].w; }
    }
    store_four(p, tl.b0 + bi, tl.t0 + r - (bi << p.tt_log2), n, v, f, rv);
  }
}

__global__ void __launch_bounds__(TC_THREADS, 1)
mimi_tc_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, const TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;                 // SWIZZLE_128B tiles need 1024 B alignment
  const bool cluster = p.ksplit > 1;                            // the CTAs of a cluster have a tile's ranges of k; one tile each
  const uint32_t sums = cluster ? base : base + (uint32_t)p.stages * p.stage_bytes;      // cluster: in the ring, which is empty by then
  const uint32_t bars = base + p.bars_at;
  const uint32_t full0 = bars, empty0 = bars + 8 * TC_MAX_STAGES, tfull0 = bars + 16 * TC_MAX_STAGES, tempty0 = tfull0 + 16;
  const uint32_t tptr = tempty0 + 16;
  uint32_t* tptr_generic = reinterpret_cast<uint32_t*>(smem_raw + (tptr - raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_tiles = p.m_tiles * p.n_tiles_n * p.ksplit;
  const uint32_t w_bytes = (uint32_t)p.NT * 128u;               // one weight tile (hi or lo)

  if (warp == 0 && lane == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_hi) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_lo) : "memory");
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, TC_EPI_WARPS);           // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tptr, p.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tptr_generic;
  pdl_trigger();                                 // the next kernel of the frame may begin its own prologue and weight prefetch

  if (warp == 0) {
    if (lane == 0) {
      // ===== producer =====
      // Programmatic dependent launch: the weights do not depend on the preceding kernel, so the first `stages` weight pairs of
      // this CTA's first tile are requested before the dependency wait (their HBM latency overlaps the predecessor's tail and
      // this kernel's own launch); the activation boxes, and everything the epilogue touches, come after it.
      int pre = 0;
      if ((int)blockIdx.x < n_tiles) {
        const Tile t0 = tile_at(p, blockIdx.x);
        const uint8_t* wsrc = p.wt + ((size_t)t0.n * p.num_kb + t0.kb0) * (size_t)(2 * w_bytes);
        for (int kb = t0.kb0; kb < t0.kb1 && pre < p.stages; ++kb, wsrc += 2 * w_bytes, ++pre) {
          mbar_expect_tx(full0 + 8 * pre, 2 * p.box_bytes + 2 * w_bytes);
          bulk_load(base + (uint32_t)pre * p.stage_bytes + 2 * p.a_bytes, wsrc, 2 * w_bytes, full0 + 8 * pre);
        }
      }
      pdl_wait();
      int s = 0; uint32_t ph = 0;
      int item = 0;
      for (int id = blockIdx.x; id < n_tiles; id += gridDim.x) {
        const Tile tl = tile_at(p, id);
        const uint8_t* wsrc = p.wt + ((size_t)tl.n * p.num_kb + tl.kb0) * (size_t)(2 * w_bytes);
        int tap, cb;
        divide(tl.kb0, p.cb_per_tap, tap, cb);
        for (int kb = tl.kb0; kb < tl.kb1; ++kb, wsrc += 2 * w_bytes, ++item) {
          const uint32_t sa = base + (uint32_t)s * p.stage_bytes;
          if (item >= pre) {
            mbar_wait(empty0 + 8 * s, ph ^ 1u);
            mbar_expect_tx(full0 + 8 * s, 2 * p.box_bytes + 2 * w_bytes);
            bulk_load(sa + 2 * p.a_bytes, wsrc, 2 * w_bytes, full0 + 8 * s);
          }
          const int row = p.row0 + tl.t0 * p.stride + tap * p.dil;
          tma_load_3d(sa, &map_hi, full0 + 8 * s, cb * TC_KB, row, tl.b0);
          tma_load_3d(sa + p.a_bytes, &map_lo, full0 + 8 * s, cb * TC_KB, row, tl.b0);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
          if (++cb == p.cb_per_tap) { cb = 0; ++tap; }
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer: the whole warp walks along, one thread issues; per k-block 4 k-steps x (hi*hi + hi*lo + lo*hi) =====
    const uint32_t idesc = make_idesc_tf32(TC_ROWS, p.swap ? p.swap : p.NT);
    // operands with the tensor core's rows (m) and columns (n), relative to a stage: hi part, and from there to the lo part
    const uint32_t a_lo = p.a_bytes >> 4, w_at = 2 * a_lo, w_lo = w_bytes >> 4;
    const uint32_t m_at = p.swap ? w_at : 0u, m_lo = p.swap ? w_lo : a_lo, n_at = p.swap ? 0u : w_at, n_lo = p.swap ? a_lo : w_lo;
    int s = 0; uint32_t ph = 0;
    int acc = 0; uint32_t acc_bits = 0u;
    for (int id = blockIdx.x; id < n_tiles; id += gridDim.x) {
      const Tile tl = tile_at(p, id);
      for (int k0 = tl.kb0; k0 < tl.kb1; k0 += TC_CHAIN) {
        mbar_wait(tempty0 + 8 * acc, ((acc_bits >> acc) & 1u) ^ 1u);
        tc_fence_after();
        const uint32_t d0 = tmem_base + (uint32_t)(acc * p.NT);
        for (int kb = k0; kb < min(tl.kb1, k0 + TC_CHAIN); ++kb) {
          mbar_wait(full0 + 8 * s, ph);
          tc_fence_after();
          const uint32_t sa = desc_low(base + (uint32_t)s * p.stage_bytes), sm = sa + m_at, sn = sa + n_at;
#pragma unroll
          for (int k = 0; k < TC_KB / 8; ++k)                // 8 tf32 = 32 bytes of K per step
            umma_tf32_split(d0, sm + 2 * k, sm + m_lo + 2 * k, sn + 2 * k, sn + n_lo + 2 * k, idesc, (kb == k0 && k == 0) ? 0u : 1u);
          commit_elected(empty0 + 8 * s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
        commit_elected(tfull0 + 8 * acc);
        acc_bits ^= 1u << acc;
        acc ^= 1;
      }
    }
    __syncwarp();
  } else {
    // ===== epilogue: TMEM lane = GEMM row = one (session, step).  The sums go through shared memory, so that what is stored and read is whole lines =====
    // (with p.swap the other way round: TMEM lane = feature, column = GEMM row; only in a cluster)
    const int ncols = p.swap ? p.swap : p.NT;
    const int q = warp & 3, sub = (warp - 2) >> 2, row = q * 32 + lane, qt = sub * 32 + lane;      // TMEM quadrant, this warp's place among its four
    const int cols = min(64, p.NT), cols4 = cols >> 2, c = qt % cols4, step = 128 / cols4;      // 64 columns at a time; where runs do not deal out evenly some threads rest
    int acc = 0; uint32_t acc_bits = 0u;
    // in a cluster every CTA finishes its share of the tile's rows: all 16 warps, whole rows of NT columns
    const int tid = threadIdx.x - 64, all4 = p.NT >> 2, c_all = tid % all4, r_all = tid / all4, step_all = 32 * TC_EPI_WARPS / all4, r_own = qt / cols4;
    const bool busy = cluster ? tid < step_all * all4 : qt < step * cols4;
    Tile tl = tile_at(p, blockIdx.x);
    int valid = valid_rows(p, tl), r = 0, r1 = 0, n = 0;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f), res = f;
    if (cluster) {
      const int lo = valid * tl.split / p.ksplit;
      r = lo + r_all;
      r1 = valid * (tl.split + 1) / p.ksplit;
      n = tl.n * p.NT + c_all * 4;
      if (busy) f = feature_terms(p, n);
    }
    pdl_wait();                                  // outputs and residuals may still be in use by the predecessor
    for (int id = blockIdx.x; id < n_tiles; id += gridDim.x) {
      if (id != (int)blockIdx.x) { tl = tile_at(p, id); valid = valid_rows(p, tl); }
      const int n_base = tl.n * p.NT;
      const bool whole = tl.kb1 - tl.kb0 <= TC_CHAIN;
      if (!cluster) {
        r = q * 32 + r_own;
        r1 = min(valid, q * 32 + 32);
        n = n_base + c * 4;
        if (busy) f = feature_terms(p, n);
      }
      if (busy) res = residual_of(p, tl, r, r1, n);
      float sum[2][16];                          // this warp's runs of 16 columns, sub * 16 and 64 + sub * 16, where the chain is too long for the tensor core
      for (int k0 = tl.kb0; !whole && k0 < tl.kb1; k0 += TC_CHAIN) {
        mbar_wait(tfull0 + 8 * acc, (acc_bits >> acc) & 1u);
        tc_fence_after();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c0 = u * 64 + sub * 16;
          if (c0 < ncols) {
            uint32_t v[16];
            __syncwarp();
            tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * p.NT + c0), v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[u][j] = k0 == tl.kb0 ? __uint_as_float(v[j]) : sum[u][j] + __uint_as_float(v[j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
        acc_bits ^= 1u << acc;
        acc ^= 1;
      }
      if (whole) {
        mbar_wait(tfull0 + 8 * acc, (acc_bits >> acc) & 1u);
        tc_fence_after();
      }
#pragma unroll 1
      for (int u = 0; u * 64 < ncols; ++u) {      // 64 columns at a time; a cluster's all lie in shared memory together
        const int c0 = u * 64 + sub * 16, left = cluster ? p.NT : min(64, p.NT - u * 64);
        if (c0 < ncols) {
          float v[16];
          if (whole) {
            uint32_t t[16];
            __syncwarp();
            tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * p.NT + c0), t);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(t[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = u == 0 ? sum[0][j] : sum[1][j];
          }
          if (p.swap) {
            const uint32_t at = sums + (uint32_t)c0 * (TC_ROWS * 4) + (row & 3) * 4;      // as four_at has it, with 128 features: c0 is a multiple of 16
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (c0 + j < valid) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (uint32_t)j * (TC_ROWS * 4) + (((row >> 2) ^ (j & 7)) << 4)), "f"(v[j]) : "memory");
          } else if (row < valid) {
#pragma unroll
            for (int j = 0; j < 4; ++j) sts_four(four_at(sums, row, (cluster ? c0 >> 2 : sub * 4) + j, left >> 2), v + 4 * j);
          }
        }
        if (!cluster) {
          asm volatile("bar.sync %0, 128;" ::"r"(1 + q) : "memory");
          if (busy && c * 4 < left) {
            if (u > 0) {
              n = n_base + u * 64 + c * 4;
              f = feature_terms(p, n);
              res = residual_of(p, tl, r, r1, n);
            }
            finish_rows(p, false, sums, tl, r, r1, step, c, left >> 2, n, f, res);
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + q) : "memory");
        }
      }
      if (whole) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
        acc_bits ^= 1u << acc;
        acc ^= 1;
      }
    }
    if (cluster) {
      __syncwarp();
      cluster_sync();
      if (busy) finish_rows(p, true, sums, tl, r, r1, step_all, c_all, all4, n, f, res);
    }
  }
  if (cluster) {
    __syncwarp();
    if (warp < 2) cluster_sync();
    cluster_meet();                              // nobody leaves while its sums are read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, p.tmem_cols);
}

// load-time: w fp32 [N][n_taps * Cin] -> [n_tile][kb][hi | lo][NT rows][32] in the SWIZZLE_128B layout
// (16-byte chunk c of row r at r * 128 + ((c ^ (r & 7)) << 4)); rows beyond N are zero
__global__ void tc_pack_kernel(const float* __restrict__ w, float4* __restrict__ out, int N, int K, int NT, int n_tiles_n, int num_kb) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;      // one 16-byte chunk (4 floats) of a hi tile
  const long long per_tile = (long long)NT * 8;
  const long long total = (long long)n_tiles_n * num_kb * per_tile;
  if (idx >= total) return;
  const int chunk = (int)(idx % per_tile);
  long long t = idx / per_tile;
  const int kb = (int)(t % num_kb);
  const int nt = (int)(t / num_kb);
  const int r = chunk >> 3, cpos = chunk & 7;
  const int csrc = cpos ^ (r & 7);
  const int n = nt * NT + r, k = kb * TC_KB + csrc * 4;
  float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
  if (n < N) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (k + i < K) split_tf32(w[(long long)n * K + k + i], hi[i], lo[i]);
  }
  const long long o = (((long long)nt * num_kb + kb) * 2) * per_tile + chunk;
  out[o] = make_float4(hi[0], hi[1], hi[2], hi[3]);
  out[o + per_tile] = make_float4(lo[0], lo[1], lo[2], lo[3]);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;

}  // namespace

bool tc_pdl() {
  static const bool on = [] { const char* e = getenv("B200_MIMI_PDL"); return !e || atoi(e) != 0; }();
  return on;
}

int tc_init() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    B200_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
    if (!fn || qres != cudaDriverEntryPointSuccess) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  static std::atomic<uint64_t> limits{0};
  return allow_smem(limits, TC_SMEM + 1024 + 16 * TC_MAX_STAGES + 64, mimi_tc_kernel);
}

static int pick_nt(int N) { return N >= TC_MAX_NT ? TC_MAX_NT : N; }

size_t tc_packed_bytes(int N, int Cin, int n_taps) {
  const int NT = pick_nt(N), n_tiles = (N + NT - 1) / NT, num_kb = n_taps * (Cin / TC_KB);
  return (size_t)n_tiles * num_kb * 2 * NT * 128;
}

int tc_pack_weights(const float* w_dev, void* out_dev, int N, int Cin, int n_taps, cudaStream_t st) {
  if (Cin % TC_KB || N % 16 || (N > TC_MAX_NT && N % TC_MAX_NT))
    B200_FAIL(B200_ERR_SHAPE, "tc_pack_weights: Cin %d must be a multiple of 32, N %d a multiple of 16 (of 128 above 128)", Cin, N);
  const int NT = pick_nt(N), n_tiles = (N + NT - 1) / NT, num_kb = n_taps * (Cin / TC_KB);
  const long long total = (long long)n_tiles * num_kb * NT * 8;
  tc_pack_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(w_dev, static_cast<float4*>(out_dev), N, n_taps * Cin, NT, n_tiles, num_kb);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("tc_pack");
}

int tc_make_map(CUtensorMap* m, const float* base, int Cin, long long rows_per_session, long long sb_elems, int n_sessions, int tt,
                int bb, int stride) {
  B200_TRY(tc_init());
  cuuint64_t dims[3] = {(cuuint64_t)Cin, (cuuint64_t)rows_per_session, (cuuint64_t)n_sessions};
  cuuint64_t strides[2] = {(cuuint64_t)Cin * 4, (cuuint64_t)sb_elems * 4};
  cuuint32_t box[3] = {(cuuint32_t)TC_KB, (cuuint32_t)(tt * stride), (cuuint32_t)(bb < n_sessions ? bb : n_sessions)};      // tc_plan: box_bytes
  cuuint32_t estr[3] = {1, (cuuint32_t)stride, 1};
  if (box[1] > 256 || box[2] > 256) B200_FAIL(B200_ERR_SHAPE, "tc_make_map: box %u x %u exceeds the TMA limit of 256", box[1], box[2]);
  CUresult r = g_encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d): Cin %d rows %lld sessions %d box %u/%u/%u stride %d", (int)r, Cin,
              rows_per_session, n_sessions, box[0], box[1], box[2], stride);
  return B200_OK;
}

// Fills the launch plan of a layer for `n_sessions` sessions of T output steps each (linear: n_sessions = 1, T = tokens).
// The caller has set the static fields, the tensor maps and the epilogue pointers of L.p.
int tc_plan(TcLayer& L, int n_sessions, int T, int sms) {
  TcParams& p = L.p;
  p.n_sessions = n_sessions; p.T = T;
  p.tt_log2 = 0; p.tiles_per_group = (T + p.tt - 1) / p.tt; p.cb_per_tap = L.Cin / TC_KB;
  while ((1 << p.tt_log2) < p.tt) ++p.tt_log2;
  if (p.tt * p.bb != TC_ROWS) B200_FAIL(B200_ERR_INVALID, "tc_plan: tile %d x %d is not 128 rows", p.tt, p.bb);
  if (p.bb > 1 && T % p.tt) B200_FAIL(B200_ERR_INVALID, "tc_plan: %d steps in tiles of %d", T, p.tt);
  const int tpg = (T + p.tt - 1) / p.tt, groups = (n_sessions + p.bb - 1) / p.bb;
  p.m_tiles = tpg * groups;
  p.n_taps = L.n_taps; p.dil = L.dil; p.stride = L.stride; p.Cin = L.Cin;
  p.wt = L.wt; p.NT = L.NT; p.n_tiles_n = L.n_tiles_n; p.num_kb = L.num_kb; p.N = L.N;
  p.bias = L.bias; p.bias_mod = L.bias_mod > 0 ? L.bias_mod : L.N;
  // few tiles: k cut over the CTAs of a cluster, as far as the clusters fit the chip side by side (of one CTA per SM: 74 of two, .., 15 of eight)
  static const int fit[TC_MAX_SPLIT + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  int ks = 1;
  const long long mn = (long long)p.m_tiles * p.n_tiles_n;
  for (int c = 2; c <= TC_MAX_SPLIT; ++c)
    if (mn * 148 <= (long long)fit[c] * sms && p.num_kb >= (p.num_kb < 8 ? c : 2 * c) && (p.num_kb + c - 1) / c < (p.num_kb + ks - 1) / ks) ks = c;
  p.kb_per_split = (p.num_kb + ks - 1) / ks;
  p.ksplit = ks;
  while ((p.ksplit - 1) * p.kb_per_split >= p.num_kb) { --p.ksplit; }
  // where fewer than 128 rows of a tile can exist a stage holds only those: the products read what lies behind them as the other rows, whose sums nobody takes
  p.box_bytes = (uint32_t)(p.tt * (p.bb < n_sessions ? p.bb : n_sessions)) * TC_KB * 4u;
  p.a_bytes = (p.box_bytes + 1023u) / 1024u * 1024u;
  p.stage_bytes = 2 * p.a_bytes + 2 * (uint32_t)p.NT * 128u;
  // few rows against 128 features: the features are the tensor core's rows, and the product costs what the rows there are cost
  const int rows16 = (int)(p.box_bytes / (TC_KB * 4u) + 15) / 16 * 16;
  p.swap = p.ksplit > 1 && p.NT == TC_ROWS && rows16 < TC_ROWS ? rows16 : 0;
  const int sums = p.ksplit > 1 ? 0 : TC_ROWS * (p.NT < 64 ? p.NT : 64) * 4;      // a cluster's lie in the ring: TC_ROWS x NT x 4 <= 2 stages
  int stages = (TC_SMEM - sums - (int)A_TILE_BYTES) / (int)p.stage_bytes;      // 128 rows from the last stage's on have to be shared memory too
  if (2 * p.a_bytes == 2 * A_TILE_BYTES) stages = (TC_SMEM - sums) / (int)p.stage_bytes;
  if (stages > TC_MAX_STAGES) stages = TC_MAX_STAGES;
  p.stages = stages;
  p.bars_at = (uint32_t)stages * p.stage_bytes + (uint32_t)sums;
  uint32_t cols = 32;
  while (cols < (uint32_t)(2 * p.NT)) cols <<= 1;
  p.tmem_cols = cols;
  const long long tiles = mn * p.ksplit;
  L.grid = (int)(p.ksplit > 1 || tiles < sms ? tiles : sms);
  const size_t reach = (size_t)(stages - 1) * p.stage_bytes + p.a_bytes + A_TILE_BYTES;
  L.smem = std::max<size_t>(p.bars_at + 16 * TC_MAX_STAGES + 64, reach) + 1024;
  return B200_OK;
}

int tc_launch(const TcLayer& L, cudaStream_t st) {
  // programmatic dependent launch (B200_MIMI_PDL=0: off): the kernel may start while its predecessor drains; it requests its
  // first weight tiles, then waits (griddepcontrol.wait) before it reads an activation or writes anything
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)L.grid); cfg.blockDim = dim3(TC_THREADS); cfg.dynamicSmemBytes = L.smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (tc_pdl()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (L.p.ksplit > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)L.p.ksplit; attr[n].val.clusterDim.y = 1; attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr; cfg.numAttrs = (unsigned)n;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, mimi_tc_kernel, L.map_hi, L.map_lo, L.p);
  if (le != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "mimi_tc launch failed: %s", cudaGetErrorString(le));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("mimi_tc");
}

}  // namespace mtc
}  // namespace b200
