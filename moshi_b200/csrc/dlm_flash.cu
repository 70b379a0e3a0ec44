// Causal softmax attention of many queries of one request on the 5th-generation tensor cores, head size 128, one sink logit per head.
//
// A CTA owns 128 queries of one head and walks the keys in tiles of 128.  Scores S = Q K^T and the sum O += P V are tcgen05.mma with fp32
// accumulators in TMEM (two score buffers and O: 384 of 512 columns), operands by TMA in SWIZZLE_128B (the values arrive transposed, so
// that both products read K-major operands).  Warp 0 fetches, warp 1 issues the products (the scores of tile i + 1 before the sum of tile
// i), warps 2-5 hold one query per thread: a row's 128 scores in registers, running maximum and sum in fp32, the weights in bf16 through
// shared memory.  O is rescaled only when a row's maximum grew by more than 8 in base 2: a weight of up to 256 has
// the relative error of one below 1, and the final division refers to the same maximum.  The longest tiles start first.
//
// A key tile takes about 3800 cycles, of which the tensor pipe and the exponentials' unit are each active a good quarter (2048 tokens, 16 heads): the bound is
// the chain of the four softmax warps, one per scheduler, whose latencies nothing hides; then the second wave (256 CTAs on 148 SMs).
// A wait that lasts longer than ten seconds raises the caller's error flag and the kernel winds down.
#include "dlm_flash.cuh"

#include <cuda.h>

#include "tc_prims.cuh"

namespace b200 {
namespace dlm {

namespace {

using namespace tcp;

constexpr int THREADS = 192, ROWS = 128, KEYS = 128;
constexpr uint32_t HALF = ROWS * 128;        // 128 rows of 64 bf16
constexpr uint32_t TILE = 2 * HALF;          // 128 x 128 bf16 as two halves along k
constexpr int STAGES = 2;                    // of K and of V each
constexpr uint32_t SMEM = TILE * (1 + 2 * STAGES + 1) + 1024 + 256;
constexpr float LOG2E = 1.4426950408889634f;

struct FlashP {
  const float* sink; __nv_bfloat16* out; long long ldo;
  int T, pos0, H, q_tiles; float scale2;     // scale2 = scale * log2(e)
  int* err;
};

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
#define FLASH_R32(r, o) "=r"((r)[o]), "=r"((r)[o + 1]), "=r"((r)[o + 2]), "=r"((r)[o + 3]), "=r"((r)[o + 4]), "=r"((r)[o + 5]), "=r"((r)[o + 6]), "=r"((r)[o + 7])
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : FLASH_R32(r, 0), FLASH_R32(r, 8), FLASH_R32(r, 16), FLASH_R32(r, 24) : "r"(taddr));
}
#undef FLASH_R32
#define FLASH_R32(r, o) "r"((r)[o]), "r"((r)[o + 1]), "r"((r)[o + 2]), "r"((r)[o + 3]), "r"((r)[o + 4]), "r"((r)[o + 5]), "r"((r)[o + 6]), "r"((r)[o + 7])
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), FLASH_R32(r, 0), FLASH_R32(r, 8), FLASH_R32(r, 16), FLASH_R32(r, 24) : "memory");
}
#undef FLASH_R32
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__global__ void __launch_bounds__(THREADS, 1)
flash_attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const FlashP p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int quit;
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t sq = base, sk = base + TILE, sv = sk + STAGES * TILE, sp = sv + STAGES * TILE, bars = sp + TILE;
  const uint32_t q_full = bars, k_full = bars + 8, k_empty = k_full + 8 * STAGES, v_full = k_empty + 8 * STAGES, v_empty = v_full + 8 * STAGES, s_full = v_empty + 8 * STAGES, s_free = s_full + 16,
                 p_full = s_free + 16, o_done = p_full + 8, tptr = o_done + 8;      // o_done: the sum over a tile is in O, its weights are free
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int qt = p.q_tiles - 1 - (int)blockIdx.x / p.H, h = (int)blockIdx.x % p.H;
  const int q0 = qt * ROWS, last_row = min(q0 + ROWS, p.T) - 1;
  const int n = (p.pos0 + last_row) / KEYS + 1;      // key tiles

  if (threadIdx.x == 0) {
    quit = 0;
    mbar_init(q_full, 1);
    for (int s = 0; s < STAGES; ++s) { mbar_init(k_full + 8 * s, 1); mbar_init(k_empty + 8 * s, 1); mbar_init(v_full + 8 * s, 1); mbar_init(v_empty + 8 * s, 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(s_full + 8 * s, 1); mbar_init(s_free + 8 * s, 4); }
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tptr, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<const uint32_t*>(smem_raw + (tptr - raw));
  const uint32_t tmem_o = tmem + 256;
  pdl_trigger();
  pdl_wait();

  // both loops are walked by their whole warps, and one thread issues (tc_prims.cuh)
  if (warp == 0) {
    auto load = [&](uint32_t dst, const CUtensorMap* m, uint32_t bar, int c, int r) {      // two halves along the inner dimension
      if (elected()) {
        mbar_expect_tx(bar, TILE);
        tma_load_2d(dst, m, bar, c, r);
        tma_load_2d(dst + HALF, m, bar, c + 64, r);
      }
      __syncwarp();
    };
    load(sq, &map_q, q_full, h * FLASH_D, q0);
    bool ok = true;
    int s = 0; uint32_t ph = 0;
    for (int i = 0; ok && i < n; ++i) {
      // a stage's keys are free once its scores are there, its values once their sum is
      if (!warp_wait(k_empty + 8 * s, ph ^ 1u, &quit)) { ok = false; break; }
      load(sk + s * TILE, &map_k, k_full + 8 * s, h * FLASH_D, i * KEYS);
      if (!warp_wait(v_empty + 8 * s, ph ^ 1u, &quit)) { ok = false; break; }
      load(sv + s * TILE, &map_v, v_full + 8 * s, i * KEYS, h * FLASH_D);
      if (++s == STAGES) { s = 0; ph ^= 1u; }
    }
    if (!ok) {                               // let copies in flight land before the block ends
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc(ROWS, 128);
    auto product = [&](uint32_t d, uint32_t a, uint32_t b, bool add) {      // 128 x 128 x 128, in two halves of k
      const uint32_t da = desc_low(a), to = desc_low(b) - da;
      umma_block<1>(d, da, to, idesc, add ? 1u : 0u);
      umma_block<1>(d, da + (HALF >> 4), to, idesc, 1u);
    };
    int ks = 0; uint32_t kph = 0;            // stage and phase of the next keys
    auto scores = [&](int i) {
      const int b = i & 1;
      if (!warp_wait(k_full + 8 * ks, kph, &quit)) return false;
      if (!warp_wait(s_free + 8 * b, ((uint32_t)(i >> 1) & 1u) ^ 1u, &quit)) return false;
      tc_fence_after();
      product(tmem + b * 128, sq, sk + ks * TILE, false);
      commit_elected(k_empty + 8 * ks);
      commit_elected(s_full + 8 * b);
      if (++ks == STAGES) { ks = 0; kph ^= 1u; }
      return true;
    };
    bool ok = warp_wait(q_full, 0, &quit) && scores(0);
    int s = 0; uint32_t ph = 0;
    for (int i = 0; ok && i < n; ++i) {
      if (i + 1 < n) ok = scores(i + 1);
      ok = ok && warp_wait(v_full + 8 * s, ph, &quit) && warp_wait(p_full, (uint32_t)i & 1u, &quit);
      if (!ok) break;
      tc_fence_after();
      product(tmem_o, sp, sv + s * TILE, i > 0);
      commit_elected(v_empty + 8 * s);
      commit_elected(o_done);
      if (++s == STAGES) { s = 0; ph ^= 1u; }
    }
    __syncwarp();
  } else {
    const int q4 = warp & 3, row = q4 * 32 + lane, pos = p.pos0 + q0 + row;
    const uint32_t lanes = (uint32_t)(q4 * 32) << 16;
    uint8_t* prow = smem_raw + (sp - raw) + row * 128;
    float m = -INFINITY, sum = 0.f;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int b = i & 1;
      ok = wait_or_quit(s_full + 8 * b, (uint32_t)(i >> 1) & 1u, &quit);
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      tc_fence_after();
      uint32_t r[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tmem + lanes + b * 128 + c * 32, r + c * 32);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free + 8 * b);
      const int k0 = i * KEYS;
      if (k0 + KEYS - 1 > p.pos0 + q0) {     // the diagonal: keys behind the query's position
#pragma unroll
        for (int j = 0; j < 128; ++j)
          if (k0 + j > pos) r[j] = 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < 128; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(r[j]));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale2;      // scale2 > 0
      float factor = 1.f;
      const bool grow = top > m + 8.f;
      if (grow) { factor = exp2f(m - top); m = top; sum *= factor; }
      const bool rescale = __any_sync(0xffffffffu, grow) && i > 0;
      const float off = m == -INFINITY ? 0.f : m;
      float add[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t w[64];
#pragma unroll
      for (int j = 0; j < 128; j += 2) {
        const float e0 = exp2f(fmaf(__uint_as_float(r[j]), p.scale2, -off)), e1 = exp2f(fmaf(__uint_as_float(r[j + 1]), p.scale2, -off));
        add[(j >> 1) & 3] += e0 + e1;
        w[j >> 1] = pack2(e0, e1);
      }
      sum += (add[0] + add[1]) + (add[2] + add[3]);
      if (i > 0) {                           // the sum over the previous tile has read its weights and settled in O
        ok = wait_or_quit(o_done, (uint32_t)(i - 1) & 1u, &quit);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        tc_fence_after();
      }
      if (rescale) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tmem_o + lanes + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * factor);
          tmem_st32(tmem_o + lanes + c * 32, o);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
#pragma unroll
      for (int c = 0; c < 16; ++c)           // 16-byte piece c of the row: half c / 8, piece c % 8 swizzled by the row
        *reinterpret_cast<uint4*>(prow + (c >> 3) * HALF + (((c & 7) ^ (row & 7)) << 4)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok) {
      ok = wait_or_quit(o_done, (uint32_t)(n - 1) & 1u, &quit);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok) {
      tc_fence_after();
      if (p.sink) sum += exp2f(p.sink[h] * LOG2E - m);
      const float inv = 1.f / sum;
      __nv_bfloat16* out = p.out + (long long)(q0 + row) * p.ldo + h * FLASH_D;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        __syncwarp();
        tmem_ld32(tmem_o + lanes + c * 32, o);
        tmem_ld_wait();
        if (q0 + row < p.T) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 v;
            v.x = pack2(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv);
            v.y = pack2(__uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
            v.z = pack2(__uint_as_float(o[j + 4]) * inv, __uint_as_float(o[j + 5]) * inv);
            v.w = pack2(__uint_as_float(o[j + 6]) * inv, __uint_as_float(o[j + 7]) * inv);
            *reinterpret_cast<uint4*>(out + c * 32 + j) = v;
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 512);
  if (threadIdx.x == 0 && quit && p.err) atomicOr(p.err, FLASH_ERR_WAIT);
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int make_map(CUtensorMap* m, const void* ptr, long long rows, long long cols, long long ld) {
  static const EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  if (!fn) B200_FAIL(B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64, 128}, est[2] = {1, 1};
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, est, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) B200_FAIL(B200_ERR_CUDA, "attention: tensor map of %lld x %lld (ld %lld) refused (%d)", rows, cols, ld, (int)r);
  return B200_OK;
}

}  // namespace

bool flash_supported(const FlashAttn& a) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.vt) | reinterpret_cast<uintptr_t>(a.out);
  return a.T >= 1 && a.pos0 >= 0 && a.H >= 1 && a.scale > 0.f && (bases & 15) == 0 && ((a.ldq | a.ldk | a.ldv | a.ldo) & 7) == 0 && a.ldv >= a.pos0 + a.T;
}

int flash_attention(const FlashAttn& a, cudaStream_t st) {
  if (!flash_supported(a)) B200_FAIL(B200_ERR_SHAPE, "attention: unsupported shape (T %d, position %d, %d heads)", a.T, a.pos0, a.H);
  const long long ctx = (long long)a.pos0 + a.T;
  CUtensorMap mq, mk, mv;
  B200_TRY(make_map(&mq, a.q, a.T, (long long)a.H * FLASH_D, a.ldq));
  B200_TRY(make_map(&mk, a.k, ctx, (long long)a.H * FLASH_D, a.ldk));
  B200_TRY(make_map(&mv, a.vt, (long long)a.H * FLASH_D, ctx, a.ldv));
  static std::atomic<uint64_t> limits{0};
  B200_TRY(allow_smem(limits, (int)SMEM, flash_attention_kernel));
  FlashP p;
  p.sink = a.sink; p.out = a.out; p.ldo = a.ldo; p.T = a.T; p.pos0 = a.pos0; p.H = a.H; p.q_tiles = ceil_div(a.T, ROWS); p.scale2 = a.scale * LOG2E; p.err = a.err;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(p.q_tiles * a.H)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, flash_attention_kernel, mq, mk, mv, p);
  if (e != cudaSuccess) B200_FAIL(B200_ERR_CUDA, "flash_attention launch failed: %s", cudaGetErrorString(e));
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_launch("flash_attention");
}

}  // namespace dlm
}  // namespace b200

using namespace b200;

extern "C" int b200_op_prefill_attention(const void* q_dev, const void* k_dev, const void* vt_dev, const float* sink_dev, void* out_dev, int T, int H, int pos0,
                                         int ldv, float scale, void* stream) {
  if (!q_dev || !k_dev || !vt_dev || !out_dev) B200_FAIL(B200_ERR_INVALID, "op_prefill_attention: null pointer");
  dlm::FlashAttn a;
  a.q = static_cast<const __nv_bfloat16*>(q_dev); a.ldq = (long long)H * dlm::FLASH_D; a.k = static_cast<const __nv_bfloat16*>(k_dev); a.ldk = a.ldq;
  a.vt = static_cast<const __nv_bfloat16*>(vt_dev); a.ldv = ldv; a.sink = sink_dev; a.out = static_cast<__nv_bfloat16*>(out_dev); a.ldo = a.ldq;
  a.T = T; a.pos0 = pos0; a.H = H; a.scale = scale; a.err = nullptr;
  return dlm::flash_attention(a, static_cast<cudaStream_t>(stream));
}
