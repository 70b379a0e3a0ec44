// The depformer of a frame for up to 16 sessions: one persistent cooperative kernel like dep_fused_kernel, with the weights going through
// registers (gemm_reg.cu) instead of shared memory and TMEM.  Included by dep_fused.cu behind DepParams.
//
// What bounds a frame here is the chain: 8 sub-steps x 6 layers x 4 products, each of which has to see all of the one before.  So a layer is five
// phases, and a phase is a grid barrier, one L2 round trip for the activations, a few products and one exchange inside the CTA:
//   * a product's 16-row groups are dealt to the CTAs whole; the eight warps of a CTA share a group's k and add their sums in shared memory,
//     so no partial sum leaves an SM (dep_fused_kernel exchanges split-K partials through L2 and needs a phase of its own to add them);
//   * every thread asks for its weights of the NEXT product before it enters the barrier.  They are meant for registers, but 255 do not hold all that
//     is live across the sampler and the long product: with one block of 8 sessions 158 words per thread go through local memory, with two 317;
//   * RMSNorm is repeated by every CTA on its way to shared memory (B rows of 2 KB), residual, gating and bf16 roundings sit in the epilogues.
//
// Frame of 1 session 2.0 (as a chain of launches) -> 1.35 ms, 8 sessions 2.6 (dep_fused_kernel) -> 1.39, 16 sessions 2.7 -> 1.8 (1.48 and 1.98 for 1
// and 16 with sampling): 8 x (2 + 5 x 6) = 256 barriers of about 5 us, of which the release of the epilogue's stores, the counter and the poll take half.
//
// A barrier that is not met within ten seconds ends the kernel; the frame's remaining tokens are then the frame's before.  It raises ERR_WAIT, and a
// word on the host that the handle's next call looks at without a synchronisation.
#pragma once

constexpr int REG_B = 16;                    // sessions at most
constexpr int REG_FRAGS = 8;                 // (group, k-block, gate / value) fragments a warp holds: 4 pieces each
constexpr int REG_GROUPS = 2;                // 16-row groups per CTA at most
constexpr int REG_KB_SHORT = 2, REG_KB_LONG = 6;      // k-blocks per warp: dd <= 1024, F <= 3072

struct RegW { uint4 f[REG_FRAGS][4]; };

__device__ __forceinline__ uint4 reg_ldw(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void reg_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// all CTAs meet; false: not within the limit.  DIAG: with time stamps and a limit of the caller's, in a kernel of its own (in the one kernel the
// tests for them cost 0.13 us per barrier, 33 us per frame of 16 sessions).
template <bool DIAG>
__device__ __forceinline__ bool reg_grid_sync(const DepParams& p, unsigned& epoch, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    epoch += 1;
    const unsigned target = epoch * gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.bar) : "memory");
    unsigned spins = 0;
    uint64_t t0 = 0;
    int met = 1;
    while (ld_acquire(p.bar) < target) {
      if ((++spins & (DIAG ? p.wait_mask : 4095u)) == 0u) {
        const uint64_t now = global_timer_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > (DIAG ? p.wait_ns : WAIT_LIMIT_NS)) { met = 0; break; }
      }
    }
    *ok = met;
  }
  __syncthreads();
  if (DIAG && p.trace != nullptr && threadIdx.x == 0 && blockIdx.x == 0 && epoch < (unsigned)DEP_TRACE_SLOTS) p.trace[epoch] = global_timer_ns();
  return *ok != 0;
}

// this warp's fragments of a product: groups blockIdx.x, + gridDim.x; k-blocks warp * KBW ..
template <int A, int KBW, int G>
__device__ __forceinline__ void reg_load(RegW& w, const uint8_t* wt, int groups, int num_kb) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int gi = 0; gi < G; ++gi) {
    const int grp = blockIdx.x + gi * gridDim.x;
    if (grp < groups) {
      const uint4* base = reinterpret_cast<const uint4*>(wt) + (size_t)(grp >> 3) * num_kb * (A * 1024) + ((grp & 7) * 16 + g) * 8;
#pragma unroll
      for (int j = 0; j < KBW; ++j) {
        const int kb = warp * KBW + j;
        if (kb < num_kb) {
#pragma unroll
          for (int a = 0; a < A; ++a) {
            uint4 (&f)[4] = w.f[(gi * KBW + j) * A + a];
            const uint4* s = base + (size_t)(kb * A + a) * 1024;
            f[0] = reg_ldw(s + (t ^ g)); f[1] = reg_ldw(s + 64 + (t ^ g));
            f[2] = reg_ldw(s + ((t + 4) ^ g)); f[3] = reg_ldw(s + 64 + ((t + 4) ^ g));
          }
        }
      }
    }
  }
}

// sums of this CTA's groups over all of k -> red[(gi * A + a)][warp][16 rows][8 NT + 1]; x(m, byte) gives 16 bytes of row m
template <int A, int KBW, int G, int NT, typename X>
__device__ __forceinline__ void reg_product(const RegW& w, int groups, int num_kb, float* red, X x) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  if ((int)blockIdx.x >= groups) return;
  float acc[G][A][NT][4];
#pragma unroll
  for (int gi = 0; gi < G; ++gi)
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int n = 0; n < NT; ++n) acc[gi][a][n][0] = acc[gi][a][n][1] = acc[gi][a][n][2] = acc[gi][a][n][3] = 0.f;
  constexpr int AHEAD = NT == 1 || KBW <= 2 ? KBW : 2;      // activations in flight: what the registers beside the weights hold
#pragma unroll
  for (int j0 = 0; j0 < KBW; j0 += AHEAD) {
    uint4 xb[AHEAD][2][NT];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int n = 0; n < NT; ++n)
          if (warp * KBW + j0 + j < num_kb) xb[j][h][n] = x(8 * n + g, (warp * KBW + j0 + j) * 128 + h * 64 + t * 16);
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      if (warp * KBW + j0 + j >= num_kb) break;
#pragma unroll
      for (int gi = 0; gi < G; ++gi) {
        if ((int)(blockIdx.x + gi * gridDim.x) >= groups) break;
#pragma unroll
        for (int a = 0; a < A; ++a) {
          const uint4 (&f)[4] = w.f[(gi * KBW + j0 + j) * A + a];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              reg_mma(acc[gi][a][n], f[2 * h].x, f[2 * h + 1].x, f[2 * h].y, f[2 * h + 1].y, xb[j][h][n].x, xb[j][h][n].y);
              reg_mma(acc[gi][a][n], f[2 * h].z, f[2 * h + 1].z, f[2 * h].w, f[2 * h + 1].w, xb[j][h][n].z, xb[j][h][n].w);
            }
        }
      }
    }
  }
  constexpr int LD = 8 * NT + 1;
#pragma unroll
  for (int gi = 0; gi < G; ++gi)
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) red[(((gi * A + a) * 8 + warp) * 16 + g + (e >> 1) * 8) * LD + 8 * n + 2 * t + (e & 1)] = acc[gi][a][n][e];
}

// out(m, n, sum, second sum) for every result of this CTA's groups; the warps' sums are added in warp order
template <int A, int G, int NT, typename F>
__device__ __forceinline__ void reg_epilogue(const float* red, int groups, int B, F out) {
  __syncthreads();
  constexpr int LD = 8 * NT + 1;
  for (int i = threadIdx.x; i < G * 16 * 8 * NT; i += THREADS) {
    const int row = i & 15, m = (i >> 4) % (8 * NT), gi = i / (128 * NT), grp = blockIdx.x + gi * gridDim.x;
    if (m >= B || grp >= groups) continue;
    float v[2] = {0.f, 0.f};
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int q = 0; q < 8; ++q) v[a] += red[(((gi * A + a) * 8 + q) * 16 + row) * LD + m];
    out(m, grp * 16 + row, v[0], v[1]);
  }
}

// rows of x -> shared memory, normed when alpha is given (same roundings as row_phase)
template <int NT>
__device__ __forceinline__ void reg_stage(const DepParams& p, const bf16* alpha, uint8_t* xs, int xs_ld) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < NT; ++r) {
    const int m = warp + 8 * r;
    if (m >= p.B) break;
    uint4 v[4];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (lane + 32 * i) * 8;
      if (c < p.dd) {
        v[i] = __ldcg(reinterpret_cast<const uint4*>(p.x + (long long)m * p.dd + c));
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v[i]);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); ss += f.x * f.x + f.y * f.y; }
      }
    }
    const float rs = alpha ? rsqrtf(1e-8f + warp_sum(ss) / (float)p.dd) : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (lane + 32 * i) * 8;
      if (c < p.dd) {
        if (alpha) {
          const uint4 av = __ldg(reinterpret_cast<const uint4*>(alpha + c));
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v[i]);
          const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&av);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h[e]), q = __bfloat1622float2(a[e]);
            h[e] = __floats2bfloat162_rn(f.x * (q.x * rs), f.y * (q.y * rs));
          }
        }
        *reinterpret_cast<uint4*>(xs + m * xs_ld + c * 2) = v[i];
      }
    }
  }
  __syncthreads();
}

// KV append and attention over step + 1 keys, one warp per (session, head); a lane reads back only what it wrote itself
__device__ __forceinline__ void reg_attention(const DepParams& p, const bf16* qkv, int layer, int step) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, C = p.dd;
  for (int it = blockIdx.x + warp * gridDim.x; it < p.B * p.H; it += gridDim.x * (THREADS / 32)) {
    const int b = it / p.H, h = it - b * p.H;
    const unsigned* src = reinterpret_cast<const unsigned*>(qkv + (long long)b * 3 * C + h * DD) + lane;
    const unsigned qw = __ldcg(src), kw = __ldcg(src + C / 2), vw = __ldcg(src + C);
    unsigned* kc = reinterpret_cast<unsigned*>(p.kc[layer] + (long long)it * p.dep_q * DD) + lane;
    unsigned* vc = reinterpret_cast<unsigned*>(p.vc[layer] + (long long)it * p.dep_q * DD) + lane;
    unsigned ko[lm::DEP_MAX_Q], vo[lm::DEP_MAX_Q];
#pragma unroll
    for (int j = 0; j < lm::DEP_MAX_Q; ++j)
      if (j < step) { ko[j] = kc[j * (DD / 2)]; vo[j] = vc[j * (DD / 2)]; }
    kc[step * (DD / 2)] = kw;
    vc[step * (DD / 2)] = vw;
    const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qw));
    float sc[lm::DEP_MAX_Q], mx = -INFINITY, sum = 0.f;
#pragma unroll
    for (int j = 0; j < lm::DEP_MAX_Q; ++j) {
      if (j <= step) {
        const unsigned w = j == step ? kw : ko[j];
        const float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
        sc[j] = warp_sum(q.x * k.x + q.y * k.y) * 0.125f;
        mx = fmaxf(mx, sc[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < lm::DEP_MAX_Q; ++j)
      if (j <= step) { sc[j] = expf(sc[j] - mx); sum += sc[j]; }
    const float inv = 1.f / sum;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int j = 0; j < lm::DEP_MAX_Q; ++j) {
      if (j <= step) {
        const unsigned w = j == step ? vw : vo[j];
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
        a0 = fmaf(sc[j] * inv, v.x, a0);
        a1 = fmaf(sc[j] * inv, v.y, a1);
      }
    }
    *reinterpret_cast<__nv_bfloat162*>(p.ao + (long long)b * C + h * DD + 2 * lane) = __floats2bfloat162_rn(a0, a1);
  }
}

template <int NT, bool DIAG>
__global__ void __launch_bounds__(THREADS, 1) dep_reg_kernel(const DepParams p, bf16* qkv) {
  extern __shared__ __align__(16) uint8_t reg_smem[];
  __shared__ int ok;
  const int xs_ld = p.dd * 2 + 64;           // rows 64 bytes apart modulo 128: the eight lanes of a 16-byte read phase meet no bank twice
  uint8_t* xs = reg_smem;
  float* red = reinterpret_cast<float*>(reg_smem + 8 * NT * xs_ld);
  for (int i = threadIdx.x * 16; i < 8 * NT * xs_ld; i += THREADS * 16) *reinterpret_cast<uint4*>(xs + i) = make_uint4(0u, 0u, 0u, 0u);
  const int kd = p.dd / 64, kf = (p.F + 63) / 64, gd = p.dd / 16, gin = 3 * p.dd / 16, gf = p.F / 16, gh = (p.card + 15) / 16;
  unsigned epoch = 0;
  if (DIAG && p.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0) p.trace[0] = global_timer_ns();
  RegW w;
  auto shared_x = [&](int m, int byte) { return *reinterpret_cast<const uint4*>(xs + m * xs_ld + byte); };
  auto global_x = [&](const bf16* buf, int K) {
    return [=](int m, int byte) {
      if (m >= p.B || byte >= 2 * K) return make_uint4(0u, 0u, 0u, 0u);
      return __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(buf + (long long)m * K) + byte));
    };
  };
  auto add_to_x = [&](int m, int n, float v, float) {
    bf16* x = p.x + (long long)m * p.dd + n;
    const unsigned short old = __ldcg(reinterpret_cast<const unsigned short*>(x));
    *x = f2bf(__bfloat162float(__ushort_as_bfloat16(old)) + rbf(v));      // x_orig + update, both bf16 (transformer.py:769,777)
  };
  reg_load<1, REG_KB_SHORT, 2>(w, p.w[0].in_w, gin, kd);
  for (int k = 0; k < p.dep_q; ++k) {
    input_rows(p, k);
    if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
    for (int l = 0; l < p.L; ++l) {
      const DepLayerW lw = p.w[k * p.L + l];
      reg_stage<NT>(p, p.n1[l], xs, xs_ld);
      reg_product<1, REG_KB_SHORT, 2, NT>(w, gin, kd, red, shared_x);
      reg_epilogue<1, 2, NT>(red, gin, p.B, [&](int m, int n, float v, float) { qkv[(long long)m * 3 * p.dd + n] = f2bf(v); });
      reg_load<1, REG_KB_SHORT, 1>(w, lw.out_w, gd, kd);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
      reg_attention(p, qkv, l, k);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
      reg_product<1, REG_KB_SHORT, 1, NT>(w, gd, kd, red, global_x(p.ao, p.dd));
      reg_epilogue<1, 1, NT>(red, gd, p.B, add_to_x);
      reg_load<2, REG_KB_SHORT, 2>(w, lw.lin_in, gf, kd);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
      reg_stage<NT>(p, p.n2[l], xs, xs_ld);
      reg_product<2, REG_KB_SHORT, 2, NT>(w, gf, kd, red, shared_x);
      reg_epilogue<2, 2, NT>(red, gf, p.B, [&](int m, int n, float g, float u) {      // gating.py:18-20
        g = rbf(g); u = rbf(u);
        p.hbuf[(long long)m * p.F + n] = f2bf(rbf(g / (1.f + expf(-g))) * u);
      });
      reg_load<1, REG_KB_LONG, 1>(w, lw.lin_out, gd, kf);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
      reg_product<1, REG_KB_LONG, 1, NT>(w, gd, kf, red, global_x(p.hbuf, p.F));
      reg_epilogue<1, 1, NT>(red, gd, p.B, add_to_x);
      if (l + 1 < p.L) reg_load<1, REG_KB_SHORT, 2>(w, p.w[k * p.L + l + 1].in_w, gin, kd);
      else reg_load<1, REG_KB_SHORT, 2>(w, p.heads[k], gh, kd);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
    }
    if (!ok) break;
    reg_stage<NT>(p, nullptr, xs, xs_ld);    // depformer_norms is Identity (lm.py:197-198): the head reads x itself
    reg_product<1, REG_KB_SHORT, 2, NT>(w, gh, kd, red, shared_x);
    reg_epilogue<1, 2, NT>(red, gh, p.B, [&](int m, int n, float v, float) {
      if (n < p.card) p.logits[((long long)k * p.B + m) * p.card + n] = f2bf(v);
    });
    if (k + 1 < p.dep_q) reg_load<1, REG_KB_SHORT, 2>(w, p.w[(k + 1) * p.L].in_w, gin, kd);
    if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
    for (int m = blockIdx.x; m < p.B; m += gridDim.x) {      // the next sub-step's input rows are the same rows of the same CTA
      lm::sample_row(p.logits + ((long long)k * p.B + m) * p.card, p.noise + (long long)m * p.noise_ld + p.noise_off + (long long)k * p.ka,
                     p.audio_tokens + (long long)k * p.B + m, p.card, p.use_sampling, p.temp, p.top_k);
      __syncthreads();
    }
  }
  if (threadIdx.x == 0 && !ok) {
    if (p.err) atomicOr(p.err, lm::ERR_WAIT);
    if (p.gave_up) {
      *p.gave_up = 1;
      __threadfence_system();
    }
  }
}

typedef void (*DepRegKernel)(const DepParams, bf16*);
inline DepRegKernel dep_reg_pick(int nt, bool diag) {
  return nt == 1 ? (diag ? dep_reg_kernel<1, true> : dep_reg_kernel<1, false>) : (diag ? dep_reg_kernel<2, true> : dep_reg_kernel<2, false>);
}
inline size_t dep_reg_smem(int nt, int dd) { return (size_t)8 * nt * (dd * 2 + 64) + (size_t)4 * 8 * 16 * (8 * nt + 1) * 4; }
inline bool dep_reg_takes(const DepFusedConfig& c, int grid) {
  return c.B <= REG_B && c.dd % 64 == 0 && c.dd <= REG_KB_SHORT * 8 * 64 && c.F % 16 == 0 && c.F <= REG_KB_LONG * 8 * 64 && 3 * c.dd / 16 <= REG_GROUPS * grid &&
         c.F / 16 <= REG_GROUPS * grid && (c.card + 15) / 16 <= REG_GROUPS * grid && c.dd / 16 <= grid;
}
