// The depformer of a frame for up to 16 sessions: one persistent cooperative kernel like dep_fused_kernel, with mma.sync fragments instead of tcgen05
// tiles and the weights as one stream per warp (as in gemm_row.cu).  Included by dep_fused.cu behind DepParams.
//
// What bounds a frame here is the chain: 8 sub-steps x 6 layers x 4 products, each of which has to see all of the one before.  So a layer is five
// phases, and a phase is a grid barrier, one L2 round trip for the activations, a few products and one exchange inside the CTA:
//   * a product's rows are dealt to the CTAs in units of 8, whole k each; the sixteen warps of a CTA share the k-blocks and add their sums in shared
//     memory, so no partial sum leaves an SM (dep_fused_kernel exchanges split-K partials through L2 and needs a phase of its own to add them);
//   * every warp asks for its weights with cp.async up to four pairs of units x 64 k ahead, through all products, layers and sub-steps and across the
//     barriers.  (Held in registers they did not fit: 632 to 1268 bytes per thread went through local memory, and a spilled load has to
//     arrive before the thread can go on to the barrier.  Of
//     what is left 12 bytes per thread are spilled for up to 8 sessions, 120 for up to 16.)
//   * a warp has one k-block of the width, so its share of the RMSNorm is what it multiplies: the sums of squares meet in shared memory; residual, gating
//     and bf16 roundings sit in the epilogues; old keys and values of the attention are asked for before the barrier.
//
// A frame with sampling: 1 session 1.48 ms with the weights in registers -> 1.09, 16 sessions 1.98 -> 1.33: 8 x (2 + 5 x 6) = 256 barriers of 3 to 5 us at one
// session (in_proj with its norm 4.9 us, attention 2.9, out_proj 2.9, gated input with its norm 5.1, linear_out 4.0), sampling 15.6 us a sub-step.
//
// A barrier that is not met within ten seconds ends the kernel; the frame's remaining tokens are then the frame's before.  It raises ERR_WAIT, and a
// word on the host that the handle's next call looks at without a synchronisation.
#pragma once

constexpr int REG_B = 16;                    // sessions at most
constexpr int REG_THREADS = 512, REG_WARPS = 16;
constexpr int REG_SLOTS = 4;                 // pairs of units under way per warp
constexpr int REG_KC = 3;                    // k-blocks of a warp at most: F <= 3072; of the width one
constexpr int REG_SUBS = 8;                  // 8-row pieces (gate and value rows apart) of a product per CTA at most
constexpr int REG_UNIT = 8, REG_UNIT_BYTES = 1024;
constexpr uint32_t REG_SLOT_BYTES = REG_WARPS * 2 * REG_UNIT_BYTES;
enum { REG_IN = 0, REG_OUT = 1, REG_GATE = 2, REG_LINEAR_OUT = 3, REG_HEAD = 4, REG_KINDS = 5 };

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

// this CTA's share of a product: `units` whole units of 8 rows from `first` on
struct RegPart { int num_kb, gated, first, units; };
__device__ __forceinline__ int reg_subs(const RegPart& p) { return p.units << p.gated; }
__device__ __forceinline__ RegPart reg_part(int num_kb, int gated, int rows) {
  const unsigned n = (rows + REG_UNIT - 1) / REG_UNIT, c = blockIdx.x, ctas = gridDim.x;
  RegPart p;
  p.num_kb = num_kb; p.gated = gated; p.first = (int)(n * c / ctas); p.units = (int)(n * (c + 1) / ctas) - p.first;
  return p;
}

// The stream of one warp through the frame: weights w[0 .. n) in the order of use, `per` to a sub-step (four a layer, then the head); a slot holds a pair of
// 8-row pieces of one k-block.
struct RegStream {
  const RegPart* parts; const uint8_t* const* w;
  int n, per;
  uint32_t ring, slot = 0;
  int at = -1, pos = -1, sub = 0, subs = 0, j = 0, nj = 0, first = 0, gated = 0;
  uint32_t tile_bytes = 0;
  const uint8_t* base = nullptr;                 // the next k-block asked for (null: none left)

  __device__ __forceinline__ void open() {       // the next product of which this warp has something
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
    do {
      if (++at >= n) { base = nullptr; return; }
      if (++pos == per) pos = 0;
      const RegPart& p = parts[pos == per - 1 ? REG_HEAD : (pos & 3)];
      gated = p.gated; first = p.first;
      subs = reg_subs(p);
      nj = (p.num_kb - warp + REG_WARPS - 1) / REG_WARPS;
      tile_bytes = (uint32_t)p.num_kb << (14 + gated);
    } while (subs <= 0 || nj <= 0);
    base = w[at] + (size_t)(first >> 4) * tile_bytes + ((uint32_t)(warp * TILE_BYTES) << gated) + lane * 16;
    first &= 15;
    sub = 0; j = 0;
  }
  __device__ __forceinline__ void ask(uint32_t to_slot) {
    if (base) {
      const uint32_t step = (uint32_t)(REG_WARPS * TILE_BYTES) << gated, to = ring + to_slot + (threadIdx.x & 31) * 16;
      const int u0 = first + (sub >> gated), u1 = u0 + 1;
      const uint8_t* s = base + ((u0 >> 4) * tile_bytes + (u0 & 15) * REG_UNIT_BYTES);
      rows::copy16(to, s);
      rows::copy16(to + 512, s + 512);
      if (sub + 1 < subs) {
        s = gated ? s + TILE_BYTES : base + ((u1 >> 4) * tile_bytes + (u1 & 15) * REG_UNIT_BYTES);
        rows::copy16(to + 1024, s);
        rows::copy16(to + 1536, s + 512);
      }
      base += step;
      if (++j == nj) {
        j = 0;
        sub += 2;
        if (sub < subs) base -= (uint32_t)nj * step;
        else open();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // the next pair of 8 rows x 64 k: pieces t and t + 4 of row rows::row_of(g) of either
  __device__ __forceinline__ void take(uint4 (&a)[2], uint4 (&b)[2]) {
    const int lane = threadIdx.x & 31, r = rows::row_of(lane >> 2);
    const uint32_t row = ring + slot + r * 128, c = (uint32_t)((lane & 3) ^ r) << 4;
    asm volatile("cp.async.wait_group %0;" ::"n"(REG_SLOTS - 1) : "memory");
    __syncwarp();
    a[0] = rows::lds16(row + c); a[1] = rows::lds16(row + (c ^ 64));
    b[0] = rows::lds16(row + 1024 + c); b[1] = rows::lds16(row + 1024 + (c ^ 64));
    __syncwarp();
    ask(slot);
    slot = slot + REG_SLOT_BYTES == REG_SLOTS * REG_SLOT_BYTES ? 0u : slot + REG_SLOT_BYTES;
  }
};

// This warp's sums of a product -> red[(warp * subs + sub) * B + session][8 rows].  The activations x[B][K] are B fragments: pieces t and t + 4 of a k-block
// of sessions g (and 8 + g).  normed: RMSNorm with alpha (this warp's pieces of it) on the way; all threads meet once for it.  The second sub of a
// last odd pair is whatever its slot held before; its sums are not stored.
template <int NT>
__device__ __forceinline__ void reg_product(RegStream& st, const RegPart& p, const bf16* x, int K, int B, bool normed, const uint4 (&alpha)[2], float (*s_sq)[REG_WARPS], float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int subs = reg_subs(p), num_kb = p.num_kb;
  uint4 xb[REG_KC][NT][2];
#pragma unroll
  for (int i = 0; i < REG_KC; ++i)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = (warp + i * REG_WARPS) * 64 + h * 32 + t * 8;
        xb[i][n][h] = 8 * n + g < B && k < K ? __ldcg(reinterpret_cast<const uint4*>(x + (long long)(8 * n + g) * K + k)) : make_uint4(0u, 0u, 0u, 0u);
      }
  if (normed) {                                  // one k-block per warp
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float q = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&xb[0][n][h]);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(v[e]); q += f.x * f.x + f.y * f.y; }
      }
      q += __shfl_xor_sync(0xffffffffu, q, 1);
      q += __shfl_xor_sync(0xffffffffu, q, 2);
      if (t == 0) s_sq[8 * n + g][warp] = q;
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float q = 0.f;
#pragma unroll
      for (int w = 0; w < REG_WARPS; w += 4) {
        const float4 v = *reinterpret_cast<const float4*>(&s_sq[8 * n + g][w]);
        q += v.x; q += v.y; q += v.z; q += v.w;
      }
      const float rs = rsqrtf(1e-8f + q / (float)K);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        __nv_bfloat162* v = reinterpret_cast<__nv_bfloat162*>(&xb[0][n][h]);
        const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&alpha[h]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(v[e]), r = __bfloat1622float2(a[e]);
          v[e] = __floats2bfloat162_rn(f.x * (r.x * rs), f.y * (r.y * rs));
        }
      }
    }
  }
  float* mine = red + ((warp * subs) * B + 2 * t) * 8 + rows::row_of(g);
#pragma unroll 1
  for (int sub = 0; sub < subs; sub += 2) {
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
    for (int i = 0; i < REG_KC; ++i) {
      if (warp + i * REG_WARPS >= num_kb) break;
      uint4 a[2], b[2];
      st.take(a, b);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          rows::mma_step(acc[n], a[h].x, b[h].x, a[h].y, b[h].y, xb[i][n][h].x, xb[i][n][h].y);
          rows::mma_step(acc[n], a[h].z, b[h].z, a[h].w, b[h].w, xb[i][n][h].z, xb[i][n][h].w);
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (8 * n + 2 * t + (e & 1) < B && sub + (e >> 1) < subs) mine[((sub + (e >> 1)) * B + 8 * n + (e & 1)) * 8] = acc[n][e];
  }
  __syncthreads();
}
// the warps' sums in warp order
__device__ __forceinline__ float reg_total(const float* red, int subs, int B, int sub, int m, int row) {
  float v = 0.f;
#pragma unroll
  for (int w = 0; w < REG_WARPS; ++w) v += red[((w * subs + sub) * B + m) * 8 + row];
  return v;
}

template <int NT, bool DIAG>
__global__ void __launch_bounds__(REG_THREADS, 1) dep_reg_kernel(const DepParams p, bf16* qkv) {
  extern __shared__ __align__(16) uint8_t reg_smem[];
  __shared__ int ok;
  __shared__ RegPart parts[REG_KINDS];
  __shared__ __align__(16) float s_sq[8 * NT][REG_WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = lane & 3, B = p.B, dd = p.dd;
  const int per = 4 * p.L + 1, n_w = p.dep_q * per;
  const uint8_t** weights = reinterpret_cast<const uint8_t**>(reg_smem + REG_SLOTS * REG_SLOT_BYTES);
  float* red = reinterpret_cast<float*>(reg_smem + REG_SLOTS * REG_SLOT_BYTES + ((size_t)n_w * 8 + 15) / 16 * 16);
  for (int i = tid; i < n_w; i += REG_THREADS) {
    const int k = i / per, r = i - k * per;
    const DepLayerW* lw = p.w + k * p.L + (r >> 2);
    weights[i] = r == per - 1 ? p.heads[k] : (r & 3) == REG_IN ? lw->in_w : (r & 3) == REG_OUT ? lw->out_w : (r & 3) == REG_GATE ? lw->lin_in : lw->lin_out;
  }
  if (tid == 0) {
    ok = 1;
    const int kd = dd / 64, kf = (p.F + 63) / 64;
    parts[REG_IN] = reg_part(kd, 0, 3 * dd);
    parts[REG_OUT] = reg_part(kd, 0, dd);
    parts[REG_GATE] = reg_part(kd, 1, p.F);
    parts[REG_LINEAR_OUT] = reg_part(kf, 0, dd);
    parts[REG_HEAD] = reg_part(kd, 0, p.card);
  }
  __syncthreads();
  RegStream st;
  st.parts = parts; st.w = weights; st.n = n_w; st.per = per; st.ring = smem_u32(reg_smem) + warp * 2 * REG_UNIT_BYTES;
  st.open();
#pragma unroll 1
  for (int s = 0; s < REG_SLOTS; ++s) st.ask((uint32_t)s * REG_SLOT_BYTES);
  unsigned epoch = 0;
  if (DIAG && p.trace != nullptr && blockIdx.x == 0 && tid == 0) p.trace[0] = global_timer_ns();
  uint4 alpha[2];
  auto norm_of = [&](const bf16* a) {            // this warp's pieces of a norm, before the barrier in front of its product
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = warp * 64 + h * 32 + t * 8;
      alpha[h] = k < dd ? __ldg(reinterpret_cast<const uint4*>(a + k)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  for (int k = 0; k < p.dep_q; ++k) {
    input_rows<REG_THREADS>(p, k);
    norm_of(p.n1[0]);
    if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
#pragma unroll 1
    for (int i = 0; i < per; ++i) {
      const int kind = i == per - 1 ? REG_HEAD : (i & 3), l = i >> 2;
      const RegPart& a = parts[kind];
      const int rows = a.units * REG_UNIT, row0 = a.first * REG_UNIT;
      const bool adds = kind == REG_OUT || kind == REG_LINEAR_OUT;
      const int m0 = rows > 0 ? tid / rows : 0, r0 = tid - m0 * rows;      // this thread's first result
      unsigned short old = 0;
      if (adds && tid < rows * B) old = __ldcg(reinterpret_cast<const unsigned short*>(p.x + (long long)m0 * dd + row0 + r0));
      // depformer_norms is Identity (lm.py:197-198): the head reads x itself
      reg_product<NT>(st, a, kind == REG_OUT ? p.ao : kind == REG_LINEAR_OUT ? p.hbuf : p.x, kind == REG_LINEAR_OUT ? p.F : dd, B, kind == REG_IN || kind == REG_GATE, alpha, s_sq, red);
      for (int o = tid; o < rows * B; o += REG_THREADS) {
        const int m = o / rows, r = o - m * rows, n = row0 + r;
        if (kind == REG_GATE) {                  // gating.py:18-20
          const float g = rbf(reg_total(red, 2 * a.units, B, 2 * (r >> 3), m, r & 7)), u = rbf(reg_total(red, 2 * a.units, B, 2 * (r >> 3) + 1, m, r & 7));
          if (n < p.F) p.hbuf[(long long)m * p.F + n] = f2bf(rbf(g / (1.f + expf(-g))) * u);
          continue;
        }
        const float v = reg_total(red, a.units, B, r >> 3, m, r & 7);
        if (kind == REG_IN) qkv[(long long)m * 3 * dd + n] = f2bf(v);
        else if (kind == REG_HEAD) {
          if (n < p.card) p.logits[((long long)k * B + m) * p.card + n] = f2bf(v);
        } else {                                 // x_orig + update, both bf16 (transformer.py:769,777)
          bf16* x = p.x + (long long)m * dd + n;
          if (o != tid) old = __ldcg(reinterpret_cast<const unsigned short*>(x));
          *x = f2bf(__bfloat162float(__ushort_as_bfloat16(old)) + rbf(v));
        }
      }
      if (kind == REG_IN) {
        // KV append and attention over k + 1 keys, one warp per (session, head); a lane reads back only what it wrote itself, so before the barrier
        const int C = dd, it = blockIdx.x + warp * gridDim.x, b = it / p.H, h = it - b * p.H;
        const bool some = it < B * p.H;
        unsigned ko[lm::DEP_MAX_Q], vo[lm::DEP_MAX_Q];
        unsigned *kc = nullptr, *vc = nullptr;
        if (some) {
          kc = reinterpret_cast<unsigned*>(p.kc[l] + (long long)it * p.dep_q * DD) + lane;
          vc = reinterpret_cast<unsigned*>(p.vc[l] + (long long)it * p.dep_q * DD) + lane;
#pragma unroll
          for (int j = 0; j < lm::DEP_MAX_Q; ++j)
            if (j < k) { ko[j] = kc[j * (DD / 2)]; vo[j] = vc[j * (DD / 2)]; }
        }
        if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
        if (some) {
          const unsigned* src = reinterpret_cast<const unsigned*>(qkv + (long long)b * 3 * C + h * DD) + lane;
          const unsigned qw = __ldcg(src), kw = __ldcg(src + C / 2), vw = __ldcg(src + C);
          kc[k * (DD / 2)] = kw;
          vc[k * (DD / 2)] = vw;
          const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qw));
          float sc[lm::DEP_MAX_Q], mx = -INFINITY, sum = 0.f;
#pragma unroll
          for (int j = 0; j < lm::DEP_MAX_Q; ++j) {
            if (j <= k) {
              const unsigned w = j == k ? kw : ko[j];
              const float2 kv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
              sc[j] = warp_sum(q.x * kv.x + q.y * kv.y) * 0.125f;
              mx = fmaxf(mx, sc[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < lm::DEP_MAX_Q; ++j)
            if (j <= k) { sc[j] = expf(sc[j] - mx); sum += sc[j]; }
          const float inv = 1.f / sum;
          float a0 = 0.f, a1 = 0.f;
#pragma unroll
          for (int j = 0; j < lm::DEP_MAX_Q; ++j) {
            if (j <= k) {
              const unsigned w = j == k ? vw : vo[j];
              const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
              a0 = fmaf(sc[j] * inv, v.x, a0);
              a1 = fmaf(sc[j] * inv, v.y, a1);
            }
          }
          *reinterpret_cast<__nv_bfloat162*>(p.ao + (long long)b * C + h * DD + 2 * lane) = __floats2bfloat162_rn(a0, a1);
        }
      }
      if (kind == REG_OUT) norm_of(p.n2[l]);
      else if (kind == REG_LINEAR_OUT && l + 1 < p.L) norm_of(p.n1[l + 1]);
      if (!reg_grid_sync<DIAG>(p, epoch, &ok)) break;
    }
    if (!ok) break;
    for (int m = blockIdx.x; m < B; m += gridDim.x) {      // the next sub-step's input rows are the same rows of the same CTA
      lm::sample_row<REG_THREADS>(p.logits + ((long long)k * B + m) * p.card, p.noise + (long long)m * p.noise_ld + p.noise_off + (long long)k * p.ka,
                                  p.audio_tokens + (long long)k * B + m, p.card, p.use_sampling, p.temp, p.top_k);
      __syncthreads();
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (tid == 0 && !ok) {
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
// 8-row pieces of the fullest CTA in the largest product
inline int dep_reg_subs(const DepFusedConfig& c, int grid) {
  auto per_cta = [&](int rows) { return ((rows + REG_UNIT - 1) / REG_UNIT + grid - 1) / grid; };
  return std::max(std::max(per_cta(3 * c.dd), 2 * per_cta(c.F)), per_cta(c.card));
}
inline size_t dep_reg_smem(const DepFusedConfig& c, int grid) {
  return (size_t)REG_SLOTS * REG_SLOT_BYTES + ((size_t)c.dep_q * (4 * c.L + 1) * 8 + 15) / 16 * 16 + (size_t)REG_WARPS * dep_reg_subs(c, grid) * c.B * REG_UNIT * 4;
}
inline bool dep_reg_takes(const DepFusedConfig& c, int grid) {
  return c.B <= REG_B && c.dd % 64 == 0 && c.dd <= REG_WARPS * 64 && c.F % 8 == 0 && c.F <= REG_KC * REG_WARPS * 64 && grid >= 1 && dep_reg_subs(c, grid) <= REG_SUBS &&
         c.B * (c.dd / DD) <= REG_WARPS * grid && dep_reg_smem(c, grid) <= SMEM_LIMIT;
}
