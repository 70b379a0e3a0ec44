// The depformer of a frame for up to 16 sessions: one persistent cooperative kernel like dep_fused_kernel, with mma.sync fragments instead of tcgen05
// tiles and the weights as one stream per warp (as in gemm_row.cu).  Included by dep_fused.cu behind DepParams.
//
// What bounds a frame here is the chain: 8 sub-steps x 6 layers x 4 products, each of which has to see all of the one before.  So a layer is five
// phases, and a phase is an exchange with all CTAs, a few products and one exchange inside the CTA:
//   * a product's rows are dealt to the CTAs in units of 8, whole k each; the sixteen warps of a CTA share the k-blocks and add their sums in shared
//     memory, so no partial sum leaves an SM (dep_fused_kernel exchanges split-K partials through L2 and needs a phase of its own to add them);
//   * up to 8 sessions there is no barrier: what a step writes carries the step's number word by word (reg_put), and who needs it asks for just that until it is there.  A
//     buffer is written again only by a CTA that has seen results for which its last readers had to be done (x: of the products that read it; qkv: of the attention; ao and h:
//     of the products behind them), so nothing is overwritten that somebody still reads.  Above 8 sessions twice the bytes from L2 into every SM cost more than the barrier
//     (16 sessions: 4.6 ms a step of the 7B instead of 4.4), which stays there in front of the products; the attention, a warp of which reads one head, takes words;
//   * every warp asks for its weights up to four pairs of units x 64 k ahead, through all products, layers and sub-steps and across the exchanges, by bulk copies from a list
//     that is made once: the addresses worked out on the way and four 16-byte copies per lane took 0.4 us of a pair's 0.7;
//   * a warp has one k-block of the width, so its share of the RMSNorm is what it multiplies: the sums of squares meet in shared memory; residual, gating
//     and bf16 roundings sit in the epilogues; old keys and values of the attention are asked for before the wait, its scores are summed over the lanes side by side;
//   * the activations of a k-block are in registers while the next ones are under way, and the attention keeps as many keys as there are sub-steps (8, or up to 16): with all
//     k-blocks and 16 keys the kernel spilled.
//
// A step of the 7B with sampling (all but the depformer unchanged), ms, barriers and 16-byte copies / so: 1 session 3.59 / 3.32, 2 3.64 / 3.44, 8 3.83 / 3.61, 9 4.08 / 3.99, 16 4.43 /
// 4.29.  Words that straddle lines (a buffer that begins off a border of 128 bytes) cost 0.3 ms of it.  Of a layer's 15 us at one session the waits for other CTAs' words are about 5,
// norms 1.6, products 6, the rest sums and epilogues.
//
// Whoever waits for ten seconds in vain stops waiting; the CTA agrees on it at the end of a product, ends, and so do the others.  The frame's remaining tokens are then the
// frame's before.  It raises ERR_WAIT, and a word on the host that the handle's next call looks at without a synchronisation.
#pragma once

constexpr int REG_B = 16;                    // sessions at most
constexpr int REG_THREADS = 512, REG_WARPS = 16;
constexpr int REG_SLOTS = 4;                 // pairs of units under way per warp
constexpr int REG_KC = 3;                    // k-blocks of a warp at most: F <= 3072; of the width one
constexpr int REG_SUBS = 8;                  // 8-row pieces (gate and value rows apart) of a product per CTA at most
constexpr int REG_UNIT = 8, REG_UNIT_BYTES = 1024;
constexpr uint32_t REG_SLOT_BYTES = REG_WARPS * 2 * REG_UNIT_BYTES;
enum { REG_IN = 0, REG_OUT = 1, REG_GATE = 2, REG_LINEAR_OUT = 3, REG_HEAD = 4, REG_KINDS = 5 };

// What passes from CTA to CTA goes as words of 8 bytes, two bf16 and the number of the step that wrote them, written and read whole: a reader asks for its words until their
// numbers are the step's, and what it has then is the data.
constexpr int REG_WORD = 8;
struct RegWords {                                // [session][pair of elements] of what a frame's steps pass on, zero at launch; above 8 sessions pairs without a number but for qkv
  uint64_t *qkv, *meet, *x, *ao, *h, *logits;    // one allocation; meet: the barrier's count, in a line of its own
  const uint8_t* const* w;                       // addresses of the frame's weights, four a layer and the head, sub-step after sub-step (null: they lie in shared memory)
};
template <int NT>
__device__ __forceinline__ void reg_put(uint64_t* base, long long i, unsigned pair, unsigned step) {
  if constexpr (NT > 1) reinterpret_cast<unsigned*>(base)[i] = pair;
  else asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(base + i), "l"((uint64_t)step << 32 | pair) : "memory");
}
__device__ __forceinline__ void reg_get2(const uint64_t* at, uint64_t& a, uint64_t& b) {      // two words; `at` on a border of 16 bytes
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(at) : "memory");
}
__device__ __forceinline__ uint64_t reg_get(const uint64_t* at) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(at) : "memory");
  return v;
}
__device__ __forceinline__ bool reg_new(uint64_t word, unsigned step) { return (unsigned)(word >> 32) == step; }
__device__ __forceinline__ unsigned reg_pair(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&v);
}
// A thread's patience over the frame.  Once it has run out, nothing is waited for any more; the CTA agrees on it at the end of a product and leaves.  DIAG: a limit of the
// caller's, in a kernel of its own.
template <bool DIAG>
struct RegWait {
  unsigned spins = 0;
  uint64_t since = 0;
  bool lost = false;
  __device__ __forceinline__ void begin() { since = 0; }
  __device__ __forceinline__ bool again(const DepParams& p) {      // one more look? no: lost
    if (lost) return false;
    if ((++spins & (DIAG ? p.wait_mask : 4095u)) == 0u) {
      const uint64_t now = global_timer_ns();
      if (since == 0) since = now;
      else if (now - since > (DIAG ? p.wait_ns : WAIT_LIMIT_NS)) { lost = true; return false; }
    }
    return true;
  }
};

// above 8 sessions: all CTAs meet; false: not within the limit
template <bool DIAG>
__device__ __forceinline__ bool reg_grid_sync(const DepParams& p, const RegWords& io, unsigned& meets, int* ok) {
  meets += 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = meets * gridDim.x;
    unsigned* const count = reinterpret_cast<unsigned*>(io.meet);
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    RegWait<DIAG> wait;
    int met = 1;
    while (ld_acquire(count) < target)
      if (!wait.again(p)) { met = 0; break; }
    *ok = met;
  }
  __syncthreads();
  return *ok != 0;
}

__device__ __forceinline__ bool mbar_passed(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}

// one pair that a step wrote
template <int NT, bool DIAG>
__device__ __forceinline__ unsigned reg_take(const DepParams& p, RegWait<DIAG>& wait, const uint64_t* base, long long i, unsigned step) {
  if constexpr (NT > 1) return __ldcg(reinterpret_cast<const unsigned*>(base) + i);
  wait.begin();
  uint64_t w;
  do w = reg_get(base + i);
  while (!reg_new(w, step) && wait.again(p));
  return (unsigned)w;
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

// What a warp asks for in a layer, and for the head behind the last one: made once, for working it out on the way cost 0.3 us of every 1 (16 warps, each a chain of some eighty
// instructions).  A pair of 8-row pieces of one k-block, each 1024 bytes on end in memory and so one bulk copy (two that are neighbours: one together).
struct RegAsk { uint32_t at0, at1, bytes0, bytes1_kind; };      // offsets in the product's weights; bytes of the second copy (0: none) << 4 | product
constexpr int REG_ASKS = 64;                     // 5 products of at most REG_SUBS / 2 pairs and REG_KC k-blocks
static_assert(REG_KINDS * (REG_SUBS / 2) * REG_KC <= REG_ASKS, "a warp's list");

// The stream of one warp through the frame, in the order of use.  All of it is the same for the whole warp.
struct RegStream {
  const uint8_t* const* w;                       // weights of the sub-step's products: four a layer, then the head
  const RegAsk* asks;
  int layer_n, n, L, per, steps;                 // asks of a layer, and with the head's; sub-steps that are left
  uint32_t ring, bars, slot = 0, phases = 0, asked = 0;      // this warp's slots and their mbarriers; bit s: the phase slot s completes next, and whether it is under way
  int next = 0, layer = 0;

  // this warp's list (one thread)
  __device__ __forceinline__ static int list(const RegPart* parts, int warp, RegAsk* to, int* layer_n) {
    int n = 0;
#pragma unroll 1
    for (int kind = 0; kind < REG_KINDS; ++kind) {
      if (kind == REG_HEAD) *layer_n = n;
      const RegPart& p = parts[kind];
      const int subs = reg_subs(p), nj = (p.num_kb - warp + REG_WARPS - 1) / REG_WARPS;
      const uint32_t tile_bytes = (uint32_t)p.num_kb << (14 + p.gated);
#pragma unroll 1
      for (int sub = 0; sub < subs; sub += 2)
#pragma unroll 1
        for (int j = 0; j < nj; ++j) {
          const uint32_t kb = (uint32_t)((warp + j * REG_WARPS) * TILE_BYTES) << p.gated;
          const int u0 = p.first + (sub >> p.gated), u1 = u0 + 1;
          RegAsk a;
          a.at0 = kb + (uint32_t)(u0 >> 4) * tile_bytes + (u0 & 15) * REG_UNIT_BYTES;
          a.at1 = p.gated ? a.at0 + TILE_BYTES : kb + (uint32_t)(u1 >> 4) * tile_bytes + (u1 & 15) * REG_UNIT_BYTES;
          a.bytes0 = REG_UNIT_BYTES;
          uint32_t second = sub + 1 < subs ? REG_UNIT_BYTES : 0;
          if (second && a.at1 == a.at0 + REG_UNIT_BYTES) { a.bytes0 = 2 * REG_UNIT_BYTES; second = 0; }
          a.bytes1_kind = second << 4 | kind;
          to[n++] = a;
        }
    }
    return n;
  }
  __device__ __forceinline__ void open() {       // a sub-step's first
    next = 0;
    layer = layer_n > 0 ? 0 : L - 1;
  }
  __device__ __forceinline__ void ask(uint32_t s) {
    if (steps == 0) return;
    const uint4 a = *reinterpret_cast<const uint4*>(asks + next);
    const uint8_t* base = w[4 * layer + (a.w & 15)];
    if (elected()) {
      const uint32_t bar = bars + 8 * s, to = ring + s * REG_SLOT_BYTES;
      mbar_expect_tx(bar, a.z + (a.w >> 4));
      bulk_load(to, base + a.x, a.z, bar);
      if (a.w >> 4) bulk_load(to + REG_UNIT_BYTES, base + a.y, a.w >> 4, bar);
    }
    __syncwarp();
    asked |= 1u << s;
    ++next;
    if (next == layer_n && layer + 1 < L) { next = 0; ++layer; }
    if (next == n) { w += per; --steps; open(); }
  }
  // slot s has arrived (whole warps; false: not in time)
  template <bool DIAG>
  __device__ __forceinline__ bool arrived(uint32_t s, const DepParams& dep, RegWait<DIAG>& wait) {
    wait.begin();
    while (!__all_sync(0xffffffffu, mbar_passed(bars + 8 * s, (phases >> s) & 1u)))
      if (!__any_sync(0xffffffffu, wait.again(dep))) return false;
    phases ^= 1u << s;
    asked &= ~(1u << s);
    return true;
  }
  // the next pair of 8 rows x 64 k: pieces t and t + 4 of row rows::row_of(g) of either
  template <bool DIAG>
  __device__ __forceinline__ void take(uint4 (&a)[2], uint4 (&b)[2], const DepParams& dep, RegWait<DIAG>& wait) {
    const int lane = threadIdx.x & 31, r = rows::row_of(lane >> 2);
    const uint32_t row = ring + slot * REG_SLOT_BYTES + r * 128, c = (uint32_t)((lane & 3) ^ r) << 4;
    const bool here = arrived<DIAG>(slot, dep, wait);
    a[0] = rows::lds16(row + c); a[1] = rows::lds16(row + (c ^ 64));
    b[0] = rows::lds16(row + 1024 + c); b[1] = rows::lds16(row + 1024 + (c ^ 64));
    __syncwarp();
    if (here) ask(slot);
    slot = (slot + 1) % REG_SLOTS;
  }
  // no copy is under way when the kernel ends
  __device__ __forceinline__ void drain() {
#pragma unroll 1
    for (uint32_t s = 0; s < REG_SLOTS; ++s)
      if (asked >> s & 1u) {
        const uint64_t from = global_timer_ns();
        while (!mbar_passed(bars + 8 * s, (phases >> s) & 1u) && global_timer_ns() - from < WAIT_LIMIT_NS) { }
      }
  }
};

__device__ __forceinline__ void reg_stamp(const DepParams& p, unsigned step) {      // CTA 0 has what it needs of a step
  if (p.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0 && step < (unsigned)DEP_TRACE_SLOTS) p.trace[step] = global_timer_ns();
}
// This warp's sums of a product -> red[(warp * pairs of subs + sub)][8 rows][sessions, and two more against bank conflicts].  The activations x[B][K], written by `step`, are B fragments: pieces t and t + 4 of a k-block
// of sessions g (and 8 + g).  normed: RMSNorm with alpha (this warp's pieces of it) on the way.  All threads meet at least twice: the sums of the product before have been
// added up by then.  The second sub of a last odd pair is whatever its slot held before; its sums are not stored.  false: something was waited for in vain.
template <int NT, bool DIAG>
__device__ __forceinline__ bool reg_product(RegStream& st, const RegPart& p, const DepParams& dep, RegWait<DIAG>& wait, const uint64_t* x, unsigned step, int K, int B, bool normed,
                                            const uint4 (&alpha)[2], float (*s_sq)[REG_WARPS], float* red, const RegWords& io, unsigned& meets, int* met) {
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int subs = reg_subs(p), nk = (p.num_kb - warp + REG_WARPS - 1) / REG_WARPS;
  uint4 xb[NT][2];                               // of one k-block; the next one is asked for meanwhile
  auto src = [&](int i, int n, int h) {          // pair of elements that a piece begins with, -1: none
    const int k = (warp + i * REG_WARPS) * 64 + h * 32 + t * 8;
    return subs > 0 && 8 * n + g < B && k < K ? ((8 * n + g) * K + k) >> 1 : -1;
  };
  uint64_t v[NT][2][NT == 1 ? 4 : 2];
  auto request = [&](int i) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int at = src(i, n, h);
        uint64_t* w = v[n][h];
        if constexpr (NT == 1) {
          if (at >= 0) {
            reg_get2(x + at, w[0], w[1]);
            reg_get2(x + at + 2, w[2], w[3]);
          } else {
            w[0] = w[1] = w[2] = w[3] = (uint64_t)step << 32;
          }
        } else {
          w[0] = w[1] = 0;
          if (at >= 0) reg_get2(reinterpret_cast<const uint64_t*>(reinterpret_cast<const unsigned*>(x) + at), w[0], w[1]);
        }
      }
  };
  auto settle = [&](int i) {
    if constexpr (NT == 1) {
      wait.begin();
      while (true) {
        bool missing = false;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < 4; ++e) missing |= !reg_new(v[0][h][e], step);
        if (!missing || !wait.again(dep)) break;
        request(i);
      }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint64_t* w = v[n][h];
        if constexpr (NT == 1) xb[n][h] = make_uint4((unsigned)w[0], (unsigned)w[1], (unsigned)w[2], (unsigned)w[3]);
        else xb[n][h] = make_uint4((unsigned)w[0], (unsigned)(w[0] >> 32), (unsigned)w[1], (unsigned)(w[1] >> 32));
      }
    __syncwarp();
  };
  if (NT > 1 && !reg_grid_sync<DIAG>(dep, io, meets, met)) return false;
  request(0);
  settle(0);
  if (DIAG) reg_stamp(dep, step);
  if (NT == 1 && !normed) __syncthreads();
  if (normed) {                                  // one k-block per warp
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float q = 0.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&xb[n][h]);
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
        __nv_bfloat162* v = reinterpret_cast<__nv_bfloat162*>(&xb[n][h]);
        const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&alpha[h]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(v[e]), r = __bfloat1622float2(a[e]);
          v[e] = __floats2bfloat162_rn(f.x * (r.x * rs), f.y * (r.y * rs));
        }
      }
    }
  }
  float* mine = red + (warp * ((subs + 1) & ~1) * 8 + rows::row_of(g)) * (8 * NT + 2) + 2 * t;
#pragma unroll 1
  for (int sub = 0; sub < subs; sub += 2) {
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll 1
    for (int i = 0; i < nk; ++i) {
      if (i > 0) settle(i);
      else if (sub > 0 && nk > 1) { request(0); settle(0); }
      if (i + 1 < nk) request(i + 1);
      uint4 a[2], b[2];
      st.take<DIAG>(a, b, dep, wait);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          rows::mma_step(acc[n], a[h].x, b[h].x, a[h].y, b[h].y, xb[n][h].x, xb[n][h].y);
          rows::mma_step(acc[n], a[h].z, b[h].z, a[h].w, b[h].w, xb[n][h].z, xb[n][h].w);
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      *reinterpret_cast<float2*>(mine + 8 * n) = make_float2(acc[n][0], acc[n][1]);
      *reinterpret_cast<float2*>(mine + 8 * (8 * NT + 2) + 8 * n) = make_float2(acc[n][2], acc[n][3]);
    }
    mine += 2 * 8 * (8 * NT + 2);
  }
  return __syncthreads_and(!wait.lost);
}
// two rows' sums, the warps' in warp order
template <int NT>
__device__ __forceinline__ float2 reg_total(const float* red, int subs, int sub, int m, int row) {
  constexpr int LD = 8 * NT + 2;
  const int step = ((subs + 1) & ~1) * 8 * LD;
  const float* at = red + (sub * 8 + row) * LD + m;
  float2 v = make_float2(0.f, 0.f);
#pragma unroll
  for (int w = 0; w < REG_WARPS; ++w, at += step) { v.x += at[0]; v.y += at[LD]; }
  return v;
}

// x = depformer_in[k](transformer_out) + emb_k(prev)   (lm.py:475-486; token -1 -> zero row, lm_utils.py:103-121)
template <int NT>
__device__ __forceinline__ void reg_input(const DepParams& p, uint64_t* x, int k, unsigned step) {
  const long long* prev = k == 0 ? p.text_token : p.audio_tokens + (long long)(k - 1) * p.B;
  const bf16* table = p.tables[k];
  for (int m = blockIdx.x; m < p.B; m += gridDim.x) {
    const long long id = prev[m];
    const bool ok = lm::embed_id_ok(id, k == 0 ? p.text_card : p.card, p.err);
    for (int j = threadIdx.x; j < p.dd / 2; j += REG_THREADS) {
      const float2 e = ok ? __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(table + id * p.dd)[j]) : make_float2(0.f, 0.f);
      const float2 d = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(p.din + (long long)m * p.din_ld + (long long)k * p.dd)[j]);
      reg_put<NT>(x, (long long)m * (p.dd / 2) + j, reg_pair(d.x + e.x, d.y + e.y), step);
    }
  }
}

template <int NT, int MQ, bool DIAG, bool FAR>      // MQ: sub-steps at most; FAR: the addresses of the weights are read from memory
__global__ void __launch_bounds__(REG_THREADS, 1) dep_reg_kernel(const DepParams p, const RegWords io) {
  extern __shared__ __align__(128) uint8_t reg_smem[];
  __shared__ int met;
  __shared__ RegPart parts[REG_KINDS];
  __shared__ __align__(16) float s_sq[8 * NT][REG_WARPS];
  __shared__ __align__(8) uint64_t ring_bars[REG_WARPS][REG_SLOTS];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, t = lane & 3, B = p.B, dd = p.dd;
  const int per = 4 * p.L + 1, n_w = FAR ? 0 : p.dep_q * per;
  const uint8_t** weights = reinterpret_cast<const uint8_t**>(reg_smem + REG_SLOTS * REG_SLOT_BYTES + REG_WARPS * REG_ASKS * sizeof(RegAsk));
  float* red = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(weights) + ((size_t)n_w * 8 + 15) / 16 * 16);
  for (int i = tid; i < n_w; i += REG_THREADS) {
    const int k = i / per, r = i - k * per;
    const DepLayerW* lw = p.w + k * p.L + (r >> 2);
    weights[i] = r == per - 1 ? p.heads[k] : (r & 3) == REG_IN ? lw->in_w : (r & 3) == REG_OUT ? lw->out_w : (r & 3) == REG_GATE ? lw->lin_in : lw->lin_out;
  }
  if (tid == 0) {
    const int kd = dd / 64, kf = (p.F + 63) / 64;
    parts[REG_IN] = reg_part(kd, 0, 3 * dd);
    parts[REG_OUT] = reg_part(kd, 0, dd);
    parts[REG_GATE] = reg_part(kd, 1, p.F);
    parts[REG_LINEAR_OUT] = reg_part(kf, 0, dd);
    parts[REG_HEAD] = reg_part(kd, 0, p.card);
  }
  if (lane == 0) {
    for (int s = 0; s < REG_SLOTS; ++s) mbar_init(smem_u32(&ring_bars[warp][s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  RegAsk* const asks = reinterpret_cast<RegAsk*>(reg_smem + REG_SLOTS * REG_SLOT_BYTES) + warp * REG_ASKS;
  int layer_asks = 0, n_asks = 0;
  if (lane == 0) n_asks = RegStream::list(parts, warp, asks, &layer_asks);
  RegStream st;
  st.w = FAR ? io.w : weights; st.asks = asks; st.L = p.L; st.per = per;
  st.layer_n = __shfl_sync(0xffffffffu, layer_asks, 0); st.n = __shfl_sync(0xffffffffu, n_asks, 0); st.steps = st.n > 0 ? p.dep_q : 0;
  st.ring = smem_u32(reg_smem) + warp * 2 * REG_UNIT_BYTES; st.bars = smem_u32(ring_bars[warp]);
  st.open();
#pragma unroll 1
  for (uint32_t s = 0; s < REG_SLOTS; ++s) st.ask(s);
  unsigned meets = 0;                            // barriers so far
  unsigned step = 0;                             // the last step, written or (from its first reader on) waited for
  RegWait<DIAG> wait;
  bool ok = true;
  if (DIAG) reg_stamp(p, 0);
  uint4 alpha[2];
  auto norm_of = [&](const bf16* a) {            // this warp's pieces of a norm, before the barrier in front of its product
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = warp * 64 + h * 32 + t * 8;
      alpha[h] = k < dd ? __ldg(reinterpret_cast<const uint4*>(a + k)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  // a thread's pair of results of the products that add to x: it keeps their sums through the sub-step
  const int x_pairs = parts[REG_OUT].units * (REG_UNIT / 2), xm = x_pairs > 0 ? tid / x_pairs : 0, xn = parts[REG_OUT].first * (REG_UNIT / 2) + tid - xm * x_pairs;
  const bool adds_x = x_pairs > 0 && xm < B;
  const long long my_x = (long long)xm * (dd / 2) + xn;
  unsigned old = 0;
  for (int k = 0; k < p.dep_q; ++k) {
    step += 1;
    reg_input<NT>(p, io.x, k, step);
    norm_of(p.n1[0]);
#pragma unroll 1
    for (int i = 0; i < per; ++i) {
      const int kind = i == per - 1 ? REG_HEAD : (i & 3), l = i >> 2;
      const RegPart& a = parts[kind];
      const int pairs = a.units * (REG_UNIT / 2), pair0 = a.first * (REG_UNIT / 2);
      const int m0 = pairs > 0 ? tid / pairs : 0, n0 = tid - m0 * pairs, dm = pairs > 0 ? REG_THREADS / pairs : 0, dn = REG_THREADS - dm * pairs;
      // depformer_norms is Identity (lm.py:197-198): the head reads x itself
      ok = reg_product<NT, DIAG>(st, a, p, wait, kind == REG_OUT ? io.ao : kind == REG_LINEAR_OUT ? io.h : io.x, step, kind == REG_LINEAR_OUT ? p.F : dd, B,
                                 kind == REG_IN || kind == REG_GATE, alpha, s_sq, red, io, meets, &met);
      if (!ok) break;
      if (i == 0 && adds_x) {                    // the sub-step's input
        old = reg_take<NT, DIAG>(p, wait, io.x, my_x, step);
      }
      step += 1;
      if (kind == REG_OUT || kind == REG_LINEAR_OUT) {      // x_orig + update, both bf16 (transformer.py:769,777); at most one pair a thread
        if (adds_x) {
          const int r = 2 * (xn - pair0);
          const float2 v = reg_total<NT>(red, a.units, r >> 3, xm, r & 7), o = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&old));
          old = reg_pair(o.x + rbf(v.x), o.y + rbf(v.y));
          reg_put<NT>(io.x, my_x, old, step);
        }
      } else {
        int m = m0, c = n0;
#pragma unroll 1
        for (int o = tid; o < pairs * B; o += REG_THREADS, m += dm, c += dn) {
          if (o > tid && c >= pairs) { c -= pairs; ++m; }
          const int r = 2 * c, n = pair0 + c;
          if (kind == REG_GATE) {                // gating.py:18-20
            const float2 g = reg_total<NT>(red, 2 * a.units, 2 * (r >> 3), m, r & 7), u = reg_total<NT>(red, 2 * a.units, 2 * (r >> 3) + 1, m, r & 7);
            const float gx = rbf(g.x), gy = rbf(g.y);
            if (2 * n < p.F) reg_put<NT>(io.h, (long long)m * (p.F / 2) + n, reg_pair(rbf(gx / (1.f + expf(-gx))) * rbf(u.x), rbf(gy / (1.f + expf(-gy))) * rbf(u.y)), step);
            continue;
          }
          const float2 v = reg_total<NT>(red, a.units, r >> 3, m, r & 7);
          const unsigned w = reg_pair(v.x, v.y);
          if (kind == REG_IN) reg_put<1>(io.qkv, (long long)m * (3 * dd / 2) + n, w, step);
          else if (2 * n < p.card) {
            reg_put<NT>(io.logits, (long long)m * ((p.card + 7) / 8 * 4) + n, w, step);
            bf16* to = p.logits + ((long long)k * B + m) * p.card + 2 * n;
            to[0] = __ushort_as_bfloat16((unsigned short)w);
            if (2 * n + 1 < p.card) to[1] = __ushort_as_bfloat16((unsigned short)(w >> 16));
          }
        }
      }
      if (kind == REG_IN) {
        // KV append and attention over k + 1 keys, one warp per (session, head); a lane reads back only what it wrote itself, so before the wait
        const int C = dd, it = blockIdx.x + warp * gridDim.x, b = it / p.H, h = it - b * p.H;
        const bool some = it < B * p.H;
        unsigned ko[MQ], vo[MQ];
        unsigned *kc = nullptr, *vc = nullptr;
        if (some) {
          kc = reinterpret_cast<unsigned*>(p.kc[l] + (long long)it * p.dep_q * DD) + lane;
          vc = reinterpret_cast<unsigned*>(p.vc[l] + (long long)it * p.dep_q * DD) + lane;
#pragma unroll
          for (int j = 0; j < MQ; ++j)
            if (j < k) { ko[j] = kc[j * (DD / 2)]; vo[j] = vc[j * (DD / 2)]; }
        }
        if (some) {
          const long long src = (long long)b * (3 * C / 2) + h * (DD / 2) + lane;
          uint64_t w[3];
          wait.begin();
          do {
#pragma unroll
            for (int j = 0; j < 3; ++j) w[j] = reg_get(io.qkv + src + j * (C / 2));
          } while (!(reg_new(w[0], step) && reg_new(w[1], step) && reg_new(w[2], step)) && wait.again(p));
          __syncwarp();
          const unsigned qw = (unsigned)w[0], kw = (unsigned)w[1], vw = (unsigned)w[2];
          kc[k * (DD / 2)] = kw;
          vc[k * (DD / 2)] = vw;
          const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qw));
          // all keys' sums over the lanes side by side (one key after the other: 0.13 us each)
          float sc[MQ], mx = -INFINITY, sum = 0.f;
#pragma unroll
          for (int j = 0; j < MQ; ++j) {
            const unsigned w = j < k ? ko[j] : kw;
            const float2 kv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
            sc[j] = q.x * kv.x + q.y * kv.y;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < MQ; ++j) sc[j] += __shfl_xor_sync(0xffffffffu, sc[j], o);
#pragma unroll
          for (int j = 0; j < MQ; ++j)
            if (j <= k) {
              sc[j] *= 0.125f;
              mx = fmaxf(mx, sc[j]);
            }
#pragma unroll
          for (int j = 0; j < MQ; ++j)
            if (j <= k) { sc[j] = expf(sc[j] - mx); sum += sc[j]; }
          const float inv = 1.f / sum;
          float a0 = 0.f, a1 = 0.f;
#pragma unroll
          for (int j = 0; j < MQ; ++j) {
            if (j <= k) {
              const unsigned w = j == k ? vw : vo[j];
              const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
              a0 = fmaf(sc[j] * inv, v.x, a0);
              a1 = fmaf(sc[j] * inv, v.y, a1);
            }
          }
          reg_put<NT>(io.ao, (long long)b * (C / 2) + h * (DD / 2) + lane, reg_pair(a0, a1), step + 1);
        }
        if (DIAG) reg_stamp(p, step);
        step += 1;
      }
      if (kind == REG_OUT) norm_of(p.n2[l]);
      else if (kind == REG_LINEAR_OUT && l + 1 < p.L) norm_of(p.n1[l + 1]);
    }
    if (!ok) break;
    if (NT > 1 && !(ok = reg_grid_sync<DIAG>(p, io, meets, &met))) break;
    if (NT == 1) __syncthreads();                // red has been read: the row of logits goes there
    for (int m = blockIdx.x; m < B; m += gridDim.x) {      // the next sub-step's input rows are the same rows of the same CTA
      unsigned* row = reinterpret_cast<unsigned*>(red);
      for (int o = tid; o < (p.card + 1) / 2; o += REG_THREADS) row[o] = reg_take<NT, DIAG>(p, wait, io.logits, (long long)m * ((p.card + 7) / 8 * 4) + o, step);
      ok = __syncthreads_and(!wait.lost);
      if (!ok) break;
      lm::sample_row<REG_THREADS>(reinterpret_cast<const bf16*>(row), p.noise + (long long)m * p.noise_ld + p.noise_off + (long long)k * p.ka,
                                  p.audio_tokens + (long long)k * B + m, p.card, p.use_sampling, p.temp, p.top_k);
      __syncthreads();
    }
    if (DIAG) reg_stamp(p, step);
    if (!ok) break;
  }
  st.drain();
  if (tid == 0 && !ok) {
    if (p.err) atomicOr(p.err, lm::ERR_WAIT);
    if (p.gave_up) {
      *p.gave_up = 1;
      __threadfence_system();
    }
  }
}

typedef void (*DepRegKernel)(const DepParams, const RegWords);
template <int NT, int MQ, bool FAR> inline DepRegKernel dep_reg_pick(bool diag) { return diag ? dep_reg_kernel<NT, MQ, true, FAR> : dep_reg_kernel<NT, MQ, false, FAR>; }
inline DepRegKernel dep_reg_pick(int sessions, int steps, bool diag, bool far) {
  if (far) return sessions <= 8 ? dep_reg_pick<1, lm::DEP_MAX_Q, true>(diag) : dep_reg_pick<2, lm::DEP_MAX_Q, true>(diag);
  if (sessions <= 8) return steps <= 8 ? dep_reg_pick<1, 8, false>(diag) : dep_reg_pick<1, lm::DEP_MAX_Q, false>(diag);
  return steps <= 8 ? dep_reg_pick<2, 8, false>(diag) : dep_reg_pick<2, lm::DEP_MAX_Q, false>(diag);
}
// 8-row pieces of the fullest CTA in the largest product
inline int dep_reg_subs(const DepFusedConfig& c, int grid) {
  auto per_cta = [&](int rows) { return ((rows + REG_UNIT - 1) / REG_UNIT + grid - 1) / grid; };
  return std::max(std::max(per_cta(3 * c.dd), 2 * per_cta(c.F)), per_cta(c.card));
}
inline size_t dep_reg_addresses(const DepFusedConfig& c) { return ((size_t)c.dep_q * (4 * c.L + 1) * 8 + 15) / 16 * 16; }      // of the frame's weights, bytes
// Shared memory: the ring, the lists of what is asked for, the sums (or a row of logits in their place) and, where there is room, the addresses.  far: there is none, and a kernel of its
// own reads them from memory (both in one kernel: 20 us more for a step of the 7B with one session).  16 sub-steps of 140 layers of width 64, ms: 1 session 24.1, as a chain of launches
// 29.1; 8 sessions 23.7, dep_fused_kernel 53.2; 16 36.9, 54.7.
inline size_t dep_reg_smem(const DepFusedConfig& c, int grid, bool* far) {
  const size_t sums = (size_t)REG_WARPS * ((dep_reg_subs(c, grid) + 1) & ~1) * REG_UNIT * (c.B <= 8 ? 10 : 18) * 4, logits = ((size_t)c.card + 1) / 2 * 4;
  const size_t rest = (size_t)REG_SLOTS * REG_SLOT_BYTES + REG_WARPS * REG_ASKS * sizeof(RegAsk) + std::max(sums, logits);
  *far = rest + dep_reg_addresses(c) > SMEM_LIMIT;
  return rest + (*far ? 0 : dep_reg_addresses(c));
}
// Depformers so deep that their weights' addresses, the ring and the bare sums are more than shared memory holds are left to the other kernels (the 7B's widths with 16 sub-steps: from 178
// layers on at one session, from 88 at 16).
inline bool dep_reg_deep(const DepFusedConfig& c, int grid) {
  return (size_t)REG_SLOTS * REG_SLOT_BYTES + dep_reg_addresses(c) + (size_t)REG_WARPS * dep_reg_subs(c, grid) * c.B * REG_UNIT * 4 > SMEM_LIMIT;
}
// words of the qkv and the barrier's, which are zeroed above 8 sessions too, and of everything
inline size_t dep_reg_front(const DepFusedConfig& c) { return (size_t)c.B * (3 * c.dd / 2) + 16; }      // words stay on lines
inline size_t dep_reg_words(const DepFusedConfig& c) { return dep_reg_front(c) + (size_t)c.B * (c.dd / 2 + c.dd / 2 + c.F / 2 + (c.card + 7) / 8 * 4); }
inline bool dep_reg_takes(const DepFusedConfig& c, int grid) {
  bool far;
  return c.B <= REG_B && c.dd % 64 == 0 && c.dd <= REG_WARPS * 64 && c.F % 8 == 0 && c.F <= REG_KC * REG_WARPS * 64 && grid >= 1 && dep_reg_subs(c, grid) <= REG_SUBS &&
         c.B * (c.dd / DD) <= REG_WARPS * grid && !dep_reg_deep(c, grid) && dep_reg_smem(c, grid, &far) <= SMEM_LIMIT;
}
