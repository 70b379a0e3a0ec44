// sm_100a primitives shared by the tensor-core kernels (gemm_sk.cu, gemm_ns.cu, gemm_wide.cu, dlm_flash.cu, dep_fused.cu, mimi_tc.cu): mbarriers, bulk / tensor
// TMA copies, TMEM allocation, tcgen05.mma / commit / ld, UMMA descriptors, programmatic dependent launch.
#pragma once

#include <cuda.h>
#include <stdint.h>

namespace b200 {
namespace tcp {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t global_timer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait: a pipeline bug must surface as a launch failure, never as a hung GPU.  The bound is wall-clock (10 s on
// %globaltimer, sampled every 4096 polls), not a poll count: under programmatic dependent launch the consumer warps poll while
// the producer warp sits in griddepcontrol.wait for the whole predecessor kernel, and a profiler, a debugger or a
// time-sliced neighbour can stretch that by orders of magnitude without anything being wrong.
constexpr uint64_t WAIT_LIMIT_NS = 10ull * 1000ull * 1000ull * 1000ull;
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity) {
  uint32_t done, spins = 0;
  uint64_t t0 = 0;
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (!done && (++spins & 4095u) == 0u) {
      const uint64_t now = global_timer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) __trap();
    }
  } while (!done);
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Programmatic dependent launch: `pdl_wait` blocks until the preceding kernel in the stream has completed and its
// writes are visible; `pdl_trigger` lets the following kernel start its own prologue (and weight prefetch) early.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// K-major SWIZZLE_128B shared-memory matrix descriptor: start address >> 4, LBO = 1 (unused for swizzled K-major), SBO = 1024 B
// (8 rows x 128 B), descriptor version 1 (bit 46), layout type 2 = SWIZZLE_128B (bits 61-63).
__device__ __forceinline__ uint64_t make_desc(uint32_t smem_addr) {
  uint64_t d = (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// instruction descriptors: D format at bit 4 (1 = f32, 2 = s32), A / B formats at bits 7 / 10, N >> 3 at bit 17, M >> 4 at bit 24;
// both operands K-major.  kind::f16: A = B = bf16 (1); kind::tf32: A = B = tf32 (2); kind::i8: A = B = signed 8 bit (1).
__device__ __forceinline__ uint32_t make_idesc(int umma_m, int umma_n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(umma_m >> 4) << 24);
}
__device__ __forceinline__ uint32_t make_idesc_tf32(int umma_m, int umma_n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(umma_m >> 4) << 24);
}
__device__ __forceinline__ uint32_t make_idesc_i8(int umma_m, int umma_n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(umma_n >> 3) << 17) | ((uint32_t)(umma_m >> 4) << 24);
}


// ---- issue from uniform registers ----
// A copy or product takes its operands in uniform registers.  Where one thread of a warp walks a loop alone the compiler moves every operand there first, and an
// instruction goes out every 90 to 140 clocks; where the whole warp walks along (the warp's number through __shfl_sync, so that the compiler knows) and one thread
// is elected for the instruction alone, every 55.
__device__ __forceinline__ bool elected() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(r));
  return r != 0;
}
__device__ __forceinline__ void commit_elected(uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
// low word of make_desc; the high word is the same for every operand
constexpr uint32_t DESC_HIGH = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_low(uint32_t smem) { return ((smem & 0x3FFFFu) >> 4) | (1u << 16); }
// The four products of a k-block (128 bytes of k), by one thread of the warp: rows at desc a, columns w_at 16-byte pieces behind them.
#define UMMA_BLOCK(GROUP, KIND)                                                                                                                        \
  asm volatile(                                                                                                                                        \
      "{\n\t.reg .pred p, t, q;\n\t.reg .b64 a0, a1, a2, a3, w0, w1, w2, w3;\n\t"                                                                     \
      "mov.b64 a0, {%1, %11};\n\tmov.b64 a1, {%2, %11};\n\tmov.b64 a2, {%3, %11};\n\tmov.b64 a3, {%4, %11};\n\t"                                     \
      "mov.b64 w0, {%5, %11};\n\tmov.b64 w1, {%6, %11};\n\tmov.b64 w2, {%7, %11};\n\tmov.b64 w3, {%8, %11};\n\t"                                     \
      "setp.ne.b32 p, %10, 0;\n\tsetp.ne.b32 t, %11, 0;\n\telect.sync _|q, 0xffffffff;\n\t"                                                         \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], a0, w0, %9, p;\n\t"                                                                    \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], a1, w1, %9, t;\n\t"                                                                    \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], a2, w2, %9, t;\n\t"                                                                    \
      "@q tcgen05.mma.cta_group::" GROUP ".kind::" KIND " [%0], a3, w3, %9, t;\n\t}"                                                                   \
      ::"r"(d), "r"(a), "r"(a + 2), "r"(a + 4), "r"(a + 6), "r"(w), "r"(w + 2), "r"(w + 4), "r"(w + 6), "r"(idesc), "r"(accumulate), "r"(DESC_HIGH) : "memory")
template <int CG>
__device__ __forceinline__ void umma_block(uint32_t d, uint32_t a, uint32_t w_at, uint32_t idesc, uint32_t accumulate) {
  const uint32_t w = a + w_at;
  if constexpr (CG == 2) UMMA_BLOCK("2", "f16");
  else UMMA_BLOCK("1", "f16");
}
__device__ __forceinline__ void umma_block_i8(uint32_t d, uint32_t a, uint32_t w_at, uint32_t idesc, uint32_t accumulate) {
  const uint32_t w = a + w_at;
  UMMA_BLOCK("1", "i8");
}
#undef UMMA_BLOCK

}  // namespace tcp
}  // namespace b200
