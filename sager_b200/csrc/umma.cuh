// umma.cuh - the tcgen05 instructions and small helpers shared by the tensor-core kernels
// (grouped_gemm_i8.cu, tc_gemm.cu).
#pragma once

#include "q4k_common.cuh"

namespace sgr {

// Shared-memory operand descriptors (K-major) as two words; only the first depends on the tile.
//   core:     8x16-byte core matrices, the two K halves 128 bytes apart (LBO), eight-row groups 256 (SBO)
//   swizzled: rows of 128 bytes, eight-row groups 1024 bytes apart, 128-byte swizzle; + 2 per K = 16 step
__device__ __forceinline__ uint32_t umma_desc_core(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (8u << 16); }
constexpr uint32_t kDescCore = 16u | (1u << 14);
__device__ __forceinline__ uint32_t umma_desc_swizzled(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t kDescSwizzled = (1024u >> 4) | (1u << 14) | (2u << 29);
// D fp32, A and B fp16, both K-major, M = m (128, of a CTA pair 256), N = n
__device__ __forceinline__ uint32_t umma_idesc_f16(int n, int m = 128) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
// A in tensor memory (lane = row, a column holds two consecutive K values) / A in shared memory
// The whole warp runs the instruction stream, `lead` picks the lane that issues. CG = 2: the instruction of a CTA pair, issued by the
// pair's first CTA: its tensor memory and the other's hold 128 rows of A and D each, their shared memory half of B's columns each.
template <int CG = 1>
__device__ __forceinline__ void umma_ts(uint32_t lead, uint32_t tmem_d, uint32_t tmem_a, uint32_t db, uint32_t db_hi,
                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 b, {%2, %5};\n\t"
      "@q tcgen05.mma.cta_group::%7.kind::f16 [%0], [%1], b, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "r"(db), "r"(idesc), "r"(accumulate), "r"(db_hi), "r"(lead), "n"(CG)
      : "memory");
}
__device__ __forceinline__ void umma_ss(uint32_t lead, uint32_t tmem_d, uint32_t da, uint32_t db, uint32_t desc_hi,
                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(da), "r"(db), "r"(idesc), "r"(accumulate), "r"(desc_hi), "r"(lead)
      : "memory");
}
// One arrival when the MMAs issued so far have finished; CG = 2: at the barrier of this address in both CTAs.
template <int CG = 1>
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  if constexpr (CG == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
// The address of a CTA's own shared memory as it lies in the CTA of the cluster with that rank
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// (no wider scope than the CTA's is asked for: what the arrival publishes are tensor-memory stores, which the tcgen05 fences order. A
// release at cluster scope waited for every store to memory before it, 1,500 cycles an arrival.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
               ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]),
                 "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
                 "r"(v[30]), "r"(v[31])
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Bounded wait (as mbar_wait) in a handful of instructions per poll: polls return early whenever something
// happens in the barrier unit, so with two dozen waiting warps their instructions count.
__device__ __forceinline__ bool mbar_wait_tight(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b32 n;\n\tmov.b32 n, 0;\n"
      "POLL%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE%=;\n\t"
      "add.u32 n, n, 1;\n\tsetp.lt.u32 q, n, %3;\n\t@q bra POLL%=;\n"
      "DONE%=:\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(1u << 22)
      : "memory");
  return ok != 0;
}
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
// (x & mask) | bits in one instruction
__device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t mask, uint32_t bits) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(x), "r"(mask), "r"(bits));
  return d;
}
// two packed fp32: each component rounds as the scalar instruction
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(uint32_t lo, uint32_t hi) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi)); return d; }
__device__ __forceinline__ f32x2 splat2(float v) { return pack2(__float_as_uint(v), __float_as_uint(v)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ float part2(f32x2 v, int hi) {
  uint32_t a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
  return __uint_as_float(hi ? b : a);
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_or_zero(uint32_t dst, const void* src, bool there) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {    // one arrival when this thread's copies so far have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace sgr
