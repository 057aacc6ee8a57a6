// Helpers for the 5th-generation tensor cores: descriptors, MMA issue, barriers, tensor-memory moves.
#pragma once

#include "common.cuh"

namespace inq {

__device__ __forceinline__ unsigned tc_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// One lane of a converged warp.  MMAs and commits are issued as `if (tc_elect())` inside a branch that is
// uniform over the warp: the compiler then keeps descriptors and addresses in uniform registers.  Issued
// from a branch on the thread index instead, each tcgen05.mma costs about 50 cycles of issue (measured, eight
// 128 x 16 x 16 MMAs with their commit and wait: 590 against 200 cycles).
__device__ __forceinline__ unsigned tc_elect() {
  unsigned chosen;
  asm volatile("{ .reg .pred p; elect.sync _|p, 0xffffffff; selp.u32 %0, 1, 0, p; }" : "=r"(chosen));
  return chosen;
}

// 64-bit shared-memory matrix descriptor: start address, leading and stride byte offsets in 16-byte
// units, descriptor version 1, layout type (0: no swizzle, 2: 128-byte swizzle).
template <int LAYOUT = 2>
__device__ __forceinline__ unsigned long long tc_desc(unsigned saddr, unsigned lbo_bytes, unsigned sbo_bytes) {
  unsigned long long d = 0;
  d |= (unsigned long long)((saddr & 0x3FFFFu) >> 4);
  d |= (unsigned long long)(lbo_bytes >> 4) << 16;
  d |= (unsigned long long)(sbo_bytes >> 4) << 32;
  d |= 1ull << 46;
  d |= (unsigned long long)LAYOUT << 61;
  return d;
}

// Instruction descriptor of kind::f16 with fp32 accumulation: operand type, M, N; B_MN: B is MN-major.
template <bool BF16, int M, int N, bool B_MN>
__device__ __forceinline__ constexpr unsigned tc_idesc() {
  return (1u << 4) | (BF16 ? (1u << 7) | (1u << 10) : 0u) | (B_MN ? 1u << 16 : 0u) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}

// D (tensor memory) = or += A B; A from shared memory or from tensor memory, B from shared memory.
__device__ __forceinline__ void tc_mma(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
               ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_mma_ta(unsigned tmem_d, unsigned tmem_a, unsigned long long db, unsigned idesc, unsigned accumulate) {
  asm volatile("{ .reg .pred p; setp.ne.b32 p, %4, 0; tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p; }"
               ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_commit(unsigned mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_bar_init(unsigned mbar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ bool tc_try_wait(unsigned mbar, unsigned parity) {
  unsigned done;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait of a thread for a phase of a barrier.  A try sleeps for up to 4 us (measured), so 2^18 of them are
// about a second.  A wait that runs out raises the abort flag, and once the flag is raised every wait of the
// CTA ends after 16 tries (most tries that fail come back early, and reading the flag after each of them held
// up the next: 1500-token prompt of 32 heads 29.3 instead of 27.9 us,
// 2048 queries over 4096 keys of 28 heads 94.2 instead of 91.1).  The lanes of a warp wait by themselves and need not agree on the outcome, but what
// follows a wait -- elect.sync over the full mask, the .sync.aligned tensor-memory instructions -- needs all
// of them.  So a warp does not leave its loop where a wait gives up: it runs through its remaining turns,
// whose waits no longer wait, on data that nobody will use.
constexpr int kTcTries = 1 << 18;
__device__ __forceinline__ bool tc_wait(unsigned mbar, unsigned parity, volatile int* abort_flag, int tries = kTcTries) {
  for (int it = 0; it < tries; ++it) {
    if (tc_try_wait(mbar, parity)) return true;
    if ((it & 15) == 15 && *abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
// Bounded wait for work of this CTA that is in flight when its roles have ended, whatever the abort flag says.
__device__ __forceinline__ void tc_drain(unsigned mbar, unsigned parity) {
  for (int it = 0; it < kTcTries && !tc_try_wait(mbar, parity); ++it) {
  }
}

#define TC_R4(v, o) "r"((v)[o]), "r"((v)[(o) + 1]), "r"((v)[(o) + 2]), "r"((v)[(o) + 3])
#define TC_R16(v, o) TC_R4(v, o), TC_R4(v, (o) + 4), TC_R4(v, (o) + 8), TC_R4(v, (o) + 12)
#define TC_W4(v, o) "=r"((v)[o]), "=r"((v)[(o) + 1]), "=r"((v)[(o) + 2]), "=r"((v)[(o) + 3])
#define TC_W16(v, o) TC_W4(v, o), TC_W4(v, (o) + 4), TC_W4(v, (o) + 8), TC_W4(v, (o) + 12)
// 32x32b: lane i of warp w moves TMEM lane 32 (w % 4) + i, register k column k.
__device__ __forceinline__ void tc_st16(unsigned taddr, const unsigned (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), TC_R16(v, 0) : "memory");
}
// The loads do not wait: tc_wait_ld32 / tc_wait_ld16 of the loaded registers stands between a load and their first
// use.  The registers are operands of the wait, because nothing else holds arithmetic on them back behind it.
__device__ __forceinline__ void tc_ld32(unsigned taddr, unsigned (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : TC_W16(v, 0), TC_W16(v, 16) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld16(unsigned taddr, unsigned (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : TC_W16(v, 0) : "r"(taddr) : "memory");
}
#define TC_RW4(v, o) "+r"((v)[o]), "+r"((v)[(o) + 1]), "+r"((v)[(o) + 2]), "+r"((v)[(o) + 3])
#define TC_RW16(v, o) TC_RW4(v, o), TC_RW4(v, (o) + 4), TC_RW4(v, (o) + 8), TC_RW4(v, (o) + 12)
__device__ __forceinline__ void tc_wait_ld32(unsigned (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : TC_RW16(v, 0), TC_RW16(v, 16) :: "memory");
}
__device__ __forceinline__ void tc_wait_ld16(unsigned (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : TC_RW16(v, 0) :: "memory");
}

}  // namespace inq
