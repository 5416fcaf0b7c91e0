// PTX glue shared by the tcgen05 kernels: mbarriers with bounded waits,
// tcgen05 fences / commit / TMEM loads, shared-memory matrix descriptors
// and bulk (non-tensor) global -> shared copies.  No multicast form of any
// copy is used.
#pragma once

#include <cstdint>

namespace frpa {
namespace sm100 {

constexpr unsigned long long WAIT_NS = 2000000000ull;  // 2 s per bounded wait

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One arrival that also announces `bytes` of asynchronous copies.
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// One poll; the thread may be suspended until the phase completes or
// SUSPEND_NS have passed, so that waiting roles leave the issue slots and the
// load/store unit to the working ones.
constexpr uint32_t SUSPEND_NS = 20000;

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(SUSPEND_NS)
      : "memory");
  return ok != 0;
}

// Bounded wait: false (and error bit 2 set) if the phase does not complete
// within WAIT_NS or another role has already given up.  The abort flag and the
// (slow) global timer are looked at once in WAIT_POLLS polls.
constexpr int WAIT_POLLS = 32;

__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity, volatile int *abort_flag,
                                          int *err) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < WAIT_POLLS; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (global_ns() - t0 > WAIT_NS) {
      *abort_flag = 1;
      atomicOr(err, 2);
      return false;
    }
  }
}

// Waits for a phase without looking at the abort flag (used on the way out,
// for copies or MMAs already in flight); false after WAIT_NS.
__device__ __forceinline__ bool mbar_wait_quiet(unsigned long long *bar, uint32_t parity) {
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity))
    if (global_ns() - t0 > WAIT_NS) return false;
  return true;
}

// Warp-uniform bounded wait: lane 0 polls, the outcome goes to every lane,
// so a warp never splits over a timeout; __syncwarp orders the lanes' later
// reads after lane 0's acquire.
__device__ __forceinline__ bool warp_wait(unsigned long long *bar, uint32_t parity, volatile int *abort_flag,
                                          int *err, int lane) {
  int ok = 1;
  if (lane == 0) ok = mbar_wait(bar, parity, abort_flag, err) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();
  return ok != 0;
}

// The same wait by a whole warp that stays converged: every lane polls, and
// all leave together (the slow path votes too).
__device__ __forceinline__ bool warp_wait_all(unsigned long long *bar, uint32_t parity, volatile int *abort_flag,
                                              int *err) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const unsigned long long t0 = global_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < WAIT_POLLS; ++i)
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    const bool late = global_ns() - t0 > WAIT_NS;
    if (late && !*abort_flag) {
      *abort_flag = 1;
      atomicOr(err, 2);
    }
    if (__any_sync(0xffffffffu, late || *abort_flag)) return false;
  }
}

// True in one lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor: K-major, no swizzle, version 1 (sm_100);
// lbo = bytes between K-adjacent core matrices, sbo = between 8-row groups.
template <uint32_t LBO, uint32_t SBO>
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(LBO >> 4) << 16;
  d |= (uint64_t)(SBO >> 4) << 32;
  d |= (uint64_t)1 << 46;  // version
  return d;                // base offset 0, lbo mode 0, layout type 0 (no swizzle)
}

__device__ __forceinline__ void umma_commit(unsigned long long *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 8 consecutive 32-bit TMEM columns of this thread's lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// 4 consecutive 32-bit TMEM columns of this thread's lane.
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

// Bulk copy global -> this CTA's shared memory, completing `bytes` on `bar`
// (both addresses 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, unsigned long long *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

}  // namespace sm100
}  // namespace frpa
