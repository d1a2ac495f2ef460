// Shared-memory access by 32-bit shared-space address, mbarriers with bounded waits, and the bulk (TMA) copy: the
// pieces every staged kernel in this directory is built from.
#pragma once
#include "common.cuh"

namespace osmos {
namespace tma {

// no copy of a tile takes anywhere near 0.2 s: a wait that long gives up and the kernel reports it
constexpr uint64_t kWaitLimitNs = 200ull * 1000 * 1000;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ int4 lds128(uint32_t a) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 lds128f(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float ldsf(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}
// after the block's barriers are initialised, before anything (a copy included) uses them
__device__ __forceinline__ void bar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void bar_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool bar_done(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// true when the phase of `parity` has completed; gives up `limit` ns after its first look. The clock is the thread's own: of
// a warp's lanes some may give up where the phase completes in time for others.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, uint64_t limit = kWaitLimitNs) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; spin++) {
    if (bar_done(bar, parity)) return true;
    if (spin == 0) t0 = global_ns();
    else if (global_ns() - t0 > limit) return false;
  }
}
// the same for a whole warp, with one outcome for all its lanes: when one gives up, all do. What follows a wait that ran out
// - leaving for a block's barrier, or going on to the warp's next meeting - is then every lane's, and no lane waits at
// either for one that took the other way.
__device__ __forceinline__ bool bar_wait_warp(uint64_t* bar, uint32_t parity, uint64_t limit = kWaitLimitNs) {
  return __all_sync(0xFFFFFFFFu, bar_wait(bar, parity, limit));
}
// bar_wait_warp for a wait that is expected to be long (an epilogue's, through a whole K loop): the look itself may suspend the
// warp for up to 10 us at a time - it still returns when the phase completes - so that waiting costs no issue slots
__device__ __forceinline__ bool bar_wait_long(uint64_t* bar, uint32_t parity, uint64_t limit = kWaitLimitNs) {
  const uint32_t a = smem_addr(bar);
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; spin++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 10000;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (__all_sync(0xFFFFFFFFu, done)) return true;
    if (spin == 0) t0 = global_ns();
    else if (__any_sync(0xFFFFFFFFu, global_ns() - t0 > limit)) return false;
  }
}
// bar_wait_warp where the phase has most often completed already: the first look by itself (a phase that has completed: 15
// cycles, where the loop's set-up takes 54 to 110)
__device__ __forceinline__ bool bar_wait_soon(uint64_t* bar, uint32_t parity, uint64_t limit = kWaitLimitNs) {
  if (__all_sync(0xFFFFFFFFu, bar_done(bar, parity))) return true;
  return bar_wait_long(bar, parity, limit);
}
// global -> this block's shared memory, completion counted on `bar`; both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// orders this thread's earlier shared-memory accesses before the copies it issues next into the same bytes
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }


// ---- a warp's tcgen05 instructions --------------------------------------------------------------------------------------
// One elected lane issues, but the whole warp runs the code around it: the operands are then the warp's own, in uniform
// registers. Under a branch for one lane each instruction's operands are moved there by themselves - measured on products of
// 128 x n x 16, f16: 65 cycles an instruction whatever its size, against 17 (n = 16), 32 (64), 128 (256). elect.sync picks
// the same lane each time, so a commit follows the products of the lane that issued them.


__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}
// (d0, d1) += A (B0, B1) over K = 64 (accumulate 0: without the old sums), pairs of instructions of K = 16: A in tensor memory,
// 32 columns from `a` on; B0 and B1 in shared memory, b1's address 32 bytes on from b's, both a `step` on each K = 16; issuer:
// elect_one()'s
__device__ __forceinline__ void mma_f16_ts_k64(uint32_t issuer, uint32_t d0, uint32_t d1, uint32_t a, uint64_t b, uint32_t step, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred e, p, t;\n .reg .b32 a;\n .reg .b64 b, c, s;\n setp.ne.b32 e, %0, 0;\n setp.ne.b32 p, %7, 0;\n setp.eq.b32 t, %0, %0;\n"
      " cvt.u64.u32 s, %5;\n add.u64 c, %4, 2;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], %4, %6, p;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%2], [%3], c, %6, p;\n"
      " add.u32 a, %3, 8;\n add.u64 b, %4, s;\n add.u64 c, c, s;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%1], [a], b, %6, t;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%2], [a], c, %6, t;\n"
      " add.u32 a, a, 8;\n add.u64 b, b, s;\n add.u64 c, c, s;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%1], [a], b, %6, t;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%2], [a], c, %6, t;\n"
      " add.u32 a, a, 8;\n add.u64 b, b, s;\n add.u64 c, c, s;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%1], [a], b, %6, t;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%2], [a], c, %6, t;\n}\n" ::"r"(issuer),
      "r"(d0), "r"(d1), "r"(a), "l"(b), "r"(step), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier when everything the issuer has issued is done
__device__ __forceinline__ void mma_commit(uint32_t issuer, uint64_t* bar) {
  asm volatile(
      "{\n .reg .pred e;\n setp.ne.b32 e, %0, 0;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%1];\n}\n" ::"r"(issuer),
      "r"(smem_addr(bar))
      : "memory");
}

}  // namespace tma
}  // namespace osmos
