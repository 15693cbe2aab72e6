// mbarrier, TMA and tcgen05 primitives (inline PTX) shared by the sm_100a kernels.
#pragma once

#include "common.cuh"

namespace gemq {

constexpr int kSpinLimit = 1 << 18;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) {  // shared address
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) { mbar_arrive_at(smem_u32(bar)); }
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Looks once, without waiting.
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after kSpinLimit polls, records `code` and returns.  A waiting warp
// sleeps between polls so that it does not take issue slots from the warps that are working.
__device__ __forceinline__ void mbar_wait(unsigned long long* bar, uint32_t parity, int* err, int code,
                                          unsigned sleep_ns = 64, int limit = kSpinLimit) {
  if (mbar_try_wait(bar, parity)) return;
  for (int i = 0; i < limit; ++i) {
    __nanosleep(sleep_ns);
    if (mbar_try_wait(bar, parity)) return;
  }
  atomicExch(err, code);
}
// Bounded wait of a warp that sleeps in hardware until the phase ends (at most 20 us a time, about a second in
// all).  Without the time hint try_wait comes back after some tens of cycles, and warps that wait long -- for
// the end of a tile, say -- spend the issue slots of the others.
__device__ __forceinline__ bool mbar_sleep_wait(unsigned long long* bar, uint32_t parity, int* err, int code) {
  for (int i = 0; i < (1 << 16); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000)
        : "memory");
    if (ok) return true;
  }
  atomicExch(err, code);
  return false;
}
// The same behind one look, for waits that are mostly over when they begin: a try_wait with a time hint takes about 190 cycles then.
__device__ __forceinline__ bool mbar_look_wait(unsigned long long* bar, uint32_t parity, int* err, int code) {
  return mbar_test_wait(bar, parity) || mbar_sleep_wait(bar, parity, err, code);
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p) : "memory"); }
// Tiled TMA load of one box at element coordinates (x = column, y = row); x * element size
// must be a multiple of 16 bytes (it is: columns come in multiples of 32).
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}


// ---- tcgen05 (5th generation tensor cores, accumulators in tensor memory) ---------------
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory matrix descriptor of a K-major operand tile stored as rows of 128 bytes with
// the 128-byte swizzle (the layout a tiled TMA load with SWIZZLE_128B produces): 8-row groups
// are 1024 bytes apart.  `addr` = shared address of the tile (1024-byte aligned) plus the byte
// offset of the K slice inside the 128-byte row.
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3ffffu) >> 4);        // start address, bits [0,14)
  d |= static_cast<uint64_t>(1) << 16;                       // leading byte offset (unused with swizzle)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;               // stride byte offset: 8 rows x 128 B
  d |= static_cast<uint64_t>(1) << 46;                       // descriptor version of sm_100
  d |= static_cast<uint64_t>(2) << 61;                       // layout: 128-byte swizzle
  return d;
}
// Instruction descriptor of kind::f16: D fp32, A/B both f16 (fmt 0) or bf16 (fmt 1), both K-major.
__device__ __forceinline__ uint32_t umma_idesc_f16(int fmt, int M, int N) {
  return (1u << 4) | (static_cast<uint32_t>(fmt) << 7) | (static_cast<uint32_t>(fmt) << 10) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}
}  // namespace gemq
