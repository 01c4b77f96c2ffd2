// tcgen05.cuh -- tcgen05 / TMEM / TMA primitives shared by the tensor-core
// pairwise kernels (pairwise_tc.cu, pairwise_tc64.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "device_util.cuh"
#include "tile_walk.h"

namespace wmd {

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, int ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// One lane of the (converged) warp; the same lane at every call.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t on;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(on));
  return on;
}

// Issue of MMAs and commits by a whole converged warp, of which the lane with
// `on` (elect_one) executes them: the operands stay warp-uniform, so ptxas keeps
// the descriptors in uniform registers.  Issued from inside `if (lane == 0)`,
// each MMA first moved its descriptors there, and that bounded the issue: with a
// commit per 32-atom chunk 85 clocks per M128 N128 K32 MMA against 65.5 this way
// (64 is the tensor rate), 68 against 59.5 for N = 96 (an issue loop alone, all SMs).
__device__ __forceinline__ void tc_commit(uint64_t* bar, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_addr(bar)),
      "r"(on)
      : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate, uint32_t on) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}

// 32 lanes x 8 consecutive 32-bit TMEM columns -> 8 registers per thread
// (call tmem_wait_ld before using them)
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
      : "memory");
}

// Shared-memory matrix descriptor, K-major, rows of ROW bytes with the
// matching swizzle (64: SWIZZLE_64B, layout 4; 32: SWIZZLE_32B, layout 6),
// 8-row core groups 8 ROW bytes apart, sm_100 descriptor version 1.
template <int ROW>
__device__ __forceinline__ uint64_t desc_sw(const void* p) {
  static_assert(ROW == 32 || ROW == 64, "row bytes");
  const uint64_t start = (smem_addr(p) >> 4) & 0x3FFFu;
  return start | (uint64_t(1) << 16) | (uint64_t((8 * ROW) >> 4) << 32) | (uint64_t(1) << 46) |
         (uint64_t(ROW == 64 ? 4 : 6) << 61);
}

// bounded wait on an mbarrier phase (no shared abort fallback needed by
// callers other than through the flag)
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, int* status, volatile int* abort,
                                        uint64_t limit_ns) {
  return mbar_wait(bar, parity, status, kStatusTimeoutFull, abort, limit_ns);
}

}  // namespace wmd
