// Inline-PTX wrappers for sm_100a shared by the attention kernels: shared-memory barriers (mbarrier), bulk tensor
// copies (TMA), ldmatrix / movmatrix, the bf16 tensor-core instruction, a few scalar helpers.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "warp_reduce.cuh"

namespace l3ci {

constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // bound of one mbarrier wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Non-blocking: has the phase with the given parity completed?
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase with the given parity, at most kWaitLimitNs.  Warp-uniform result.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
  bool ok = mbar_try_wait(bar, parity);
  if (!__all_sync(kFullMask, ok)) {
    const unsigned long long t0 = global_ns();
    for (uint32_t it = 0;; ++it) {
      ok = mbar_try_wait(bar, parity);
      if (__all_sync(kFullMask, ok)) break;
      if ((it & 63u) == 63u) {
        const bool late = global_ns() - t0 > kWaitLimitNs;
        if (__any_sync(kFullMask, late)) return false;
      }
    }
  }
  return true;
}
// The same by one thread.
__device__ __forceinline__ bool mbar_wait_bounded_one(uint32_t bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (uint32_t it = 0;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 63u && global_ns() - t0 > kWaitLimitNs) return false;
  }
}
// Programmatic dependent launch.  pdl_wait: blocks until the kernel this one was launched behind has completed and
// its memory operations are visible (at once when the kernel was launched the plain way); everything before it may
// run while that kernel is still draining.  pdl_launch_dependents: lets the NEXT kernel of the stream be set up on the
// SMs as they come free (it stops at its own pdl_wait until this grid has completed).  A kernel that calls it first lets the chain
// of kernels behind start as far as the SMs have room, and what that may do ahead (l3ci_linear reads weights) overlaps it.
// A kernel that allocates tensor memory calls it behind the allocation.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Beginning of a kernel of many small CTAs (norms, caches, activations, recurrences): grids of few CTAs, a decode step's, let the next
// kernel start first; larger ones wait first.  CTAs that come early take places beside those that run, and the grid behind is then
// spread unevenly: back to back, residual norm of 300 rows 5.9 us instead of 4.4, 128 CTAs of the recurrent step 7.4 instead of 6.2, scans of
// 64 to 128 CTAs a fifth longer; at 8 rows a norm takes 1.5 instead of 1.7, and a product behind it has its weights.
// ahead: false where nothing may start early whatever the size.
constexpr unsigned kPdlAheadCtas = 64;
__device__ __forceinline__ void pdl_begin(bool ahead = true) {
  ahead = ahead && gridDim.x < kPdlAheadCtas;
  if (ahead) pdl_launch_dependents();
  pdl_wait();
  if (!ahead) pdl_launch_dependents();
}

__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// One tile (box) of a rank-4 tensor map into shared memory; completion is counted in bytes on `bar`.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0,
                                            int c1, int c2, int c3, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
      "l"(policy)
      : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// c += a(16x16, row) * b(16x8, col), bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Transposes an 8x8 matrix of 16-bit values held one row per 4 lanes, two values per lane.
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t ld_global_u32(const __nv_bfloat16* p) {
  return __ldg(reinterpret_cast<const uint32_t*>(p));
}


}  // namespace l3ci
