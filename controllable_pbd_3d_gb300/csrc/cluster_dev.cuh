// Device helpers of the kernels whose blocks form a thread-block cluster and
// exchange through one another's shared memory (dcg.cu, sweep.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mgpbd {
namespace cdev {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The address of this block's shared address in block `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

// Stores into another block's shared memory that complete there by counting
// their bytes on its barrier: data and signal travel together, so neither
// side needs a fence
__device__ __forceinline__ void send_f4(uint32_t addr, uint32_t bar, float x, float y, float z,
                                        float w = 0.0f) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
      ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void send_f64(uint32_t addr, uint32_t bar, double v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr),
               "d"(v), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void expect_bytes(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}

__device__ __forceinline__ bool test_phase(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// The same, but the warp may be suspended for a (bounded) while first: it leaves
// the issue slots to the others
__device__ __forceinline__ bool try_phase(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void cluster_meet() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}

}  // namespace cdev
}  // namespace mgpbd
