// Sums that the blocks of a cluster exchange: asynchronous stores into another block's shared memory which count
// their bytes on an mbarrier there. A cluster barrier behind ordinary remote stores took 1400 to 1600 clocks;
// this way a block waits for its own bytes only. The receiver announces the bytes once (expect_tx) and
// its peers write only after a cluster barrier that follows the announcement.
#pragma once
#include "tc_common.cuh"

namespace ac {

// The address of `local` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* local, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(tc::smem_u32(local)), "r"(rank));
  return a;
}
__device__ __forceinline__ void send4(uint32_t dst, uint32_t bar, float4 v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send1(uint32_t dst, uint32_t bar, float v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}
// Bounded wait for everything announced on the barrier; what the peers sent is then visible.
__device__ __forceinline__ bool wait_sent(uint64_t* bar, uint32_t parity) {
  const uint32_t addr = tc::smem_u32(bar);
  for (uint32_t i = 0; i < tc::kWaitLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

}  // namespace ac
