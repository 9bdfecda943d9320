// Barriers with bounded waits, and tensor-memory operations of kernels whose products are issued by a warp that walks
// together: every lane has the same operands, one elected lane issues.
#pragma once

#include "simt.cuh"

namespace tcgen05 {

constexpr uint32_t kWaitLimit = 1u << 22;

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_address(bar)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(shared_address(bar)) : "memory");
}
// A wait that runs out leaves EXPIRED in the status word and raises the block's flag.
template <int EXPIRED>
__device__ __forceinline__ void bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  for (uint32_t spin = 0; spin < kWaitLimit; ++spin) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(shared_address(bar)), "r"(parity) : "memory");
    if (done) return;
    if (spin > 8) __nanosleep(32);
    if ((spin & 1023u) == 1023u && *abort_flag) return;
  }
  *abort_flag = 1;
  atomicExch(status, EXPIRED);
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile(
      "{\n .reg .pred leader;\n elect.sync _|leader, 0xffffffff;\n"
      " @leader tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(shared_address(bar)) : "memory");
}
// D (tensor memory) = or += A . B with both operands in shared memory
__device__ __forceinline__ void mma_shared(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p, leader;\n elect.sync _|leader, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
      " @leader tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

}  // namespace tcgen05
