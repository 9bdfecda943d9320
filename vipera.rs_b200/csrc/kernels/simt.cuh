// Pieces of the kernels that compute in 32 bits on the CUDA cores: asynchronous copies, packed
// multiply-adds, clusters of blocks.
#pragma once

#include <atomic>

#include "common.cuh"

__device__ __forceinline__ uint32_t shared_address(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void copy_16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Two independent fused multiply-adds, each rounded as fmaf rounds.
__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float sum_of_pair(unsigned long long v) {
  return __uint_as_float(static_cast<uint32_t>(v)) + __uint_as_float(static_cast<uint32_t>(v >> 32));
}
__device__ __forceinline__ float remote_float(uint32_t address, uint32_t block) {
  float v;
  asm volatile("{\n .reg .b32 r;\n mapa.shared::cluster.u32 r, %1, %2;\n ld.shared::cluster.f32 %0, [r];\n}\n" : "=f"(v) : "r"(address), "r"(block));
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The opt-in for more than 48 KB of dynamic shared memory, asked for once per device.
struct SharedMemoryOptIn {
  std::atomic<unsigned long long> done{0};   // a bit per device
  int ask(const void* kernel, int bytes) {
    int device = 0;
    cudaError_t error = cudaGetDevice(&device);
    if (error != cudaSuccess) return static_cast<int>(error);
    const unsigned long long bit = 1ull << (device & 63);
    if (device < 64 && (done.load(std::memory_order_acquire) & bit)) return 0;
    error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (error != cudaSuccess) return static_cast<int>(error);
    done.fetch_or(bit, std::memory_order_release);
    return 0;
  }
};

// Multiprocessors of the current device, asked for once per device.
static inline int multiprocessors() {
  static std::atomic<int> counts[64];
  int device = 0, count = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return 148;
  if (device < 64 && (count = counts[device].load(std::memory_order_relaxed)) > 0) return count;
  if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || count <= 0) return 148;
  if (device < 64) counts[device].store(count, std::memory_order_relaxed);
  return count;
}

// Launch `kernel` as vipera_launch does; `cluster` > 1: in clusters of that many blocks along x.
template <typename... KernelArgs, typename... Args>
static inline int launch_in_clusters(void (*kernel)(KernelArgs...), int cluster, dim3 grid, dim3 block, size_t shared_bytes,
                                     cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = vipera_pdl_enabled() ? 1 : 0;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = cluster;
  attributes[1].val.clusterDim.y = attributes[1].val.clusterDim.z = 1;
  config.attrs = attributes;
  config.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t error = cudaLaunchKernelEx(&config, kernel, static_cast<KernelArgs>(std::forward<Args>(args))...);
  return error == cudaSuccess ? VIPERA_OK : static_cast<int>(error);
}
