// Shared-memory addresses and asynchronous global -> shared copies (cp.async).
#pragma once

#include "common.cuh"

namespace jfli {

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

template <int BYTES>
__device__ __forceinline__ void copy_async(void* smem, const void* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(smem)), "l"(global), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace jfli
