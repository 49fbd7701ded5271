// Asynchronous 16-byte copies from global to shared memory (cp.async), waited for by the warp.
#pragma once
#include <cuda_runtime.h>

namespace v3dba {

// 16 bytes global -> shared; zeros when !use.
__device__ __forceinline__ void cp16(void* dst, const void* src, bool use) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(use ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_join() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// All copies but those of the last group have arrived.
__device__ __forceinline__ void cp_join_but_last() {
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  __syncwarp();
}
// ... but those of the last N groups.
template <int N>
__device__ __forceinline__ void cp_join_but() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
  __syncwarp();
}

}  // namespace v3dba
