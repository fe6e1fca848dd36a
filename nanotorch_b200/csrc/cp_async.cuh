// cp.async wrappers: 16- and 4-byte copies from global to shared memory; a copy that is not live writes zeros.
#pragma once

#include <cstdint>

namespace ntb {

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

} // namespace ntb
