// cp.async wrappers: copies from global to shared memory that a thread issues and waits for later.  `src_bytes` 0 fills the
// destination with zeros and reads nothing.
#pragma once
#include <cuda_runtime.h>

namespace mpt {

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(src_bytes));
}
// Bytes of a 16-byte copy from where `left` floats of the row remain (none from outside it): counted in elements first, since
// four times a large extent does not fit 32 bits.
__host__ __device__ __forceinline__ int bytes16(int left) { return 4 * (left < 0 ? 0 : left > 4 ? 4 : left); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

}  // namespace mpt
