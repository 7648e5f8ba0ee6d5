// Asynchronous global -> shared copies, as hand-written inline PTX.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace mfdm {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Global -> shared asynchronous copy of 16 bytes (zeros when !ok: nothing is
// read), committed and awaited per thread.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Programmatic dependent launch. A grid launched with the attribute starts when
// every block of the grid before it on the stream has called launch_dependents()
// (or ended); wait_previous() returns when that grid has ended and its memory is
// visible. What a previous grid of the chain writes is read after it, and not
// through the read-only cache, which assumes data constant from the launch on.
__device__ __forceinline__ void launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace mfdm
