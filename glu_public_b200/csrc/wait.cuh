// What the bounded device-side waits of the cooperative kernels share.
#pragma once

#include <cuda_runtime.h>

namespace glu {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A value of the dense solve that has not been solved yet (a NaN payload no arithmetic produces),
// and the NaN stored in its place should a solved value have these bits.
constexpr long long kUnsolved = 0x7ff4a1c35e6b2d97ll;
constexpr long long kNaN = 0x7ff8000000000000ll;

// First statement of a kernel that launch_next launches (after reads of the plan's arrays at most,
// which nothing writes): waits until the kernel before it in the stream has finished and its writes
// are visible, then lets the kernel after it be placed on SMs that become free.  Every CTA passes
// here before it returns, so kernels finish in stream order.
// Such a kernel is resident while the one before it writes, so const __restrict__, which lets the
// compiler load through the read-only path and at any place in the kernel, is for the plan's
// arrays only: not for what the kernel before it in the stream, or the caller's, may have written
// (right-hand sides, solutions, matrix values as loaded, perturbations).
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace glu
