// Packed float32 arithmetic (two values in a register pair) and asynchronous copies into shared memory, for the 32-bit kernels.
//
// fma.rn.f32x2 does two float32 FMAs, each rounded like fmaf. It takes two issue cycles' worth of the FMA pipe for one issue
// slot, so that shared-memory reads and address work fit between; operands are pairs as they lie in memory.
#pragma once

#include "common.cuh"

namespace slb {

typedef unsigned long long f32x2;      // the value at the lower address in the low half

__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ f32x2 both(float v) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

__device__ __forceinline__ float low_half(f32x2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high_half(f32x2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ float halves_sum(f32x2 v) { return __fadd_rn(low_half(v), high_half(v)); }

// `bytes` of 16 (or 4) are copied, the rest of the 16 (4) are set to zero.
template <bool VEC>
__device__ __forceinline__ void copy_async(void* dst, const void* src, int bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

}  // namespace slb
