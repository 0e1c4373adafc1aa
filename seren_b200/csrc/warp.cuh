// warp.cuh - warp-wide helpers of the pair kernels: several particles share a
// warp, eight lanes each.
#pragma once

#include <cuda_runtime.h>

namespace seren {

// Sums of v0..v3 over each group of 8 lanes: lane 2k of a group (k = 0..3)
// returns the sum of vk.
template <class T>
__device__ __forceinline__ T sum4_by8(T v0, T v1, T v2, T v3, int lane) {
  const bool h4 = lane & 4, h2 = lane & 2;
  T a = h4 ? v2 : v0, b = h4 ? v3 : v1;
  a += __shfl_xor_sync(0xffffffffu, h4 ? v0 : v2, 4);
  b += __shfl_xor_sync(0xffffffffu, h4 ? v1 : v3, 4);
  T c = h2 ? b : a;
  c += __shfl_xor_sync(0xffffffffu, h2 ? a : b, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// 32 x 32 bit transposition over the warp: bit j of lane i goes to bit i of lane j
__device__ __forceinline__ unsigned warp_transpose(unsigned x, int lane) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    constexpr unsigned M[5] = {0x55555555u, 0x33333333u, 0x0f0f0f0fu, 0x00ff00ffu, 0x0000ffffu};
    const unsigned m = M[s == 16 ? 4 : s == 8 ? 3 : s == 4 ? 2 : s == 2 ? 1 : 0];
    const bool hi = lane & s;
    const unsigned y = __shfl_xor_sync(0xffffffffu, x, s);
    const unsigned t = __funnelshift_l(y, y, hi ? 32 - s : s);
    const unsigned keep = hi ? ~m : m;
    x = (x & keep) | (t & ~keep);
  }
  return x;
}

// Packed FP32: the two halves of a register pair go through one instruction
// (fma/add/mul.f32x2), so a kernel bound by its instruction count does two
// terms in the issue slots of one.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 pk1(float x) { return pk(x, x); }
__device__ __forceinline__ void unpk(f2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 fma2_rm(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float sum2(f2 v) {
  float lo, hi;
  unpk(v, lo, hi);
  return lo + hi;
}

// 1/sqrt(x) and 1/x of normal numbers (no subnormal handling)
__device__ __forceinline__ float rsqrt_n(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_n(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

}  // namespace seren
