/*
 * hm_pack.cuh - pairs of fp32 values in one 64-bit register pair and the
 * packed arithmetic of sm_100 (add / sub / mul / fma .f32x2).
 *
 * Why: the solvers' kernels are bound by instruction issue (one warp
 * instruction per scheduler and cycle), not by the fp32 lanes.  A packed
 * instruction does the work of two and takes one issue slot; it occupies
 * the fp32 lanes for two cycles (measured: 2.06 cycles against 1.10 for
 * the scalar FFMA), during which the scheduler issues loads, min / max,
 * compares and logic of the same or another warp.
 *
 * Rounding: each half is rounded exactly as the scalar operation.  But the
 * compiler contracts a packed multiply that feeds a packed add or subtract
 * into one fma, in spite of the explicit .rn and of -fmad=false (measured:
 * a quarter of random a * b + c differ from two roundings).  So a product
 * that is added or subtracted next is formed by mul2r, an fma with a -0
 * addend that the compiler cannot see through (x + -0 is x for every x,
 * zeros of both signs included).
 */
#ifndef HM_PACK_CUH
#define HM_PACK_CUH

#include <cuda_runtime.h>

namespace hm
{

struct F2
{
  unsigned long long v;
};

__device__ __forceinline__ F2 pk(float a, float b)
{
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2    pk(float2 a) { return pk(a.x, a.y); }
__device__ __forceinline__ F2    pk1(float a) { return pk(a, a); }
__device__ __forceinline__ float2 up(F2 p)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p.v));
  return r;
}
__device__ __forceinline__ float lo(F2 p) { return up(p).x; }
__device__ __forceinline__ float hi(F2 p) { return up(p).y; }

__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b)
{
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
/* a * b whose result feeds no packed add or subtract */
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
/* a * b rounded on its own; nz is (-0, -0) from a kernel argument */
__device__ __forceinline__ F2 mul2r(F2 a, F2 b, F2 nz) { return fma2(a, b, nz); }

} // namespace hm

#endif
