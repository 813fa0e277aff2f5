/*
 * hm_thermal_math.cuh - the talus exchange of one cell, bit-exact with the
 * reference's fp32 arithmetic.
 *
 * Reference: helper_thermal_exchange and the neighbour loop of
 * HighMap/src/gpu_opencl/kernels/thermal.cl:5-24,41-57 (neighbour order
 * HMAP_DI / HMAP_DJ, HighMap/include/highmap/erosion.hpp:21-22; distance
 * 1 for the four axial neighbours and 1.414 for the diagonals; rate 0.2).
 *
 * Every operation is an explicitly rounded intrinsic so the compiler cannot
 * contract a multiply into a following add: the result equals the
 * reference evaluated one rounding per operation.  The reference's
 * branches are folded:  with n = other - self,
 *     x = max(|n| - dist * talus, 0),   e = (0.2 * x) / dist,
 *     contribution = copysign(e, n),
 * which is the reference's value for every finite input (n = +0 gives
 * +e, as the reference's `else` branch does).
 *
 * Division by the diagonal distance 1.414f uses Markstein's correction of
 * the product by the correctly rounded reciprocal (P. Markstein, "Computation
 * of elementary functions on the IBM RISC System/6000 processor", IBM J.
 * Res. Dev. 34(1), 1990):  q = x * RN(1/b), r = fma(-q, b, x),
 * q' = fma(r, RN(1/b), q).  q' equals the correctly rounded x / 1.414f for
 * every normal x with a normal quotient (checked exhaustively over all
 * float mantissas; the identity is exponent independent).
 */
#ifndef HM_THERMAL_MATH_CUH
#define HM_THERMAL_MATH_CUH

#include <cfloat>

#include "hm_pack.cuh"

namespace hm
{

__device__ __forceinline__ float div_by_diag(float x)
{
  const float b = 1.414f;
  const float y = 0x1.6a17e6p-1f; /* RN(1 / 1.414f) */
  float       q = __fmul_rn(x, y);
  float       r = __fmaf_rn(-q, b, x);
  return __fmaf_rn(r, y, q);
}

__device__ __forceinline__ float exch_axial(float self, float other, float talus)
{
  float n = __fsub_rn(other, self);
  float x = fmaxf(__fsub_rn(fabsf(n), talus), 0.f);
  return copysignf(__fmul_rn(0.2f, x), n);
}

__device__ __forceinline__ float exch_diag(float self, float other, float max_dif_diag)
{
  float n = __fsub_rn(other, self);
  float x = fmaxf(__fsub_rn(fabsf(n), max_dif_diag), 0.f);
  return copysignf(div_by_diag(__fmul_rn(0.2f, x)), n);
}

/* Sum of the eight exchanges in reference order:
 * (-1,0) (0,+1) (0,-1) (+1,0) (-1,-1) (-1,+1) (+1,-1) (+1,+1)
 * with (di, dj) = (x offset, y offset).  Arguments are named by position:
 * w = (i-1, j), e = (i+1, j), n = (i, j-1), s = (i, j+1), nw = (i-1, j-1) ... */
__device__ __forceinline__ float thermal_amount(float c,
                                                float w,
                                                float s,
                                                float n,
                                                float e,
                                                float nw,
                                                float sw,
                                                float ne,
                                                float se,
                                                float talus)
{
  const float md = __fmul_rn(1.414f, talus);
  float       a = exch_axial(c, w, talus);
  a = __fadd_rn(a, exch_axial(c, s, talus));
  a = __fadd_rn(a, exch_axial(c, n, talus));
  a = __fadd_rn(a, exch_axial(c, e, talus));
  a = __fadd_rn(a, exch_diag(c, nw, md));
  a = __fadd_rn(a, exch_diag(c, sw, md));
  a = __fadd_rn(a, exch_diag(c, ne, md));
  a = __fadd_rn(a, exch_diag(c, se, md));
  return a;
}

/* Bedrock modes of the kernel templates */
enum BedMode
{
  BED_NONE = 0,
  BED_INTENDED = 1,
  BED_LITERAL = 2,
  BED_AUTO = 3
};

/* New value of an interior cell.  BED_INTENDED: max(val + amount, bedrock)
 * when val >= bedrock, else bedrock.  BED_LITERAL: max(val, bedrock), the
 * value thermal.cl:99 leaves.
 *
 * BED_AUTO is thermal_auto_bedrock (thermal.cl:102-145) with `bedrock` =
 * z0, the heights the solve started from, and `first` set on the first
 * step.  The reference keeps a bedrock grid: -FLT_MAX before the first
 * step, then max(z0, z_new) after every update, where
 * z_new = max(max(val + amount, z0), bedrock) is never below z0 (the
 * selects return z0 when val + amount is NaN).  So after a step the grid
 * holds exactly the new value, every later step finds bedrock == val and
 * passes the gate val >= bedrock, and the grid need not exist: the gate
 * becomes z0 >= -FLT_MAX (false only for cells that start NaN or -inf,
 * which then never change) and the last max takes -FLT_MAX on the first
 * step and val afterwards. */
template <int BED>
__device__ __forceinline__ float thermal_cell(float c,
                                              float w,
                                              float s,
                                              float n,
                                              float e,
                                              float nw,
                                              float sw,
                                              float ne,
                                              float se,
                                              float talus,
                                              float bedrock,
                                              bool  first = false)
{
  if (BED == BED_LITERAL) return c > bedrock ? c : bedrock;
  if (BED == BED_AUTO)
  {
    if (!(bedrock >= -FLT_MAX)) return c;
    const float x = __fadd_rn(c, thermal_amount(c, w, s, n, e, nw, sw, ne, se, talus));
    const float zn = x > bedrock ? x : bedrock;
    const float fl = first ? -FLT_MAX : c;
    return zn > fl ? zn : fl;
  }
  float out = c;
  if (BED == BED_NONE || c >= bedrock)
    out = __fadd_rn(c, thermal_amount(c, w, s, n, e, nw, sw, ne, se, talus));
  if (BED == BED_INTENDED) out = out > bedrock ? out : bedrock;
  return out;
}

/* The same for two adjacent cells at once, in packed arithmetic
 * (hm_pack.cuh): fewer issue slots per cell, the same bits.
 * Each exchange is the scalar one, operation by operation: the difference
 * of the heights, the products and the sums are packed; the absolute value
 * (packed instructions take none), the max and the sign go per half.
 * No packed product feeds a packed add or subtract directly: diag_talus2
 * forms none, and a copysign or the last fma of the division lies between
 * the others and the sum. */
__device__ __forceinline__ F2 copysign2(F2 mag, F2 sgn)
{
  /* mag is not negative */
  F2 r;
  asm("{\n.reg .b32 a, b, c, d;\nmov.b64 {a, b}, %1;\nmov.b64 {c, d}, %2;\n"
      "lop3.b32 a, a, c, 0x80000000, 0xf8;\nlop3.b32 b, b, d, 0x80000000, 0xf8;\nmov.b64 %0, {a, b};\n}"
      : "=l"(r.v)
      : "l"(mag.v), "l"(sgn.v));
  return r;
}

/* 0.2 * max(|n| - t, 0) for both halves.  (max(|n|, t) - t would leave one
 * scalar instruction per half, but is NaN for an infinite or NaN t, and
 * bounding t first is wrong where |n| is beyond the bound.) */
__device__ __forceinline__ F2 exch2(F2 n, F2 t)
{
  const float2 a = up(n);
  const float2 x = up(sub2(pk(fabsf(a.x), fabsf(a.y)), t));
  return mul2(pk(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)), pk1(0.2f));
}

__device__ __forceinline__ F2 exch_axial2(F2 self, F2 other, F2 t)
{
  const F2 n = sub2(other, self);
  return copysign2(exch2(n, t), n);
}

__device__ __forceinline__ F2 exch_diag2(F2 self, F2 other, F2 md)
{
  const F2 n = sub2(other, self);
  const F2 x = exch2(n, md);
  const F2 y = pk1(0x1.6a17e6p-1f); /* div_by_diag */
  const F2 q = mul2(x, y);
  const F2 r = fma2(q, pk1(-1.414f), x);
  return copysign2(fma2(r, y, q), n);
}

/* 1.414 t, which exch2 subtracts: two scalar products, or, PACKED, one fma
 * that cannot be contracted (mul2r; blocks are flat, so threadIdx.z is a
 * zero the compiler does not know) */
template <bool PACKED>
__device__ __forceinline__ F2 diag_talus2(F2 t)
{
  if (PACKED) return mul2r(pk1(1.414f), t, pk1(__uint_as_float(0x80000000u | threadIdx.z)));
  return pk(__fmul_rn(1.414f, lo(t)), __fmul_rn(1.414f, hi(t)));
}

__device__ __forceinline__ F2 thermal_amount2(F2 c, F2 w, F2 s, F2 n, F2 e, F2 nw, F2 sw, F2 ne, F2 se, F2 t, F2 md)
{
  F2 a = exch_axial2(c, w, t);
  a = add2(a, exch_axial2(c, s, t));
  a = add2(a, exch_axial2(c, n, t));
  a = add2(a, exch_axial2(c, e, t));
  a = add2(a, exch_diag2(c, nw, md));
  a = add2(a, exch_diag2(c, sw, md));
  a = add2(a, exch_diag2(c, ne, md));
  a = add2(a, exch_diag2(c, se, md));
  return a;
}

/* thermal_cell for two adjacent cells */
template <int BED>
__device__ __forceinline__ F2 thermal_cell2(F2 c, F2 w, F2 s, F2 n, F2 e, F2 nw, F2 sw, F2 ne, F2 se, F2 t, F2 bed,
                                            bool first)
{
  const float2 v = up(c), b = up(bed);
  if (BED == BED_LITERAL) return pk(v.x > b.x ? v.x : b.x, v.y > b.y ? v.y : b.y);
  /* (auto-bedrock's sweep has two registers too many for seven CTAs per SM
   * with the scalar products: 96 steps at 2048 x 2048 1.53 against 1.40 ms;
   * the block kernel of the other modes is 3 to 5 % faster with them) */
  const F2     md = diag_talus2<BED == BED_AUTO>(t);
  const F2     x2 = add2(c, thermal_amount2(c, w, s, n, e, nw, sw, ne, se, t, md));
  if (BED == BED_NONE) return x2;
  const float2 x = up(x2);
  /* val < bedrock leaves the bedrock, so both tests of thermal_cell end in
   * one select */
  if (BED == BED_INTENDED)
    return pk(v.x >= b.x && x.x > b.x ? x.x : b.x, v.y >= b.y && x.y > b.y ? x.y : b.y);
  const float zx = x.x > b.x ? x.x : b.x, zy = x.y > b.y ? x.y : b.y;
  const float fx = first ? -FLT_MAX : v.x, fy = first ? -FLT_MAX : v.y;
  return pk(b.x >= -FLT_MAX ? (zx > fx ? zx : fx) : v.x, b.y >= -FLT_MAX ? (zy > fy ? zy : fy) : v.y);
}

} // namespace hm

#endif
