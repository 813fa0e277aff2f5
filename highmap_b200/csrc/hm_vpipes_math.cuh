/*
 * hm_vpipes_math.cuh - per-cell arithmetic of the virtual-pipes passes,
 * rounded exactly as the reference's fp32 kernel text evaluates it.
 *
 * Reference: HighMap/src/gpu_opencl/kernels/hydraulic_vpipes.cl
 *   flow pass         :5-69     water pass  :71-116
 *   erosion pass      :118-184  advection   :186-211
 * and the host steps of HighMap/src/erosion/hydraulic_vpipes_gpu.cpp:36-55,
 * :163-169.
 *
 * Every operation is an explicitly rounded intrinsic, so no multiply is
 * contracted into an add and each result is the reference's
 * one-rounding-per-operation value.  hypot is evaluated as
 * sqrt(x*x + y*y) in fp64 (both squares exact, one rounding for the sum,
 * a correctly rounded square root, one rounding to fp32), which equals the
 * C library's correctly rounded hypotf used by the CPU oracle.  pow with
 * exponent 1 is the identity; other exponents go through fp64 pow.
 */
#ifndef HM_VPIPES_MATH_CUH
#define HM_VPIPES_MATH_CUH

#include "hm_pack.cuh"

namespace hm
{

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }
/* a / b rounded as fdiv, for dividends that are often zero: +-0 / b for
 * b > 0 (+inf included) is a itself, so it is selected instead and the
 * division is given the dividend 1 there (a zero dividend sends the whole
 * warp down the division's special-operand path).  Any other b divides. */
__device__ __forceinline__ float fdiv_z(float a, float b)
{
  const bool z = a == 0.f && b > 0.f;
  return z ? a : __fdiv_rn(z ? 1.f : a, b);
}
/* the reference's max / min as the oracle spells them: a > b ? a : b */
__device__ __forceinline__ float rmax(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float rmin(float a, float b) { return a < b ? a : b; }
/* rmax(a, b) with NaN only in b and no zeros of opposite sign (or where
 * the sign of a zero does not matter): one instruction instead of a compare
 * and a select */
__device__ __forceinline__ float rmaxn(float a, float b)
{
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ float hyp(float x, float y)
{
  /* x*x is exact in fp64, so the fma's one rounding is that of the sum */
  double dx = (double)x, dy = (double)y;
  return __double2float_rn(__dsqrt_rn(__fma_rn(dx, dx, __dmul_rn(dy, dy))));
}

/* hyp in fp32 arithmetic, with a certificate: ok is cleared where the
 * result is not proven to be hyp's, which the caller then evaluates.
 *
 * With a >= b the magnitudes, p = RN(a a) and s = RN(b b + p): s - p is
 * exact, so (b b - (s - p)) + (a a - p) is s's error up to its own rounding
 * (error-free transformations; Dekker, Numer. Math. 18, 1971).  From r ~
 * 1 / sqrt(s) and g = RN(s r), the root is g + (a a + b b - g g) r / 2 with
 * a relative error of the correction under 2^-20 (one Newton step; the
 * residual s - g g is one fma).  If the correction enlarged and reduced by
 * 1e-5 of itself gives the same float, that is the correctly rounded root,
 * which hyp's two roundings also give.  6 in 10^6 operand pairs fail; so do
 * magnitudes whose squares leave the normal range.  About as many
 * instructions as the fp64 form but none on the conversion and fp64 pipes:
 * 28 against 37 cycles per warp and scheduler.
 * rinv: r, about 1 / hyp. */
__device__ __forceinline__ float hyp_try(float x, float y, bool &ok, float &rinv)
{
  float a, b;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(a) : "f"(fabsf(x)), "f"(fabsf(y)));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(b) : "f"(fabsf(x)), "f"(fabsf(y)));
  const float p = fmul(a, a);
  const float s = __fmaf_rn(b, b, p);
  const float e = fadd(__fmaf_rn(b, b, -fsub(s, p)), __fmaf_rn(a, a, -p));
  float       r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fadd(s, 1.2e-38f)));
  const float g = fmul(s, r);
  const float d = fadd(__fmaf_rn(-g, g, s), e);
  const float lo = __fmaf_rn(d, fmul(r, 0.5f * (1.f - 1e-5f)), g), hi = __fmaf_rn(d, fmul(r, 0.5f * (1.f + 1e-5f)), g);
  /* a zero or above 1e-15 (a zero wraps around); infinities and NaN fail
   * the comparison */
  ok = ok && lo == hi && __float_as_uint(a) - 1u >= 0x26901d7cu;
  rinv = r;
  return lo;
}

/* x / h for h = hyp(1, x) from hyp_try, x >= 1e-3, r its approximate
 * reciprocal: one Newton step, the quotient and one residual correction, the
 * steps of Markstein's division (IBM J. Res. Dev. 34(1), 1990).  The Newton
 * step need not give the correctly rounded reciprocal, so the theorem does
 * not apply; the quotient was compared with the division instead, for every
 * float x from 1e-3 to 7e4 and r off by up to 3 ulp either way, and for 1.6
 * 10^8 larger x, where it is 1.  No operand can leave the normal range. */
__device__ __forceinline__ float div_hyp(float x, float h, float r)
{
  r = __fmaf_rn(r, __fmaf_rn(-h, r, 1.f), r);
  const float q = fmul(x, r);
  return __fmaf_rn(__fmaf_rn(-h, q, x), r, q);
}

template <class T> __device__ __forceinline__ T bc(float v);
template <> __device__ __forceinline__ float bc<float>(float v) { return v; }

__device__ __forceinline__ float powr(float b, float e) { return __double2float_rn(pow((double)b, (double)e)); }

/* Scalars of one vpipes call, prepared on the host with the same float
 * operations the reference performs. */
struct VpConst
{
  int   nx, ny;
  int   ld;          /* row stride of the state grids in floats (>= nx; the caller's grids have rows of nx) */
  float dt;
  float dtga;        /* dt * (gravity * pipe_area)                    */
  float pl;          /* pipe length                                    */
  float pl2;         /* pipe length squared                            */
  float c0, c1;      /* flux diffusion weights (c1 = 1 - 4 c0)         */
  float vel_floor;   /* 0.001 * water_height / dt                      */
  float water_height;
  float ratio;       /* downcutting_max_depth_ratio                     */
  float k_capacity, k_erode, k_depose, k_exp;
  float keep;        /* 1 - dt * evap_rate                              */
  float rps;         /* rain per step                                   */
  float fnx;         /* (float)nx, the slope scale of :156              */
  float nz;          /* -0, unknown to the compiler (mul2r)              */
  float rwh;         /* 1 / water_height                                 */
  int   quot_ok;     /* water_height and vel_floor in quot2's range      */
};

/* Depth at the start of a step: the stored evaporated depth, plus the
 * volume top-up of the previous step ((add * rain) / R, :167-168), plus the
 * optional per-step rain. */
template <bool MAINTAIN, bool RAIN, class T>
__device__ __forceinline__ T depth_d1(T d, T rain, float add, float rvol, float rps)
{
  T dc = d;
  if (MAINTAIN) dc = fadd(d, fdiv(fmul(bc<T>(add), rain), bc<T>(rvol)));
  if (RAIN) dc = fadd(dc, fmul(bc<T>(rps), rain));
  return dc;
}

/* Flow pass for one cell; the height differences are formed
 * as the reference subtracts them: (h0 - z_n) - d1_n.  "s" is j + 1 (the
 * reference's "top"), "n" is j - 1. */
template <bool DIFFUSION, bool PL_ONE, class T>
__device__ __forceinline__ void flow_cell(const VpConst &c,
                                          T zc, T d1c,
                                          T zw, T d1w,
                                          T ze, T d1e,
                                          T zs, T d1s,
                                          T zn, T d1n,
                                          T &fl, T &fr, T &ft, T &fb)
{
  const T zero = bc<T>(0.f);
  T       h0 = fadd(zc, d1c);
  T       dhl = fsub(fsub(h0, zw), d1w);
  T       dhr = fsub(fsub(h0, ze), d1e);
  T       dht = fsub(fsub(h0, zs), d1s);
  T       dhb = fsub(fsub(h0, zn), d1n);
  const T dtga = bc<T>(c.dtga);
  T       ql = fmul(dtga, dhl), qr = fmul(dtga, dhr), qt = fmul(dtga, dht), qb = fmul(dtga, dhb);
  if (!PL_ONE)
  {
    const T pl = bc<T>(c.pl);
    ql = fdiv(ql, pl);
    qr = fdiv(qr, pl);
    qt = fdiv(qt, pl);
    qb = fdiv(qb, pl);
  }
  /* (a flux is never -0, so neither is its sum with a product) */
  T nl = rmaxn(zero, fadd(fl, ql));
  T nr = rmaxn(zero, fadd(fr, qr));
  T nt = rmaxn(zero, fadd(ft, qt));
  T nb = rmaxn(zero, fadd(fb, qb));
  if (DIFFUSION)
  {
    const T c1 = bc<T>(c.c1);
    T       f_diff = fmul(bc<T>(c.c0), fadd(fadd(fadd(nl, nr), nt), nb));
    nl = fadd(fmul(c1, nl), f_diff);
    nr = fadd(fmul(c1, nr), f_diff);
    nt = fadd(fmul(c1, nt), f_diff);
    nb = fadd(fmul(c1, nb), f_diff);
  }
  T sum = fadd(fadd(fadd(nl, nr), nt), nb);
  /* k = sum > 1e-5 ? d1 * l * l / (sum * dt) : 0, clamped to [0, 1]; with
   * l = 1 the two products are d1 itself (x * 1 is exact for every x) */
  const T num = PL_ONE ? d1c : fmul(fmul(d1c, bc<T>(c.pl)), bc<T>(c.pl));
  /* where the quotient is discarded (sum <= 1e-5 or NaN: pits have
   * sum = 0, and d1 / 0 takes the division's special-operand path) the
   * divisor is 1 */
  const bool wet = sum > bc<T>(1e-5f);
  T          kq = fdiv(num, wet ? fmul(sum, bc<T>(c.dt)) : bc<T>(1.f));
  T          k = wet ? __saturatef(kq) : zero; /* NaN clamps to 0, as k > 0 ? k : 0 does */
  fl = fmul(nl, k);
  fr = fmul(nr, k);
  ft = fmul(nt, k);
  fb = fmul(nb, k);
}

/* Water pass for one cell: new depth d2 and velocity (u, v).
 * frw = fr(i-1, j), fle = fl(i+1, j), ftn = ft(i, j-1), fbs = fb(i, j+1). */
template <bool PL_ONE, class T>
__device__ __forceinline__ void water_cell(const VpConst &c,
                                           T d1c,
                                           T flc, T frc, T ftc, T fbc,
                                           T frw, T fle, T ftn, T fbs,
                                           T &d2, T &u, T &v)
{
  T dv = fmul(bc<T>(c.dt), fsub(fsub(fsub(fsub(fadd(fadd(fadd(frw, ftn), fle), fbs), flc), frc), ftc), fbc));
  d2 = rmaxn(bc<T>(0.f), fadd(d1c, PL_ONE ? dv : fdiv(dv, bc<T>(c.pl2))));
  T un = fmul(bc<T>(0.5f), fsub(fadd(fsub(frw, flc), frc), fle));
  T vn = fmul(bc<T>(0.5f), fsub(fadd(fsub(ftn, fbc), ftc), fbs));
  T dmean = rmaxn(bc<T>(c.vel_floor), d2);
  u = fdiv(un, dmean);
  v = fdiv(vn, dmean);
}

/* Erosion / deposition for one cell from the old z and s around it. */
template <bool KEXP_ONE, class T>
__device__ __forceinline__ void erosion_cell(const VpConst &c,
                                             T zc, T sc,
                                             T zw, T ze, T zn, T zs,
                                             T sw, T se, T sn, T ss,
                                             T d2, T u, T v,
                                             T &z_out, T &s_out)
{
  const T half = bc<T>(0.5f);
  T       dzx = fmul(half, fsub(fadd(fsub(ze, zw), se), sw));
  T       dzy = fmul(half, fsub(fadd(fsub(zs, zn), ss), sn));
  bool    ok = true;
  float   ri;
  T       speed = hyp_try(u, v, ok, ri);
  T       dzn = rmaxn(bc<T>(1e-3f), fmul(bc<T>(c.fnx), hyp_try(dzx, dzy, ok, ri)));
  T       h = hyp_try(bc<T>(1.f), dzn, ok, ri);
  T       sa = div_hyp(dzn, h, ri);
  if (!ok)
  {
    speed = hyp(u, v);
    dzn = rmaxn(bc<T>(1e-3f), fmul(bc<T>(c.fnx), hyp(dzx, dzy)));
    sa = fdiv(dzn, hyp(bc<T>(1.f), dzn));
  }
  T       salpha = rmaxn(bc<T>(0.01f), sa);
  /* d2 is zero on dry cells (about 6 % of the cells after a few hundred
   * steps of the 4096^2 benchmark, in over 90 % of the warps) */
  T       depth = rmin(fdiv_z(d2, bc<T>(c.water_height)), bc<T>(c.ratio));
  T       discharge = fmul(depth, speed);
  T       pw = KEXP_ONE ? discharge : powr(discharge, c.k_exp);
  T       capa = fmul(fmul(bc<T>(c.k_capacity), pw), salpha);
  /* erosion moves k_erode (capa - s) from z to s, deposition k_depose
   * (s - capa) from s to z: the same sums with the sign of the difference
   * in the product (rounding is symmetric) */
  T m = fmul(capa > sc ? bc<T>(c.k_erode) : bc<T>(c.k_depose), fsub(capa, sc));
  z_out = fsub(zc, m);
  s_out = fadd(sc, m);
}

/* ---- two adjacent cells in packed arithmetic (hm_pack.cuh) ------------
 * Pipe length and discharge exponent 1: the scalar passes operation by
 * operation, divisions and selects per half.  The step is bound by issue
 * slots (77 % busy at 2048 x 2048), and a packed operation takes one slot
 * for two cells: 100 steps with rain 24.5 -> 23.6 ms at 4096 x 4096, 6.70 ->
 * 6.55 ms at 2048 x 2048; with the top-up 33.0 -> 32.6 ms.  The step kernel
 * has no register to spare (48): the first two hypots of the erosion pass
 * stay per cell, because packed they cost spills and 10 % of the step. */

__device__ __forceinline__ F2 max2n(float a, F2 b)
{
  const float2 v = up(b);
  return pk(rmaxn(a, v.x), rmaxn(a, v.y));
}

/* Quotients of pairs.  y = 1 / b after one Newton step from the hardware's
 * approximation is the correctly rounded reciprocal (every mantissa was
 * compared with __frcp_rn), and one residual correction then rounds the
 * quotient correctly (Markstein, IBM J. Res. Dev. 34(1), 1990; the only
 * operands that could fail are those whose quotient lies within 4 / (2 b)
 * ulp of a midpoint, b the divisor's integer mantissa, and all 2.9e7 of
 * them were compared with the division).  That needs every intermediate in
 * the normal range: b in [2^-40, 2^60], n zero or at least 2^-60 and the
 * quotient under 2^60, which the callers check; other pairs divide.
 * 3 packed operations for two quotients where each division takes a chain
 * of its own and a branch: 100 steps with rain 23.6 -> 22.8 ms at 4096 x
 * 4096, 1.90 -> 1.85 ms at 1024 x 1024; with the top-up and a rain map 5.0
 * -> 4.87 ms at 1500 x 1500, 2.09 -> 2.05 ms at 1023 x 767. */
__device__ __forceinline__ F2 rcp2(F2 b, F2 &nb)
{
  const float2 v = up(b);
  float        y0, y1;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(v.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(v.y));
  const F2 y = pk(y0, y1);
  nb = mul2(b, pk1(-1.f));
  return fma2(y, fma2(nb, y, pk1(1.f)), y);
}
__device__ __forceinline__ F2 quot2(F2 n, F2 nb, F2 y)
{
  const F2 q = mul2(n, y);
  return fma2(fma2(nb, q, n), y, q);
}
/* least of m and the magnitude of x as an integer, a zero counting as the
 * largest; QUOT_MIN is 2^-60 so mapped */
constexpr unsigned QUOT_MIN = 0x42ffffffu; /* 2 * bits(2^-60) - 1 */
__device__ __forceinline__ unsigned quot_min(unsigned m, float x) { return min(m, 2u * __float_as_uint(x) - 1u); }
constexpr float QUOT_MAX = 1152921504606846976.f; /* 2^60 */

/* depth_d1's top-up term (add * rain) / rvol for a pair, y the reciprocal of
 * rvol and ok rvol in quot2's range */
__device__ __forceinline__ F2 top_up_pair(F2 rain, float add, float rvol, float y, bool ok)
{
  const float2 n = up(mul2(pk1(add), rain));
  const float2 q = up(quot2(pk(n), pk1(-rvol), pk1(y)));
  if (ok && quot_min(quot_min(~0u, n.x), n.y) >= QUOT_MIN && fadd(fabsf(q.x), fabsf(q.y)) < QUOT_MAX)
    return pk(copysignf(q.x, n.x), copysignf(q.y, n.y)); /* rvol > 0: the sign of n, of a zero too */
  return pk(fdiv(n.x, rvol), fdiv(n.y, rvol));
}

/* flow_cell for a pair; w and e are the pairs one column to the west and
 * to the east */
template <bool DIFFUSION>
__device__ __forceinline__ void flow_pair(const VpConst &c, F2 zc, F2 d1c, F2 zw, F2 d1w, F2 ze, F2 d1e, F2 zs, F2 d1s,
                                          F2 zn, F2 d1n, F2 &fl, F2 &fr, F2 &ft, F2 &fb)
{
  const F2 nz = pk1(c.nz), dtga = pk1(c.dtga);
  const F2 h0 = add2(zc, d1c);
  F2 nl = max2n(0.f, add2(fl, mul2r(dtga, sub2(sub2(h0, zw), d1w), nz)));
  F2 nr = max2n(0.f, add2(fr, mul2r(dtga, sub2(sub2(h0, ze), d1e), nz)));
  F2 nt = max2n(0.f, add2(ft, mul2r(dtga, sub2(sub2(h0, zs), d1s), nz)));
  F2 nb = max2n(0.f, add2(fb, mul2r(dtga, sub2(sub2(h0, zn), d1n), nz)));
  if (DIFFUSION)
  {
    const F2 c1 = pk1(c.c1);
    const F2 f_diff = mul2r(pk1(c.c0), add2(add2(add2(nl, nr), nt), nb), nz);
    nl = add2(mul2r(c1, nl, nz), f_diff);
    nr = add2(mul2r(c1, nr, nz), f_diff);
    nt = add2(mul2r(c1, nt, nz), f_diff);
    nb = add2(mul2r(c1, nb, nz), f_diff);
  }
  const F2     sum2 = add2(add2(add2(nl, nr), nt), nb);
  const float2 sum = up(sum2), den = up(mul2(sum2, pk1(c.dt))), d = up(d1c);
  const bool   wx = sum.x > 1e-5f, wy = sum.y > 1e-5f;
  /* (quot2 gains nothing here, one divisor for one quotient: 100 steps with
   * the defaults at 1024 x 1056 2.54 ms, divided 2.46) */
  const float qx = __saturatef(fdiv(d.x, wx ? den.x : 1.f)), qy = __saturatef(fdiv(d.y, wy ? den.y : 1.f));
  const F2    k = pk(wx ? qx : 0.f, wy ? qy : 0.f);
  fl = mul2(nl, k);
  fr = mul2(nr, k);
  ft = mul2(nt, k);
  fb = mul2(nb, k);
}

/* water_cell for a pair, and erosion_cell's depth ratio min(d2 /
 * water_height, ratio) */
__device__ __forceinline__ void water_pair(const VpConst &c, F2 d1c, F2 flc, F2 frc, F2 ftc, F2 fbc, F2 frw, F2 fle,
                                           F2 ftn, F2 fbs, F2 &d2, F2 &u, F2 &v, F2 &depth)
{
  const F2 half = pk1(0.5f);
  const F2 in = add2(add2(add2(frw, ftn), fle), fbs);
  d2 = max2n(0.f, add2(d1c, mul2r(pk1(c.dt), sub2(sub2(sub2(sub2(in, flc), frc), ftc), fbc), pk1(c.nz))));
  /* (the numerators before the halving: halving could round one to -0) */
  const F2 un2 = sub2(add2(sub2(frw, flc), frc), fle), vn2 = sub2(add2(sub2(ftn, fbc), ftc), fbs);
  const F2 un = mul2(half, un2), vn = mul2(half, vn2), dm = max2n(c.vel_floor, d2);
  F2       nb;
  const F2 y = rcp2(dm, nb);
  u = quot2(un, nb, y);
  v = quot2(vn, nb, y);
  F2 dq = quot2(d2, pk1(-c.water_height), pk1(c.rwh));
  unsigned m = quot_min(quot_min(quot_min(~0u, lo(d2)), hi(d2)), lo(un2));
  m = quot_min(quot_min(quot_min(m, hi(un2)), lo(vn2)), hi(vn2));
  const float t = fadd(fadd(fadd(fabsf(lo(u)), fabsf(hi(u))), fadd(fabsf(lo(v)), fabsf(hi(v)))), fadd(lo(d2), hi(d2)));
  if (!(c.quot_ok && m >= QUOT_MIN && t < QUOT_MAX))
  {
    const float2 a = up(un), b = up(vn), e = up(dm), d = up(d2);
    u = pk(fdiv(a.x, e.x), fdiv(a.y, e.y));
    v = pk(fdiv(b.x, e.x), fdiv(b.y, e.y));
    dq = pk(fdiv(d.x, c.water_height), fdiv(d.y, c.water_height));
  }
  depth = pk(rmin(lo(dq), c.ratio), rmin(hi(dq), c.ratio));
}

/* hyp_try for a pair */
__device__ __forceinline__ F2 hyp_try2(F2 x2, F2 y2, F2 nz, bool &ok, F2 &rinv)
{
  const float2 x = up(x2), y = up(y2);
  float        a0, a1, b0, b1;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(a0) : "f"(fabsf(x.x)), "f"(fabsf(y.x)));
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(a1) : "f"(fabsf(x.y)), "f"(fabsf(y.y)));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(b0) : "f"(fabsf(x.x)), "f"(fabsf(y.x)));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(b1) : "f"(fabsf(x.y)), "f"(fabsf(y.y)));
  const F2 a = pk(a0, a1), b = pk(b0, b1), m1 = pk1(-1.f);
  const F2 p = mul2r(a, a, nz);
  const F2 s = fma2(b, b, p);
  const F2 e = add2(fma2(b, b, sub2(p, s)), fma2(a, a, mul2(p, m1)));
  const float2 st = up(add2(s, pk1(1.2e-38f)));
  float        r0, r1;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(st.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(st.y));
  const F2     r = pk(r0, r1);
  const F2     g = mul2(s, r);
  const F2     d = add2(fma2(mul2(g, m1), g, s), e);
  const F2     l2 = fma2(d, mul2(r, pk1(0.5f * (1.f - 1e-5f))), g);
  const float2 lo = up(l2), hi = up(fma2(d, mul2(r, pk1(0.5f * (1.f + 1e-5f))), g));
  ok = ok && lo.x == hi.x && lo.y == hi.y && __float_as_uint(a0) - 1u >= 0x26901d7cu &&
       __float_as_uint(a1) - 1u >= 0x26901d7cu;
  rinv = r;
  return l2;
}

/* erosion_cell for a pair; depth from water_pair */
__device__ __forceinline__ void erosion_pair(const VpConst &c, F2 zc, F2 sc, F2 zw, F2 ze, F2 zn, F2 zs, F2 sw, F2 se,
                                             F2 sn, F2 ss, F2 depth, F2 u, F2 v, F2 &z_out, F2 &s_out)
{
  const F2 nz = pk1(c.nz), half = pk1(0.5f);
  const F2 dzx = mul2(half, sub2(add2(sub2(ze, zw), se), sw));
  const F2 dzy = mul2(half, sub2(add2(sub2(zs, zn), ss), sn));
  bool     ok = true;
  float    r0, r1;
  F2       r;
  F2       speed = pk(hyp_try(lo(u), lo(v), ok, r0), hyp_try(hi(u), hi(v), ok, r1));
  F2       dzn = max2n(1e-3f, mul2(pk1(c.fnx), pk(hyp_try(lo(dzx), lo(dzy), ok, r0), hyp_try(hi(dzx), hi(dzy), ok, r1))));
  const F2 h = hyp_try2(pk1(1.f), dzn, nz, ok, r);
  /* div_hyp */
  const F2 nh = mul2(h, pk1(-1.f));
  r = fma2(r, fma2(nh, r, pk1(1.f)), r);
  F2 sa = mul2(dzn, r);
  sa = fma2(fma2(nh, sa, dzn), r, sa);
  if (!ok)
  {
    const float2 uu = up(u), vv = up(v), gx = up(dzx), gy = up(dzy);
    speed = pk(hyp(uu.x, vv.x), hyp(uu.y, vv.y));
    const float n0 = rmaxn(1e-3f, fmul(c.fnx, hyp(gx.x, gy.x))), n1 = rmaxn(1e-3f, fmul(c.fnx, hyp(gx.y, gy.y)));
    sa = pk(fdiv(n0, hyp(1.f, n0)), fdiv(n1, hyp(1.f, n1)));
  }
  const F2     capa = mul2r(mul2(pk1(c.k_capacity), mul2(depth, speed)), max2n(0.01f, sa), nz);
  const float2 cp = up(capa), s = up(sc);
  const F2     kk = pk(cp.x > s.x ? c.k_erode : c.k_depose, cp.y > s.y ? c.k_erode : c.k_depose);
  const F2     m = mul2r(kk, sub2(capa, sc), nz);
  z_out = sub2(zc, m);
  s_out = add2(sc, m);
}

/* Mirror an unnormalised coordinate with period 2 * n (texel units):
 * |x - 2n * rint(x / 2n)|.  For |x| <= n the quotient rounds to at most
 * 1/2 in magnitude and rint gives +-0, so the result is |x| exactly; the
 * division is skipped there. */
__device__ __forceinline__ float mirror_coord(float x, int n)
{
  const float ax = fabsf(x);
  if (ax <= (float)n) return ax;
  float period = (float)(2 * n);
  float r = rintf(fdiv(x, period));
  return fabsf(fsub(x, fmul(period, r)));
}

/* Bilinear sample weights and texel indices of the linear sampler at
 * (x, y): texel centres at k + 0.5, mirrored repeat, indices clamped. */
struct Tap
{
  int   i0, i1, j0, j1;
  float a, b;
};

__device__ __forceinline__ Tap linear_tap(float x, float y, int nx, int ny)
{
  float xm = fsub(mirror_coord(x, nx), 0.5f);
  float ym = fsub(mirror_coord(y, ny), 0.5f);
  float fx = floorf(xm), fy = floorf(ym);
  Tap   t;
  t.a = fsub(xm, fx);
  t.b = fsub(ym, fy);
  /* after mirroring fx lies in [-1, nx - 1]; the clamp only matters for
   * coordinates too large to mirror exactly and keeps the taps in the grid */
  t.i0 = (int)fminf(fmaxf(fx, -1.f), (float)(nx - 1));
  t.j0 = (int)fminf(fmaxf(fy, -1.f), (float)(ny - 1));
  t.i1 = t.i0 + 1;
  t.j1 = t.j0 + 1;
  t.i0 = t.i0 < 0 ? 0 : t.i0;
  t.j0 = t.j0 < 0 ? 0 : t.j0;
  t.i1 = t.i1 > nx - 1 ? nx - 1 : t.i1;
  t.j1 = t.j1 > ny - 1 ? ny - 1 : t.j1;
  return t;
}

__device__ __forceinline__ float blend(const Tap &t, float s00, float s10, float s01, float s11)
{
  float oma = fsub(1.f, t.a), omb = fsub(1.f, t.b);
  float r = fmul(fmul(oma, omb), s00);
  r = fadd(r, fmul(fmul(t.a, omb), s10));
  r = fadd(r, fmul(fmul(oma, t.b), s01));
  r = fadd(r, fmul(fmul(t.a, t.b), s11));
  return r;
}

} // namespace hm

#endif
