/*
 * hm_vflow.cu - flow_simulation_viscous on sm_100a: water spreading over a
 * fixed terrain as a viscous thin film.
 *
 * Replaces HighMap/src/hydrology/flow_simulation.cpp:112-157 and its
 * kernel shallow_viscous_flow.cl.  Per step (h_in -> h_out, clamp-to-edge
 * reads):
 *   M_face = ((h + h_n) / 2)^power / viscosity       for the four faces,
 *   q = -M (H_n - H_c), H = h + z,
 *   h' = max(0, h - dt ((q_e - q_w) + q_n - q_s)),
 * and every 10 steps, before the step, dt = 0.2 / max(hmax^power /
 * viscosity, 1e-6) (helper_vflow_compute_adaptive_dt, :16-24; the caller's
 * dt is replaced before the first step).  Afterwards the dry-out of
 * water_depth.cpp:40-66.
 *
 * The reference round-trips the depth to the host around every step and
 * takes hmax on the host; here the depth stays in HBM and dt is formed on
 * the device: the launch that ends a group of 10 steps also takes the max
 * over order-preserving integer keys of the depth (exact for negative
 * values too), and its last CTA turns it into the next group's dt.  pow is
 * evaluated in fp64 and rounded once to fp32, which equals the host's powf
 * except where the exact power lies within about 2^-52 of a float rounding
 * boundary.
 *
 * Powers that are multiples of 1/2 from 1 to 4 (the default is 2.5) are
 * x^floor times sqrt(x) in fp64, at most five roundings of 2^-53: the same
 * accuracy at a fifth of pow's instructions.  Those with a square root
 * come from fp32 pairs where the rounding to fp32 is certain (nearly
 * always), off the fp64 pipe and its conversions.
 *
 * Kernels
 *   k_vflow_block  up to VB_TMAX steps per launch on a 64 x 32 tile in
 *                  registers (the layout of hm_thermal_block.cuh: a warp
 *                  owns two rows, two columns per lane), up to 1.5 M
 *                  cells, where a step's launch (4.1 us of host time) is
 *                  longer than its arithmetic: 512^2, power 2.5, 200
 *                  steps 2.51 ms with one step per launch and pow, 0.76 ms
 *                  here (0.86 with the powers in fp64).
 *   k_vflow_step   one step, a 32 x 8 tile in shared memory (larger grids).
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hm_chain.cuh"
#include "hm_internal.h"
#include "hm_vpipes.h"
#include "hm_vpipes_math.cuh"

namespace hm
{

namespace
{

constexpr int VF_NT = 256;
constexpr int VF_GRID = 148 * 8;

/* float -> unsigned key that orders like the values (negatives below
 * positives), and back */
__device__ __forceinline__ unsigned fkey(float v)
{
  const unsigned b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float funkey(unsigned k)
{
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

/* device scalars of a solve: the running max key, the CTAs done, the key
 * of the last finished max and the time step */
struct VfScalars
{
  unsigned slot, ticket, hmax;
  float    dt;
};

/* power 0: the general pow; else twice the power, an integer in 2 .. 8 */
struct VfConst
{
  float viscosity, power;
  int   half;
};

/* x^1.5, x^2.5 or x^3.5 (half 3, 5, 7) rounded as vf_pow rounds them, from
 * fp32 arithmetic in unevaluated sums of two (error-free products;
 * Dekker, Numer. Math. 18, 1971): the root is g + d r / 2 with g = RN(x r),
 * r ~ 1 / sqrt(x), d = x - g g; the power is (h + l)(g + c).  Relative
 * error under 2^-41; ok is cleared unless the float is the same 2^-40 to
 * either side (3 in 10^5 fail), and for x outside [1e-8, 1e8] but 0. */
__device__ __forceinline__ float half_pow_try(float x, int half, bool &ok)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fadd(x, 1.2e-38f)));
  const float g = fmul(x, r);
  const float cr = fmul(fmul(0.5f, r), __fmaf_rn(-g, g, x));
  float       h = x, l = 0.f;
  if (half > 3)
  {
    h = fmul(x, x);
    l = __fmaf_rn(x, x, -h);
    if (half > 5)
    {
      const float h3 = fmul(h, x);
      l = __fmaf_rn(l, x, __fmaf_rn(h, x, -h3));
      h = h3;
    }
  }
  const float p = fmul(h, g);
  const float lo = __fmaf_rn(l, g, __fmaf_rn(h, cr, __fmaf_rn(h, g, -p)));
  const float p1 = fadd(p, __fmaf_rn(p, 0x1p-40f, lo)), p2 = fadd(p, __fmaf_rn(p, -0x1p-40f, lo));
  ok = p1 == p2 && ((x >= 1e-8f && x <= 1e8f) || x == 0.f);
  return p1;
}

/* x^power in fp64, rounded once (header) */
__device__ __forceinline__ float vf_pow(float xf, const VfConst &c)
{
  if (c.half == 0) return powr(xf, c.power);
  if ((c.half & 1) && c.half > 1)
  {
    bool        ok;
    const float p = half_pow_try(xf, c.half, ok);
    if (ok) return p;
  }
  const double x = (double)xf, x2 = __dmul_rn(x, x); /* the square is exact */
  double       r = c.half & 4 ? x2 : 1.0;            /* x^2 of 4 .. 7 halves */
  if (c.half == 8) r = __dmul_rn(x2, x2);
  else if (c.half & 2) r = c.half & 4 ? __dmul_rn(x2, x) : x;
  if (c.half & 1) r = __dmul_rn(r, __dsqrt_rn(x));
  return __double2float_rn(r);
}

__device__ __forceinline__ float face_mobility(float h, float hn, const VfConst &c)
{
  const float p = vf_pow(fmul(0.5f, fadd(h, hn)), c);
  return c.viscosity == 1.f ? p : fdiv(p, c.viscosity); /* p / 1 is p */
}

/* The CTA's part of the max of h, m = the thread's greatest key; the last
 * CTA stores the key, forms dt = 0.2 / fmax(hmax^power / viscosity, 1e-6)
 * and re-arms the slot for the next max. */
__device__ __forceinline__ void vf_max_commit(unsigned m, VfScalars *sc, unsigned nblocks, const VfConst &c)
{
  m = __reduce_max_sync(0xffffffffu, m);
  const unsigned tid = threadIdx.y * blockDim.x + threadIdx.x;
  if ((tid & 31u) == 0) atomicMax(&sc->slot, m);
  __threadfence();
  __syncthreads();
  if (tid != 0) return;
  if (atomicAdd(&sc->ticket, 1u) != nblocks - 1u) return;
  __threadfence();
  const unsigned key = atomicExch(&sc->slot, 0u);
  sc->hmax = key;
  const float p = vf_pow(funkey(key), c);
  sc->dt = fdiv(0.2f, fmaxf(fdiv(p, c.viscosity), 1e-6f));
  sc->ticket = 0u;
}

/* h = water_height * depth_map, its max and the first time step */
__global__ void __launch_bounds__(VF_NT) k_vflow_init(float *__restrict__ h, const float *__restrict__ depth_map,
                                                      float water_height, size_t n, VfScalars *sc, VfConst c)
{
  unsigned m = 0u;
  for (size_t k = blockIdx.x * (size_t)VF_NT + threadIdx.x; k < n; k += (size_t)gridDim.x * VF_NT)
  {
    const float v = __fmul_rn(water_height, depth_map[k]);
    /* the reference's maximum starts at the first cell and takes what is
     * greater: a NaN counts there and is passed over elsewhere (steps leave
     * no NaN) */
    const unsigned key = v == v ? fkey(v) : (k == 0 ? ~0u : 0u);
    h[k] = v;
    m = key > m ? key : m;
  }
  vf_max_commit(m, sc, gridDim.x, c);
}

/* One step over a 32 x 8 tile.  Each face mobility is evaluated once, by
 * the thread of the cell west / south of it (plus the tile's west and
 * south edges), into shared memory; a face is the same value for the two
 * cells it separates (fadd is commutative), so this equals evaluating it
 * from both sides, at about half the pow calls.  Faces on the grid's edge
 * pair a cell with itself, as the clamped reads do.  GENERAL: a power that
 * needs pow, without the code of the half-integer ones beside it (power 2.2,
 * 20 steps at 2048 x 2048 2.48 -> 2.35 ms). */
constexpr int VT_X = 32, VT_Y = 8;

template <bool GENERAL>
__global__ void __launch_bounds__(VT_X *VT_Y) k_vflow_step(const float *__restrict__ z, const float *hin,
                                                          float *__restrict__ hout, int nx, int ny, VfScalars *sc,
                                                          VfConst c, int want_max)
{
  if (GENERAL) c.half = 0;
  __shared__ float me[VT_Y][VT_X + 1]; /* me[ty][tx + 1]: east face of (tx, ty); [ty][0]: west edge  */
  __shared__ float mn[VT_Y + 1][VT_X]; /* mn[ty + 1][tx]: north face of (tx, ty); [0][tx]: south edge */
  chain_wait();
  hin = produced(hin);
  const int  tx = threadIdx.x, ty = threadIdx.y;
  const int  i = blockIdx.x * VT_X + tx, j = blockIdx.y * VT_Y + ty;
  const bool in = i < nx && j < ny;
  const int  ic = in ? i : 0, jc = in ? j : 0;
  const size_t k = (size_t)jc * nx + ic;
  const size_t ke = ic < nx - 1 ? k + 1 : k, kw = ic > 0 ? k - 1 : k;
  const size_t kn = jc < ny - 1 ? k + nx : k, ks = jc > 0 ? k - nx : k; /* j + 1, j - 1 */
  const float  h = hin[k];
  const float  hxp = hin[ke], hxm = hin[kw], hyp = hin[kn], hym = hin[ks];
  if (in)
  {
    me[ty][tx + 1] = face_mobility(h, hxp, c);
    mn[ty + 1][tx] = face_mobility(h, hyp, c);
    if (tx == 0) me[ty][0] = face_mobility(h, hxm, c);
    if (ty == 0) mn[0][tx] = face_mobility(h, hym, c);
  }
  __syncthreads();
  unsigned key = 0u;
  if (in)
  {
    const float dt = sc->dt;
    const float zc = z[k];
    const float Hc = fadd(h, zc);
    const float Hxp = fadd(hxp, z[ke]), Hxm = fadd(hxm, z[kw]), Hyp = fadd(hyp, z[kn]), Hym = fadd(hym, z[ks]);
    const float Mp = me[ty][tx + 1], Mm = me[ty][tx], Myp = mn[ty + 1][tx], Mym = mn[ty][tx];
    const float qxp = fmul(-Mp, fsub(Hxp, Hc));
    const float qxm = fmul(-Mm, fsub(Hc, Hxm));
    const float qyp = fmul(-Myp, fsub(Hyp, Hc));
    const float qym = fmul(-Mym, fsub(Hc, Hym));
    const float dhdt = -fsub(fadd(fsub(qxp, qxm), qyp), qym);
    const float o = fmaxf(0.f, fadd(h, fmul(dt, dhdt)));
    hout[k] = o;
    key = fkey(o);
  }
  if (want_max) vf_max_commit(key, sc, gridDim.x * gridDim.y, c);
}

/* T steps on a tile of 64 columns x 32 rows.  Warp w holds rows 2 w and
 * 2 w + 1 and reads the rows above and below them from shared memory; the
 * terrain around the cells is loaded once for all steps.  Vertical faces
 * are evaluated by the row below them (three per column and step for two
 * rows), horizontal ones by the cell west of them, the value shuffled
 * east.  The halo is that of hm_thermal_block.cuh, one cell per step. */
constexpr int VB_NW = 16, VB_NT = 32 * VB_NW, VB_TY = 2 * VB_NW, VB_TMAX = 5;

template <bool VEC>
__device__ __forceinline__ float2 vb_load(const float *row, int x0, int x1)
{
  return VEC ? *reinterpret_cast<const float2 *>(row + x0) : make_float2(row[x0], row[x1]);
}

template <bool VEC>
__global__ void __launch_bounds__(VB_NT)
    k_vflow_block(const float *__restrict__ z, const float *hin, float *__restrict__ hout, int nx, int ny,
                  VfScalars *sc, VfConst c, int T, int want_max)
{
  __shared__ float2 rows[2][VB_NW][2][32];
  const int  HL = (T + 1) >> 1, W = 64 - 4 * HL;
  const int  lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int  gx = blockIdx.x * W - 2 * HL + 2 * lane;
  const int  j0 = blockIdx.y * (VB_TY - 2 * T) - T + 2 * wp; /* first of the warp's two rows */
  const int  x0 = min(max(gx, 0), VEC ? nx - 2 : nx - 1), x1 = min(max(gx + 1, 0), nx - 1);
  /* the warp's rows are 1, 2 of these; 0 and 3 are their neighbours */
  float2     h[4], zr[4];
  float      zw[2], ze[2]; /* terrain west of the pair and east of it */
#pragma unroll
  for (int q = 0; q < 4; q++)
  {
    const size_t o = (size_t)min(max(j0 + q - 1, 0), ny - 1) * nx;
    zr[q] = vb_load<VEC>(z + o, x0, x1);
    if (q == 1 || q == 2)
    {
      zw[q - 1] = __ldg(z + o + min(max(gx - 1, 0), nx - 1));
      ze[q - 1] = __ldg(z + o + min(max(gx + 2, 0), nx - 1));
    }
  }
  chain_wait();
  hin = produced(hin);
#pragma unroll
  for (int q = 1; q < 3; q++) h[q] = vb_load<VEC>(hin + (size_t)min(max(j0 + q - 1, 0), ny - 1) * nx, x0, x1);
  const float dt = sc->dt;
  const bool  wedge = gx == 0, e0 = gx == nx - 1, e1 = gx + 1 == nx - 1;
  for (int t = 0; t < T; t++)
  {
    const int par = t & 1;
    rows[par][wp][0][lane] = h[1];
    rows[par][wp][1][lane] = h[2];
    __syncthreads();
    if (2 * wp + 1 <= t || 2 * wp >= VB_TY - 1 - t) continue; /* halo rows that are done */
    h[0] = rows[par][max(wp - 1, 0)][1][lane];
    h[3] = rows[par][min(wp + 1, VB_NW - 1)][0][lane];
    /* clamped reads: the row outside the grid is the edge row */
    if (j0 == 0) h[0] = h[1];
    if (j0 == -1) h[1] = h[2];
    if (j0 == ny - 1) h[2] = h[1];
    if (j0 + 1 == ny - 1) h[3] = h[2];
    /* vertical faces below row 1, between rows 1 and 2, above row 2 */
    float2 my[3];
#pragma unroll
    for (int q = 0; q < 3; q++)
      my[q] = make_float2(face_mobility(h[q].x, h[q + 1].x, c), face_mobility(h[q].y, h[q + 1].y, c));
    float2 o[2];
#pragma unroll
    for (int q = 1; q < 3; q++)
    {
      const float2 hc = h[q];
      float        hw = __shfl_up_sync(0xffffffffu, hc.y, 1), he = __shfl_down_sync(0xffffffffu, hc.x, 1);
      if (wedge) hw = hc.x;
      if (e1) he = hc.y;
      const float hm = e0 ? hc.x : hc.y; /* east of the first column */
      const float mx = face_mobility(hc.x, hm, c), mxe = face_mobility(hc.y, he, c);
      float       mxw = __shfl_up_sync(0xffffffffu, mxe, 1);
      if (wedge) mxw = face_mobility(hw, hc.x, c);
      const float Hc0 = fadd(hc.x, zr[q].x), Hc1 = fadd(hc.y, zr[q].y);
      const float Hw = fadd(hw, zw[q - 1]), He = fadd(he, ze[q - 1]), Hm = fadd(hm, zr[q].y);
      const float Hn0 = fadd(h[q + 1].x, zr[q + 1].x), Hn1 = fadd(h[q + 1].y, zr[q + 1].y);
      const float Hs0 = fadd(h[q - 1].x, zr[q - 1].x), Hs1 = fadd(h[q - 1].y, zr[q - 1].y);
      auto cell = [&](float hh, float Hc, float He_, float Hw_, float Hn, float Hs, float Me, float Mw, float Mn,
                      float Ms) {
        const float qxp = fmul(-Me, fsub(He_, Hc)), qxm = fmul(-Mw, fsub(Hc, Hw_));
        const float qyp = fmul(-Mn, fsub(Hn, Hc)), qym = fmul(-Ms, fsub(Hc, Hs));
        return fmaxf(0.f, fadd(hh, fmul(dt, -fsub(fadd(fsub(qxp, qxm), qyp), qym))));
      };
      o[q - 1].x = cell(hc.x, Hc0, Hm, Hw, Hn0, Hs0, mx, mxw, my[q].x, my[q - 1].x);
      o[q - 1].y = cell(hc.y, Hc1, He, Hc0, Hn1, Hs1, mxe, mx, my[q].y, my[q - 1].y);
    }
    h[1] = o[0];
    h[2] = o[1];
  }
  unsigned key = 0u;
  if (lane >= HL && lane < 32 - HL && gx < nx)
  {
#pragma unroll
    for (int q = 0; q < 2; q++)
    {
      const int tr = 2 * wp + q, j = j0 + q;
      if (tr < T || tr >= VB_TY - T || j >= ny) continue;
      float       *p = hout + (size_t)j * nx + gx;
      const float2 v = h[q + 1];
      if (VEC) *reinterpret_cast<float2 *>(p) = v;
      else
      {
        p[0] = v.x;
        if (gx + 1 < nx) p[1] = v.y;
      }
      const unsigned k0 = fkey(v.x), k1 = gx + 1 < nx ? fkey(v.y) : 0u;
      key = max(key, max(k0, k1));
    }
  }
  if (want_max) vf_max_commit(key, sc, gridDim.x * gridDim.y, c);
}

/* water_depth_dry_out: h -= ratio * hmax, then max(0, h) */
__global__ void __launch_bounds__(VF_NT) k_vflow_dry_out(const float *h, VfScalars *sc,
                                                         float ratio, float *__restrict__ out, size_t n)
{
  chain_wait();
  h = produced(h);
  const float drop = fmul(ratio, funkey(sc->hmax));
  for (size_t k = blockIdx.x * (size_t)VF_NT + threadIdx.x; k < n; k += (size_t)gridDim.x * VF_NT)
  {
    const float w = fsub(h[k], drop);
    out[k] = 0.f < w ? w : 0.f;
  }
}

} // namespace

size_t vflow_scratch_bytes(int nx, int ny)
{
  /* two depth grids, then the scalars */
  return 2 * align_up((size_t)nx * ny, 64) * sizeof(float) + 256;
}

int vflow_check_args(const float *z, const float *depth_map, const float *out, int nx, int ny, int iterations)
{
  if (!z || !depth_map || !out) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation_viscous: NULL grid");
  if (nx < 1 || ny < 1) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation_viscous: nx and ny must be >= 1");
  if ((long long)nx * (long long)ny > (1ll << 34))
    return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation_viscous: grid larger than 2^34 cells");
  if (iterations < 0) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation_viscous: iterations < 0");
  if ((ny + VT_Y - 1) / VT_Y > 65535)
    return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation_viscous: ny larger than 524280 rows");
  return HM_OK;
}

int vflow_core(const float *z, int nx, int ny, float water_height, const float *depth_map, int iterations,
               float dt, float dry_out_ratio, float viscosity, float power, float *water_depth, void *scratch,
               cudaStream_t s)
{
  const size_t n = (size_t)nx * ny;
  const size_t na = align_up(n, 64);
  float       *hA = (float *)scratch, *hB = hA + na;
  VfScalars   *sc = (VfScalars *)(hB + na);
  VfConst      c{viscosity, power, 0};
  for (int half = 2; half <= 8; half++)
    if (power == 0.5f * (float)half) c.half = half;
  (void)dt; /* replaced before the first step */
  HM_CUDA_TRY(cudaMemsetAsync(sc, 0, sizeof(VfScalars), s));
  k_vflow_init<<<VF_GRID, VF_NT, 0, s>>>(hA, depth_map, water_height, n, sc, c);
  HM_LAUNCH_CHECK("k_vflow_init");
  /* Steps per launch: 5 up to 1.5 M cells (two launches per time step
   * update), one above and for the powers that need pow, where the halo's
   * arithmetic (1.8 x at 5) costs more than the launches (power 2.2,
   * 224 x 129: 8.9 us per step with 5, 7.4 with one). */
  const int  per = c.half != 0 && n <= 1500000 ? VB_TMAX : 1;
  auto       al8 = [](const void *p) { return ((uintptr_t)p & 7u) == 0; };
  float     *cur = hA, *nxt = hB;
  for (int it = 0; it < iterations;)
  {
    const int  T = std::min(per, std::min(10 - it % 10, iterations - it));
    const bool last = it + T == iterations;
    /* the depth's max is needed before every tenth step and by the dry-out */
    const int  want_max = ((it + T) % 10 == 0 && !last) || (last && dry_out_ratio != 0.f);
    if (last && dry_out_ratio == 0.f && water_depth != z) nxt = water_depth;
    if (per == 1)
    {
      const dim3 tiles((nx + VT_X - 1) / VT_X, (ny + VT_Y - 1) / VT_Y);
      chain_launch(it > 0, c.half ? k_vflow_step<false> : k_vflow_step<true>, tiles, dim3(VT_X, VT_Y), s, z, cur, nxt, nx, ny, sc, c, want_max);
      HM_LAUNCH_CHECK("k_vflow_step");
    }
    else
    {
      const int  w = 64 - 4 * ((T + 1) / 2), hgt = VB_TY - 2 * T;
      const dim3 tiles((nx + w - 1) / w, (ny + hgt - 1) / hgt);
      const bool vec = nx % 2 == 0 && al8(z) && al8(cur) && al8(nxt);
      chain_launch(it > 0, vec ? k_vflow_block<true> : k_vflow_block<false>, tiles, dim3(VB_NT), s, z, cur, nxt, nx, ny,
                   sc, c, T, want_max);
      HM_LAUNCH_CHECK("k_vflow_block");
    }
    float *t = cur;
    cur = nxt;
    nxt = t;
    it += T;
  }
  if (dry_out_ratio != 0.f)
  {
    chain_launch(iterations > 0, k_vflow_dry_out, dim3(VF_GRID), dim3(VF_NT), s, cur, sc, dry_out_ratio, water_depth, n);
    HM_LAUNCH_CHECK("k_vflow_dry_out");
  }
  else if (cur != water_depth)
    HM_CUDA_TRY(cudaMemcpyAsync(water_depth, cur, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
  return HM_OK;
}

} // namespace hm
