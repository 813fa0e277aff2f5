/*
 * hm_thermal_sweep.cuh - one Jacobi step of the talus exchange for the 32
 * columns of one warp, walking down a range of rows.  Used by the plain
 * one-step kernel (hm_thermal.cu) and by the thermal tiles of the batched
 * form (hm_batch.cu).
 *
 * Every row of z is loaded once per warp (lanes 0 and 31 also load the
 * column just outside the warp) and the west / east neighbours come from
 * warp shuffles, so a cell costs two coalesced loads per 32 cells instead
 * of nine loads.  The loads of P rows (z, talus, bedrock; a template
 * parameter) are issued before any of them is used, which keeps enough
 * bytes in flight to cover the HBM latency: the plain kernels take 8 (4
 * row pairs), the batched form's persistent kernel fewer, as its
 * occupancy hides the latency instead.  z is read by plain loads (the
 * launch before may have written it, hm_chain.cuh), talus and bedrock,
 * constant for the whole solve, by non-coherent ones.  Cell rule and border copies as the reference kernel
 * (HighMap/src/gpu_opencl/kernels/thermal.cl:26-100, Jacobi form; border
 * copies _common_index.cl:106-132).
 */
#ifndef HM_THERMAL_SWEEP_CUH
#define HM_THERMAL_SWEEP_CUH

#include "hm_thermal_math.cuh"

namespace hm
{

constexpr int SW_P = 8; /* rows whose loads are issued together */

/* Cell rules of the sweeps: R::cell(c, w, s, n, e, nw, sw, ne, se, talus,
 * extra, first, param) is the new value of an interior cell from its 3 x 3
 * neighbourhood (named by position: w = (i-1, j), s = (i, j+1), n =
 * (i, j-1), ...), its talus, the value of the optional per-cell grid
 * `extra` (R::EXTRA), the first-step flag and a scalar parameter;
 * R::pair is the same for two adjacent cells at once (hm_pack.cuh). */
template <int BED>
struct TalusExchange
{
  static constexpr bool EXTRA = BED != BED_NONE;
  __device__ static __forceinline__ float cell(float c, float w, float s, float n, float e, float nw, float sw,
                                               float ne, float se, float t, float x, bool first, float)
  {
    return thermal_cell<BED>(c, w, s, n, e, nw, sw, ne, se, t, x, first);
  }
  __device__ static __forceinline__ F2 pair(F2 c, F2 w, F2 s, F2 n, F2 e, F2 nw, F2 sw, F2 ne, F2 se, F2 t, F2 x,
                                            bool first, float)
  {
    return thermal_cell2<BED>(c, w, s, n, e, nw, sw, ne, se, t, x, first);
  }
};

/* Columns wx .. wx+31 (lane = column; columns past nx only feed the
 * shuffles), output rows y0 .. y1-1, the loads of P rows in flight
 * together.  The whole warp must call it. */
template <bool TMAP, class R, int P = SW_P>
__device__ __forceinline__ void thermal_sweep_warp(const float *a,
                                                   float *__restrict__ b,
                                                   int nx,
                                                   int ny,
                                                   const float *__restrict__ talus,
                                                   float talus_value,
                                                   const float *__restrict__ bedrock,
                                                   int first,
                                                   int wx,
                                                   int y0,
                                                   int y1,
                                                   float param = 0.f)
{
  const int  lane = threadIdx.x & 31;
  const int  gx = wx + lane;
  const bool live = gx < nx;
  const int  gxc = live ? gx : nx - 1;
  /* lanes 0 and 31 also load the column west / east of the warp */
  const int  hx = lane == 0 ? max(wx - 1, 0) : (lane == 31 ? min(wx + 32, nx - 1) : gxc);

  float vc[P + 2], vl[P + 2], vr[P + 2];
  {
    const float *r0 = a + (size_t)max(y0 - 1, 0) * nx, *r1 = a + (size_t)y0 * nx;
    vc[0] = r0[gxc];
    vl[0] = r0[hx];
    vc[1] = r1[gxc];
    vl[1] = r1[hx];
#pragma unroll
    for (int q = 0; q < 2; q++)
    {
      const float up = __shfl_up_sync(0xffffffffu, vc[q], 1), dn = __shfl_down_sync(0xffffffffu, vc[q], 1);
      vr[q] = lane == 31 ? vl[q] : dn;
      vl[q] = lane == 0 ? vl[q] : up;
    }
  }
  for (int j0 = y0; j0 < y1; j0 += P)
  {
    float tl[P], bd[P];
#pragma unroll
    for (int q = 0; q < P; q++)
    {
      const float *r = a + (size_t)min(j0 + 1 + q, ny - 1) * nx;
      vc[q + 2] = r[gxc];
      vl[q + 2] = r[hx]; /* the halo value until the shuffles below */
      const size_t o = (size_t)min(j0 + q, ny - 1) * nx + gxc;
      tl[q] = TMAP ? __ldg(talus + o) : talus_value;
      bd[q] = R::EXTRA ? __ldg(bedrock + o) : 0.f;
    }
#pragma unroll
    for (int q = 2; q < P + 2; q++)
    {
      const float up = __shfl_up_sync(0xffffffffu, vc[q], 1), dn = __shfl_down_sync(0xffffffffu, vc[q], 1);
      vr[q] = lane == 31 ? vl[q] : dn;
      vl[q] = lane == 0 ? vl[q] : up;
    }
#pragma unroll
    for (int q = 0; q < P; q++)
    {
      const int j = j0 + q;
      if (!live || j >= y1) continue;
      float out;
      /* apply_boundaries, _common_index.cl:106-132 */
      if (gx == 0) out = vr[q + 1];
      else if (gx == nx - 1) out = vl[q + 1];
      else if (j == 0) out = vc[q + 2];
      else if (j == ny - 1) out = vc[q];
      else
        out = R::cell(vc[q + 1], vl[q + 1], vc[q + 2], vc[q], vr[q + 1], vl[q], vl[q + 2], vr[q], vr[q + 2], tl[q],
                      bd[q], first != 0, param);
      b[(size_t)j * nx + gx] = out;
    }
    vc[0] = vc[P];
    vl[0] = vl[P];
    vr[0] = vr[P];
    vc[1] = vc[P + 1];
    vl[1] = vl[P + 1];
    vr[1] = vr[P + 1];
  }
}


/* The same sweep with two adjacent columns per lane (a warp owns the 64
 * columns wx .. wx+63): z, talus and bedrock move as 8-byte pairs, one
 * pair of shuffles per row serves both cells, and the cell rule runs on
 * both in packed arithmetic (R::pair).  Needs an even nx and 8-byte aligned
 * grids; identical bits to thermal_sweep_warp. */
constexpr int S2_P = 4; /* rows whose loads are issued together */

__device__ __forceinline__ F2 ldg2(const float *p)
{
  F2 r;
  r.v = __ldg(reinterpret_cast<const unsigned long long *>(p));
  return r;
}
__device__ __forceinline__ F2 ld2(const float *p)
{
  F2 r;
  r.v = *reinterpret_cast<const unsigned long long *>(p);
  return r;
}
__device__ __forceinline__ void st2(float *p, F2 v) { *reinterpret_cast<unsigned long long *>(p) = v.v; }

/* One row of a lane's column pair: the pair (x, y), the pair one column to
 * the west (w, x) and the pair one column to the east (y, e). */
struct PairRow
{
  F2 c, w, e;
};

/* the shifted pairs of a row from the neighbouring lanes' pairs; halo is
 * the column just outside the warp on lanes 0 and 31 */
__device__ __forceinline__ void pair_exchange(PairRow &r, int lane, float halo)
{
  const float2 c = up(r.c);
  const float  wv = __shfl_up_sync(0xffffffffu, c.y, 1), ev = __shfl_down_sync(0xffffffffu, c.x, 1);
  r.w = pk(lane == 0 ? halo : wv, c.x);
  r.e = pk(c.y, lane == 31 ? halo : ev);
}

template <bool TMAP, class R, int P = S2_P>
__device__ __forceinline__ void thermal_sweep2_warp(const float *a,
                                                    float *__restrict__ b,
                                                    int nx,
                                                    int ny,
                                                    const float *__restrict__ talus,
                                                    float talus_value,
                                                    const float *__restrict__ bedrock,
                                                    int first,
                                                    int wx,
                                                    int y0,
                                                    int y1,
                                                    float param = 0.f)
{
  const int  lane = threadIdx.x & 31;
  const int  gx = wx + 2 * lane; /* first of the lane's two columns (nx is even) */
  const bool live = gx < nx;
  const int  gxc = live ? gx : nx - 2;
  /* lanes 0 and 31 also load the column west / east of the warp */
  const int  hx = lane == 0 ? max(wx - 1, 0) : (lane == 31 ? min(wx + 64, nx - 1) : gxc);

  PairRow    v[P + 2];
  float      halo[P + 2];
  const bool halo_lane = lane == 0 || lane == 31;
  auto load = [&](int r, int q) {
    const float *row = a + (size_t)r * nx;
    v[q].c = ld2(row + gxc);
    halo[q] = halo_lane ? row[hx] : 0.f;
  };
  load(max(y0 - 1, 0), 0);
  load(y0, 1);
  pair_exchange(v[0], lane, halo[0]);
  pair_exchange(v[1], lane, halo[1]);
  for (int j0 = y0; j0 < y1; j0 += P)
  {
    F2 tl[P], bd[P];
#pragma unroll
    for (int q = 0; q < P; q++)
    {
      load(min(j0 + 1 + q, ny - 1), q + 2);
      const size_t o = (size_t)min(j0 + q, ny - 1) * nx + gxc;
      tl[q] = TMAP ? ldg2(talus + o) : pk1(talus_value);
      bd[q] = R::EXTRA ? ldg2(bedrock + o) : pk1(0.f);
    }
#pragma unroll
    for (int q = 2; q < P + 2; q++) pair_exchange(v[q], lane, halo[q]);
    auto cell2 = [&](int q) {
      return R::pair(v[q + 1].c, v[q + 1].w, v[q + 2].c, v[q].c, v[q + 1].e, v[q].w, v[q + 2].w, v[q].e, v[q + 2].e,
                     tl[q], bd[q], first != 0, param);
    };
    /* a warp whose columns and rows are all interior: no border tests
     * (10 % of the step at 4096^2) */
    if (wx > 0 && wx + 64 < nx && j0 > 0 && j0 + P < ny - 1 && j0 + P <= y1)
    {
#pragma unroll
      for (int q = 0; q < P; q++) st2(b + (size_t)(j0 + q) * nx + gx, cell2(q));
    }
    else
    {
#pragma unroll
      for (int q = 0; q < P; q++)
      {
        const int j = j0 + q;
        if (!live || j >= y1) continue;
        /* apply_boundaries, _common_index.cl:106-132: rows 0 and ny - 1
         * copy their inward row, then columns 0 and nx - 1 their inward
         * column */
        F2 out = j == 0 ? v[q + 2].c : (j == ny - 1 ? v[q].c : cell2(q));
        if (gx == 0) out = pk(hi(v[q + 1].c), hi(out));
        if (gx + 1 == nx - 1) out = pk(lo(out), lo(v[q + 1].c));
        st2(b + (size_t)j * nx + gx, out);
      }
    }
    v[0] = v[P];
    v[1] = v[P + 1];
  }
}

} // namespace hm

#endif
