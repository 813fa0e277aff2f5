/*
 * hm_thermal_block.cuh - T Jacobi steps of a 3 x 3 cell rule in one launch
 * (temporal blocking in registers), for the talus exchange and the sibling
 * stencils.
 *
 * A CTA of 16 warps holds a tile of 64 columns x 16 ROWS rows in registers:
 * a warp owns ROWS whole rows, two columns per lane.  Per step, the row
 * above and below a warp's rows come from its neighbours through shared
 * memory (two 8-byte stores and two loads per lane, one barrier) and the
 * west / east columns from two shuffles per row; talus and bedrock are
 * read once for all T steps.  The tile carries a halo of T rows and of T
 * columns (rounded up to a lane), which shrinks by one cell per step.
 *
 * Why: up to about 1.5 M cells a one-step launch is not bound by its
 * arithmetic but by the launch (4.1 us of host time each) and by one
 * warp's walk down its rows: 6.3 us per step from 64^2 to 512^2, 8.3 us at
 * 1024^2.  Here a step inside the launch takes 0.65 us (ROWS 1) or 1.1 us
 * (ROWS 2) on one CTA per SM.  Measured, 48 steps, talus map and bedrock:
 * 1.1 us per step at 64^2, 1.3 at 256^2, 2.0 at 512^2, 5.3 at 1024^2, 6.2
 * at 1200^2 (one step per launch, chained: 4.8, 5.9, 6.0, 6.6, 7.9).  Above,
 * the recomputed halo costs more than the launch: 15.5 against 13.9 us at
 * 2048^2, 62 against 52 us at 4096^2.
 *
 * Every cell follows the one-step rule (border copies of
 * _common_index.cl:106-132, then the cell rule), so T steps here are T
 * one-step launches bit for bit.
 */
#ifndef HM_THERMAL_BLOCK_CUH
#define HM_THERMAL_BLOCK_CUH

#include <cstdint>

#include "hm_chain.cuh"
#include "hm_thermal_sweep.cuh"

namespace hm
{

constexpr int TBK_NW = 16;            /* warps per CTA             */
constexpr int TBK_NT = 32 * TBK_NW;   /* threads per CTA           */
constexpr int TBK_TMAX = 8;           /* most steps per launch     */

/* output columns and rows of a tile that advances T steps */
constexpr int tbk_cols(int T) { return 64 - 4 * ((T + 1) / 2); }
constexpr int tbk_rows(int rows, int T) { return TBK_NW * rows - 2 * T; }

/* the shifted pairs of a row from the neighbouring lanes' pairs; lanes 0
 * and 31 get their own values, which only feed halo columns */
__device__ __forceinline__ void pair_shift(PairRow &r)
{
  const float2 c = up(r.c);
  r.w = pk(__shfl_up_sync(0xffffffffu, c.y, 1), c.x);
  r.e = pk(c.y, __shfl_down_sync(0xffffffffu, c.x, 1));
}

/* a lane's two columns of a row: one 8-byte load (VEC: nx even, 8-byte
 * aligned grid, x0 even), or one by one */
template <bool VEC>
__device__ __forceinline__ F2 pair_load(const float *row, int x0, int x1)
{
  return VEC ? ld2(row + x0) : pk(row[x0], row[x1]);
}
/* the same for a grid no launch of the chain writes */
template <bool VEC>
__device__ __forceinline__ F2 pair_ldg(const float *row, int x0, int x1)
{
  return VEC ? ldg2(row + x0) : pk(__ldg(row + x0), __ldg(row + x1));
}

/* Tile bx of the block's row of tiles: T steps from a into b.  talus and extra are loaded before
 * the wait for the launch before (hm_chain.cuh).  Loads are clamped to the grid;
 * what lies outside only feeds halo cells, since border cells copy their
 * inward neighbour. */
template <bool TMAP, class R, int ROWS, bool VEC>
__device__ __forceinline__ void thermal_block(const float *a,
                                              float *__restrict__ b,
                                              int nx,
                                              int ny,
                                              const float *__restrict__ talus,
                                              float talus_value,
                                              const float *__restrict__ extra,
                                              int T,
                                              int bx,
                                              bool first,
                                              float param = 0.f)
{
  constexpr int TY = TBK_NW * ROWS;
  __shared__ F2 rows[2][TBK_NW][2][32]; /* [step parity][warp][its first, last row][lane] */
  const int  HL = (T + 1) >> 1, W = 64 - 4 * HL;
  const int  lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int  c0 = bx * W - 2 * HL, gx = c0 + 2 * lane;
  /* first row of the tile's output; tbk_grid folds a grid's y into z */
  const unsigned y0 = (blockIdx.y + blockIdx.z * gridDim.y) * (unsigned)(TY - 2 * T);
  if (y0 >= (unsigned)ny) return;        /* the whole CTA: a block that the fold adds */
  const int  r0 = (int)y0 - T;           /* first row of the tile */
  const int  j0 = r0 + wp * ROWS;        /* first row of the warp */
  const int  x0 = min(max(gx, 0), VEC ? nx - 2 : nx - 1), x1 = min(max(gx + 1, 0), nx - 1);
  const bool edge = c0 <= 0 || c0 + 64 >= nx || r0 <= 0 || r0 + TY >= ny;

  PairRow v[ROWS + 2]; /* v[0], v[ROWS + 1]: rows of the warps above and below */
  F2      tl[ROWS], ex[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; q++)
  {
    const size_t o = (size_t)min(max(j0 + q, 0), ny - 1) * nx;
    tl[q] = TMAP ? pair_ldg<VEC>(talus + o, x0, x1) : pk1(talus_value);
    ex[q] = R::EXTRA ? pair_ldg<VEC>(extra + o, x0, x1) : pk1(0.f);
  }
  chain_wait();
  a = produced(a);
#pragma unroll
  for (int q = 0; q < ROWS; q++)
    v[q + 1].c = pair_load<VEC>(a + (size_t)min(max(j0 + q, 0), ny - 1) * nx, x0, x1);
  for (int t = 0; t < T; t++)
  {
    const int par = t & 1;
    rows[par][wp][0][lane] = v[1].c;
    rows[par][wp][1][lane] = v[ROWS].c;
    __syncthreads();
    /* rows t + 1 .. TY - 2 - t of the tile are still needed */
    if (wp * ROWS + ROWS - 1 <= t || wp * ROWS >= TY - 1 - t) continue;
    v[0].c = rows[par][max(wp - 1, 0)][1][lane];
    v[ROWS + 1].c = rows[par][min(wp + 1, TBK_NW - 1)][0][lane];
#pragma unroll
    for (int q = 0; q < ROWS + 2; q++) pair_shift(v[q]);
    F2 o[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; q++)
    {
      o[q] = R::pair(v[q + 1].c, v[q + 1].w, v[q + 2].c, v[q].c, v[q + 1].e, v[q].w, v[q + 2].w, v[q].e, v[q + 2].e,
                     tl[q], ex[q], first && t == 0, param);
      if (edge)
      {
        /* apply_boundaries: rows, then columns, which win at the corners */
        const int j = j0 + q;
        if (j == 0) o[q] = v[q + 2].c;
        else if (j == ny - 1) o[q] = v[q].c;
        if (gx == 0) o[q] = pk(hi(v[q + 1].c), hi(o[q]));
        if (gx == nx - 1) o[q] = pk(lo(v[q + 1].w), hi(o[q]));
        if (gx + 1 == nx - 1) o[q] = pk(lo(o[q]), lo(v[q + 1].c));
      }
    }
#pragma unroll
    for (int q = 0; q < ROWS; q++) v[q + 1].c = o[q];
  }
  if (lane < HL || lane >= 32 - HL || gx >= nx) return;
#pragma unroll
  for (int q = 0; q < ROWS; q++)
  {
    const int tr = wp * ROWS + q, j = j0 + q;
    if (tr < T || tr >= TY - T || j >= ny) continue;
    float *p = b + (size_t)j * nx + gx;
    if (VEC) st2(p, v[q + 1].c);
    else
    {
      p[0] = lo(v[q + 1].c);
      if (gx + 1 < nx) p[1] = hi(v[q + 1].c);
    }
  }
}

/* Steps per launch and rows per warp of a solve; T 1 is the one-step sweep. */
struct BlockPlan
{
  int T, rows, launches;
};

/* (a grid has at most 65535 blocks in y) */
inline dim3 tbk_grid(int nx, int ny, const BlockPlan &p)
{
  const int w = tbk_cols(p.T), h = tbk_rows(p.rows, p.T);
  const int gy = (ny + h - 1) / h;
  return dim3((nx + w - 1) / w, gy < 65535 ? gy : 65535, (gy + 65534) / 65535);
}

/* `iterations` steps in launches of at most T, the count rounded up so that
 * the result ends in the first buffer (even) or not (odd), which saves a
 * copy of the grid; the launches share the steps evenly */
inline BlockPlan block_split(int iterations, int T, int rows, bool even)
{
  int n = (iterations + T - 1) / T;
  if ((n & 1) != (even ? 0 : 1) && n < iterations) n++;
  return BlockPlan{(iterations + n - 1) / n, rows, n};
}

/* The library's choice by grid size.  Over 1.5 M cells: one step per
 * launch (figures above).  Below: the least modelled time over T and ROWS,
 * launches x max(4.1, 2 + T (s + k c)) us with k CTAs on the fullest SM,
 * s + c = 0.65, c = 0.45 for ROWS 1 and s + c = 1.1, c = 0.8 for ROWS 2, a
 * fit within 10 % of the times measured at 64^2, 256^2, 513 x 257, 512^2,
 * 1025 x 769 and 1024^2 for T = 2 .. 8.
 *
 * Two shapes fill the tiles badly.  Grids of up to 32 rows are compared
 * with one step per launch (5 us and 2 per million cells; odd widths, whose
 * warps take 32 columns and load 8 rows at a time, 6 per million cells of at
 * least 8 rows): 10 steps, blocked and not, 350000 x 4 187 and 68 us,
 * 466666 x 3 412 and 240, 87500 x 16 109 and 86, 43750 x 32 117 and 90, but
 * 3000 x 20 24 and 69 and 19781 x 63 78 and 127.  Grids of 3 or 4 columns
 * take one step per launch from 150000 rows on: 3 x 466666 1.30 and 0.99 ms,
 * 3 x 30000 116 and 142 us. */
inline BlockPlan block_pick(int nx, int ny, int iterations, bool even)
{
  if (iterations < 2 || (long long)nx * ny > 1500000) return BlockPlan{1, 0, iterations};
  BlockPlan best{1, 0, iterations};
  double    best_us = 1e30;
  for (int rows = 1; rows <= 2; rows++)
    for (int T = 2; T <= TBK_TMAX && tbk_rows(rows, T) >= 4; T++)
    {
      const BlockPlan p = block_split(iterations, T, rows, even);
      if (p.T < 2) continue;
      const dim3   g = tbk_grid(nx, ny, p);
      const int    k = (int)((g.x * g.y * g.z + 147) / 148);
      const double s = rows == 1 ? 0.20 : 0.30, c = rows == 1 ? 0.45 : 0.80;
      const double us = 2.0 + p.T * (s + k * c);
      const double total = p.launches * (us > 4.1 ? us : 4.1);
      if (total < best_us)
      {
        best_us = total;
        best = p;
      }
    }
  const double sweep_us = nx % 2 == 0 ? 5.0 + 2e-6 * nx * ny : 5.0 + 6e-6 * nx * (ny < 8 ? 8 : ny);
  if (ny <= 32 ? iterations * sweep_us < best_us : nx <= 4 && ny >= 150000) return BlockPlan{1, 0, iterations};
  return best;
}

/* a depth T >= 2 asked for by the caller or the launch-shape table; `rows`
 * is its tile height (16 or 32, 0: 32), raised where T needs more */
inline BlockPlan block_fixed(int T, int rows, int iterations, bool even)
{
  const int r = rows > 0 && rows <= TBK_NW && tbk_rows(1, T) >= 4 ? 1 : 2;
  return block_split(iterations, T, r, even);
}

/* the steps launch l of a plan advances */
inline int block_steps(const BlockPlan &p, int iterations, int l)
{
  /* the first `iterations mod launches` launches take one step more */
  return iterations / p.launches + (l < iterations % p.launches ? 1 : 0);
}

} // namespace hm

#endif
