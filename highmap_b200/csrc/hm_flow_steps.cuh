/*
 * hm_flow_steps.cuh - T steps of the flow-only virtual-pipes model in one
 * launch: a tile and a halo of 2 T cells stay in shared memory between the
 * steps.
 *
 * Why: a single flow step moves 44 bytes a cell and computes little; the
 * grids of ordinary calls sit in L2, so a step's time is the latency of
 * fetching a tile, its stores and the launch.  T steps per launch pay these
 * once, for halo cells computed again (T = 2: 1.19 times the cells).  100
 * steps, one per launch, then T = 2, 3, 4: 256 x 256 0.41 -> 0.26, 0.23,
 * 0.22 ms; 1024 x 1024 1.11 -> 0.91, 1.05, 1.08 ms; 1921 x 1080 2.26 ->
 * 1.70, 2.01, 2.06 ms; 4096 x 4096 14.2 -> 11.5, 14.4, 15.1 ms.  Hence 2.
 *
 * A step's new flux needs z and d of the cell and its neighbours and its own
 * old flux; the new depth needs its own old depth and the new fluxes of the
 * cell and its neighbours.  So both are updated in place, with a barrier
 * between the two passes.  Step t of T computes fluxes on the tile and a
 * ring of 2 (T - t) + 1 cells and depths on a ring of 2 (T - t); neighbours
 * outside the grid are the edge cell itself, by clamped indices (cells
 * outside the grid are never read).
 */
#ifndef HM_FLOW_STEPS_CUH
#define HM_FLOW_STEPS_CUH

#include "hm_chain.cuh"
#include "hm_tma.cuh"
#include "hm_vpipes_tiled.cuh"

namespace hm
{

/* steps per launch */
constexpr int FLOW_T = 2;

/* 512 threads per tile instead of 256 by the number of tiles.  Up to two
 * tiles per SM a launch's time is one CTA's chain of passes, which twice the
 * warps shorten (100 steps at 256 x 256 0.243 -> 0.217 ms).  Up to four
 * (592), the CTAs of two launches fit side by side at 256 threads and the
 * next launch's start is hidden (420 x 480 0.344 against 0.376 ms); above
 * that they no longer do, and the 512-thread form fills the SMs with half
 * the CTAs (540 x 560 0.594 -> 0.426 ms, 660 x 700 0.615 -> 0.542 ms, 800 x
 * 760 0.677 -> 0.666 ms) until the waves are many (2048 x 2048 3.13 against
 * 3.32 ms). */
constexpr bool flow_steps_wide(unsigned tiles) { return tiles <= 296 || (tiles > 592 && tiles <= 1480); }

/* tensor maps of one state copy: boxes of W x ZH (z, d) and W x FH (fluxes) */
struct FlowMaps
{
  CUtensorMap z, d, fl, fr, ft, fb;
};

template <int T>
struct FlowTile
{
  static constexpr int HX = (2 * T + 3) / 4 * 4; /* staged columns west of the tile (boxes start on 16 bytes) */
  static constexpr int W = FT_TX + 2 * HX;
  static constexpr int ZH = FT_TY + 4 * T; /* rows y0 - 2 T .. */
  static constexpr int FH = ZH - 2;        /* rows y0 - 2 T + 1 .. */
  struct Plane
  {
    alignas(128) float v[FH * W];
  };
  alignas(128) float z[ZH * W];
  alignas(128) float d[ZH * W];
  Plane              f[4];
  uint64_t           bar;
  static constexpr unsigned BYTES = 4u * W * (2u * ZH + 4u * FH);
};

template <int T, bool DIFF, bool INNER, int NT>
__device__ __forceinline__ void flow_steps_tile(const VpStateOut &out, const VpConst &c, bool vec_, int x0, int y0,
                                                FlowTile<T> &sm)
{
  using L = FlowTile<T>;
  constexpr int W = L::W;
  const int     nx = c.nx, ny = c.ny;
#pragma unroll
  for (int t = 1; t <= T; t++)
  {
    {
      const int h = 2 * (T - t) + 1, np = FT_TX / 2 + h + 1, nr = FT_TY + 2 * h;
      for (int e = threadIdx.x; e < np * nr; e += NT)
      {
        const int r = e / np, p = e - r * np;
        const int gy = y0 - h + r, gx = x0 - (h + 1) + 2 * p;
        if (!INNER && (gx < 0 || gx >= nx || gy < 0 || gy >= ny)) continue;
        const int    k = (2 * T - h + r) * W + L::HX - (h + 1) + 2 * p, kf = k - W;
        const int    kn = INNER || gy > 0 ? k - W : k, ks = INNER || gy + 1 < ny ? k + W : k;
        const float2 zc = lds2(&sm.z[k]), dc = lds2(&sm.d[k]);
        const float2 zn = lds2(&sm.z[kn]), dn = lds2(&sm.d[kn]), zs = lds2(&sm.z[ks]), ds = lds2(&sm.d[ks]);
        const int    kw = INNER || gx > 0 ? k - 1 : k;
        const bool   second = INNER || gx + 1 < nx;
        const int    ke0 = second ? k + 1 : k, ke1 = INNER || gx + 2 < nx ? k + 2 : k + 1;
        F2           l = pk(lds2(&sm.f[0].v[kf])), rr = pk(lds2(&sm.f[1].v[kf])), tt = pk(lds2(&sm.f[2].v[kf])),
           b = pk(lds2(&sm.f[3].v[kf]));
        const F2 ze = INNER ? pk(zc.y, sm.z[ke1]) : pk(sm.z[ke0], sm.z[ke1]);
        const F2 de = INNER ? pk(dc.y, sm.d[ke1]) : pk(sm.d[ke0], sm.d[ke1]);
        flow_pair<DIFF>(c, pk(zc), pk(dc), pk(sm.z[kw], zc.x), pk(sm.d[kw], dc.x), ze, de, pk(zs), pk(ds), pk(zn), pk(dn),
                        l, rr, tt, b);
        sts2(&sm.f[0].v[kf], lo(l), hi(l));
        sts2(&sm.f[1].v[kf], lo(rr), hi(rr));
        sts2(&sm.f[2].v[kf], lo(tt), hi(tt));
        sts2(&sm.f[3].v[kf], lo(b), hi(b));
      }
    }
    __syncthreads();
    {
      const int g = 2 * (T - t), np = FT_TX / 2 + g, nr = FT_TY + 2 * g;
      for (int e = threadIdx.x; e < np * nr; e += NT)
      {
        const int r = e / np, p = e - r * np;
        const int gy = y0 - g + r, gx = x0 - g + 2 * p;
        if (!INNER && (gx < 0 || gx >= nx || gy < 0 || gy >= ny)) continue;
        const int    k = (2 * T - g + r) * W + L::HX - g + 2 * p, kf = k - W;
        const bool   second = INNER || gx + 1 < nx;
        const int    kn = INNER || gy > 0 ? kf - W : kf, ks = INNER || gy + 1 < ny ? kf + W : kf;
        const int    kw = INNER || gx > 0 ? kf - 1 : kf;
        const int    ke0 = second ? kf + 1 : kf, ke1 = INNER || gx + 2 < nx ? kf + 2 : kf + 1;
        const float2 l = lds2(&sm.f[0].v[kf]), rr = lds2(&sm.f[1].v[kf]), tt = lds2(&sm.f[2].v[kf]),
                     b = lds2(&sm.f[3].v[kf]);
        const F2 fle = INNER ? pk(l.y, sm.f[0].v[ke1]) : pk(sm.f[0].v[ke0], sm.f[0].v[ke1]);
        F2       d2, u, v, dr;
        water_pair(c, pk(lds2(&sm.d[k])), pk(l), pk(rr), pk(tt), pk(b), pk(sm.f[1].v[kw], rr.x), fle,
                   pk(lds2(&sm.f[2].v[kn])), pk(lds2(&sm.f[3].v[ks])), d2, u, v, dr);
        if (t < T) sts2(&sm.d[k], lo(d2), hi(d2));
        else
        {
          const size_t q = (size_t)gy * c.ld + gx;
          const bool   vec = INNER || vec_;
          st_pair(out.fl, q, l.x, l.y, second, vec);
          st_pair(out.fr, q, rr.x, rr.y, second, vec);
          st_pair(out.ft, q, tt.x, tt.y, second, vec);
          st_pair(out.fb, q, b.x, b.y, second, vec);
          st_pair(out.d, q, lo(d2), hi(d2), second, vec);
        }
      }
    }
    if (t < T) __syncthreads();
  }
}

/* A tile whose loads time out sets bit 0 of sc->error and writes nothing
 * (HOOK: the form for the test hook, hm_debug_tma_expect_extra, whose
 * barrier expects bytes that never come; the hook's count as an argument
 * cost 1 to 2 % of a call from 256^2 to 540 x 560).
 * 32 registers: eight CTAs (of 256 threads) per SM instead of six cover more of the waits
 * (513 x 511 0.50 -> 0.40 ms, 4096 x 4096 11.65 -> 11.50 ms). */
template <int T, bool DIFF, int NT, bool HOOK = false>
__global__ void __launch_bounds__(NT, 2048 / NT)
    k_flow_steps(VpStateOut out, int vec, const __grid_constant__ FlowMaps maps, VpConst c, VpScalars *sc)
{
  using L = FlowTile<T>;
  __shared__ L sm;
  const int    x0 = blockIdx.x * FT_TX, y0 = blockIdx.y * FT_TY;
  if (threadIdx.x == 0)
  {
    mbar_init(&sm.bar, 1);
    mbar_fence_init();
    tma_prefetch_map(&maps.z);
    tma_prefetch_map(&maps.d);
    tma_prefetch_map(&maps.fl);
    tma_prefetch_map(&maps.fr);
    tma_prefetch_map(&maps.ft);
    tma_prefetch_map(&maps.fb);
  }
  chain_wait(); /* the launch before has written the grids */
  __syncthreads();
  if (threadIdx.x == 0)
  {
    mbar_arrive_expect_tx(&sm.bar, L::BYTES + (HOOK ? 16u : 0u));
    tma_load_2d(sm.z, &maps.z, x0 - L::HX, y0 - 2 * T, &sm.bar);
    tma_load_2d(sm.d, &maps.d, x0 - L::HX, y0 - 2 * T, &sm.bar);
    tma_load_2d(sm.f[0].v, &maps.fl, x0 - L::HX, y0 - 2 * T + 1, &sm.bar);
    tma_load_2d(sm.f[1].v, &maps.fr, x0 - L::HX, y0 - 2 * T + 1, &sm.bar);
    tma_load_2d(sm.f[2].v, &maps.ft, x0 - L::HX, y0 - 2 * T + 1, &sm.bar);
    tma_load_2d(sm.f[3].v, &maps.fb, x0 - L::HX, y0 - 2 * T + 1, &sm.bar);
  }
  bool ok = mbar_wait_bounded(&sm.bar, 0);
  if (!ok) ok = mbar_wait_bounded(&sm.bar, 0); /* loads still in flight: give them a second window */
  if (!__syncthreads_and(ok))
  {
    if (threadIdx.x == 0) atomicOr(&sc->error, 1u);
    return;
  }
  if (vec && x0 >= 2 * T && x0 + FT_TX + 2 * T <= c.nx && y0 >= 2 * T && y0 + FT_TY + 2 * T <= c.ny)
    flow_steps_tile<T, DIFF, true, NT>(out, c, true, x0, y0, sm);
  else
    flow_steps_tile<T, DIFF, false, NT>(out, c, vec != 0, x0, y0, sm);
}

} // namespace hm

#endif
