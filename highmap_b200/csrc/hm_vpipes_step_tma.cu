/*
 * hm_vpipes_step_tma.cu - instances of k_vp_step_tma (the previous step's
 * advection and this step's flow, water and erosion in one TMA-staged
 * tile, hm_vpipes_tiled.cuh) for every option word of the erosion steps,
 * and their launcher.  A translation unit of its own so the instances
 * compile in parallel with the rest of the library.
 */
#include <cuda_runtime.h>

#include "hm_internal.h"
#include "hm_vpipes_tiled.cuh"

namespace hm
{

namespace
{
template <bool M, int F> struct StepKernel
{
  static auto fn() { return &k_vp_step_tma<M, F>; }
};
/* the wide form and the one of six CTAs per SM have fixed options only */
template <bool M, int F> struct WideKernel
{
  static auto fn() { return &k_vp_step_tma<M, F, (F & FWE_GENERIC) ? FT_NT : FT_WIDE, (F & FWE_GENERIC) ? 5 : 2>; }
};
template <bool M, int F> struct SixKernel
{
  static auto fn() { return &k_vp_step_tma<M, F, FT_NT, (F & FWE_GENERIC) ? 5 : 6>; }
};
} // namespace

int launch_step_tma(const FweIo &io, const FweMaps &maps, const AdvMaps &am, const VpConst &c, VpScalars *sc,
                    double *partials, dim3 grid, cudaStream_t s)
{
  const int  flags = fwe_flags(io, c);
  const bool wide = grid.x * grid.y <= FT_WIDE_TILES && !(flags & FWE_GENERIC);
  auto       launch = [&](auto kernel) -> int {
    chain_launch(true, kernel, grid, dim3(wide ? FT_WIDE : FT_NT), s, io, maps, am, c, sc, partials);
    HM_LAUNCH_CHECK("k_vp_step_tma");
    return HM_OK;
  };
  if (wide) return step_dispatch<WideKernel>(io.maintain != 0, flags, launch);
  if (grid.x * grid.y > FT_FIVE_TILES) return step_dispatch<SixKernel>(io.maintain != 0, flags, launch);
  return step_dispatch<StepKernel>(io.maintain != 0, flags, launch);
}

} // namespace hm
