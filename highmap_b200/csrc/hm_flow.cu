/*
 * hm_flow.cu - flow_simulation on sm_100a: the water-only use of the
 * virtual-pipes model.
 *
 * Replaces HighMap/src/hydrology/flow_simulation.cpp:26-110, which runs
 * the flow and water passes of hydraulic_vpipes.cl (:5-116) on a fixed
 * terrain with host round trips around every pass, then the optional
 * dry-out of HighMap/src/hydrology/water_depth.cpp:40-66.  Here the steps
 * are the tiled vpipes kernels in their flow-only form (FWE_FLOWONLY:
 * flow, water, no erosion or advection, depth and fluxes written), the
 * state stays in HBM, and the dry-out is a max reduction plus one
 * elementwise pass.  Where a tile's boxes fit the grid the steps go in
 * pairs (hm_flow_steps.cuh).
 *
 * State: depth and the four fluxes in two copies (A, B); the terrain is
 * read in place, or from a copy where its rows miss the TMA rules (the
 * state's rows are then padded to a multiple of 4 floats).  Gravity, pipe area and
 * pipe length are 1, evaporation 0, as in the reference's kernels.
 */
#include <cuda_runtime.h>

#include <cstdint>

#include "hm_flow_steps.cuh"
#include "hm_internal.h"
#include "hm_vpipes.h"
#include "hm_vpipes_tiled.cuh"

namespace hm
{

namespace
{

/* grid-stride index q of nx-float rows as an index of ld-float rows */
__device__ __forceinline__ size_t padded_index(size_t q, int nx, int ld)
{
  return ld == nx ? q : q + (q / (size_t)nx) * (size_t)(ld - nx);
}

/* d = water_height * depth_map, fluxes of copy A 0; the terrain into zc
 * where it is copied */
__global__ void k_flow_init(float *__restrict__ d, const float *__restrict__ depth_map, float water_height,
                            float *__restrict__ fl, float *__restrict__ fr, float *__restrict__ ft,
                            float *__restrict__ fb, const float *__restrict__ z, float *__restrict__ zc, size_t n,
                            int nx, int ld)
{
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
  {
    const size_t k = padded_index(q, nx, ld);
    d[k] = __fmul_rn(water_height, depth_map[q]);
    fl[k] = fr[k] = ft[k] = fb[k] = 0.f;
    if (zc) zc[k] = z[q];
  }
}

/* max of the depth (Array::max); depths are >= 0 (or -0), so the bit
 * patterns of the non-negative values order like the values */
__global__ void k_flow_max(const float *__restrict__ d, size_t n, unsigned *__restrict__ out, int nx, int ld)
{
  unsigned m = 0u;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
  {
    const float v = d[padded_index(k, nx, ld)];
    const unsigned b = v > 0.f ? __float_as_uint(v) : 0u;
    m = b > m ? b : m;
  }
  for (int o = 16; o > 0; o >>= 1)
  {
    const unsigned t = __shfl_xor_sync(0xffffffffu, m, o);
    m = t > m ? t : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

/* water_depth_dry_out (water_depth.cpp:59-64): d = max(0, d - ratio * dmax),
 * written to the output */
__global__ void k_flow_dry_out(const float *__restrict__ d, const unsigned *__restrict__ dmax_bits, float ratio,
                               float *__restrict__ out, size_t n, int nx, int ld)
{
  const float drop = __fmul_rn(ratio, __uint_as_float(*dmax_bits));
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
  {
    const float w = __fsub_rn(d[padded_index(k, nx, ld)], drop);
    out[k] = 0.f < w ? w : 0.f;
  }
}

} // namespace

/* maps of one state copy for k_flow_steps<T>; false if a box is larger than
 * the grid (the caller has checked the TMA rules with fwe_maps) */
template <int T>
static bool flow_maps(const VpFields &f, int nx, int ny, int ld, FlowMaps *m)
{
  using L = FlowTile<T>;
  if (nx < L::W || ny < L::ZH) return false;
  auto map = [&](CUtensorMap *q, const float *p, int rows) { return encode_grid_map(q, p, nx, ny, ld, rows, L::W); };
  return map(&m->z, f.z, L::ZH) && map(&m->d, f.d, L::ZH) && map(&m->fl, f.fl, L::FH) && map(&m->fr, f.fr, L::FH) &&
         map(&m->ft, f.ft, L::FH) && map(&m->fb, f.fb, L::FH);
}

static size_t flow_state_floats(int nx, int ny, bool padded)
{
  return align_up((padded ? align_up((size_t)nx, 4) : (size_t)nx) * ny, 64);
}

bool flow_wants_padding(const float *z, int nx, int ny, int iterations)
{
  /* one step: the terrain's copy costs more than it wins on small grids
   * (255 x 257 26.7 -> 28.2 us; 601 x 599 6 % faster) */
  return (iterations > 1 || (iterations == 1 && (long long)nx * ny >= 100000)) && nx >= 40 && ny >= FT_H2 && (long long)nx * ny <= (1ll << 28) &&
         (nx % 4 != 0 || ((uintptr_t)z & 15u) != 0);
}

size_t flow_scratch_bytes(int nx, int ny, bool padded)
{
  /* depth and fluxes of two copies, the terrain's copy, a max slot, the
   * scalar block (its error word records TMA load timeouts) */
  return flow_state_floats(nx, ny, padded) * sizeof(float) * 11 + 256 + align_up(sizeof(VpScalars), 256);
}

int flow_check_args(const float *z, const float *depth_map, const float *out, int nx, int ny, int iterations,
                    float dt)
{
  if (!z || !depth_map || !out) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation: NULL grid");
  if (nx < 1 || ny < 1) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation: nx and ny must be >= 1");
  if ((long long)nx * (long long)ny > (1ll << 32))
    return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation: grid larger than 2^32 cells");
  if (iterations < 0) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation: iterations < 0");
  if (!(dt != 0.f)) return fail(HM_ERR_INVALID_ARGUMENT, "flow_simulation: dt must be non-zero");
  return HM_OK;
}

int flow_simulation_core(const float *z, int nx, int ny, float water_height, const float *depth_map, int iterations,
                         float dt, int flux_diffusion, float flux_diffusion_strength, float dry_out_ratio,
                         float *water_depth, void *scratch, cudaStream_t s, bool padded)
{
  const size_t n = (size_t)nx * ny;
  const size_t na = flow_state_floats(nx, ny, padded);
  const int    ld = padded ? (int)align_up((size_t)nx, 4) : nx;
  float       *base = (float *)scratch;
  float       *dA = base, *dB = base + na, *zc = padded ? base + 10 * na : nullptr;
  float       *zt = padded ? zc : const_cast<float *>(z); /* read only */
  unsigned    *dmax = (unsigned *)(base + 11 * na);
  VpScalars   *sc = (VpScalars *)((char *)(base + 11 * na) + 256);
  VpFields     A{zt, dA, nullptr, base + 2 * na, base + 3 * na, base + 4 * na, base + 5 * na};
  VpFields     B{zt, dB, nullptr, base + 6 * na, base + 7 * na, base + 8 * na, base + 9 * na};

  hm_vpipes_params p;
  hm_vpipes_default_params(&p);
  p.water_height = water_height;
  p.dt = dt;
  p.flux_diffusion = flux_diffusion != 0;
  p.flux_diffusion_strength = flux_diffusion_strength;
  p.evap_rate = 0.f;
  p.maintain_water_volume = 0;
  VpConst c = vpipes_consts(nx, ny, p);
  c.ld = ld;

  HM_CUDA_TRY(cudaMemsetAsync(sc, 0, sizeof(VpScalars), s));
  k_flow_init<<<592, 256, 0, s>>>(dA, depth_map, water_height, A.fl, A.fr, A.ft, A.fb, z, zc, n, nx, ld);
  HM_LAUNCH_CHECK("k_flow_init");

  FweIo io;
  memset(&io, 0, sizeof io);
  io.diffusion = p.flux_diffusion;
  io.pl_one = 1;
  io.kexp_one = 1;
  io.flow_only = 1;
  {
    auto al8 = [](const void *q) { return ((uintptr_t)q & 7u) == 0; };
    const void *outs[] = {A.d, A.fl, A.fr, A.ft, A.fb, B.d, B.fl, B.fr, B.ft, B.fb};
    bool        ok = ld % 2 == 0;
    for (const void *q : outs) ok = ok && al8(q);
    io.vec = ok ? 1 : 0;
  }
  io.tma_extra_tx = tma_extra_tx();
  FweMaps    maps[2];
  const bool tma = fwe_maps(A, nx, ny, ld, &maps[0]) && fwe_maps(B, nx, ny, ld, &maps[1]);
  const dim3 g1((nx + FT_TX - 1) / FT_TX, (ny + FT_TY - 1) / FT_TY);
  VpFields  *cur = &A, *nxt = &B;
  /* FLOW_T steps per launch; the remainder, and grids smaller than their
   * boxes, a step at a time */
  FlowMaps   fm[2];
  const bool blocked = tma && iterations >= FLOW_T && flow_maps<FLOW_T>(A, nx, ny, ld, &fm[0]) &&
                       flow_maps<FLOW_T>(B, nx, ny, ld, &fm[1]);
  const bool wide = flow_steps_wide(g1.x * g1.y);
  auto       kernel = wide ? (io.diffusion ? k_flow_steps<FLOW_T, true, FT_WIDE> : k_flow_steps<FLOW_T, false, FT_WIDE>)
                           : (io.diffusion ? k_flow_steps<FLOW_T, true, FT_NT> : k_flow_steps<FLOW_T, false, FT_NT>);
  if (io.tma_extra_tx)
    kernel = wide ? (io.diffusion ? k_flow_steps<FLOW_T, true, FT_WIDE, true> : k_flow_steps<FLOW_T, false, FT_WIDE, true>)
                  : (io.diffusion ? k_flow_steps<FLOW_T, true, FT_NT, true> : k_flow_steps<FLOW_T, false, FT_NT, true>);
  int        it = 0;
  for (; blocked && it + FLOW_T <= iterations; it += FLOW_T)
  {
    const VpStateOut o{nxt->z, nxt->d, nxt->s, nxt->fl, nxt->fr, nxt->ft, nxt->fb, nullptr, nullptr};
    chain_launch(it > 0, kernel, g1, wide ? FT_WIDE : FT_NT, s, o, io.vec, fm[cur == &A ? 0 : 1], c, sc);
    HM_LAUNCH_CHECK("k_flow_steps");
    VpFields *t = cur;
    cur = nxt;
    nxt = t;
  }
  for (; it < iterations; it++)
  {
    io.in = VpState{cur->z, cur->d, cur->s, cur->fl, cur->fr, cur->ft, cur->fb};
    io.out = VpStateOut{nxt->z, nxt->d, nxt->s, nxt->fl, nxt->fr, nxt->ft, nxt->fb, nullptr, nullptr};
    io.parity = it & 1;
    const int rc = tma ? launch_fwe_tma(io, maps[cur == &A ? 0 : 1], c, sc, nullptr, g1, s, it > 0)
                       : launch_fwe_cp_async(io, c, sc, nullptr, g1, s, it > 0);
    if (rc) return rc;
    VpFields *t = cur;
    cur = nxt;
    nxt = t;
  }
  if (dry_out_ratio != 0.f)
  {
    HM_CUDA_TRY(cudaMemsetAsync(dmax, 0, sizeof(unsigned), s));
    k_flow_max<<<592, 256, 0, s>>>(cur->d, n, dmax, nx, ld);
    HM_LAUNCH_CHECK("k_flow_max");
    k_flow_dry_out<<<592, 256, 0, s>>>(cur->d, dmax, dry_out_ratio, water_depth, n, nx, ld);
    HM_LAUNCH_CHECK("k_flow_dry_out");
  }
  else if (ld != nx)
    HM_CUDA_TRY(cudaMemcpy2DAsync(water_depth, (size_t)nx * sizeof(float), cur->d, (size_t)ld * sizeof(float),
                                  (size_t)nx * sizeof(float), ny, cudaMemcpyDeviceToDevice, s));
  else
    HM_CUDA_TRY(cudaMemcpyAsync(water_depth, cur->d, n * sizeof(float), cudaMemcpyDeviceToDevice, s));
  return HM_OK;
}

const unsigned *flow_error_word(const void *scratch, int nx, int ny, bool padded)
{
  const size_t na = flow_state_floats(nx, ny, padded);
  return &((const VpScalars *)((const char *)((const float *)scratch + 11 * na) + 256))->error;
}

} // namespace hm
