/*
 * hm_thermal.cu - talus thermal erosion on sm_100a.
 *
 * Replaces the host loop of HighMap/src/erosion/thermal_gpu.cpp:17-96 and
 * the OpenCL kernels thermal / thermal_with_bedrock
 * (HighMap/src/gpu_opencl/kernels/thermal.cl:26-100).
 *
 * Device data: z, talus and bedrock stay in HBM for the whole call; steps
 * ping-pong between z and one workspace grid (Jacobi), or, where the input
 * heights are needed to the end (deposition map, mask, auto-bedrock),
 * between two workspace grids, so that no copy of them is made.  After the
 * steps: extrapolate_borders (HighMap/src/boundary/boundary.cpp:19-41) on
 * the outer ring, then, when asked, the deposition map max(z - z0, 0)
 * (HighMap/src/range/range.cpp:253-262) and the mask blend
 * lerp(z0, z, mask) (HighMap/include/highmap/operator.hpp:405-418), all in
 * one kernel that also brings the result to z.
 *
 * Kernels
 *   k_thermal_sweep2  one step per launch: a warp walks down rows of 64
 *                     columns (two per lane), neighbours by warp shuffles;
 *                     reads z, talus and bedrock once, writes z: 12 B/cell
 *                     (16 B with bedrock).  Even nx, 8-byte aligned grids.
 *   k_thermal_sweep   the same with one column per lane (any grid).
 *   k_thermal_block   up to 8 steps per launch (temporal blocking,
 *                     hm_thermal_block.cuh): the choice up to 1.5 M cells.
 *   k_thermal_out     border, deposition map and mask blend from the last
 *                     step's grid into z.
 *   k_border          the border alone, in place.
 *   k_extrapolate(_n), k_thermal_final   the same in place, border first
 *                     (grids under 4 cells a side, deeper borders, the
 *                     batched form).
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "hm_internal.h"
#include "hm_thermal.h"
#include "hm_thermal_block.cuh"
#include "hm_thermal_math.cuh"
#include "hm_thermal_sweep.cuh"
#include "hm_tune.h"

namespace hm
{

/* ------------------------------------------------------------------ */
/* one step per launch, column sweep                                  */
/* ------------------------------------------------------------------ */

constexpr int SW_NT = 256; /* 8 warps; a warp owns 32 columns              */
constexpr int SW_H = 16;   /* output rows per CTA (a multiple of SW_P)      */

/* One Jacobi step, a warp per 32 columns and SW_H rows
 * (hm_thermal_sweep.cuh). */
template <bool TMAP, int BED>
__global__ void __launch_bounds__(SW_NT)
    k_thermal_sweep(const float *a,
                    float *__restrict__ b,
                    int nx,
                    int ny,
                    const float *__restrict__ talus,
                    float talus_value,
                    const float *__restrict__ bedrock,
                    int first)
{
  chain_wait();
  a = produced(a);
  const int wx = (blockIdx.x * (SW_NT / 32) + (threadIdx.x >> 5)) * 32;
  if (wx >= nx) return; /* the whole warp: no CTA barrier in this kernel */
  const int y0 = blockIdx.y * SW_H;
  thermal_sweep_warp<TMAP, TalusExchange<BED>>(a, b, nx, ny, talus, talus_value, bedrock, first, wx, y0, min(ny, y0 + SW_H));
}

/* One Jacobi step, a warp per 64 columns (two per lane) and SW_H rows
 * (hm_thermal_sweep.cuh); even nx, 8-byte aligned grids. */
constexpr int S2_NT = 128; /* 4 warps; a warp owns 64 columns */

template <bool TMAP, int BED>
__global__ void __launch_bounds__(S2_NT)
    k_thermal_sweep2(const float *a,
                     float *__restrict__ b,
                     int nx,
                     int ny,
                     const float *__restrict__ talus,
                     float talus_value,
                     const float *__restrict__ bedrock,
                     int first)
{
  chain_wait();
  a = produced(a);
  const int wx = (blockIdx.x * (S2_NT / 32) + (threadIdx.x >> 5)) * 64;
  if (wx >= nx) return; /* the whole warp: no CTA barrier in this kernel */
  const int y0 = blockIdx.y * SW_H;
  thermal_sweep2_warp<TMAP, TalusExchange<BED>>(a, b, nx, ny, talus, talus_value, bedrock, first, wx, y0, min(ny, y0 + SW_H));
}

/* ------------------------------------------------------------------ */
/* several steps per launch (temporal blocking)                       */
/* ------------------------------------------------------------------ */

template <bool TMAP, int BED, int ROWS, bool VEC>
__global__ void __launch_bounds__(TBK_NT)
    k_thermal_block(const float *a,
                    float *__restrict__ b,
                    int nx,
                    int ny,
                    const float *__restrict__ talus,
                    float talus_value,
                    const float *__restrict__ bedrock,
                    int T,
                    int first)
{
  thermal_block<TMAP, TalusExchange<BED>, ROWS, VEC>(a, b, nx, ny, talus, talus_value, bedrock, T, blockIdx.x,
                                                     first != 0);
}

/* ------------------------------------------------------------------ */
/* borders and finalisation                                           */
/* ------------------------------------------------------------------ */

/* extrapolate_borders(z, 1, 0): columns first, then rows, as the loops of
 * boundary.cpp:26-40 order them (the row pass reads the column pass's
 * corner values). */
__global__ void __launch_bounds__(1024) k_extrapolate(float *z, int nx, int ny)
{
  for (int j = threadIdx.x; j < ny; j += blockDim.x)
  {
    float *r = z + (size_t)j * nx;
    r[0] = __fsub_rn(__fmul_rn(2.f, r[1]), r[2]);
    r[nx - 1] = __fsub_rn(__fmul_rn(2.f, r[nx - 2]), r[nx - 3]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nx; i += blockDim.x)
  {
    z[i] = __fsub_rn(__fmul_rn(2.f, z[(size_t)nx + i]), z[(size_t)2 * nx + i]);
    size_t l = (size_t)(ny - 1) * nx + i;
    z[l] = __fsub_rn(__fmul_rn(2.f, z[l - nx]), z[l - 2 * (size_t)nx]);
  }
}

/* extrapolate_borders(z, nb, 0) for nb > 1 (boundary.cpp:19-41): per row,
 * for k = nb-1 .. 0, column k from columns k+1, k+2, then column nx-1-k
 * from its two inward neighbours; then the same per column over the rows.
 * One thread walks one row (then one column) in the reference's order, so
 * rows narrower than 2 nb + 2, where the two sides meet, match too. */
__global__ void __launch_bounds__(1024) k_extrapolate_n(float *z, int nx, int ny, int nb)
{
  for (int j = threadIdx.x; j < ny; j += blockDim.x)
  {
    float *r = z + (size_t)j * nx;
    for (int k = nb - 1; k > -1; k--)
    {
      r[k] = __fsub_rn(__fmul_rn(2.f, r[k + 1]), r[k + 2]);
      r[nx - 1 - k] = __fsub_rn(__fmul_rn(2.f, r[nx - 2 - k]), r[nx - 3 - k]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nx; i += blockDim.x)
    for (int k = nb - 1; k > -1; k--)
    {
      z[(size_t)k * nx + i] = __fsub_rn(__fmul_rn(2.f, z[(size_t)(k + 1) * nx + i]), z[(size_t)(k + 2) * nx + i]);
      z[(size_t)(ny - 1 - k) * nx + i] =
          __fsub_rn(__fmul_rn(2.f, z[(size_t)(ny - 2 - k) * nx + i]), z[(size_t)(ny - 3 - k) * nx + i]);
    }
}

__global__ void k_thermal_final(float *__restrict__ z,
                                const float *__restrict__ z0,
                                float *__restrict__ depo,
                                const float *__restrict__ mask,
                                size_t n,
                                int depo_abs)
{
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
  {
    float r = z[k];
    float o = z0[k];
    if (depo)
    {
      float dz = __fsub_rn(r, o);
      depo[k] = depo_abs ? fabsf(dz) : (dz > 0.f ? dz : 0.f);
    }
    if (mask)
    {
      float m = mask[k];
      z[k] = __fadd_rn(__fmul_rn(o, __fsub_rn(1.f, m)), __fmul_rn(r, m));
    }
  }
}

/* Cell (i, j) of extrapolate_borders(s, 1, 0) for grids of at least 4 x 4,
 * where every border cell is a function of interior cells alone: columns
 * from the two inward ones of their row, then rows from the two inward
 * rows (whose end cells are the column pass's). */
__device__ __forceinline__ float bordered_row(const float *r, int i, int nx)
{
  if (i == 0) return __fsub_rn(__fmul_rn(2.f, r[1]), r[2]);
  if (i == nx - 1) return __fsub_rn(__fmul_rn(2.f, r[nx - 2]), r[nx - 3]);
  return r[i];
}
__device__ __forceinline__ float bordered(const float *s, int i, int j, int nx, int ny)
{
  if (j == 0 || j == ny - 1)
  {
    const float *r1 = s + (size_t)(j == 0 ? 1 : ny - 2) * nx, *r2 = s + (size_t)(j == 0 ? 2 : ny - 3) * nx;
    return __fsub_rn(__fmul_rn(2.f, bordered_row(r1, i, nx)), bordered_row(r2, i, nx));
  }
  return bordered_row(s + (size_t)j * nx, i, nx);
}

/* the outer ring in place: one thread per border cell; only interior cells
 * are read and only border cells written */
__global__ void __launch_bounds__(256) k_border(float *z, int nx, int ny)
{
  const long long n = 2ll * nx + 2ll * (ny - 2);
  chain_wait();
  for (long long k = blockIdx.x * 256ll + threadIdx.x; k < n; k += gridDim.x * 256ll)
  {
    int i, j;
    if (k < 2ll * nx)
    {
      j = k < nx ? 0 : ny - 1;
      i = (int)(k < nx ? k : k - nx);
    }
    else
    {
      const long long m = k - 2ll * nx;
      j = 1 + (int)(m >> 1);
      i = (m & 1) ? nx - 1 : 0;
    }
    z[(size_t)j * nx + i] = bordered(z, i, j, nx, ny);
  }
}

/* The result of a solve from its last grid s (not z): border, deposition
 * map against the input heights z still holds, mask blend; 256 cells of a
 * row per CTA and turn, the loads of four turns in flight: with a row per
 * CTA one step at 4096 x 4096 took 139 us, with a deposition map 153; now 104
 * and 118. */
__global__ void __launch_bounds__(256)
    k_thermal_out(const float *s, float *__restrict__ z, float *__restrict__ depo,
                  const float *__restrict__ mask, int nx, int ny, int depo_abs)
{
  const int i = blockIdx.x * 256 + threadIdx.x;
  chain_wait();
  s = produced(s);
  if (i >= nx) return;
#pragma unroll 4
  for (int j = blockIdx.y; j < ny; j += gridDim.y)
  {
    const size_t k = (size_t)j * nx + i;
    const float  r = bordered(s, i, j, nx, ny);
    if (!depo && !mask)
    {
      z[k] = r;
      continue;
    }
    const float o = z[k];
    if (depo)
    {
      const float dz = __fsub_rn(r, o);
      depo[k] = depo_abs ? fabsf(dz) : (dz > 0.f ? dz : 0.f);
    }
    if (mask)
    {
      const float m = mask[k];
      z[k] = __fadd_rn(__fmul_rn(o, __fsub_rn(1.f, m)), __fmul_rn(r, m));
    }
    else
      z[k] = r;
  }
}

/* ------------------------------------------------------------------ */
/* host side                                                          */
/* ------------------------------------------------------------------ */

static int num_sms(int device)
{
  static int cached[64] = {0};
  if (device >= 0 && device < 64 && cached[device]) return cached[device];
  int n = 0;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
  if (n <= 0) n = 148;
  if (device >= 0 && device < 64) cached[device] = n;
  return n;
}

/* kernel bedrock mode: auto (bed = z0) or the caller's bedrock grid */
static int kernel_bed_mode(const float *bed, int bed_mode, bool auto_bed)
{
  if (auto_bed) return BED_AUTO;
  return bed ? (bed_mode == HM_BEDROCK_LITERAL ? BED_LITERAL : BED_INTENDED) : BED_NONE;
}

/* one Jacobi step: the column-pair sweep where the grid allows 8-byte
 * access (even nx, 8-byte aligned grids), else the one-column sweep */
template <bool TMAP, int BED>
static void launch_step(const float *a, float *b, int nx, int ny, const float *talus, float tv,
                        const float *bed, int first, cudaStream_t s, bool chained)
{
  auto al8 = [](const void *p) { return ((uintptr_t)p & 7u) == 0; };
  if (nx % 2 == 0 && al8(a) && al8(b) && (!TMAP || al8(talus)) && (BED == BED_NONE || al8(bed)))
  {
    dim3 grid((nx + 2 * S2_NT - 1) / (2 * S2_NT), (ny + SW_H - 1) / SW_H);
    chain_launch(chained, k_thermal_sweep2<TMAP, BED>, grid, dim3(S2_NT), s, a, b, nx, ny, talus, tv, bed, first);
    return;
  }
  dim3 grid((nx + SW_NT - 1) / SW_NT, (ny + SW_H - 1) / SW_H);
  chain_launch(chained, k_thermal_sweep<TMAP, BED>, grid, dim3(SW_NT), s, a, b, nx, ny, talus, tv, bed, first);
}

template <bool TMAP>
static void step_dispatch_t(const float *a, float *b, int nx, int ny, const float *talus, float tv,
                            const float *bed, int mode, int first, cudaStream_t s, bool chained)
{
  switch (mode)
  {
  case BED_NONE: launch_step<TMAP, BED_NONE>(a, b, nx, ny, talus, tv, bed, first, s, chained); break;
  case BED_INTENDED: launch_step<TMAP, BED_INTENDED>(a, b, nx, ny, talus, tv, bed, first, s, chained); break;
  case BED_LITERAL: launch_step<TMAP, BED_LITERAL>(a, b, nx, ny, talus, tv, bed, first, s, chained); break;
  default: launch_step<TMAP, BED_AUTO>(a, b, nx, ny, talus, tv, bed, first, s, chained); break;
  }
}

static void step_dispatch(const float *a, float *b, int nx, int ny, const float *talus, float tv,
                          const float *bed, int mode, int first, cudaStream_t s, bool chained)
{
  if (talus) step_dispatch_t<true>(a, b, nx, ny, talus, tv, bed, mode, first, s, chained);
  else step_dispatch_t<false>(a, b, nx, ny, talus, tv, bed, mode, first, s, chained);
}

/* post-processing of a finished thermal solve (z holds the last step):
 * border extrapolation (nbuffer cells deep), then the deposition map (max(z - z0, 0), or
 * |z - z0| with depo_abs) and the mask blend when asked (z0 = the input
 * heights) */
int thermal_finish(int device, float *z, int nx, int ny, const float *z0, float *depo, const float *mask,
                   cudaStream_t s, bool depo_abs, int nbuffer)
{
  if (nbuffer > 1)
  {
    k_extrapolate_n<<<1, 1024, 0, s>>>(z, nx, ny, nbuffer);
    HM_LAUNCH_CHECK("k_extrapolate_n");
  }
  else
  {
    k_extrapolate<<<1, 1024, 0, s>>>(z, nx, ny);
    HM_LAUNCH_CHECK("k_extrapolate");
  }
  if (depo || mask)
  {
    k_thermal_final<<<num_sms(device) * 8, 256, 0, s>>>(z, z0, depo, mask, (size_t)nx * ny, depo_abs ? 1 : 0);
    HM_LAUNCH_CHECK("k_thermal_final");
  }
  return HM_OK;
}

int thermal_out(const float *src, float *z, int nx, int ny, float *depo, const float *mask, cudaStream_t s,
                bool depo_abs, bool chained)
{
  if (src == z && !depo && !mask && nx >= 4 && ny >= 4)
  {
    const long long n = 2ll * nx + 2ll * (ny - 2);
    chain_launch(chained, k_border, dim3((unsigned)((n + 255) / 256)), dim3(256), s, z, nx, ny);
    HM_LAUNCH_CHECK("k_border");
    return HM_OK;
  }
  /* the heights alone on a large grid: a copy and the border (a call of one
   * step at 4096 x 4096 93 against 104 us, at 3000 x 2000 51 against 47) */
  if (!depo && !mask && (long long)nx * ny > (1ll << 23))
  {
    HM_CUDA_TRY(cudaMemcpyAsync(z, src, (size_t)nx * ny * sizeof(float), cudaMemcpyDeviceToDevice, s));
    return thermal_out(z, z, nx, ny, nullptr, nullptr, s, depo_abs, false);
  }
  /* about 64 CTAs per SM, which take every so many rows */
  const int gx = (nx + 255) / 256, gy = std::min(ny, std::max(1, 64 * 148 / gx));
  chain_launch(chained, k_thermal_out, dim3(gx, gy), dim3(256), s, src, z, depo, mask, nx, ny, depo_abs ? 1 : 0);
  HM_LAUNCH_CHECK("k_thermal_out");
  return HM_OK;
}

template <bool TMAP, int BED>
static void launch_block(const float *a, float *b, int nx, int ny, const float *talus, float tv, const float *bed,
                         int T, int rows, int first, cudaStream_t s, bool chained)
{
  auto       al8 = [](const void *p) { return ((uintptr_t)p & 7u) == 0; };
  const bool vec = nx % 2 == 0 && al8(a) && al8(b) && (!TMAP || al8(talus)) && (BED == BED_NONE || al8(bed));
  const dim3 g = tbk_grid(nx, ny, BlockPlan{T, rows, 1});
  auto       k = rows == 1 ? (vec ? k_thermal_block<TMAP, BED, 1, true> : k_thermal_block<TMAP, BED, 1, false>)
                           : (vec ? k_thermal_block<TMAP, BED, 2, true> : k_thermal_block<TMAP, BED, 2, false>);
  chain_launch(chained, k, g, dim3(TBK_NT), s, a, b, nx, ny, talus, tv, bed, T, first);
}

template <bool TMAP>
static void block_dispatch_t(const float *a, float *b, int nx, int ny, const float *talus, float tv,
                             const float *bed, int mode, int T, int rows, int first, cudaStream_t s, bool chained)
{
  switch (mode)
  {
  case BED_NONE: launch_block<TMAP, BED_NONE>(a, b, nx, ny, talus, tv, bed, T, rows, first, s, chained); break;
  case BED_INTENDED: launch_block<TMAP, BED_INTENDED>(a, b, nx, ny, talus, tv, bed, T, rows, first, s, chained); break;
  case BED_LITERAL: launch_block<TMAP, BED_LITERAL>(a, b, nx, ny, talus, tv, bed, T, rows, first, s, chained); break;
  default: launch_block<TMAP, BED_AUTO>(a, b, nx, ny, talus, tv, bed, T, rows, first, s, chained); break;
  }
}

static void block_dispatch(const float *a, float *b, int nx, int ny, const float *talus, float tv, const float *bed,
                           int mode, int T, int rows, int first, cudaStream_t s, bool chained)
{
  if (talus) block_dispatch_t<true>(a, b, nx, ny, talus, tv, bed, mode, T, rows, first, s, chained);
  else block_dispatch_t<false>(a, b, nx, ny, talus, tv, bed, mode, T, rows, first, s, chained);
}

static int g_tb_rows = 0; /* tile rows of the blocked kernel (hm_thermal_set_launch); 0 = built-in */

int thermal_check_args(const float *z, int nx, int ny, int iterations, const hm_thermal_options *o)
{
  if (!z) return fail(HM_ERR_INVALID_ARGUMENT, "thermal: z is NULL");
  if (nx < 3 || ny < 3) return fail(HM_ERR_INVALID_ARGUMENT, "thermal: nx and ny must be >= 3");
  if ((long long)nx * (long long)ny > (1ll << 34))
    return fail(HM_ERR_INVALID_ARGUMENT, "thermal: grid larger than 2^34 cells");
  if (iterations < 0) return fail(HM_ERR_INVALID_ARGUMENT, "thermal: iterations < 0");
  if (o && o->bedrock_mode != HM_BEDROCK_INTENDED && o->bedrock_mode != HM_BEDROCK_LITERAL)
    return fail(HM_ERR_INVALID_ARGUMENT, "thermal: unknown bedrock_mode");
  if (o && o->time_block < 0) return fail(HM_ERR_INVALID_ARGUMENT, "thermal: time_block < 0");
  return HM_OK;
}

size_t thermal_scratch_floats(int nx, int ny, bool need_z0)
{
  size_t n = align_up((size_t)nx * ny, 64);
  return n * (need_z0 ? 2 : 1);
}

int thermal_core(int device,
                 float *z,
                 int nx,
                 int ny,
                 const float *talus,
                 float talus_value,
                 int iterations,
                 const float *bedrock,
                 float *depo,
                 const float *mask,
                 const hm_thermal_options *opts,
                 float *scratch_buf,
                 cudaStream_t s,
                 bool auto_bed,
                 bool chained)
{
  hm_thermal_options o;
  hm_thermal_default_options(&o);
  if (opts) o = *opts;
  const bool   keep_z = depo || mask || auto_bed; /* z holds the input heights to the end */
  const size_t na = align_up((size_t)nx * ny, 64);
  /* the grids the launches write in turn */
  float       *buf[2] = {scratch_buf, keep_z ? scratch_buf + na : z};
  (void)device;

  /* steps per launch: 1 runs the one-step kernel, 2..8 the blocked kernel;
   * 0 takes the tuned choice for this grid, else block_pick's.  Without
   * the input heights to keep, an even number of launches ends in z. */
  BlockPlan plan;
  int       tb = o.time_block, rows = g_tb_rows;
  TuneEntry e;
  if (tb == 0 && tuned_thermal(nx, ny, &e))
  {
    tb = e.block;
    if (rows == 0) rows = e.rows;
  }
  if (tb == 0) plan = block_pick(nx, ny, iterations, !keep_z);
  else if (tb == 1 || iterations == 0) plan = BlockPlan{1, 0, iterations};
  else plan = block_fixed(tb > TBK_TMAX ? TBK_TMAX : tb, rows, iterations, !keep_z);
  /* auto-bedrock reads the input heights as its bedrock */
  const int    mode = kernel_bed_mode(bedrock, o.bedrock_mode, auto_bed);
  const float *bed = auto_bed ? z : bedrock;
  const float *src = z;
  for (int l = 0; l < plan.launches; l++)
  {
    float *dst = buf[l & 1];
    /* (a plan asked for goes on past the rows a launch of the sweep takes) */
    if (plan.T == 1 && (plan.rows == 0 || ny <= 65535 * SW_H))
    {
      step_dispatch(src, dst, nx, ny, talus, talus_value, bed, mode, l == 0, s, chained || l > 0);
      HM_LAUNCH_CHECK("k_thermal_sweep");
    }
    else
    {
      block_dispatch(src, dst, nx, ny, talus, talus_value, bed, mode, block_steps(plan, iterations, l), plan.rows,
                     l == 0, s, chained || l > 0);
      HM_LAUNCH_CHECK("k_thermal_block");
    }
    src = dst;
  }
  /* in place, or on a grid too narrow for k_thermal_out: border first,
   * then the rest against a copy of the input heights */
  if (nx < 4 || ny < 4 || (src == z && (depo || mask)))
  {
    const size_t bytes = (size_t)nx * ny * sizeof(float);
    float       *z0 = nullptr;
    if (depo || mask)
    {
      z0 = src == buf[0] ? buf[1] : buf[0];
      HM_CUDA_TRY(cudaMemcpyAsync(z0, z, bytes, cudaMemcpyDeviceToDevice, s));
    }
    if (src != z) HM_CUDA_TRY(cudaMemcpyAsync(z, src, bytes, cudaMemcpyDeviceToDevice, s));
    return thermal_finish(device, z, nx, ny, z0, depo, mask, s);
  }
  return thermal_out(src, z, nx, ny, depo, mask, s, false, chained || plan.launches > 0);
}

} // namespace hm

extern "C" int hm_thermal_set_launch(int rows)
{
  hm::clear_error();
  if (rows != 0 && (rows < 8 || rows > 4096))
    return hm::fail(HM_ERR_INVALID_ARGUMENT, "hm_thermal_set_launch: rows must be 0 or in [8, 4096]");
  hm::g_tb_rows = rows;
  return HM_OK;
}

extern "C" void hm_thermal_default_options(hm_thermal_options *opts)
{
  if (!opts) return;
  opts->bedrock_mode = HM_BEDROCK_INTENDED;
  opts->time_block = 0;
}
