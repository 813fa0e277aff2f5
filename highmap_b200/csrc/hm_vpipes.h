/* hm_vpipes.h - internal entry points of hm_vpipes.cu */
#ifndef HM_VPIPES_H
#define HM_VPIPES_H

#include <cuda_runtime.h>

#include "hm_erosion.h"

namespace hm
{
int    vpipes_check_args(const float *z, int nx, int ny, const hm_vpipes_params *p);
/* Whether a solve should keep its state in rows padded to a multiple of 4
 * floats, with copies of z and of the copied_outputs among sediment, vel_u
 * and vel_v: where nx or z miss the TMA rules, the copies (8 B per cell in
 * and out each) buy the TMA-staged kernels for every step:
 * 1023 x 767, rain map and top-up, 50 steps, 1575 us with clamped 4-byte
 * copies, 1394 us padded.  The copies take the time of a few launches or of
 * a few steps: with all outputs, cp.async tiles and padded, 255 x 257 8 steps
 * 93 and 104 us, 50 steps 1.09x; 601 x 599 2 steps 0.89x, 4 steps 0.97x, 8
 * steps 1.03x; 2047 x 2049 2 steps 0.86x, 4 steps 1.01x, 8 steps 1.15x.  So
 * from 1.2 M cell-steps on, and between 5 (4 from a million cells on) and 20
 * steps; with z alone, 3
 * steps (1.01x and 1.13x at the two smaller and the largest).  Not above 2^28
 * cells, so that memory limits stay where they are, nor where another kernel
 * is asked for or tuned. */
bool   vpipes_wants_padding(const float *z, int nx, int ny, int iterations, int copied_outputs);
size_t vpipes_scratch_bytes(int nx, int ny, bool padded);
/* Device pointers; ordered on s.  rain and the outputs are nullable. */
int    vpipes_core(float *z, int nx, int ny, const hm_vpipes_params &p, const float *rain, float *water_depth,
                   float *sediment, float *vel_u, float *vel_v, void *scratch_buf, cudaStream_t s, bool padded);
struct VpFields;
struct VpScalars;
struct VpConst;
VpConst vpipes_consts(int nx, int ny, const hm_vpipes_params &p);
/* initial state of copy A (depth, with the first step's rain where
 * first_rain is set; zero sediment and fluxes; z from z_in where given) in
 * rows of ld floats (0: nx), and V0, R */
int     vpipes_init(const VpFields &A, const float *rain, int nx, int ny, float init_depth, VpScalars *sc,
                    double *partials, cudaStream_t s, float first_rain, const float *z_in = nullptr, int ld = 0);
/* device address of the solve's error word (bit 0: a tile's TMA loads
 * timed out and the tile was skipped) inside the scratch of vpipes_core */
const unsigned *vpipes_error_word(const void *scratch_buf, int nx, int ny, bool padded);
/* what hm_debug_tma_expect_extra has set */
unsigned        tma_extra_tx();
/* flow_simulation (hm_flow.cu): device pointers, ordered on s; scratch of
 * flow_scratch_bytes; water_depth receives the final depth */
int             flow_check_args(const float *z, const float *depth_map, const float *out, int nx, int ny,
                                int iterations, float dt);
bool            flow_wants_padding(const float *z, int nx, int ny, int iterations); /* as vpipes_wants_padding */
size_t          flow_scratch_bytes(int nx, int ny, bool padded);
int             flow_simulation_core(const float *z, int nx, int ny, float water_height, const float *depth_map,
                                     int iterations, float dt, int flux_diffusion, float flux_diffusion_strength,
                                     float dry_out_ratio, float *water_depth, void *scratch, cudaStream_t s,
                                     bool padded);
const unsigned *flow_error_word(const void *scratch, int nx, int ny, bool padded);
/* flow_simulation_viscous (hm_vflow.cu): device pointers, ordered on s;
 * scratch of vflow_scratch_bytes; water_depth receives the final depth */
int             vflow_check_args(const float *z, const float *depth_map, const float *out, int nx, int ny,
                                 int iterations);
size_t          vflow_scratch_bytes(int nx, int ny);
int             vflow_core(const float *z, int nx, int ny, float water_height, const float *depth_map, int iterations,
                           float dt, float dry_out_ratio, float viscosity, float power, float *water_depth,
                           void *scratch, cudaStream_t s);
/* fp64 partial-sum slots vpipes_init needs */
size_t  vpipes_init_partials();
/* water-depth output: stored depth (rows of ld floats, 0: nx) plus the
 * top-up of the last step */
int     vpipes_final_depth(const float *d, const float *rain, const VpScalars *sc, int parity, bool maintain,
                           float *out, int nx, int ny, cudaStream_t s, int ld = 0);
} // namespace hm

#endif
