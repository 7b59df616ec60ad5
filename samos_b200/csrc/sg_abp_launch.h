// sg_abp_launch.h -- launch interface of the specialised active-Brownian step
// kernels.  Each shape / aligner pair is compiled in a unit of its own
// (sg_abp_*.cu), so the kernel variants build side by side.
#pragma once
#include "sg_abp.cuh"

namespace sg {

struct AbpLaunch {
  const AbpParams* abp;  // per replica
  AbpParams abp0;        // replica 0's, passed by value to the by-value variants
  const int* blk_rep;
  const Clock* clk;
  const D4 *Gin, *Hin;
  D4 *Gout, *Hout;
  Dyn cur;
  Stat st;
  NbList nl;
  int *rebuild, *status;
  int apply_e1, last;
  bool energy, self_propulsion;
  double* epart;
  int nblocks;
  const uint8_t* lane_order;
  const int *tile_n, *tile_slot;
  const uint16_t* nbpos;
  int nrep, variant, device;
  cudaStream_t stream;
};

void launch_abp_plane_none(const AbpLaunch& L);
void launch_abp_plane_polar(const AbpLaunch& L);
void launch_abp_plane_nematic(const AbpLaunch& L);
void launch_abp_sphere_none(const AbpLaunch& L);
void launch_abp_sphere_polar(const AbpLaunch& L);
void launch_abp_sphere_nematic(const AbpLaunch& L);

}  // namespace sg
