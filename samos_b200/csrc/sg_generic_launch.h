// sg_generic_launch.h -- launch interface of the generic fused step (sg_generic.cu).
#pragma once
#include "sg_kernels.cuh"

namespace sg {

struct GenericLaunch {
  const Program* prog;
  const Replica* reps;
  const int* blk_rep;
  const Clock* clk;
  Dyn cur, alt;
  Stat st;
  NbList nl;
  int *rebuild, *status;
  double dt_global;
  int apply_e1;
  bool energy;
  double* epart;
  int nblocks, slots;
  const uint8_t* gmask;
  const int* grank;
  int minb;  // blocks per SM of the launch bounds, 6 or 8
  cudaStream_t stream;
};

void launch_generic_step(const GenericLaunch& L);

}  // namespace sg
