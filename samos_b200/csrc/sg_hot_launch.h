// sg_hot_launch.h -- launch interface of the packed step kernel (sg_hot_step.cu).
#pragma once
#include "sg_hot.cuh"

namespace sg {

struct HotLaunch {
  const Program* prog;
  const Replica* reps;
  const int* blk_rep;
  const Clock* clk;
  const D4 *Gin, *Hin;
  D4 *Gout, *Hout;
  Dyn cur;
  Stat st;
  NbList nl;
  int *rebuild, *status;
  double dt_global;
  int apply_e1, last;
  bool energy;
  double* epart;
  int nblocks;
  cudaStream_t stream;
};

void launch_hot_step(const HotLaunch& L, int shape);

}  // namespace sg
