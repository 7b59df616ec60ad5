// sg_hot_step.cu -- launches of the packed step kernel (k_hot_step): programs of
// one lj, morse or gaussian potential and at most one aligner under `brownian`
// with their kinds fixed, every other program through the component loops.  By
// kinds alone: the fixed kernel was the faster one at every size (500,009
// particles with morse + polar: 81 -> 46 us a step); steps that report energies
// are one in a run and keep the loops.
#include "sg_hot_launch.h"

namespace sg {

template <int SHAPE, bool ENERGY, int PAIR, int ALIGN>
static void launch(const HotLaunch& L) {
  k_hot_step<SHAPE, ENERGY, PAIR, ALIGN><<<L.nblocks, BLOCK, 0, L.stream>>>(
      *L.prog, L.reps, L.blk_rep, L.clk, L.Gin, L.Gout, L.Hin, L.Hout, L.cur, L.st, L.nl, L.rebuild, L.status,
      L.dt_global, L.apply_e1, L.last, L.epart, L.nblocks);
}

template <int SHAPE, int PAIR>
static void launch_align(const HotLaunch& L) {
  const Program& P = *L.prog;
  if (P.nalign == 0) launch<SHAPE, false, PAIR, HOT_ALIGN_NONE>(L);
  else if (P.align[0].kind == ALIGN_POLAR) launch<SHAPE, false, PAIR, ALIGN_POLAR>(L);
  else launch<SHAPE, false, PAIR, ALIGN_NEMATIC>(L);
}

template <int SHAPE>
static void launch_shape(const HotLaunch& L) {
  const Program& P = *L.prog;
  if (L.energy) return launch<SHAPE, true, HOT_ANY, HOT_ANY>(L);
  const bool one = P.ntypes == 1 && P.npair == 1 && P.nalign <= 1 && P.ninteg == 1 && P.integ[0].kind == INT_BROWNIAN;
  if (one && P.pair[0].kind == PAIR_LJ) return launch_align<SHAPE, PAIR_LJ>(L);
  if (one && P.pair[0].kind == PAIR_MORSE) return launch_align<SHAPE, PAIR_MORSE>(L);
  if (one && P.pair[0].kind == PAIR_GAUSSIAN) return launch_align<SHAPE, PAIR_GAUSSIAN>(L);
  launch<SHAPE, false, HOT_ANY, HOT_ANY>(L);
}

void launch_hot_step(const HotLaunch& L, int shape) {
  if (shape == HOT_PLANE) launch_shape<HOT_PLANE>(L);
  else launch_shape<HOT_SPHERE>(L);
}

}  // namespace sg
