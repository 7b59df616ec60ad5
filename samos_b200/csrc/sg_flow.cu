// sg_flow.cu -- the two-launch Langevin / NVE / FIRE step: kernel instances and
// their launches.
#include "sg_flow.cuh"

namespace sg {

static __global__ void k_flow_const(Program P, const Replica* reps, int nrep, FlowConst* fc) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrep) return;
  const double* ip = reps[r].integ_p[0];
  const double dt = ip[0], gamma = ip[9], T = P.integ[0].temp.min_val;
  FlowConst c;
  c.exp_dt = exp(-gamma * dt);
  c.B = P.integ[0].method == LANGEVIN_BBK ? sqrt(2.0 * T * dt * gamma) : sqrt(T * (1.0 - exp(-2.0 * gamma * dt)));
  c.draws = langevin_draws(P.integ[0], ip, 0, reps[r].n);
  fc[r] = c;
}

cudaError_t flow_const(const Program& P, const Replica* reps, int nrep, FlowConst* fc, cudaStream_t stream) {
  k_flow_const<<<(nrep + 63) / 64, 64, 0, stream>>>(P, reps, nrep, fc);
  return cudaGetLastError();
}

// Kernel instances: one pair potential of one particle type with its kind (and
// the aligner's, which only NVE integrates) known at compile time; everything
// else through the program's loops.
FlowKind flow_kind(const Program& P) {
  FlowKind K;
  K.integ = P.integ[0].kind == INT_LANGEVIN ? FLOW_LANGEVIN : P.integ[0].kind == INT_NVE ? FLOW_NVE : FLOW_FIRE;
  const bool one = P.ntypes == 1 && P.npair == 1;
  K.pair = one ? P.pair[0].kind : FLOW_ANY;
  K.align = ABP_ALIGN_NONE;
  if (K.integ == FLOW_NVE) {
    K.align = P.nalign == 0 ? ABP_ALIGN_NONE : P.nalign == 1 ? P.align[0].kind : FLOW_ANY;
    if (K.pair != PAIR_SOFT && !(K.pair == PAIR_LJ && K.align == ABP_ALIGN_NONE)) K.pair = FLOW_ANY;
    if (K.pair == FLOW_ANY || K.align == FLOW_ANY) K.pair = K.align = FLOW_ANY;
  }
  if (K.integ == FLOW_FIRE && K.pair != PAIR_SOFT) K.pair = FLOW_ANY;
  return K;
}

// calls f with the instance's constants
template <class F>
static cudaError_t flow_dispatch(const FlowKind& K, F&& f) {
#define FLOW_CASE(I, Q, A) \
  if (K.integ == I && K.pair == Q && K.align == A) return f.template operator()<I, Q, A>();
  FLOW_CASE(FLOW_LANGEVIN, PAIR_SOFT, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_LANGEVIN, PAIR_LJ, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_LANGEVIN, PAIR_MORSE, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_LANGEVIN, PAIR_GAUSSIAN, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_LANGEVIN, FLOW_ANY, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_NVE, PAIR_SOFT, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_NVE, PAIR_SOFT, ALIGN_POLAR)
  FLOW_CASE(FLOW_NVE, PAIR_SOFT, ALIGN_NEMATIC)
  FLOW_CASE(FLOW_NVE, PAIR_LJ, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_NVE, FLOW_ANY, FLOW_ANY)
  FLOW_CASE(FLOW_FIRE, PAIR_SOFT, ABP_ALIGN_NONE)
  FLOW_CASE(FLOW_FIRE, FLOW_ANY, ABP_ALIGN_NONE)
#undef FLOW_CASE
  return cudaErrorInvalidValue;
}

struct LaunchForce {
  const Program& P;
  const FlowArgs& A;
  cudaStream_t stream;
  template <int I, int Q, int L> cudaError_t operator()() const {
    k_flow_force<I, Q, L><<<A.nblist, BLOCK, 0, stream>>>(P, A);
    return cudaGetLastError();
  }
};

struct LaunchBegin {
  const Program& P;
  const FlowArgs& A;
  const RebuildArgs& B;
  D4 *G0, *G1;
  int sort_every, tail, begin, pre, nsteps, grid;
  cudaStream_t stream;
  template <int I, int Q, int L> cudaError_t operator()() const {
    LaunchBegin a = *this;
    void* args[] = {const_cast<Program*>(&P), const_cast<FlowArgs*>(&A), const_cast<RebuildArgs*>(&B), &a.G0, &a.G1,
                    &a.sort_every, &a.tail, &a.begin, &a.pre, &a.nsteps};
    return cudaLaunchCooperativeKernel((const void*)k_flow_begin<I, Q, L>, dim3(grid), dim3(BLOCK), args, 0, stream);
  }
};

struct BeginBlocks {
  int* per;
  template <int I, int Q, int L> cudaError_t operator()() const {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, (const void*)k_flow_begin<I, Q, L>, BLOCK, 0);
  }
};

cudaError_t flow_force(const FlowKind& K, const Program& P, const FlowArgs& A, cudaStream_t stream) {
  return flow_dispatch(K, LaunchForce{P, A, stream});
}

cudaError_t flow_begin(const FlowKind& K, const Program& P, const FlowArgs& A, const RebuildArgs& B, int sort_every,
                       bool tail, bool begin, bool pre, int nsteps, D4* G0, D4* G1, int grid, cudaStream_t stream) {
  return flow_dispatch(K, LaunchBegin{P, A, B, G0, G1, sort_every, tail, begin, pre, nsteps, grid, stream});
}

cudaError_t flow_begin_occupancy(const FlowKind& K, int* blocks_per_sm) {
  return flow_dispatch(K, BeginBlocks{blocks_per_sm});
}

struct LaunchRun {
  const Program& P;
  const FlowArgs& A;
  const RebuildArgs& B;
  D4 *G0, *G1;
  unsigned long long* word;
  int nsteps, grid;
  cudaStream_t stream;
  template <int I, int Q, int L> cudaError_t operator()() const {
    LaunchRun a = *this;
    void* args[] = {const_cast<Program*>(&P), const_cast<FlowArgs*>(&A), const_cast<RebuildArgs*>(&B), &a.G0, &a.G1,
                    &a.word, &a.nsteps};
    return cudaLaunchCooperativeKernel((const void*)k_flow_run<I, Q, L>, dim3(grid), dim3(BLOCK), args, 0, stream);
  }
};

struct RunBlocks {
  int* per;
  template <int I, int Q, int L> cudaError_t operator()() const {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, (const void*)k_flow_run<I, Q, L>, BLOCK, 0);
  }
};

cudaError_t flow_run(const FlowKind& K, const Program& P, const FlowArgs& A, const RebuildArgs& B, D4* G0, D4* G1,
                     unsigned long long* word, int nsteps, int grid, cudaStream_t stream) {
  return flow_dispatch(K, LaunchRun{P, A, B, G0, G1, word, nsteps, grid, stream});
}

cudaError_t flow_run_occupancy(const FlowKind& K, int* blocks_per_sm) {
  return flow_dispatch(K, RunBlocks{blocks_per_sm});
}

}  // namespace sg
