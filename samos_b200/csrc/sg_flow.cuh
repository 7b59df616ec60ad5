// sg_flow.cuh -- Langevin (BAOAB, BBK), NVE and FIRE steps on a periodic plane
// in two launches (sm_100a).
//
// The unfused path moves every field of a particle through memory four or five
// times a step (two integrator halves, the force pass, FIRE's mixing, the step
// counters), each in a launch of its own.  Here a step is
//   k_flow_force   force pass, second half, skin test (FIRE: its sums and control)
//   k_flow_begin   counters, rebuild of flagged replicas, first half of the next step
// on the packed records G = {x, y, nx, ny} and the few fields that the plane
// leaves free: z = zpos, v_z = f_z = n_z = 0 hold exactly after every enforce.
// k_flow_begin is cooperative, since a rebuild passes through grid barriers;
// after one the forces are evaluated again with the new lists before the next
// step begins, as the unfused path does (the sums' order follows the lists).
// Operation order as in sg_kernels.cuh: same bits.
#pragma once
#include "sg_rebuild.cuh"

namespace sg {

enum { FLOW_LANGEVIN = 0, FLOW_NVE = 1, FLOW_FIRE = 2 };
constexpr int FLOW_ANY = -2;  // pair kind or aligner taken from the program (several components, types)

// per-replica constants of a Langevin integrator at constant temperature
// (integrator_langevin.cpp:63-75, 203-210): exp(-gamma dt), the noise amplitude,
// draws per step
struct FlowConst { double exp_dt, B; uint64_t draws; };

struct FlowArgs {
  const Replica* reps;
  const int* blk_rep;
  Clock* clk;
  const D4* Gin;  // k_flow_force
  D4* G;          // records written (k_flow_force: NVE, FIRE) and moved on (k_flow_begin)
  Dyn d;
  Stat st;
  NbList nl;
  int *rebuild, *status;
  const FlowConst* fc;
  double* Rn;
  // FIRE
  double *epart, *part, *alpha_mix, *terms;
  const int *rep_blk0, *rep_nblk;
  int* fire_cnt;
  int nblocks, terms_stride, driver;
  const int* blist;  // blocks taking part (null: all)
  int nblist;
};

// launch interface (sg_flow.cu)
struct FlowKind { int integ, pair, align; };
FlowKind flow_kind(const Program& P);
cudaError_t flow_const(const Program& P, const Replica* reps, int nrep, FlowConst* fc, cudaStream_t stream);
cudaError_t flow_force(const FlowKind& K, const Program& P, const FlowArgs& A, cudaStream_t stream);
cudaError_t flow_begin(const FlowKind& K, const Program& P, const FlowArgs& A, const RebuildArgs& B, int sort_every,
                       bool tail, bool begin, bool pre, int grid, cudaStream_t stream);
cudaError_t flow_begin_blocks(const FlowKind& K, int* blocks_per_sm);

// ---------------------------------------------------------------------------
// forces (and torque) of slot k, neighbours in list order; PAIR / ALIGN fixed
// at compile time for one component of one type, else the program's loops
// (compute_ft).  COH: records and lists may have been written by this kernel.
// ---------------------------------------------------------------------------
template <int PAIR, int ALIGN, bool ENERGY, bool COH>
__device__ __forceinline__ void flow_gather(const Program& P, const Replica& R, const D4* G, const Stat& st,
                                            const NbList& nl, int k, const D4& me, double& fx, double& fy, double& tz,
                                            double (&e)[MAX_PAIR]) {
  constexpr bool ONE = PAIR != FLOW_ANY;
  Part m;
  m.r = st.r[k];
  m.type = !ONE && P.ntypes > 1 ? st.type[k] : 1;
  const int cnt = nl.cnt[k], lo = nl.lo[k];
  const int npair = ONE ? 1 : P.npair;
  const int nalign = ALIGN == FLOW_ANY ? P.nalign : ALIGN == ABP_ALIGN_NONE ? 0 : 1;
  const int nloops = npair > nalign ? npair : nalign;
  fx = fy = tz = 0.0;
  for (int c = 0; c < nloops; c++) {
    const bool hp = ONE || c < npair, ha = c < nalign;
    PairComp pc = P.pair[hp ? c : 0];
    if (ONE) pc.kind = PAIR;
    const int akind = ALIGN == FLOW_ANY ? (ha ? P.align[c].kind : -1) : ALIGN;
    const bool app = ha && P.align[c].has_pp;
    double Jg = ha ? R.align_J[c] : 0.0;
    if (akind == ALIGN_NEMATIC) Jg = 2.0 * Jg;
    const double rcg = ha ? R.align_rcut[c] : 0.0;
    const double* g = R.pair_g[hp ? c : 0];
    // the next entry's record is requested before this one is used
    int j = 0 < cnt ? ld_int<COH>(nl.nb + k) : k;
    int jn = 1 < cnt ? ld_int<COH>(nl.nb + (size_t)nl.stride + k) : k;
    D4 nx = ld_rec<COH>(G + j);
    for (int q = 0; q < cnt; q++) {
      const D4 o4 = nx;
      const int jq = j;
      if (q + 1 < cnt) {
        j = jn;
        nx = ld_rec<COH>(G + j);
        jn = q + 2 < cnt ? ld_int<COH>(nl.nb + (size_t)(q + 2) * nl.stride + k) : k;
      }
      Nb o;
      if (pc.use_radii) o.r = st.r[jq];
      o.type = !ONE && P.ntypes > 1 ? st.type[jq] : 1;
      double dx = o4.x - me.x, dy = o4.y - me.y;
      if (dx > R.xhi) dx -= R.Lx; else if (dx < R.xlo) dx += R.Lx;
      if (dy > R.yhi) dy -= R.Ly; else if (dy < R.ylo) dy += R.Ly;
      const double r_sq = dx * dx + dy * dy;
      const bool upper = q >= lo;
      if (hp) {
        double ff, pe;
        if (pair_term(pc, g, ONE ? 1 : P.ntypes, m, o, r_sq, 1.0, ff, pe)) {
          fx -= ff * dx; fy -= ff * dy;
          if (ENERGY && upper) e[c] += pe;
        }
      }
      if (ha) {
        double J = Jg, rcut = rcg;
        if (app) {
          const double* t = P.align[c].table + ((size_t)(m.type - 1) * P.ntypes + (size_t)(o.type - 1)) * 2;
          J = t[0]; rcut = t[1];
        }
        if (r_sq <= rcut * rcut) {
          const double tau_z = me.z * o4.w - me.w * o4.z;
          if (akind == ALIGN_POLAR) tz += J * tau_z;
          else tz += J * (me.z * o4.z + me.w * o4.w) * tau_z;
        }
      }
    }
  }
}

// ConstraintPlane::enforce on the free fields (plane_enforce)
__device__ __forceinline__ void flow_enforce(const Replica& R, D4& g, int& dix, int& diy) {
  if (g.x <= R.xlo) { g.x += R.Lx; dix--; } else if (g.x > R.xhi) { g.x -= R.Lx; dix++; }
  if (g.y <= R.ylo) { g.y += R.Ly; diy--; } else if (g.y > R.yhi) { g.y -= R.Ly; diy++; }
  const double nn = g.z * g.z + g.w * g.w;
  const double inv = nn != 0.0 ? inv_len(nn) : 1.0;
  g.z *= inv; g.w *= inv;
}

__device__ __forceinline__ bool flow_left_skin(const Replica& R, const NbList& nl, int k, const D4& g) {
  double dx = nl.ox[k] - g.x, dy = nl.oy[k] - g.y;
  if (dx > R.xhi) dx -= R.Lx; else if (dx < R.xlo) dx += R.Lx;
  if (dy > R.yhi) dy -= R.Ly; else if (dy < R.ylo) dy += R.Ly;
  return !(dx * dx + dy * dy < 0.25 * R.pad * R.pad);
}

// ---------------------------------------------------------------------------
// Force pass and second half of a step.
// ---------------------------------------------------------------------------
template <int INTEG, int PAIR, int ALIGN>
__global__ void __launch_bounds__(BLOCK, 8)
k_flow_force(const __grid_constant__ Program P, const __grid_constant__ FlowArgs A) {
  const int bid = A.blist ? A.blist[blockIdx.x] : (int)blockIdx.x;
  const int r = A.blk_rep[bid];
  const Clock& C = A.clk[r];
  if (C.halt) return;
  if (INTEG == FLOW_FIRE && C.fire_conv_step >= 0) return;  // frozen (its partials are kept)
  const Replica& R = A.reps[r];
  const int k = bid * BLOCK + threadIdx.x;
  const double* ip = R.integ_p[0];
  double e[MAX_PAIR];
#pragma unroll
  for (int i = 0; i < MAX_PAIR; i++) e[i] = 0.0;
  double v3[3] = {0.0, 0.0, 0.0}, fmax2 = 0.0;
  if (k - R.off < R.n) {
    D4 g = ldg4(A.Gin + k);
    double fx, fy, tz;
    flow_gather<PAIR, ALIGN, INTEG == FLOW_FIRE, false>(P, R, A.Gin, A.st, A.nl, k, g, fx, fy, tz, e);
    A.d.fx[k] = fx; A.d.fy[k] = fy;
    double vx = A.d.vx[k], vy = A.d.vy[k];
    int dix = 0, diy = 0;
    if (INTEG == FLOW_LANGEVIN) {
      const double dt = ip[0], dt2 = 0.5 * dt, mass = A.st.mass[k];
      if (P.integ[0].method == LANGEVIN_BBK) {  // integrator_langevin.cpp:232-252
        const double gamma = ip[9], B = A.fc[r].B;
        const double one_div_one_p_dt2 = 1.0 / (1.0 + gamma * dt2);
        const double dt2_over_mass = dt2 / mass;
        vx = one_div_one_p_dt2 * (vx + dt2_over_mass * fx);
        vy = one_div_one_p_dt2 * (vy + dt2_over_mass * fy);
        if (B != 0.0) {
          const double stoch_fact = 0.5 * B * one_div_one_p_dt2 / sqrt(mass);
          const uint64_t c0 = C.ctr[0] + (uint64_t)A.st.id[k] * 3u;
          const size_t gi = (size_t)R.off + (size_t)A.st.id[k];
          const double rx = noise_gauss(R.seed[0], c0 + 0), ry = noise_gauss(R.seed[0], c0 + 1);
          A.Rn[3 * gi + 0] = rx; A.Rn[3 * gi + 1] = ry; A.Rn[3 * gi + 2] = noise_gauss(R.seed[0], c0 + 2);
          vx += stoch_fact * rx; vy += stoch_fact * ry;
          A.d.age[k] += dt;
        }
      } else {  // BAOAB, integrator_langevin.cpp:104-111
        const double fact = mass == 1.0 ? dt2 : dt2 / mass;
        vx += fact * fx; vy += fact * fy;
        A.d.age[k] += dt;
      }
    } else if (INTEG == FLOW_NVE) {  // nve.cpp:93-120
      const double dt = ip[0], dt_2 = 0.5 * dt;
      const bool has_limit = ip[12] != 0.0, has_theta = ip[14] != 0.0;
      const double limit = ip[13], theta_limit = ip[15];
      vx += dt_2 * fx; vy += dt_2 * fy;
      if (has_limit) {
        const double v = sqrt(vx * vx + vy * vy);
        if (v * dt > limit) {
          vx = vx / v * limit / dt;
          vy = vy / v * limit / dt;
        }
      }
      flow_enforce(R, g, dix, diy);
      double omega = A.d.omega[k] + dt_2 * (0.0 + tz);
      if (has_limit && has_theta && fabs(omega) * dt > theta_limit) omega = sign_of(omega) * theta_limit / dt;
      A.d.omega[k] = omega;
      A.d.tz[k] = tz;
      A.d.age[k] += dt;
      stg4(A.G + k, g);
    } else {  // k_fire_b
      const double dt_2 = 0.5 * C.fire_dt;
      vx += dt_2 * fx; vy += dt_2 * fy;
      v3[0] = vx * fx + vy * fy;
      v3[1] = fx * fx + fy * fy;
      fmax2 = v3[1];
      v3[2] = vx * vx + vy * vy;
      if (A.terms) {
        const size_t q = (size_t)R.off + (size_t)A.st.id[k];
        A.terms[q] = v3[0]; A.terms[(size_t)A.terms_stride + q] = v3[1]; A.terms[(size_t)2 * A.terms_stride + q] = v3[2];
      }
      flow_enforce(R, g, dix, diy);
      stg4(A.G + k, g);
    }
    A.d.vx[k] = vx; A.d.vy[k] = vy;
    if (dix) A.d.ix[k] += dix;
    if (diy) A.d.iy[k] += diy;
    // skin test: no position changes between here and the next step's first half
    if (flow_left_skin(R, A.nl, k, g) && A.rebuild[r] == 0) atomicOr(&A.rebuild[r], 1);
    if (!(isfinite(g.x) && isfinite(g.y))) atomicOr(A.status, ST_NONFINITE);
  }
  if (INTEG != FLOW_FIRE) return;
  // FIRE: energies and sums per block, then the control in the replica's last block (k_fire_b)
  {
    constexpr int NE = PAIR == FLOW_ANY ? MAX_PAIR : 1;
    double ev[NE];
#pragma unroll
    for (int i = 0; i < NE; i++) ev[i] = e[i];
    block_reduce_store<NE>(ev, A.epart, A.nblocks, bid);
  }
  block_reduce_store<3>(v3, A.part, A.nblocks, bid);
  for (int o = 16; o > 0; o >>= 1) fmax2 = fmax(fmax2, __shfl_down_sync(0xffffffffu, fmax2, o));
  __shared__ double shm[BLOCK / 32];
  if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = fmax2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int i = 0; i < BLOCK / 32; i++) m = fmax(m, shm[i]);
    A.part[(size_t)3 * A.nblocks + bid] = m;
  }
  __shared__ int amlast;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) amlast = atomicAdd(&A.fire_cnt[r], 1) == A.rep_nblk[r] - 1;
  __syncthreads();
  if (!amlast) return;
  __threadfence();
  double sums[5];
  fire_sums(P, A.part, A.epart, A.nblocks, A.rep_blk0[r], A.rep_nblk[r], sums);
  if (A.terms && threadIdx.x < 32) {
    double o[3];
    fire_ordered_sums(A.terms, A.terms_stride, R.off, R.n, o);
    if (threadIdx.x == 0) { sums[0] = o[0]; sums[1] = o[1]; sums[2] = o[2]; }
  }
  if (threadIdx.x == 0) {
    fire_control(R, A.clk[r], r, 0, sums, A.driver, A.alpha_mix);
    A.fire_cnt[r] = 0;
  }
}

// FIRE velocity mixing and the P <= 0 restart (k_fire_d)
__device__ __forceinline__ void flow_mix(const FlowArgs& A, const Clock& C, int r, int k, double fx, double fy, double& vx,
                                         double& vy) {
  if (C.fire_converged) return;
  const double a = A.alpha_mix[r];
  const double inv_Fnorm = 1.0 / C.fire_F;
  const double fact_1 = 1.0 - a;
  const double fact_2 = a * inv_Fnorm * C.fire_V;
  vx = fact_1 * vx + fact_2 * fx;
  vy = fact_1 * vy + fact_2 * fy;
  if (!(C.fire_P > 0.0)) { vx = 0.0; vy = 0.0; }
}

// First half of a step for slot k (k_langevin_a, k_nve_a, k_fire_d and
// k_fire_a): pre, the start-of-step enforce is still to come; mix, FIRE's mixing.
template <int INTEG>
__device__ __forceinline__ void flow_first_half(const Program& P, const FlowArgs& A, const Replica& R, const Clock& C,
                                                int r, int k, bool pre, bool mix, uint64_t base) {
  D4 g = ld4(A.G + k);
  const double* ip = R.integ_p[0];
  const double fx = A.d.fx[k], fy = A.d.fy[k];
  double vx = A.d.vx[k], vy = A.d.vy[k];
  int dix = 0, diy = 0;
  if (INTEG == FLOW_FIRE && mix) flow_mix(A, C, r, k, fx, fy, vx, vy);
  if (pre) flow_enforce(R, g, dix, diy);
  if (INTEG == FLOW_LANGEVIN) {
    const double dt = ip[0], dt2 = 0.5 * dt, mass = A.st.mass[k];
    const double B = A.fc[r].B;
    const uint64_t id = (uint64_t)A.st.id[k];
    if (P.integ[0].method == LANGEVIN_BBK) {  // integrator_langevin.cpp:203-223
      const double gamma = ip[9];
      const double one_m_dt2 = 1.0 - gamma * dt2;
      const double dt2_over_mass = dt2 / mass;
      vx = one_m_dt2 * vx + dt2_over_mass * fx;
      vy = one_m_dt2 * vy + dt2_over_mass * fy;
      if (B != 0.0) {
        const double stoch_fact = 0.5 * B / sqrt(mass);
        const size_t gi = (size_t)R.off + id;
        vx += stoch_fact * A.Rn[3 * gi + 0];
        vy += stoch_fact * A.Rn[3 * gi + 1];
      }
      g.x += dt * vx; g.y += dt * vy;
      flow_enforce(R, g, dix, diy);
    } else {  // BAOAB, integrator_langevin.cpp:63-95
      const double exp_dt = A.fc[r].exp_dt;
      const double fact = mass == 1.0 ? dt2 : dt2 / mass;
      vx += fact * fx; vy += fact * fy;
      g.x += dt2 * vx; g.y += dt2 * vy;
      flow_enforce(R, g, dix, diy);
      vx *= exp_dt; vy *= exp_dt;
      if (B != 0.0) {
        const double stoch_fact = mass == 1.0 ? B : B / sqrt(mass);
        const uint64_t c0 = base + id * 3u;  // the third draw moves v_z, which the enforce clears
        vx += stoch_fact * noise_gauss(R.seed[0], c0 + 0);
        vy += stoch_fact * noise_gauss(R.seed[0], c0 + 1);
      }
      g.x += dt2 * vx; g.y += dt2 * vy;
      flow_enforce(R, g, dix, diy);
    }
  } else if (INTEG == FLOW_NVE) {
    const double dt = ip[0], dt_2 = 0.5 * dt;
    const bool has_limit = ip[12] != 0.0, has_theta = ip[14] != 0.0;
    const double limit = ip[13], theta_limit = ip[15];
    vx += dt_2 * fx; vy += dt_2 * fy;  // nve.cpp:49-55
    flow_enforce(R, g, dix, diy);
    const double omega = A.d.omega[k] + dt_2 * (0.0 + A.d.tz[k]);
    double dx = dt * vx, dy = dt * vy;  // nve.cpp:57-76
    if (has_limit) {
      const double dr = sqrt(dx * dx + dy * dy);
      if (dr > limit) { dx = limit * dx / dr; dy = limit * dy / dr; }
    }
    g.x += dx; g.y += dy;
    flow_enforce(R, g, dix, diy);
    double dtheta = dt * omega;  // nve.cpp:78-86
    if (has_theta && fabs(dtheta) > theta_limit) dtheta = sign_of(dtheta) * theta_limit;
    const double cs = cos(dtheta), sn = sin(dtheta);
    set_unit(cs * g.z + -sn * g.w, sn * g.z + cs * g.w, g.z, g.w);
    A.d.omega[k] = omega;
  } else {
    const double dt = C.fire_dt, dt_2 = 0.5 * dt;
    vx += dt_2 * fx; vy += dt_2 * fy;
    g.x += dt * vx; g.y += dt * vy;
    flow_enforce(R, g, dix, diy);
    // no aligner: the torque is 0, and so the half kick of omega
    const double dtheta = dt * (A.d.omega[k] + dt_2 * 0.0);
    const double cs = cos(dtheta), sn = sin(dtheta);
    set_unit(cs * g.z + -sn * g.w, sn * g.z + cs * g.w, g.z, g.w);
  }
  stg4(A.G + k, g);
  A.d.vx[k] = vx; A.d.vy[k] = vy;
  if (dix) A.d.ix[k] += dix;
  if (diy) A.d.iy[k] += diy;
}

// Counters and rebuild of the step just done (tail), first half of the next
// (begin; without a tail, pre says whether its enforce is still to come).
// executed[1]: the last tail rebuilt lists and left the forces as they were.
template <int INTEG, int PAIR, int ALIGN>
__global__ void __launch_bounds__(BLOCK, 8)
k_flow_begin(const __grid_constant__ Program P, const __grid_constant__ FlowArgs A, const __grid_constant__ RebuildArgs B,
             int sort_every, int tail, int begin, int pre) {
  __shared__ RebuildList L;
  const int t = threadIdx.x;
  if (B.clk[0].halt) return;  // set between launches only
  const unsigned long long t0 = global_ns();
  GridBar bar{B.bar, 0u, B.status};
  // converged replicas are frozen: a request of their last iteration is dropped
  const bool flagged = tail && rebuild_list(B, sort_every, L, INTEG == FLOW_FIRE);
  bool over = false;
  if (flagged) {
    if (INTEG == FLOW_FIRE)  // the mixing reads the forces that the rebuild replaces
      for (int v = blockIdx.x; v < L.nblk; v += gridDim.x) {
        const int s = list_find(L.blk, L.n, v), r = L.rep[s];
        const Replica& R = A.reps[r];
        const int k = R.off + (v - L.blk[s]) * BLOCK + t;
        if (k - R.off >= R.n) continue;
        double vx = A.d.vx[k], vy = A.d.vy[k];
        flow_mix(A, A.clk[r], r, k, A.d.fx[k], A.d.fy[k], vx, vy);
        A.d.vx[k] = vx; A.d.vy[k] = vy;
      }
    if (!rebuild_phases<HOT_PLANE>(B, L, bar)) return;
    if (!grid_wait(bar)) return;
    over = (__ldcg(B.bstatus) & ST_OVERFLOW) != 0;
    if (!over && begin) {
      // the start-of-step enforce, then the forces with the new lists
      for (int v = blockIdx.x; v < L.nblk; v += gridDim.x) {
        const int s = list_find(L.blk, L.n, v);
        const Replica& R = A.reps[L.rep[s]];
        const int k = R.off + (v - L.blk[s]) * BLOCK + t;
        if (k - R.off >= R.n) continue;
        D4 g = ld4(A.G + k);
        int dix = 0, diy = 0;
        flow_enforce(R, g, dix, diy);
        stg4(A.G + k, g);
        if (dix) A.d.ix[k] += dix;
        if (diy) A.d.iy[k] += diy;
      }
      if (!grid_wait(bar)) return;
      for (int v = blockIdx.x; v < L.nblk; v += gridDim.x) {
        const int s = list_find(L.blk, L.n, v);
        const Replica& R = A.reps[L.rep[s]];
        const int k = R.off + (v - L.blk[s]) * BLOCK + t;
        if (k - R.off >= R.n) continue;
        double fx, fy, tz, e[MAX_PAIR];
        const D4 g = ld4(A.G + k);
        flow_gather<PAIR, ALIGN, false, true>(P, R, A.G, A.st, A.nl, k, g, fx, fy, tz, e);
        A.d.fx[k] = fx; A.d.fy[k] = fy;
        if (INTEG == FLOW_NVE) A.d.tz[k] = tz;
      }
      if (!grid_wait(bar)) return;  // the neighbours' records move on below
    }
  }
  for (int v = blockIdx.x; v < A.nblist && (begin || INTEG == FLOW_FIRE); v += gridDim.x) {
    const int bid = A.blist ? A.blist[v] : v;
    const int r = A.blk_rep[bid];
    const Clock& C = A.clk[r];
    if (INTEG == FLOW_FIRE && C.fire_conv_step >= 0) continue;
    const Replica& R = A.reps[r];
    const int k = bid * BLOCK + t;
    if (k - R.off >= R.n) continue;
    const bool redo = flagged && __ldcg(B.rebuild + r) != 0;  // cleared by the last block below
    if (begin && !over) {
      uint64_t base = 0;
      if (INTEG == FLOW_LANGEVIN) base = C.ctr[0] + (tail ? A.fc[r].draws : 0ull);
      flow_first_half<INTEG>(P, A, R, C, r, k, tail ? !redo : pre != 0, tail && !redo, base);
    } else if (INTEG == FLOW_FIRE && !redo) {  // the step ends with its mixing
      double vx = A.d.vx[k], vy = A.d.vy[k];
      flow_mix(A, C, r, k, A.d.fx[k], A.d.fy[k], vx, vy);
      A.d.vx[k] = vx; A.d.vy[k] = vy;
    }
  }
  // the block that finishes last: every other has read the clocks and flags
  if (!tail) return;
  if (!grid_last(bar)) return;
  for (int r = t; r < B.nrep; r += BLOCK) tail_one(P, A.reps[r], A.clk[r]);
  if (t == 0) {
    B.executed[0]++;
    B.executed[1] = flagged && !begin ? 1 : 0;
  }
  if (flagged) rebuild_done(B, L, t0);
  if (INTEG == FLOW_FIRE && !over)
    for (int r = t; r < B.nrep; r += BLOCK)
      if (A.clk[r].fire_conv_step >= 0) B.rebuild[r] = 0;
}

}  // namespace sg
