// Rodas5P with a trajectory's state cut into MDX_TEAM equal blocks, one per lane
// (4 to 32 lanes, a power of two, so a trajectory never straddles a warp).
//
// For systems that repeat themselves around a ring (_cyclic.py finds them) every
// lane runs the same straight-line code on MDX_BLOCK components of its own, with
// the state, the eight stage increments and the factors in its registers; a
// neighbour's seam components come by shuffle.  The step is the thread kernel's
// (mdx_rodas5p.cuh) in fast arithmetic with its FP64 solves (MDX_WIDE_SOLVE): matrix and
// factorisation in MDX_LU_T, the factors widened once per step, everything else in
// double.  Only the order of elimination and of the error sum differ.
//
// Solves in MDX_LU_T are 7% to 30% faster and further from the FP64-LU solve than
// the team and thread kernels' own in FP32, whose elimination orders differ: Van der Pol
// rings, 512 trajectories, distance over the result's norm with FP32 / FP64 solves here and
// in the thread kernel: 32 states over [0, 100] 2.5e-4 to 3.0e-4 / 1.1e-4 and 2.2e-4 / 1.1e-4,
// 16 states over [0, 300] 1.2e-3 / 2.9e-4 to 3.9e-4 and 1.5e-3 / 3.7e-4.
//
// What bounds it: the step's dependent chain (a stage is a right-hand side, a
// tableau row, the interior's substitutions and log2(MDX_TEAM) exchanges) while
// few trajectories are left, instruction issue while the device is full.  The team
// kernel (mdx_team.cuh) factorises and solves on one lane of a trajectory out of
// shared memory; here all lanes work on every phase and nothing leaves registers.
// Calls on a B200, that kernel / this: 32-state Van der Pol ring, 8,192 trajectories,
// 110.9 / 24.0 ms (8 lanes; FP32 solves 22.4, the factorisation in FP64 too 28.3);
// 64-state Brusselator, 16,384, 16.7 / 4.0 ms (8 lanes, 255 registers and 0.8 KB of spills a
// thread; 16 lanes 4.5, 32 lanes 7.3; FP32 solves 3.1, all in FP64 4.6).
//
// The whole warp steps together: lanes whose trajectory is done step on stale
// values and commit nothing, so every shuffle names the full warp.
#pragma once
#include "mdx_common.cuh"
#include "mdx_rodas5p_coef.cuh"

namespace mdx {
namespace cyclic {

using rodas5p::coef_a;
using rodas5p::coef_c;
using rodas5p::coef_ct;
using rodas5p::coef_d;
using rodas5p::coef_h;
using rodas5p::FACTOR_MAX;
using rodas5p::FACTOR_MIN;
using rodas5p::GAMMA;

constexpr int B = MDX_BLOCK;
constexpr int Q = MDX_SEPARATORS;
constexpr int LEVELS = MDX_TEAM == 32 ? 5 : MDX_TEAM == 16 ? 4 : MDX_TEAM == 8 ? 3 : 2;
static_assert(MDX_TEAM == 4 || MDX_TEAM == 8 || MDX_TEAM == 16 || MDX_TEAM == 32, "4, 8, 16 or 32 lanes");
static_assert(MDX_TPB % 32 == 0, "blocks are whole warps");
static_assert(B * MDX_TEAM == MDX_NV && MDX_NS == MDX_NV, "equal blocks of the plain system");

struct State {
  double y[B];
  double p[MDX_LANE_PARAMS > 0 ? MDX_LANE_PARAMS : 1];
  double t, dt, err_prev, err_prev2, tf_local;
  double next_save;  // times[save_idx]: read when the cursor moves, not on every step
  int save_idx, n_steps, accepted, rejected, traj;
};

__device__ __forceinline__ Lane lane_of_thread() {
  const int lane = (int)(threadIdx.x & (MDX_TEAM - 1));
  const int base = (int)(threadIdx.x & 31u) - lane;
  return Lane{lane, base, base + ((lane + MDX_TEAM - 1) & (MDX_TEAM - 1)), base + ((lane + 1) & (MDX_TEAM - 1))};
}

// --- the separators' block tridiagonal cyclic system --------------------------------
typedef lu_t Block[Q * Q];

// c (-)= a b, all q x q.
template <bool SUBTRACT>
__device__ __forceinline__ void multiply(const Block& a, const Block& b, Block& c) {
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int j = 0; j < Q; ++j) {
      lu_t acc = SUBTRACT ? c[i * Q + j] : (lu_t)0;
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        if constexpr (SUBTRACT) acc -= a[i * Q + k] * b[k * Q + j];
        else acc += a[i * Q + k] * b[k * Q + j];
      }
      c[i * Q + j] = acc;
    }
}

// r -= a x
__device__ __forceinline__ void subtract(const double (&a)[Q * Q], const double (&x)[Q], double (&r)[Q]) {
#pragma unroll
  for (int i = 0; i < Q; ++i)
#pragma unroll
    for (int k = 0; k < Q; ++k) r[i] -= a[i * Q + k] * x[k];
}

// The inverse by Gauss-Jordan elimination in place, unpivoted like the sparse LU;
// unlike a determinant it squares no entry, so 1/(h gamma) may be as large as FP32 holds.
__device__ __forceinline__ void invert(Block& a) {
#pragma unroll
  for (int p = 0; p < Q; ++p) {
    const lu_t r = fast_recip(a[p * Q + p]);
    a[p * Q + p] = (lu_t)1;
#pragma unroll
    for (int j = 0; j < Q; ++j) a[p * Q + j] *= r;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      if (i == p) continue;
      const lu_t f = a[i * Q + p];
      a[i * Q + p] = (lu_t)0;
#pragma unroll
      for (int j = 0; j < Q; ++j) a[i * Q + j] -= f * a[p * Q + j];
    }
  }
}

__device__ __forceinline__ void from_lane(const Block& v, int src, Block& out) {
#pragma unroll
  for (int i = 0; i < Q * Q; ++i) out[i] = __shfl_sync(MDX_FULL_MASK, v[i], src);
}

// A lane's factors: its interior's, and per reduction level the multiples of the
// rows `reach` lanes to the left and right that eliminate them.
template <class T>
struct FactorsOf {
  T lu[LU_SIZE];
  T left[LEVELS][Q * Q], right[LEVELS][Q * Q];  // the last level has one partner: left only
  T inverse[Q * Q];
};
typedef FactorsOf<lu_t> Factors;    // as factorised
typedef FactorsOf<double> Solver;   // as the stages solve with them

__device__ __forceinline__ void widen(const Factors& F, Solver& S) {
#pragma unroll
  for (int i = 0; i < LU_SIZE; ++i) S.lu[i] = (double)F.lu[i];
#pragma unroll
  for (int i = 0; i < Q * Q; ++i) {
#pragma unroll
    for (int k = 0; k < LEVELS; ++k) S.left[k][i] = (double)F.left[k][i];
#pragma unroll
    for (int k = 0; k < LEVELS - 1; ++k) S.right[k][i] = (double)F.right[k][i];
    S.inverse[i] = (double)F.inverse[i];
  }
}

__device__ __forceinline__ int lane_at(const Lane& L, int offset) {
  return L.base + ((L.lane + offset) & (MDX_TEAM - 1));
}

__device__ __forceinline__ void factorize(Factors& F, const Block& next, const Lane& L) {
  eliminate(F.lu);
  Block a, b, c;
#pragma unroll
  for (int i = 0; i < Q * Q; ++i) {
    a[i] = F.lu[2 * Q * Q + i];
    b[i] = F.lu[3 * Q * Q + i];
    c[i] = next[i];
    if constexpr (HAS_INTERIOR) {
      // The next lane's interior joins its left separators, which are this lane's.
      b[i] += __shfl_sync(MDX_FULL_MASK, F.lu[i], L.right);
      c[i] += __shfl_sync(MDX_FULL_MASK, F.lu[Q * Q + i], L.right);
    }
  }
#pragma unroll
  for (int k = 0; k < LEVELS - 1; ++k) {
    const int l = lane_at(L, -(1 << k)), r = lane_at(L, 1 << k);
    Block inv, other, na, nc;
#pragma unroll
    for (int i = 0; i < Q * Q; ++i) inv[i] = b[i];
    invert(inv);
    from_lane(inv, l, other);
    multiply<false>(a, other, F.left[k]);
    from_lane(inv, r, other);
    multiply<false>(c, other, F.right[k]);
    from_lane(c, l, other);
    multiply<true>(F.left[k], other, b);
    from_lane(a, r, other);
    multiply<true>(F.right[k], other, b);
    from_lane(a, l, other);
    multiply<false>(F.left[k], other, na);
    from_lane(c, r, other);
    multiply<false>(F.right[k], other, nc);
#pragma unroll
    for (int i = 0; i < Q * Q; ++i) {
      a[i] = -na[i];
      c[i] = -nc[i];
    }
  }
  // Half a turn away both neighbours are the same lane.
  const int partner = lane_at(L, MDX_TEAM / 2);
  Block inv, other;
#pragma unroll
  for (int i = 0; i < Q * Q; ++i) {
    a[i] += c[i];
    inv[i] = b[i];
  }
  invert(inv);
  from_lane(inv, partner, other);
  multiply<false>(a, other, F.left[LEVELS - 1]);
  from_lane(a, partner, other);
  multiply<true>(F.left[LEVELS - 1], other, b);
#pragma unroll
  for (int i = 0; i < Q * Q; ++i) F.inverse[i] = b[i];
  invert(F.inverse);
}

__device__ __forceinline__ void solve(const Solver& F, double (&r)[B], const Lane& L) {
  double left[Q], x[Q], xl[Q], xr[Q];
  if constexpr (HAS_INTERIOR) {
#pragma unroll
    for (int s = 0; s < Q; ++s) left[s] = 0.0;
    interior_forward(F.lu, r, left);
  }
#pragma unroll
  for (int s = 0; s < Q; ++s) {
    x[s] = r[separator(s)];
    if constexpr (HAS_INTERIOR) x[s] += __shfl_sync(MDX_FULL_MASK, left[s], L.right);
  }
#pragma unroll
  for (int k = 0; k < LEVELS - 1; ++k) {
    const int l = lane_at(L, -(1 << k)), rt = lane_at(L, 1 << k);
#pragma unroll
    for (int s = 0; s < Q; ++s) {
      xl[s] = __shfl_sync(MDX_FULL_MASK, x[s], l);
      xr[s] = __shfl_sync(MDX_FULL_MASK, x[s], rt);
    }
    subtract(F.left[k], xl, x);
    subtract(F.right[k], xr, x);
  }
  const int partner = lane_at(L, MDX_TEAM / 2);
#pragma unroll
  for (int s = 0; s < Q; ++s) xl[s] = __shfl_sync(MDX_FULL_MASK, x[s], partner);
  subtract(F.left[LEVELS - 1], xl, x);
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    double acc = F.inverse[i * Q] * x[0];
#pragma unroll
    for (int k = 1; k < Q; ++k) acc += F.inverse[i * Q + k] * x[k];
    r[separator(i)] = acc;
  }
  if constexpr (HAS_INTERIOR) {
#pragma unroll
    for (int s = 0; s < Q; ++s) left[s] = __shfl_sync(MDX_FULL_MASK, r[separator(s)], L.left);
    interior_backward(F.lu, r, left);
  }
}

// --- the solver ------------------------------------------------------------------------
__device__ __forceinline__ size_t hist_index(const MdxSolveArgs& a, int traj, int s, const Lane& L) {
  return ((size_t)traj * (size_t)a.n_save_hist + (size_t)s) * (size_t)MDX_NV + (size_t)(L.lane * B);
}

__device__ __forceinline__ double weight(const MdxSolveArgs& a, int traj, int j) {
#if MDX_WEIGHTS_RUNTIME
  return a.weights[(size_t)traj * MDX_NV + j];
#else
  (void)a; (void)traj; (void)j;
  return 1.0;
#endif
}

// A state to step on before a lane has had a trajectory.
__device__ __forceinline__ void rest(State& st) {
#pragma unroll
  for (int j = 0; j < B; ++j) st.y[j] = 0.0;
#pragma unroll
  for (int k = 0; k < MDX_LANE_PARAMS; ++k) st.p[k] = 0.0;
  st.t = st.tf_local = st.next_save = 0.0;
  st.dt = st.err_prev = st.err_prev2 = 1.0;
  st.save_idx = st.n_steps = st.accepted = st.rejected = st.traj = 0;
}

__device__ __forceinline__ void init(State& st, const MdxSolveArgs& a, int traj, const Lane& L) {
  st.traj = traj;
  const double* y0 = a.y0 + (size_t)traj * MDX_NV + L.lane * B;
  double* row = a.hist + hist_index(a, traj, 0, L);
#pragma unroll
  for (int j = 0; j < B; ++j) {
    st.y[j] = y0[j];
    row[j] = st.y[j];
  }
#pragma unroll
  for (int k = 0; k < MDX_LANE_PARAMS; ++k) st.p[k] = a.params[(size_t)traj * MDX_NP + param_column(k, L.lane)];
  const double t0 = a.times[0];
  const double tf = a.times[a.n_save - 1];
  st.t = t0;
  st.dt = a.dt0 > 0.0 ? a.dt0 : (tf - t0) * 1e-6;
  st.save_idx = 1;
  st.next_save = a.times[a.n_save > 1 ? 1 : 0];
  st.n_steps = 0;
  st.accepted = 0;
  st.rejected = 0;
  st.err_prev = 1.0;
  st.err_prev2 = 1.0;
#if MDX_TF_INDEX >= 0
  st.tf_local = a.params[(size_t)traj * MDX_NP + MDX_TF_INDEX];
#else
  st.tf_local = tf;
#endif
}

__device__ __forceinline__ bool running(const State& st, const MdxSolveArgs& a) {
  return st.save_idx < a.n_save && st.t < st.tf_local && st.n_steps < a.max_steps;
}

// Stage S: its right-hand side from f (in `work`) and the tableau row, then the solve.
template <int S, class DT>
__device__ __forceinline__ void stage(const Solver& F, double (&k)[8][B], const double (&work)[B], const DT& dT,
                                      double dt_use, double inv_dt, const Lane& L) {
  double r[B];
#pragma unroll
  for (int j = 0; j < B; ++j) {
    double value = work[j];
#if !MDX_AUTONOMOUS
    if constexpr (coef_d(S) != 0.0) value += dt_use * coef_d(S) * dT[j];
#else
    (void)dt_use; (void)dT;
#endif
    if constexpr (S > 0) {
      double acc = coef_c(S, 0) * k[0][j];
#pragma unroll
      for (int m = 1; m < S; ++m) acc += coef_c(S, m) * k[m][j];
      value += acc * inv_dt;
    }
    r[j] = value;
  }
  solve(F, r, L);
#pragma unroll
  for (int j = 0; j < B; ++j) k[S][j] = r[j];
}

template <int S>
__device__ __forceinline__ void advance(double (&u)[B], const State& st, const double (&k)[8][B]) {
#pragma unroll
  for (int j = 0; j < B; ++j) {
    double acc = coef_a(S, 0) * k[0][j];
#pragma unroll
    for (int m = 1; m <= S; ++m) acc += coef_a(S, m) * k[m][j];
    u[j] = st.y[j] + acc;
  }
}

// One attempted step of every lane; lanes that are not `active` commit nothing.
__device__ __forceinline__ void step(State& st, const MdxSolveArgs& a, const Lane& L, bool active) {
  double dt_use = st.dt;
  if (dt_use > st.tf_local - st.t) dt_use = st.tf_local - st.t;
  if (dt_use < 1e-30) dt_use = 1e-30;
  const double t = st.t;
  const double t_end = t + dt_use;
  const double inv_dt = recip_newton(dt_use);

  Factors factors;
  Block next;
  matrix(st.y, t, st.p, inv_dt * (1.0 / GAMMA), factors.lu, next, L);
  double dT[B];
#if !MDX_AUTONOMOUS
  time_derivative(st.y, t, st.p, dT, L);
#endif
  factorize(factors, next, L);
  Solver F;
  widen(factors, F);

  double k[8][B];
  double u[B], work[B];
  rhs(st.y, t, st.p, work, L);
  stage<0>(F, k, work, dT, dt_use, inv_dt, L);
  advance<0>(u, st, k);
  rhs(u, t + coef_ct(0) * dt_use, st.p, work, L);
  stage<1>(F, k, work, dT, dt_use, inv_dt, L);
  advance<1>(u, st, k);
  rhs(u, t + coef_ct(1) * dt_use, st.p, work, L);
  stage<2>(F, k, work, dT, dt_use, inv_dt, L);
  advance<2>(u, st, k);
  rhs(u, t + coef_ct(2) * dt_use, st.p, work, L);
  stage<3>(F, k, work, dT, dt_use, inv_dt, L);
  advance<3>(u, st, k);
  rhs(u, t + coef_ct(3) * dt_use, st.p, work, L);
  stage<4>(F, k, work, dT, dt_use, inv_dt, L);
  advance<4>(u, st, k);
  rhs(u, t_end, st.p, work, L);
  stage<5>(F, k, work, dT, dt_use, inv_dt, L);
#pragma unroll
  for (int j = 0; j < B; ++j) u[j] += k[5][j];
  rhs(u, t_end, st.p, work, L);
  stage<6>(F, k, work, dT, dt_use, inv_dt, L);
#pragma unroll
  for (int j = 0; j < B; ++j) u[j] += k[6][j];
  rhs(u, t_end, st.p, work, L);
  stage<7>(F, k, work, dT, dt_use, inv_dt, L);

  // Weighted mean square of k8: a lane's own components, then over the lanes in
  // pairs, which leaves the same bits on every lane of a trajectory.
  double err = 0.0;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const double k7 = k[7][j];
    const double y_new = u[j] + k7;
    const double scale = a.atol + a.rtol * pymax(fabs(st.y[j]), fabs(y_new));
    const double r = weight(a, st.traj, L.lane * B + j) * k7 * recip_newton(scale);
    err += r * r;
  }
#pragma unroll
  for (int d = 1; d < MDX_TEAM; d *= 2) err += __shfl_xor_sync(MDX_FULL_MASK, err, d);
  const double err_sq = err * (1.0 / MDX_NERR);
  const bool accept = err_sq <= 1.0;
  double safe_err;
  double factor = controller_factor_sq(err_sq, st.err_prev, st.err_prev2, MDX_E1, MDX_E2, MDX_E3,
                                       MDX_USE_E2, MDX_USE_E3, safe_err);
  if (factor < FACTOR_MIN) factor = FACTOR_MIN;
  else if (factor > FACTOR_MAX) factor = FACTOR_MAX;
  if (!active) return;
  st.dt = dt_use * factor;
  if (accept) {
    st.err_prev2 = st.err_prev;
    st.err_prev = safe_err;
    const double t_new = t + dt_use;
    while (st.save_idx < a.n_save && save_reached(st.next_save, t_new)) {
      // The thread kernel's dense output: eight weights shared by every component.
      const double theta = (st.next_save - t) * inv_dt;
      const double theta1 = 1.0 - theta;
      double w[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) w[m] = coef_h(0, m) + theta * (coef_h(1, m) + theta * coef_h(2, m));
      double* row = a.hist + hist_index(a, st.traj, st.save_idx, L);
#pragma unroll
      for (int j = 0; j < B; ++j) {
        double hsum = w[0] * k[0][j];
#pragma unroll
        for (int m = 1; m < 8; ++m) hsum += w[m] * k[m][j];
        const double y_new = u[j] + k[7][j];
        row[j] = theta1 * st.y[j] + theta * (y_new + theta1 * hsum);
      }
      ++st.save_idx;
      if (st.save_idx < a.n_save) st.next_save = a.times[st.save_idx];
    }
#pragma unroll
    for (int j = 0; j < B; ++j) st.y[j] = u[j] + k[7][j];
    st.t += dt_use;
    ++st.accepted;
  } else {
    ++st.rejected;
  }
  ++st.n_steps;
}

// Ends the trajectories of the lanes where `done`; the whole warp comes here.
__device__ __forceinline__ void finish(State& st, const MdxSolveArgs& a, const Lane& L, bool done) {
  bool bad = false;
#pragma unroll
  for (int j = 0; j < B; ++j) bad |= !isfinite(st.y[j]);
  const unsigned bads = __ballot_sync(MDX_FULL_MASK, bad) >> L.base;
  if (done) {
    const bool hit_max = st.save_idx < a.n_save && st.t < st.tf_local;
    // Saves past this trajectory's end hold its final state (modax/rodas5P.py:991-1002).
    for (; st.save_idx < a.n_save; ++st.save_idx) {
      double* row = a.hist + hist_index(a, st.traj, st.save_idx, L);
#pragma unroll
      for (int j = 0; j < B; ++j) row[j] = st.y[j];
    }
    if (L.lane == 0) {
      a.accepted[st.traj] = st.accepted;
      a.rejected[st.traj] = st.rejected;
      a.loop_steps[st.traj] = st.n_steps;
      const bool any = (bads & (0xffffffffu >> (32 - MDX_TEAM))) != 0u;
      if (a.status)
        a.status[st.traj] = (hit_max ? MDX_STATUS_MAX_STEPS : MDX_STATUS_OK) | (any ? MDX_STATUS_NONFINITE : 0);
    }
  }
  __syncwarp();
  if (a.hist_host != nullptr && done) {
    // The barrier ordered every lane's history stores before these L2 reads.
    const size_t row = (size_t)a.n_save_hist * (size_t)MDX_NV;
    const double* src = a.hist + (size_t)st.traj * row;
    double* dst = a.hist_host + (size_t)st.traj * row;
    for (size_t i = L.lane; i < row; i += MDX_TEAM) dst[i] = __ldcg(src + i);
  }
}

#if MDX_STAGED
// A stopped trajectory's record: its scalars, then the state; every lane has the scalars.
constexpr int RECORD = RECORD_SCALARS + MDX_NV;
__device__ __forceinline__ void save(const State& st, double* rec, const Lane& L) {
  if (L.lane == 0) save_scalars(st, rec);
#pragma unroll
  for (int j = 0; j < B; ++j) rec[RECORD_SCALARS + L.lane * B + j] = st.y[j];
}
__device__ __forceinline__ void load(State& st, const MdxSolveArgs& a, const double* rec, int traj, const Lane& L) {
  st.traj = traj;
#pragma unroll
  for (int j = 0; j < B; ++j) st.y[j] = rec[RECORD_SCALARS + L.lane * B + j];
#pragma unroll
  for (int k = 0; k < MDX_LANE_PARAMS; ++k) st.p[k] = a.params[(size_t)traj * MDX_NP + param_column(k, L.lane)];
#if MDX_TF_INDEX >= 0
  st.tf_local = a.params[(size_t)traj * MDX_NP + MDX_TF_INDEX];
#else
  st.tf_local = a.times[a.n_save - 1];
#endif
  load_scalars(st, a, rec);
}

// The two stages of mdx_entry.cuh's mdx_solve_staged, a trajectory per team.
__device__ __forceinline__ void solve_staged(const MdxSolveArgs& a, const MdxStageArgs& b) {
  const Lane L = lane_of_thread();
  State st;
  rest(st);
  bool active = false, drained = false;
  while (true) {
    const bool whole = active && !running(st, a);
    if (__any_sync(MDX_FULL_MASK, whole)) finish(st, a, L, whole);
    if (b.slice > 0 && active && (whole || st.n_steps >= b.slice)) {
      if (L.lane == 0) b.remaining[st.traj] = whole ? 0 : steps_to_go(a.times[0], st.t, st.tf_local, st.n_steps);
      if (!whole) save(st, b.records + (size_t)st.traj * RECORD, L);
      active = false;
    }
    active = active && !whole;
    if (__any_sync(MDX_FULL_MASK, !active && !drained)) {
      int slot = 0;
      if (!active && !drained && L.lane == 0) slot = atomicAdd(a.work_counter, 1);
      slot = __shfl_sync(MDX_FULL_MASK, slot, L.base);
      if (!active && !drained) {
        if (slot >= a.n_traj) {
          drained = true;
        } else {
          const int traj = a.order ? a.order[slot] : slot;
          if (b.slice > 0) {
            init(st, a, traj, L);
            active = true;
          } else if (b.remaining[traj] > 0) {
            load(st, a, b.records + (size_t)traj * RECORD, traj, L);
            active = true;
          } else {
            drained = true;  // finished ones come last in the order
          }
        }
      }
      continue;
    }
    if (!__any_sync(MDX_FULL_MASK, active)) break;
    step(st, a, L, active);
  }
}
#endif

// REFILL: lanes whose trajectory ends take the next one off the queue (one
// atomicAdd per trajectory, by its first lane); nothing waits on anything.
template <bool REFILL>
__device__ __forceinline__ void solve_warp(const MdxSolveArgs& a) {
  const Lane L = lane_of_thread();
  State st;
  rest(st);
  bool active = false, drained = false;
  if (!REFILL) {
    const int traj = (int)((blockIdx.x * MDX_TPB + threadIdx.x) / MDX_TEAM);
    active = traj < a.n_traj;
    if (active) init(st, a, traj, L);
    drained = true;
  }
  while (true) {
    const bool done = active && !running(st, a);
    if (__any_sync(MDX_FULL_MASK, done)) {
      finish(st, a, L, done);
      active = active && !done;
    }
    if (REFILL && __any_sync(MDX_FULL_MASK, !active && !drained)) {
      int slot = 0;
      if (!active && !drained && L.lane == 0) slot = atomicAdd(a.work_counter, 1);
      slot = __shfl_sync(MDX_FULL_MASK, slot, L.base);
      if (!active && !drained) {
        if (slot < a.n_traj) {
          init(st, a, a.order ? a.order[slot] : slot, L);
          active = true;
        } else {
          drained = true;
        }
      }
      continue;  // a trajectory may end where it begins
    }
    if (!__any_sync(MDX_FULL_MASK, active)) break;
    step(st, a, L, active);
  }
}

}  // namespace cyclic
}  // namespace mdx

extern "C" __global__ void __launch_bounds__(MDX_TPB, MDX_MIN_BLOCKS) mdx_solve_plain(const MdxSolveArgs a) {
  mdx::cyclic::solve_warp<false>(a);
}

extern "C" __global__ void __launch_bounds__(MDX_TPB, MDX_MIN_BLOCKS) mdx_solve_persistent(const MdxSolveArgs a) {
  mdx::cyclic::solve_warp<true>(a);
}

#if MDX_STAGED
extern "C" __global__ void __launch_bounds__(MDX_TPB, MDX_MIN_BLOCKS)
mdx_solve_staged(const MdxSolveArgs a, const MdxStageArgs b) {
  mdx::cyclic::solve_staged(a, b);
}
#endif
