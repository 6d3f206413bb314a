// Shared device helpers for the ensemble ODE kernels (sm_100a, NVRTC-compiled).
//
// Every kernel runs one trajectory per thread.  A problem header generated on
// the host (menodax_b200/_codegen.py) defines the sizes, the traced right-hand
// side and its derivatives as force-inlined templates; with every component
// index a compile-time constant the per-trajectory vectors live in registers.
#pragma once
#include "mdx_args.h"

#define MDX_FULL_MASK 0xffffffffu

#ifndef MDX_TPB
#define MDX_TPB 32
#endif
#ifndef MDX_MIN_BLOCKS
#define MDX_MIN_BLOCKS 1
#endif

namespace mdx {

// Python's max(a, b) on floats: the first argument unless the second is larger.
// It differs from fmax only on NaN, where the reference's comparison semantics
// (modax/rodas5P.py:907, modax/tsit5.py:297) are kept.
__device__ __forceinline__ double pymax(double a, double b) { return b > a ? b : a; }

__device__ __forceinline__ bool finite(double x) { return isfinite(x); }

__device__ __forceinline__ double nan_value() { return __longlong_as_double(0x7ff8000000000000LL); }

// x^e for the step-size factor in the fast path: the factor is a heuristic that
// is clamped to [0.2, 6] and multiplied by 0.9, so float precision (relative
// error ~1e-6) is ample; __powf is two special-function-unit instructions.
__device__ __forceinline__ double fast_pow(double x, double e) {
  return (double)__powf((float)x, (float)e);
}

// 1/x for the fast path's LU pivots.  In single precision the approximate
// reciprocal (__fdividef: within 2 ulp for |x| in [2^-126, 2^126], 1/0 = inf),
// whose error is below the FP32 factorisation's own rounding; double pivots keep
// the IEEE division.
__device__ __forceinline__ float fast_recip(float x) { return __fdividef(1.0f, x); }
__device__ __forceinline__ double fast_recip(double x) { return 1.0 / x; }

// 1/s in double for the fast path (the step's 1/h, the error scales): the
// single-precision reciprocal as a seed, refined by one Newton-Raphson step
// y <- y + y (1 - s y), which squares the seed's relative error (~1e-7 ->
// ~1e-14).  Values outside float's normal range keep the IEEE division.
__device__ __forceinline__ double recip_newton(double s) {
  if (s >= 1e-37 && s <= 1e37) {
    const double y = (double)__fdividef(1.0f, (float)s);
    return fma(y, fma(-s, y, 1.0), y);
  }
  return 1.0 / s;
}

// a / d from r = 1/d rounded to nearest, for a divisor used again and again:
// quotient, exact residual, correction (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. R&D 34, 1990).  The
// result is the rounded quotient save where the exact one lies within rounding
// of the residual's correction of a midpoint.  Three dependent multiply-adds, 25
// cycles on a B200, against 125 for a double division.  d = 0 and overflowing
// quotients give NaN where a division gives an infinity; both reject a step.  An
// infinite divisor goes in as d = r = 0 (and gives 0).
template <typename T>
__device__ __forceinline__ T div_by(T a, T d, T r) {
  const T q = a * r;
  return fma(fma(-q, d, a), r, q);
}

// x^(-1/K), K even, for x in [1e-36, 1e36]: a float power as seed (relative error
// about 1e-6) and two Newton steps y <- y + y (1 - x y^K) / K, each of which
// squares the relative error times (K + 1) / 2, so the result is good to a few
// rounding errors.
template <int K>
__device__ __forceinline__ double inverse_root(double x) {
  static_assert(K == 10 || K == 12, "the embedded error's two orders");
  double y = (double)__powf((float)x, -1.0f / (float)K);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double y2 = y * y, y4 = y2 * y2, y8 = y4 * y4;
    const double yk = y8 * (K == 10 ? y2 : y4);
    y = fma(y * (1.0 / K), fma(-x, yk, 1.0), y);
  }
  return y;
}

// Step-size controller (modax/rodas5P.py:913-928, modax/tsit5.py:383-398) on the
// sum of the squared scaled errors: accept on a norm (its root mean) of at most
// one, clamp the norm into [1e-18, 1e18] (NaN counts as huge), form the PID factor
// from the error history; the caller clamps the factor.  E1, E2 and E3 are
// compile-time constants.  The default I-controller (E1 = -1/ORDER, no history)
// needs only norm^(-1/ORDER) = mean^(-1/(2 ORDER)), taken by inverse_root of the
// mean: neither the square root nor the double power, which alone cost about 860
// dependent cycles of a step (a step of Tsit5 on three states took 2,300).  Lorenz
// by Tsit5, calls on a B200: 250,007 trajectories 1,177 -> 947 us, 4,096 286 -> 199
// us; Robertson in 64 bits, 20,001 trajectories, 648 -> 590 us.  Its
// accept test is the norm's: the rounded root of a double is at most one exactly
// when the double is at most 1 + 2^-52.  A mean below 1e-36 clamps with zero: the
// factor is far past the caller's largest either way.
template <int ORDER>
__device__ __forceinline__ double controller_factor(double err_sum, double n_err, double err_prev,
                                                    double err_prev2, double e1, double e2, double e3,
                                                    bool use_e2, bool use_e3, bool& accept,
                                                    double& safe_err) {
  const double mean = div_by(err_sum, n_err, 1.0 / n_err);
  if (e1 == -1.0 / ORDER && !use_e2 && !use_e3) {
    accept = mean <= 1.0 + 2.220446049250313e-16;
    safe_err = 1e36;  // NaN too
    if (mean <= 1e36) safe_err = mean < 1e-36 ? 1e-36 : mean;
    return 0.9 * inverse_root<2 * ORDER>(safe_err);
  }
  const double err_norm = sqrt(mean);
  accept = err_norm <= 1.0 && !isnan(err_norm);
  if (isnan(err_norm) || err_norm > 1e18) {
    safe_err = 1e18;
  } else if (err_norm == 0.0) {
    safe_err = 1e-18;
  } else {
    safe_err = err_norm;
  }
  double factor = 0.9 * pow(safe_err, e1);
  if (use_e2) factor = factor * pow(err_prev, e2);
  if (use_e3) factor = factor * pow(err_prev2, e3);
  return factor;
}

// The fast path's controller on the SQUARED weighted RMS error: the step is
// accepted on err^2 <= 1 and err^e = (err^2)^(e/2), so no square root is taken.
// The error history is kept squared too.  The clamp is [1e-36, 1e36] on err^2
// (the reference's [1e-18, 1e18] on err), applied below as well as at zero so
// that every power is taken of a normal float.
__device__ __forceinline__ double controller_factor_sq(double err_sq, double prev_sq, double prev2_sq,
                                                       double e1, double e2, double e3, bool use_e2,
                                                       bool use_e3, double& safe_sq) {
  if (isnan(err_sq) || err_sq > 1e36) {
    safe_sq = 1e36;
  } else if (err_sq < 1e-36) {
    safe_sq = 1e-36;
  } else {
    safe_sq = err_sq;
  }
  double factor = 0.9 * fast_pow(safe_sq, 0.5 * e1);
  if (use_e2) factor = factor * fast_pow(prev_sq, 0.5 * e2);
  if (use_e3) factor = factor * fast_pow(prev2_sq, 0.5 * e3);
  return factor;
}

// True when save time `ts` is reached by a step ending at `t_new`
// (modax/rodas5P.py:933-935): the 1e-12 relative slack keeps a save that
// rounding puts a hair past the end of the step from being missed.
__device__ __forceinline__ bool save_reached(double ts, double t_new) {
  return ts <= t_new + 1e-12 * pymax(1.0, fabs(ts));
}

#ifndef MDX_STAGED
#define MDX_STAGED 0
#endif

// What a trajectory that stopped after `steps` attempted steps at t still has to take,
// if it goes on at its average pace: what the second stage is ordered by.
__device__ __forceinline__ int steps_to_go(double t0, double t, double tf, int steps) {
  const double more = (tf - t) / (t - t0) * (double)steps;
  return more >= 1.0 ? (more < 1e9 ? (int)more : 1000000000) : 1;
}

// The scalars of a stopped trajectory's state, six doubles of its record.
constexpr int RECORD_SCALARS = 6;
template <class S>
__device__ __forceinline__ void save_scalars(const S& st, double* rec) {
  rec[0] = st.t;
  rec[1] = st.dt;
  rec[2] = st.err_prev;
  rec[3] = st.err_prev2;
  int* counts = reinterpret_cast<int*>(rec + 4);
  counts[0] = st.save_idx;
  counts[1] = st.n_steps;
  counts[2] = st.accepted;
  counts[3] = st.rejected;
}
template <class S>
__device__ __forceinline__ void load_scalars(S& st, const MdxSolveArgs& a, const double* rec) {
  st.t = rec[0];
  st.dt = rec[1];
  st.err_prev = rec[2];
  st.err_prev2 = rec[3];
  const int* counts = reinterpret_cast<const int*>(rec + 4);
  st.save_idx = counts[0];
  st.n_steps = counts[1];
  st.accepted = counts[2];
  st.rejected = counts[3];
  if (st.save_idx < a.n_save) st.next_save = a.times[st.save_idx];
}

#ifndef MDX_CKPT_SEG
#define MDX_CKPT_SEG 1
#endif

// Checkpoint layout of a MDX_CHECKPOINT solve: a row per trajectory, in it a record per
// MDX_CKPT_SEG accepted steps: the first one's start (t, y), then the sizes h of all (fewer
// in a capacity's last record).  The reverse pass replays a segment from its start
// state.  A row is contiguous because lanes do not stay in step: with a row per step a
// warp's writes and reads went to as many pages as it has lanes, gigabytes apart, here
// they stay in a page or two and a two-state step is one 32-byte sector.  65,536
// gradients of a stiff oscillator over 1,500 steps on a B200: forward 3.93 -> 3.49 ms,
// reverse 2.65 -> 2.57, the call 7.0 to 19.8 ms (by where the buffer came to lie) ->
// 6.4 to 6.7.
__host__ __device__ __forceinline__ size_t ckpt_row(long long capacity) {
  const size_t segments = (size_t)((capacity + MDX_CKPT_SEG - 1) / MDX_CKPT_SEG);
  return (size_t)capacity + segments * (size_t)(MDX_NV + 1);
}

template <class T>  // double or const double
__device__ __forceinline__ T* ckpt_record(T* ckpt, long long capacity, int seg, int traj) {
  return ckpt + (size_t)traj * ckpt_row(capacity) + (size_t)seg * (size_t)(MDX_NV + 1 + MDX_CKPT_SEG);
}

template <class Y>
__device__ __forceinline__ void ckpt_write(const MdxSolveArgs& a, int traj, int m, double t, double h, const Y& y) {
  double* rec = ckpt_record(a.ckpt, a.ckpt_capacity, m / MDX_CKPT_SEG, traj);
  if (m % MDX_CKPT_SEG == 0) {
    rec[0] = t;
#pragma unroll
    for (int j = 0; j < MDX_NV; ++j) rec[1 + j] = y[j];
  }
  rec[MDX_NV + 1 + m % MDX_CKPT_SEG] = h;
}

}  // namespace mdx
