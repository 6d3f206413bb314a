// Dense LU with partial pivoting, one n x n system per thread, row-major.
//
// The algorithm is the reference's dense_lu_solver (modax/rodas5P.py:167-238):
// right-looking elimination, the largest remaining entry of the column as pivot,
// whole-row swaps recorded in ipiv, a zero pivot left alone (the Rosenbrock-W
// step controller rejects what comes out of it).  Arithmetic follows the
// reference's mixed typing: the multipliers and the rank-one update are formed in
// double and stored in the LU type T; the substitutions run in T.
//
// For N <= MDX_DENSE_UNROLL_MAX every index is a compile-time constant: the row
// swaps become predicated selects over the candidate rows, so the matrix stays in
// registers.  Larger systems use plain loops and the compiler places the matrix in
// local memory.
//
// With RECIP the matrix has N more entries, lu[N * N + i] = 1/U_ii, and the
// substitutions' divisions by U_ii go through div_by (the same rounding, 25 dependent
// cycles instead of a double division's 125).  Eight stages of N divisions, each on
// the step's dependent chain, were half of a 64-bit step of three states.  Calls on
// a B200: Robertson FP64, 20,001 trajectories, 590 -> 446 us; 65,536 adjoint
// gradients of a stiff oscillator 11.1 -> 8.1 ms, forward-sensitivity ones 4.2 -> 3.2 ms.
#pragma once
#include "mdx_common.cuh"

#ifndef MDX_DENSE_UNROLL_MAX
#define MDX_DENSE_UNROLL_MAX 12
#endif

namespace mdx {

template <typename T>
__device__ __forceinline__ void swap_vals(T& a, T& b) { T c = a; a = b; b = c; }

// Keeps pivot i's reciprocal; an infinite pivot becomes the zero pair that div_by
// takes for it.
template <int N, typename T, class LU>
__device__ __forceinline__ void keep_reciprocal(LU& lu, int i, double inv_piv) {
  const T r = (T)inv_piv;
  lu[N * N + i] = r;
  if (r == T(0)) lu[i * N + i] = T(0);
}

template <int N, typename T, bool RECIP, class LU, class IP>
__device__ __forceinline__ void dense_factorize_unrolled(LU& lu, IP& ipiv) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T max_val = fabs(lu[i * N + i]);
    int pivot = i;
#pragma unroll
    for (int k = i + 1; k < N; ++k) {
      const T v = fabs(lu[k * N + i]);
      if (v > max_val) { max_val = v; pivot = k; }
    }
    ipiv[i] = pivot;
#pragma unroll
    for (int k = i + 1; k < N; ++k) {
      if (pivot == k) {
#pragma unroll
        for (int j = 0; j < N; ++j) swap_vals(lu[i * N + j], lu[k * N + j]);
      }
    }
    const T piv = lu[i * N + i];
    const double inv_piv = 1.0 / (double)piv;
    if (piv != T(0)) {
#pragma unroll
      for (int k = i + 1; k < N; ++k) {
        const double factor = (double)lu[k * N + i] * inv_piv;
        lu[k * N + i] = (T)factor;
#pragma unroll
        for (int j = i + 1; j < N; ++j)
          lu[k * N + j] = (T)((double)lu[k * N + j] - factor * (double)lu[i * N + j]);
      }
    }
    if constexpr (RECIP) keep_reciprocal<N, T>(lu, i, inv_piv);
  }
}

template <int N, typename T, bool RECIP, class LU, class IP>
__device__ __forceinline__ void dense_factorize_loops(LU& lu, IP& ipiv) {
#pragma unroll 1
  for (int i = 0; i < N; ++i) {
    T max_val = fabs(lu[i * N + i]);
    int pivot = i;
    for (int k = i + 1; k < N; ++k) {
      const T v = fabs(lu[k * N + i]);
      if (v > max_val) { max_val = v; pivot = k; }
    }
    ipiv[i] = pivot;
    if (pivot != i) {
      for (int j = 0; j < N; ++j) swap_vals(lu[i * N + j], lu[pivot * N + j]);
    }
    const T piv = lu[i * N + i];
    const double inv_piv = 1.0 / (double)piv;
    if (piv != T(0)) {
#pragma unroll 1
      for (int k = i + 1; k < N; ++k) {
        const double factor = (double)lu[k * N + i] * inv_piv;
        lu[k * N + i] = (T)factor;
#pragma unroll 4
        for (int j = i + 1; j < N; ++j)
          lu[k * N + j] = (T)((double)lu[k * N + j] - factor * (double)lu[i * N + j]);
      }
    }
    if constexpr (RECIP) keep_reciprocal<N, T>(lu, i, inv_piv);
  }
}

template <int N, typename T, bool RECIP = false, class LU, class IP>
__device__ __forceinline__ void dense_factorize(LU& lu, IP& ipiv) {
  if constexpr (N <= MDX_DENSE_UNROLL_MAX) dense_factorize_unrolled<N, T, RECIP>(lu, ipiv);
  else dense_factorize_loops<N, T, RECIP>(lu, ipiv);
}

// acc / U_ii
template <int N, typename T, bool RECIP, class LU>
__device__ __forceinline__ T over_pivot(T acc, const LU& lu, int i) {
  if constexpr (RECIP) return div_by<T>(acc, lu[i * N + i], lu[N * N + i]);
  else return acc / lu[i * N + i];
}

// M x = rhs in place: forward through L applying the pivots as they come, then
// back through U (modax/rodas5P.py:218-236).
template <int N, typename T, bool RECIP = false, class LU, class IP, class R>
__device__ __forceinline__ void dense_solve(const LU& lu, const IP& ipiv, R& rhs) {
  if constexpr (N <= MDX_DENSE_UNROLL_MAX) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int pivot = ipiv[i];
#pragma unroll
      for (int k = i + 1; k < N; ++k)
        if (pivot == k) swap_vals(rhs[i], rhs[k]);
      T acc = rhs[i];
#pragma unroll
      for (int j = 0; j < i; ++j) acc -= lu[i * N + j] * rhs[j];
      rhs[i] = acc;
    }
#pragma unroll
    for (int i = N - 1; i >= 0; --i) {
      T acc = rhs[i];
#pragma unroll
      for (int j = i + 1; j < N; ++j) acc -= lu[i * N + j] * rhs[j];
      rhs[i] = over_pivot<N, T, RECIP>(acc, lu, i);
    }
  } else {
#pragma unroll 1
    for (int i = 0; i < N; ++i) {
      const int pivot = ipiv[i];
      if (pivot != i) swap_vals(rhs[i], rhs[pivot]);
      T acc = rhs[i];
      for (int j = 0; j < i; ++j) acc -= lu[i * N + j] * rhs[j];
      rhs[i] = acc;
    }
#pragma unroll 1
    for (int i = N - 1; i >= 0; --i) {
      T acc = rhs[i];
      for (int j = i + 1; j < N; ++j) acc -= lu[i * N + j] * rhs[j];
      rhs[i] = over_pivot<N, T, RECIP>(acc, lu, i);
    }
  }
}

// M^T x = rhs in place, for the discrete adjoint.  With M = P^-1 L U (P the
// product of the recorded row swaps): U^T z = rhs, L^T w = z, then the swaps
// undone in reverse order.
template <int N, typename T, bool RECIP = false, class LU, class IP, class R>
__device__ __forceinline__ void dense_solve_t(const LU& lu, const IP& ipiv, R& rhs) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T acc = rhs[i];
#pragma unroll
    for (int k = 0; k < i; ++k) acc -= lu[k * N + i] * rhs[k];
    rhs[i] = over_pivot<N, T, RECIP>(acc, lu, i);
  }
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    T acc = rhs[i];
#pragma unroll
    for (int k = i + 1; k < N; ++k) acc -= lu[k * N + i] * rhs[k];
    rhs[i] = acc;
  }
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    const int pivot = ipiv[i];
    if constexpr (N <= MDX_DENSE_UNROLL_MAX) {
#pragma unroll
      for (int k = i + 1; k < N; ++k)
        if (pivot == k) swap_vals(rhs[i], rhs[k]);
    } else {
      if (pivot != i) swap_vals(rhs[i], rhs[pivot]);
    }
  }
}

// --- fast arithmetic (MDX_FAST): the FP32-LU path of the persistent kernel ------
// The factorisation runs entirely in T (no double multipliers, no conversions),
// the row swaps are folded into a permutation `perm` (perm[i] = the original
// row that ends at position i) so a solve permutes its right-hand side with
// selects instead of branches, and the diagonal is left holding 1/U_ii (the
// approximate reciprocal fast_recip) so the back substitution multiplies.  Same algorithm, different rounding: the FP32
// path is held to accuracy against the FP64 oracle, not to the reference's bits.
template <int N, typename T, class LU, class IP>
__device__ __forceinline__ void dense_factorize_fast(LU& lu, IP& perm) {
  static_assert(N <= MDX_DENSE_UNROLL_MAX, "the fast dense LU is for register-resident systems");
#pragma unroll
  for (int i = 0; i < N; ++i) perm[i] = i;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T max_val = fabs(lu[i * N + i]);
    int pivot = i;
#pragma unroll
    for (int k = i + 1; k < N; ++k) {
      const T v = fabs(lu[k * N + i]);
      if (v > max_val) { max_val = v; pivot = k; }
    }
#pragma unroll
    for (int k = i + 1; k < N; ++k) {
      const bool sw = pivot == k;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const T a = lu[i * N + j], b = lu[k * N + j];
        lu[i * N + j] = sw ? b : a;
        lu[k * N + j] = sw ? a : b;
      }
      const int pa = perm[i], pb = perm[k];
      perm[i] = sw ? pb : pa;
      perm[k] = sw ? pa : pb;
    }
    const T piv = lu[i * N + i];
    const T recip = fast_recip(piv);
    const T inv_piv = piv != T(0) ? recip : T(0);
#pragma unroll
    for (int k = i + 1; k < N; ++k) {
      const T factor = lu[k * N + i] * inv_piv;
      lu[k * N + i] = factor;
#pragma unroll
      for (int j = i + 1; j < N; ++j) lu[k * N + j] -= factor * lu[i * N + j];
    }
    lu[i * N + i] = recip;
  }
}

template <int N, typename T, class LU, class IP, class R>
__device__ __forceinline__ void dense_solve_fast(const LU& lu, const IP& perm, R& rhs) {
  T x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T v = rhs[0];
#pragma unroll
    for (int k = 1; k < N; ++k) v = perm[i] == k ? rhs[k] : v;
    x[i] = v;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T acc = x[i];
#pragma unroll
    for (int j = 0; j < i; ++j) acc -= lu[i * N + j] * x[j];
    x[i] = acc;
  }
  // Back substitution takes each row's terms latest-solved last (descending
  // column), so a row waits on one FMA after its last input.
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    T acc = x[i];
#pragma unroll
    for (int j = N - 1; j > i; --j) acc -= lu[i * N + j] * x[j];
    x[i] = acc * lu[i * N + i];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) rhs[i] = x[i];
}

// Transposed solve for the fast factorisation: M^T x = b with M = P^T L U.
template <int N, typename T, class LU, class IP, class R>
__device__ __forceinline__ void dense_solve_t_fast(const LU& lu, const IP& perm, R& rhs) {
  T z[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    T acc = rhs[i];
#pragma unroll
    for (int k = 0; k < i; ++k) acc -= lu[k * N + i] * z[k];
    z[i] = acc * lu[i * N + i];
  }
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    T acc = z[i];
#pragma unroll
    for (int k = i + 1; k < N; ++k) acc -= lu[k * N + i] * z[k];
    z[i] = acc;
  }
  // x[perm[i]] = z[i]
#pragma unroll
  for (int j = 0; j < N; ++j) {
    T v = z[0];
#pragma unroll
    for (int i = 1; i < N; ++i) v = perm[i] == j ? z[i] : v;
    rhs[j] = perm[0] == j ? z[0] : v;
  }
}

// --- systems of up to three states in fast arithmetic -------------------------------
// The matrix is inverted in place in double: a solve is then N independent rows of N
// multiply-adds instead of a permutation and two substitutions, each row of which waits
// for the one before.  One and two states by cofactors, whose only cancellation is the
// determinant's.  Cofactors of three states cancel twice: for one fast reaction
// A + B <-> C, M = I + s u v^T, they are off by eps s^2 where an LU is by eps s, and at
// s = 1e9 a solve took 15 times the steps.  So three states take one elimination step and
// the cofactors of the two rows that remain, and lose what an LU does.  The remaining
// rows are kept times the pivot: one reciprocal serves pivot and determinant, and all but
// it and a multiply-add per entry is done while it is under way.  A determinant past the
// double range would make a zero inverse, whose zero increments pass any error test; it
// becomes NaN, which the controller rejects.
//
// The pivot is the first row's entry unless another's is over eight times as large, which
// the exponents tell: rows in the order of an unconditional partial pivoting cost every
// step 48 selects (3.5% of a solve).  Robertson on a B200, one launch, cofactors /
// this: 1 trajectory 142 / 145 us, 65,536 370 / 374.  Pivoted LUs with FP32 factors in
// place of both, and 1/h in the matrix (mdx_rodas5p.cuh), made the calls 218 and 524 us,
// cofactors 159 and 484.
constexpr int CLOSED_INVERSE_MAX = 3;

__device__ __forceinline__ double inverse_or_nan(double det) { return finite(det) ? 1.0 / det : nan_value(); }

// The exponent and leading 20 bits of |x|.
__device__ __forceinline__ unsigned magnitude_word(double x) {
  unsigned long long bits;
  memcpy(&bits, &x, sizeof bits);
  return (unsigned)(bits >> 32) & 0x7fffffffu;
}

__device__ __forceinline__ void swap_if(bool yes, double& a, double& b) {
  const double c = yes ? b : a;
  b = yes ? a : b;
  a = c;
}

// The inverse of a 3 x 3 matrix with m[0] as the first pivot.
template <class M, class X>
__device__ __forceinline__ void inverse_by_first_pivot(const M& m, X& x) {
  const double a = m[0];
  // a times the rows that remain; their determinant is a times the matrix's.
  const double s00 = a * m[4] - m[3] * m[1], s01 = a * m[5] - m[3] * m[2];
  const double s10 = a * m[7] - m[6] * m[1], s11 = a * m[8] - m[6] * m[2];
  const double det = s00 * s11 - s01 * s10;
  const double q = inverse_or_nan(a * det);
  const double left0 = s11 * m[3] - s01 * m[6], left1 = s00 * m[6] - s10 * m[3];
  const double top0 = m[1] * s11 - m[2] * s10, top1 = m[2] * s00 - m[1] * s01;
  const double corner = det + (m[1] * left0 + m[2] * left1);
  const double r = a * q, ar = (a * a) * q;
  x[0] = corner * q;
  x[1] = -top0 * r;
  x[2] = -top1 * r;
  x[3] = -left0 * r;
  x[4] = s11 * ar;
  x[5] = -s01 * ar;
  x[6] = -left1 * r;
  x[7] = -s10 * ar;
  x[8] = s00 * ar;
}

template <int N, class M>
__device__ __forceinline__ void closed_inverse(M& m) {
  static_assert(N <= CLOSED_INVERSE_MAX, "closed forms of up to three states");
  if constexpr (N == 1) {
    m[0] = inverse_or_nan(m[0]);
  } else if constexpr (N == 2) {
    const double r = inverse_or_nan(m[0] * m[3] - m[1] * m[2]);
    const double first = m[0];
    m[0] = m[3] * r;
    m[1] = -m[1] * r;
    m[2] = -m[2] * r;
    m[3] = first * r;
  } else {
    double x[N * N];
    inverse_by_first_pivot(m, x);
    const unsigned w0 = magnitude_word(m[0]), w1 = magnitude_word(m[3]), w2 = magnitude_word(m[6]);
    if ((w1 > w2 ? w1 : w2) > w0 + (3u << 20)) {  // 2^3 times m[0]
      // The largest entry's row first; the inverse's columns go back the same way.
      const bool second = fabs(m[3]) > fabs(m[0]);
#pragma unroll
      for (int j = 0; j < 3; ++j) swap_if(second, m[j], m[3 + j]);
      const bool third = fabs(m[6]) > fabs(m[0]);
#pragma unroll
      for (int j = 0; j < 3; ++j) swap_if(third, m[j], m[6 + j]);
      inverse_by_first_pivot(m, x);
#pragma unroll
      for (int i = 0; i < 3; ++i) swap_if(third, x[3 * i], x[3 * i + 2]);
#pragma unroll
      for (int i = 0; i < 3; ++i) swap_if(second, x[3 * i], x[3 * i + 1]);
    }
#pragma unroll
    for (int i = 0; i < N * N; ++i) m[i] = x[i];
  }
}

// x = M^-1 b and (TRANSPOSED) x = M^-T b, in place.
template <int N, bool TRANSPOSED, class M, class R>
__device__ __forceinline__ void inverse_solve(const M& m, R& rhs) {
  double x[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    x[i] = m[TRANSPOSED ? i : i * N] * rhs[0];
#pragma unroll
    for (int j = 1; j < N; ++j) x[i] += m[TRANSPOSED ? j * N + i : i * N + j] * rhs[j];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) rhs[i] = x[i];
}

}  // namespace mdx
