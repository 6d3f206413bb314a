// The team kernel's dense matrix inverted in registers (MDX_TEAM_INVERSE).
//
// Lane l of a team keeps rows l, l + MDX_TEAM, ... of M.  Gauss-Jordan elimination
// with partial pivoting inverts M in place: per column one max-reduction finds the
// pivot row, its owner writes it to shared memory, and every lane updates its rows
// with one multiply-add per entry.  A solve is then a row of independent
// multiply-adds against the right-hand side, read from shared memory four values
// at a time, where substitutions are a chain of 2 n dependent exchanges.
//
// What bounds it: issue (n rows of n multiply-adds per column, n^3 in all against
// the 2/3 n^3 of a factorisation, at one shared-memory access per four of them
// instead of 1.25 per one in mdx_team_lu.cuh).  The dense Brusselator on a B200, LU in
// shared memory / inverse here, each at its best team: 32 states, 1 trajectory 3.7 /
// 0.92 ms, 256 4.2 / 1.02, 4,097 7.6 / 3.8, 16,384 28.1 / 12.8; 16 states, 4,097 2.7 /
// 1.18; 64 states, 4,097 44.6 / 17.9.  The LU stays for matrices whose rows do not
// fit the registers (team_inverse_fits) and for the reference's arithmetic.
//
// Rows stay where they are: `column[q]` is the column whose pivot row q was, so row
// q of the inverse gives that component, and pivots are not applied until the end
// (`scale[q]`).  Columns rotate one place left per step, which keeps every register
// index literal in a loop that is not unrolled: the eliminated column is always the
// first.  A row of zeros for a pivot gives infinities and NaN; the step is rejected.
#pragma once

namespace mdx {
namespace team {

constexpr int ROWS = (MDX_NV + MDX_TEAM - 1) / MDX_TEAM;  // rows a lane keeps
constexpr int PADDED = (MDX_NV + 3) / 4 * 4;              // a vector read four at a time

struct Inverse {
  lu_t a[ROWS][MDX_NV];
  lu_t scale[ROWS];
  int column[ROWS];
  double k[8][ROWS];  // the lane's own components of the stage increments, widened once
};

// Two vectors at the front of the matrix's shared memory, free once its rows are in
// registers: 16-byte aligned, one ahead of the other's readers.  The offset is reckoned
// in integers: a pointer rounded up by a cast is no longer known to point to shared
// memory, and its loads, then generic ones, were what the inversion waited for.
__device__ __forceinline__ lu_t* exchange(Slice& s, int which) {
  const unsigned at = (threadIdx.x / MDX_TEAM) * (unsigned)MDX_TEAM_SLICE_BYTES
                      + (unsigned)((const char*)s.lu - (const char*)&s);
  return s.lu + ((0u - at) & 15u) / (unsigned)sizeof(lu_t) + which * (PADDED + 4);
}
static_assert(4 * MDX_TEAM_LU_SIZE >= 16 + 8 * (PADDED + 4), "the matrix's memory holds both vectors");

struct __align__(16) Four { lu_t v[4]; };

__device__ __forceinline__ void invert(Slice& s, Inverse& m, const Lanes& L) {
  bool used[ROWS];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const int row = L.lane + q * MDX_TEAM;
    used[q] = row >= MDX_NV;
    m.column[q] = 0;
    m.scale[q] = (lu_t)0;
#pragma unroll
    for (int j = 0; j < MDX_NV; ++j) m.a[q][j] = used[q] ? (lu_t)0 : s.lu[row * MDX_TEAM_LDA + j];
  }
  __syncwarp(L.mask);
#pragma unroll 1
  for (int i = 0; i < MDX_NV; ++i) {
    // The largest remaining entry, its row number in the low bits: magnitudes are
    // told apart to one part in 2^17.
    unsigned best = 0;
    lu_t recip[ROWS];  // every row's, ready before the search has found the pivot
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      recip[q] = fast_recip(m.a[q][0]);
      const unsigned key = (__float_as_uint(fabsf(m.a[q][0])) & ~63u) | (unsigned)(63 - (L.lane + q * MDX_TEAM));
      if (!used[q] && key > best) best = key;
    }
    best = __reduce_max_sync(L.mask, best);
    const int pivot = 63 - (int)(best & 63u);
    lu_t* const x = exchange(s, i & 1);
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      if (pivot == L.lane + q * MDX_TEAM) {
        // The row as the next columns' order has it, then the pivot's reciprocal.
        Four* const out = reinterpret_cast<Four*>(x);
#pragma unroll
        for (int j = 0; j < PADDED; j += 4) {
          Four f;
#pragma unroll
          for (int e = 0; e < 4; ++e) f.v[e] = m.a[q][j + e + 1 < MDX_NV ? j + e + 1 : 0];
          out[j / 4] = f;
        }
        x[PADDED] = recip[q];
      }
    }
    __syncwarp(L.mask);
    const lu_t inv = x[PADDED];
    lu_t f[ROWS], first[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const bool mine = pivot == L.lane + q * MDX_TEAM;
      f[q] = mine ? (lu_t)0 : m.a[q][0] * inv;
      first[q] = mine ? (lu_t)1 : -f[q];
      if (mine) {
        used[q] = true;
        m.scale[q] = inv;
        m.column[q] = i;
      }
    }
    const Four* const in = reinterpret_cast<const Four*>(x);
#pragma unroll
    for (int j = 0; j < PADDED; j += 4) {
      const Four p = in[j / 4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (j + e + 1 < MDX_NV) {
#pragma unroll
          for (int q = 0; q < ROWS; ++q) m.a[q][j + e] = m.a[q][j + e + 1] - f[q] * p.v[e];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < ROWS; ++q) m.a[q][MDX_NV - 1] = first[q];
  }
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
#pragma unroll
    for (int j = 0; j < MDX_NV; ++j) m.a[q][j] *= m.scale[q];
  }
  // The last column's readers are done before a solve writes its vector there.
  __syncwarp(L.mask);
}

// out = M^-1 b: `b[q]` is the component of this lane's row q; the row's result is
// component column[q].
__device__ __forceinline__ void apply(Slice& s, const Inverse& m, const lu_t (&b)[ROWS], lu_t* out, const Lanes& L) {
  lu_t* const x = exchange(s, 0);
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
    if (L.lane + q * MDX_TEAM < MDX_NV) x[m.column[q]] = b[q];
  __syncwarp(L.mask);
  lu_t acc[ROWS][4];  // four chains: a solve waits for a quarter of its row's multiply-adds
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[q][e] = (lu_t)0;
  const Four* const in = reinterpret_cast<const Four*>(x);
#pragma unroll
  for (int j = 0; j < PADDED; j += 4) {
    const Four p = in[j / 4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (j + e < MDX_NV) {
#pragma unroll
        for (int q = 0; q < ROWS; ++q) acc[q][e] += m.a[q][j + e] * p.v[e];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < ROWS; ++q)
    if (L.lane + q * MDX_TEAM < MDX_NV) out[m.column[q]] = (acc[q][0] + acc[q][1]) + (acc[q][2] + acc[q][3]);
  __syncwarp(L.mask);
}

}  // namespace team
}  // namespace mdx
