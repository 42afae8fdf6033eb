// Partition solver: the GB300 engine for systems of any size (not only powers
// of two), used by the generic solve, the large-system and ragged paths and
// the refinement loop.  It has no counterpart kernel in the reference; its
// oracle is the same gold Thomas solver (tridiagonal_gold.h:26-44).
//
// A system's rows are cut into contiguous chunks, one per lane (thread).  The
// last row of chunk j is its separator s_j; the other rows are interior.
//   1. Chunk elimination (sequential, in registers): a downward Thomas-like
//      sweep over the interior rows gives, per row i,
//          x_i + c'_i x_{i+1} + a'_i s_{j-1} = d'_i
//      (one reciprocal and six flops per row).  A division-free upward pass
//      expresses the first interior row as x = D - C s_j - A s_{j-1}; the
//      last interior row is already in that form.
//   2. Separator system: substituting the neighbouring interior rows into the
//      separator's equation couples s_j to s_{j-1} and s_{j+1} only: a
//      tridiagonal system with one row per lane, solved by PCR over the warp's
//      lanes (shuffles; lanes past the system are identity rows).
//   3. Back substitution: x_{k-1} = s_j, x_i = d'_i - c'_i x_{i+1} - a'_i s_{j-1}.
// a[0] and c[n-1] are ignored (treated as zero), as the gold solver does.
//
// Lanes own an odd number of rows (kk), so lane l reading row l*kk + i of a
// dense shared-memory copy of the system hits 32 distinct banks.
#pragma once
#include "tridi_device.cuh"

namespace tridi {

template <class T, int K>
struct Chunk {
  T cp[K], ap[K], dp[K];  // normalised downward elimination of the interior rows
  Row<T> sep;             // separator row (the chunk's last row)
  T fD, fC, fA;           // first interior row:  x = fD - fC s_j - fA s_{j-1}
  T lD, lC, lA;           // last interior row (row k-2), same form
};

// Eliminates the lane's k rows (0 <= k <= K), interior row i of the chunk being
// row(i), its last row sep.  first/last: the chunk holds the system's
// first/last row.
template <class T, int K, class RowAt>
__device__ __forceinline__ void chunk_eliminate_rows(Chunk<T, K>& ch, int k, bool first, bool last, const RowAt& row,
                                                     const Row<T>& sep) {
  T cprev = T(0), aprev = T(0), dprev = T(0);
#pragma unroll
  for (int i = 0; i < K; ++i) {
    if (i < k - 1) {
      const Row<T> r = row(i);
      const T a = (i == 0 && first) ? T(0) : r.a;
      tdiv3(r.c, i == 0 ? a : -a * aprev, r.d - a * dprev, r.b - a * cprev, ch.cp[i], ch.ap[i], ch.dp[i]);
      cprev = ch.cp[i];
      aprev = ch.ap[i];
      dprev = ch.dp[i];
    }
  }
  // Upward, division free: coefficients of the first interior row.  Seeded
  // with the separator itself (x_{k-1} = s_j: D = 0, C = -1, A = 0), so the
  // step at row k-2 yields exactly (d', c', a') of that row, and a chunk with
  // no interior row keeps (0, -1, 0): the row after the left separator is s_j.
  T D = T(0), C = T(-1), A = T(0);
#pragma unroll
  for (int i = K - 1; i >= 0; --i) {
    if (i <= k - 2) {
      D = ch.dp[i] - ch.cp[i] * D;
      C = -ch.cp[i] * C;
      A = ch.ap[i] - ch.cp[i] * A;
    }
  }
  ch.fD = D; ch.fC = C; ch.fA = A;
  if (k >= 2) {
    ch.lD = dprev; ch.lC = cprev; ch.lA = aprev;
  } else {  // no interior row: the row before the separator is s_{j-1}
    ch.lD = T(0); ch.lC = T(0); ch.lA = T(-1);
  }
  if (k >= 1) {
    ch.sep = sep;
    if (k == 1 && first) ch.sep.a = T(0);
    if (last) ch.sep.c = T(0);
  } else {  // lane past the end of the system: identity separator
    ch.sep = Row<T>{T(0), T(1), T(0), T(0)};
  }
}

// Rows (pa[i*rs], pb[i*rs], pc[i*rs], pd[i*rs]).  PREFETCH (for global-memory
// rows): all k rows are loaded into registers before the dependent elimination
// chain starts, so their loads overlap.
template <class T, int K, bool PREFETCH = false>
__device__ __forceinline__ void chunk_eliminate(Chunk<T, K>& ch, int k, bool first, bool last, const T* pa,
                                                const T* pb, const T* pc, const T* pd, long rs = 1) {
  T qa[PREFETCH ? K : 1], qb[PREFETCH ? K : 1], qc[PREFETCH ? K : 1], qd[PREFETCH ? K : 1];
  if constexpr (PREFETCH) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (i < k - 1) {
        qa[i] = pa[i * rs]; qb[i] = pb[i * rs]; qc[i] = pc[i * rs]; qd[i] = pd[i * rs];
      }
    }
  }
  Row<T> sep{};
  if (k >= 1) {
    const long o = (long)(k - 1) * rs;
    sep = Row<T>{pa[o], pb[o], pc[o], pd[o]};
  }
  chunk_eliminate_rows<T, K>(
      ch, k, first, last,
      [&](int i) {
        if constexpr (PREFETCH) return Row<T>{qa[i], qb[i], qc[i], qd[i]};
        else return Row<T>{pa[i * rs], pb[i * rs], pc[i * rs], pd[i * rs]};
      },
      sep);
}

// The same with the right-hand sides in registers (a correction's residuals).
template <class T, int K>
__device__ __forceinline__ void chunk_eliminate_rhs(Chunk<T, K>& ch, int k, bool first, bool last, const T* pa,
                                                    const T* pb, const T* pc, const T (&rhs)[K]) {
  Row<T> sep{};
  if (k >= 1) sep = Row<T>{pa[k - 1], pb[k - 1], pc[k - 1], T(0)};
#pragma unroll
  for (int i = 0; i < K; ++i)
    if (i == k - 1) sep.d = rhs[i];
  chunk_eliminate_rows<T, K>(
      ch, k, first, last, [&](int i) { return Row<T>{pa[i], pb[i], pc[i], rhs[i]}; }, sep);
}

// Summary of a chunk eliminated in shared memory: what the separator system
// and the back substitution need besides the rows themselves.
template <class T>
struct ChunkSummary {
  Row<T> sep;
  T fD, fC, fA;
  T lD, lC, lA;
};

// The right-hand side of row i as staged (rhs(i, a, b, c, d) = d).  A
// right-hand side functor is told the chunk's first row (start) and then
// called for the chunk's rows in order.
struct RhsStaged {
  __device__ __forceinline__ void start(int) const {}
  template <class T>
  __device__ __forceinline__ T operator()(int, T, T, T, T d) const {
    return d;
  }
};

// chunk_eliminate on rows held in shared memory (no size bound, K-free):
// interior rows i < k-1 get (a, c, d) overwritten by (ap, cp, dp), so the
// back substitution reads them again instead of holding 3k registers.
// Row i's right-hand side is rhs(i, a_i, b_i, c_i, d_i) of its staged values
// (a correction solve forms its residual there, as the row is eliminated).
// RS: words from one row to the next.
template <class T, int RS = 1, class Rhs = RhsStaged>
__device__ __forceinline__ void chunk_eliminate_smem(ChunkSummary<T>& cs, int k, bool first, bool last,
                                                     T* __restrict__ sa, const T* __restrict__ sb,
                                                     T* __restrict__ sc, T* __restrict__ sd,
                                                     const Rhs& rhs = Rhs()) {
  T cprev = T(0), aprev = T(0), dprev = T(0);
  const auto step = [&](int i, T a0, T b0, T c0, T r) {
    const T a = (i == 0 && first) ? T(0) : a0;
    T cn, an, dn;
    tdiv3(c0, i == 0 ? a : -a * aprev, r - a * dprev, b0 - a * cprev, cn, an, dn);
    sa[i * RS] = an; sc[i * RS] = cn; sd[i * RS] = dn;
    cprev = cn; aprev = an; dprev = dn;
  };
#pragma unroll 4
  for (int i = 0; i < k - 1; ++i) {
    const T a0 = sa[i * RS], b0 = sb[i * RS], c0 = sc[i * RS];
    step(i, a0, b0, c0, rhs(i, a0, b0, c0, sd[i * RS]));
  }
  T D = T(0), C = T(-1), A = T(0);
#pragma unroll 4
  for (int i = k - 2; i >= 0; --i) {
    const T c = sc[i * RS];
    D = sd[i * RS] - c * D;
    C = -c * C;
    A = sa[i * RS] - c * A;
  }
  cs.fD = D; cs.fC = C; cs.fA = A;
  if (k >= 2) {
    cs.lD = dprev; cs.lC = cprev; cs.lA = aprev;
  } else {
    cs.lD = T(0); cs.lC = T(0); cs.lA = T(-1);
  }
  if (k >= 1) {
    const T a0 = sa[(k - 1) * RS], b0 = sb[(k - 1) * RS], c0 = sc[(k - 1) * RS];
    cs.sep = Row<T>{a0, b0, c0, rhs(k - 1, a0, b0, c0, sd[(k - 1) * RS])};
    if (k == 1 && first) cs.sep.a = T(0);
    if (last) cs.sep.c = T(0);
  } else {
    cs.sep = Row<T>{T(0), T(1), T(0), T(0)};
  }
}

template <class T>
__device__ __forceinline__ Row<T> separator_row_s(const ChunkSummary<T>& cs, T nD, T nC, T nA) {
  const Row<T>& s = cs.sep;
  return Row<T>{-s.a * cs.lA, s.b - s.a * cs.lC - s.c * nA, -s.c * nC, s.d - s.a * cs.lD - s.c * nD};
}

// Back substitution of a chunk eliminated by chunk_eliminate_smem: emit(i, x_i)
// for every row i < k of the chunk, last row first.
// (emit writes to arrays other than sa, sc, sd.)
template <class T, int RS = 1, class Emit>
__device__ __forceinline__ void chunk_back_smem(int k, T sj, T sl, const T* __restrict__ sa,
                                                const T* __restrict__ sc, const T* __restrict__ sd, Emit& emit) {
  if (k >= 1) emit(k - 1, sj);
  T xn = sj;
#pragma unroll 4
  for (int i = k - 2; i >= 0; --i) {
    xn = sd[i * RS] - sc[i * RS] * xn - sa[i * RS] * sl;
    emit(i, xn);
  }
}

// ---- a chunk in shared memory, eliminated once for two right-hand sides ----
// chunk_factor_smem leaves 1 / p_i over b, with the pivots p_i (the separator
// row's b becomes 1; a, c and d stay), and the chunk's summary, accumulated on
// the way (chunk_eliminate_smem reads the rows again for it): with c' = c / p and
// P the product of the -c' before it, a block of four rows adds P times its own
// D = d'_0 - c'_0 (d'_1 - c'_1 (d'_2 - c'_2 d'_3)), and A likewise, so that the
// sums' roundings are those of the few blocks that P leaves large (summed row by
// row, the error of a refined batch grew by half).  chunk_between_smem then
// solves between the separators.  For a second right-hand side a / p goes over
// a, c / p over c and g = r / p anywhere: chunk_rhs_smem gives its D and last
// d', chunk_between_scaled_smem its unknowns.  (With the scaled rows in the first
// solve as well, both solves carry the same rounding in the matrix, and the
// refined error grew by 6%.)
__device__ __forceinline__ void chunk_factor_smem(ChunkSummary<float>& cs, int k, bool first, bool last,
                                                  float* __restrict__ sa, float* __restrict__ sb,
                                                  const float* __restrict__ sc, const float* __restrict__ sd) {
  float cprev = 0.f, aprev = -1.f, dprev = 0.f, P = 1.f, D = 0.f, A = 0.f;
  if (first && k >= 1) sa[0] = 0.f;
  const auto step = [&](int i) {
    const float a = sa[i];
    const float inv = tdiv(1.f, sb[i] - a * cprev);
    cprev = sc[i] * inv;
    aprev = -a * aprev * inv;
    dprev = (sd[i] - a * dprev) * inv;
    sb[i] = inv;
  };
  int i = 0;
  for (; i + 4 < k; i += 4) {
    float c[4], a[4], d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      step(i + q);
      c[q] = cprev; a[q] = aprev; d[q] = dprev;
    }
    D += P * (d[0] - c[0] * (d[1] - c[1] * (d[2] - c[2] * d[3])));
    A += P * (a[0] - c[0] * (a[1] - c[1] * (a[2] - c[2] * a[3])));
    P *= (c[0] * c[1]) * (c[2] * c[3]);
  }
  for (; i < k - 1; ++i) {
    step(i);
    D += P * dprev;
    A += P * aprev;
    P *= -cprev;
  }
  cs.fD = D; cs.fC = -P; cs.fA = A;
  cs.lD = dprev; cs.lC = cprev; cs.lA = aprev;
  cs.sep = Row<float>{0.f, 1.f, 0.f, 0.f};
  if (k >= 1) {
    cs.sep = Row<float>{sa[k - 1], sb[k - 1], last ? 0.f : sc[k - 1], sd[k - 1]};
    sb[k - 1] = 1.f;
  }
}

// The chunk's unknowns over d, between sl (the row before it) and sj (its last).
__device__ __forceinline__ void chunk_between_smem(int k, float sj, float sl, const float* __restrict__ sa,
                                                   const float* __restrict__ inv, const float* __restrict__ sc,
                                                   float* __restrict__ sd) {
  float v = sl;
#pragma unroll 4
  for (int i = 0; i < k - 1; ++i) {
    v = (sd[i] - sa[i] * v) * inv[i];
    sd[i] = v;
  }
  if (k >= 1) sd[k - 1] = sj;
  v = sj;
#pragma unroll 4
  for (int i = k - 2; i >= 0; --i) {
    v = sd[i] - sc[i] * v * inv[i];
    sd[i] = v;
  }
}

// The first row's D and the last interior row's d' of a right-hand side g
// (divided by the pivots, as sa is).
__device__ __forceinline__ void chunk_rhs_smem(int k, const float* __restrict__ sa, const float* __restrict__ sc,
                                               const float* __restrict__ g, float& fD, float& lD) {
  float P = 1.f, D = 0.f, dprev = 0.f;
  int i = 0;
  for (; i + 4 < k; i += 4) {
    float c[4], d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      d[q] = dprev = g[i + q] - sa[i + q] * dprev;
      c[q] = sc[i + q];
    }
    D += P * (d[0] - c[0] * (d[1] - c[1] * (d[2] - c[2] * d[3])));
    P *= (c[0] * c[1]) * (c[2] * c[3]);
  }
  for (; i < k - 1; ++i) {
    dprev = g[i] - sa[i] * dprev;
    D += P * dprev;
    P *= -sc[i];
  }
  fD = D; lD = dprev;
}

__device__ __forceinline__ void chunk_between_scaled_smem(int k, float sj, float sl, const float* __restrict__ sa,
                                                          const float* __restrict__ sc, float* __restrict__ g) {
  float v = sl;
#pragma unroll 4
  for (int i = 0; i < k - 1; ++i) {
    v = g[i] - sa[i] * v;
    g[i] = v;
  }
  if (k >= 1) g[k - 1] = sj;
  v = sj;
#pragma unroll 4
  for (int i = k - 2; i >= 0; --i) {
    v = g[i] - sc[i] * v;
    g[i] = v;
  }
}

// The chunk's unknowns between its known neighbours -- sl the row before it, sj
// its last row -- from its rows as they were read: a Thomas sweep over the
// interior rows (the coupling to sl goes to the right-hand side), 3 operations
// and 2 quotients a row where the elimination above takes 8 and 3.
template <class T, int K, bool PREFETCH = false>
__device__ __forceinline__ void chunk_between(int k, bool first, T sl, T sj, const T* pa, const T* pb, const T* pc,
                                              const T* pd, long rs, T (&x)[K]) {
  T qa[PREFETCH ? K : 1], qb[PREFETCH ? K : 1], qc[PREFETCH ? K : 1], qd[PREFETCH ? K : 1];
  if constexpr (PREFETCH) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (i < k - 1) {
        qa[i] = pa[i * rs]; qb[i] = pb[i * rs]; qc[i] = pc[i * rs]; qd[i] = pd[i * rs];
      }
    }
  }
  T cp[K], cprev = T(0), dprev = sl;  // row 0's left neighbour: x = sl - 0 x
#pragma unroll
  for (int i = 0; i < K; ++i) {
    if (i < k - 1) {
      const Row<T> r = PREFETCH ? Row<T>{qa[PREFETCH ? i : 0], qb[PREFETCH ? i : 0], qc[PREFETCH ? i : 0],
                                         qd[PREFETCH ? i : 0]}
                                : Row<T>{pa[i * rs], pb[i * rs], pc[i * rs], pd[i * rs]};
      const T a = (i == 0 && first) ? T(0) : r.a;
      tdiv2(r.c, r.d - a * dprev, i == 0 ? r.b : r.b - a * cprev, cp[i], x[i]);
      cprev = cp[i];
      dprev = x[i];
    }
  }
  T xn = sj;
#pragma unroll
  for (int i = K - 1; i >= 0; --i) {
    if (i <= k - 2) {
      xn = x[i] - cp[i] * xn;
      x[i] = xn;
    } else {
      x[i] = sj;
    }
  }
}

// The lane's row of the separator system, given the next chunk's first
// interior row (nD, nC, nA).
template <class T, int K>
__device__ __forceinline__ Row<T> separator_row(const Chunk<T, K>& ch, T nD, T nC, T nA) {
  const Row<T>& s = ch.sep;
  return Row<T>{-s.a * ch.lA, s.b - s.a * ch.lC - s.c * nA, -s.c * nC, s.d - s.a * ch.lD - s.c * nD};
}

// PCR over the 32 lanes of a warp (one row per lane, identity rows outside):
// returns the lane's unknown.
template <class T>
__device__ __forceinline__ T warp_pcr32(Row<T> r) {
  const int lane = threadIdx.x & 31;
  const Row<T> id{T(0), T(1), T(0), T(0)};
#pragma unroll
  for (int dl = 1; dl < 32; dl *= 2) {
    Row<T> L = shfl_up(r, dl, 32);
    Row<T> R = shfl_down(r, dl, 32);
    if (lane < dl) L = id;
    if (lane + dl > 31) R = id;
    r = reduce_row(r, L, R);
  }
  return tdiv(r.d, r.b);
}

// Back substitution of the lane's chunk: sj its separator, sl the left one.
template <class T, int K>
__device__ __forceinline__ void chunk_back(const Chunk<T, K>& ch, int k, T sj, T sl, T (&x)[K]) {
  T xn = sj;
#pragma unroll
  for (int i = K - 1; i >= 0; --i) {
    xn = (i <= k - 2) ? ch.dp[i] - ch.cp[i] * xn - ch.ap[i] * sl : sj;
    x[i] = xn;
  }
}

// Same, handing each unknown to emit(i, x_i) (i < k) as soon as it is known.
template <class T, int K, class Emit>
__device__ __forceinline__ void chunk_back_emit(const Chunk<T, K>& ch, int k, T sj, T sl, Emit& emit) {
  T xn = sj;
#pragma unroll
  for (int i = K - 1; i >= 0; --i) {
    xn = (i <= k - 2) ? ch.dp[i] - ch.cp[i] * xn - ch.ap[i] * sl : sj;
    if (i < k) emit(i, xn);
  }
}

}  // namespace tridi
