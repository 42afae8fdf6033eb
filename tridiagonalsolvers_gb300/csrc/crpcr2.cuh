// CR levels, PCR and back substitutions on rows held in a warp's registers,
// one system (or what is left of one) a warp: shared by crpcr2.cu and
// crpcr_wide.cu.
#pragma once
#include "hybrid.cuh"
#include "pcr_twophase.cuh"

namespace tridi {
namespace pcr2 {

// One CR level of the lane's K unnormalised rows (local rows 0..K-1 of a
// contiguous block): the odd rows 2j+1 eliminate their even neighbours (the
// last one's right neighbour, row K of the block, is the next lane's row 0:
// one shuffle; lane 31's has c = 0 and contributes nothing).  The K/2 new
// rows land in (na, nb, nc, nd).
template <int K>
__device__ __forceinline__ void cr_level(const float (&a)[K], const float (&b)[K], const float (&c)[K],
                                         const float (&d)[K], float (&na)[K / 2], float (&nb)[K / 2],
                                         float (&nc)[K / 2], float (&nd)[K / 2]) {
  const float ra = __shfl_down_sync(kFull, a[0], 1), rb = __shfl_down_sync(kFull, b[0], 1);
  const float rc = __shfl_down_sync(kFull, c[0], 1), rd = __shfl_down_sync(kFull, d[0], 1);
#pragma unroll
  for (int j = 0; j < K / 2; ++j) {
    const int q = 2 * j + 1;
    const float aR = q + 1 < K ? a[q + 1] : ra, bR = q + 1 < K ? b[q + 1] : rb;
    const float cR = q + 1 < K ? c[q + 1] : rc, dR = q + 1 < K ? d[q + 1] : rd;
    const float k1 = tdiv(a[q], b[q - 1]);
    const float k2 = tdiv(c[q], bR);
    na[j] = -a[q - 1] * k1;
    nb[j] = b[q] - c[q - 1] * k1 - aR * k2;
    nc[j] = -cR * k2;
    nd[j] = d[q] - d[q - 1] * k1 - dR * k2;
  }
}

// The even rows of a CR level given x of the odd ones (xo[j] = x of row 2j+1
// of the lane's block): x[2j] = (d - a x[2j-1] - c x[2j+1]) / b, row -1 the
// previous lane's last odd row (zero for lane 0, whose first row has a = 0).
template <int K>
__device__ __forceinline__ void cr_back(const float (&a)[K], const float (&b)[K], const float (&c)[K],
                                        const float (&d)[K], const float (&xo)[K / 2], float (&x)[K], int lane) {
  float xprev = __shfl_up_sync(kFull, xo[K / 2 - 1], 1);
  if (lane == 0) xprev = 0.0f;
#pragma unroll
  for (int j = 0; j < K / 2; ++j) {
    x[2 * j] = (d[2 * j] - a[2 * j] * xprev - c[2 * j] * xo[j]) * rcp_approx(b[2 * j]);
    x[2 * j + 1] = xo[j];
    xprev = xo[j];
  }
}

// The same level with the even rows normalised first, (ea, ec, ed) = (a, c, d)
// / b of row 2j: one reciprocal per even row instead of two per odd row, and
// the back substitution (cr_back_norm) needs none.  The eliminations then
// take the form me - a_q L' - c_q R' with normalised neighbours, which rounds
// differently from CR's own divisions (used where crpcr switches above 2).
template <int K>
__device__ __forceinline__ void cr_level_norm(const float (&a)[K], const float (&b)[K], const float (&c)[K],
                                              const float (&d)[K], float (&ea)[K / 2], float (&ec)[K / 2],
                                              float (&ed)[K / 2], float (&na)[K / 2], float (&nb)[K / 2],
                                              float (&nc)[K / 2], float (&nd)[K / 2]) {
#pragma unroll
  for (int j = 0; j < K / 2; ++j) {
    const float ib = rcp_approx(b[2 * j]);
    ea[j] = a[2 * j] * ib;
    ec[j] = c[2 * j] * ib;
    ed[j] = d[2 * j] * ib;
  }
  const float ra = __shfl_down_sync(kFull, ea[0], 1), rc = __shfl_down_sync(kFull, ec[0], 1);
  const float rd = __shfl_down_sync(kFull, ed[0], 1);
#pragma unroll
  for (int j = 0; j < K / 2; ++j) {
    const int q = 2 * j + 1;
    const float Ra = j + 1 < K / 2 ? ea[j + 1] : ra, Rc = j + 1 < K / 2 ? ec[j + 1] : rc;
    const float Rd = j + 1 < K / 2 ? ed[j + 1] : rd;
    na[j] = -a[q] * ea[j];
    nb[j] = b[q] - a[q] * ec[j] - c[q] * Ra;
    nc[j] = -c[q] * Rc;
    nd[j] = d[q] - a[q] * ed[j] - c[q] * Rd;
  }
}

template <int K>
__device__ __forceinline__ void cr_back_norm(const float (&ea)[K / 2], const float (&ec)[K / 2],
                                             const float (&ed)[K / 2], const float (&xo)[K / 2], float (&x)[K],
                                             int lane) {
  float xprev = __shfl_up_sync(kFull, xo[K / 2 - 1], 1);
  if (lane == 0) xprev = 0.0f;
#pragma unroll
  for (int j = 0; j < K / 2; ++j) {
    x[2 * j] = ed[j] - ea[j] * xprev - ec[j] * xo[j];
    x[2 * j + 1] = xo[j];
    xprev = xo[j];
  }
}

// PCR step between lanes: lane t holds rows K2 t + j, so the neighbours at
// distance K2 ld are lanes t -/+ ld in the same slot.  Lanes whose neighbour
// lies beyond the system's ends receive their own row from the shuffle: the
// coupling there is exactly zero.
template <int K2>
__device__ __forceinline__ void lane_step(NR (&w)[K2], int ld) {
#pragma unroll
  for (int j = 0; j < K2; ++j) {
    const NR L{__shfl_up_sync(kFull, w[j].a, ld), __shfl_up_sync(kFull, w[j].c, ld),
               __shfl_up_sync(kFull, w[j].d, ld)};
    const NR Rr{__shfl_down_sync(kFull, w[j].a, ld), __shfl_down_sync(kFull, w[j].c, ld),
                __shfl_down_sync(kFull, w[j].d, ld)};
    w[j] = step_both(w[j], L, Rr);
  }
}

// PCR on the rows left by the CR levels: lane t holds rows K2 t .. K2 t + K2 - 1
// (unnormalised) of the 32 K2 rows, or, after CR levels between lanes
// (LD0 = 2^levels > 1, K2 = 1), only the lanes t = LD0 j + LD0 - 1 hold a row
// (row j of 32 / LD0).  Distances below K2 run inside the lane, the others
// between lanes (lane distances LD0 .. 8), then the closing 2x2 systems
// pair lane t with lane t ^ 16 in the same slot.  x of the lane's rows out
// (meaningless on lanes that hold no row).
template <int K2, int LD0>
__device__ __forceinline__ void pcr_lanes(const float (&a)[K2], const float (&b)[K2], const float (&c)[K2],
                                          const float (&d)[K2], float (&x)[K2], int lane) {
  NR w[K2];
#pragma unroll
  for (int j = 0; j < K2; ++j) {
    const float ib = rcp_approx(b[j]);
    w[j] = NR{a[j] * ib, c[j] * ib, d[j] * ib};
  }
  if constexpr (K2 >= 2) phase_a_step<1, 32, K2>(w);
  if constexpr (K2 >= 4) phase_a_step<2, 32, K2>(w);
  if constexpr (K2 >= 8) phase_a_step<4, 32, K2>(w);
  if constexpr (K2 >= 16) phase_a_step<8, 32, K2>(w);
#pragma unroll
  for (int ld = LD0; ld < 16; ld *= 2) lane_step<K2>(w, ld);
#pragma unroll
  for (int j = 0; j < K2; ++j) {
    const NR pr = shfl_xor_nr(w[j], 16);
    const NR& u = lane < 16 ? w[j] : pr;  // row r
    const NR& l = lane < 16 ? pr : w[j];  // row r + 16 K2 (r + 16 / LD0 between lanes)
    const float xu = (u.d - u.c * l.d) * rcp_approx(fmaf(-u.c, l.a, 1.0f));
    x[j] = lane < 16 ? xu : fmaf(-l.a, xu, l.d);
  }
}

// L2 CR levels between lanes on a 32-row system held one row a lane (row t in
// lane t), the PCR of the 32 / 2^L2 rows left, and the back substitutions.
// Level i (lane stride s = 2^i) leaves the rows of lanes t with
// (t + 1) mod 2s = 0, each from its neighbours t -/+ s; every lane computes
// (the warp stays converged) and keeps the row it held at each level for the
// back substitution, where the lanes with (t + 1) mod 2s = s take x from
// lanes t -/+ s.  Active rows only ever read active rows; the last row's
// c = 0 zeroes the neighbour that lane 31 receives from itself, and the
// first row's a = 0 the one that lane s - 1 receives from itself.
template <int L2>
__device__ __forceinline__ float cr_cross(float a, float b, float c, float d, int lane) {
  float la[L2], lb[L2], lc[L2], ld[L2];
#pragma unroll
  for (int i = 0; i < L2; ++i) {
    const int s = 1 << i;
    const float aL = __shfl_up_sync(kFull, a, s), bL = __shfl_up_sync(kFull, b, s);
    const float cL = __shfl_up_sync(kFull, c, s), dL = __shfl_up_sync(kFull, d, s);
    const float aR = __shfl_down_sync(kFull, a, s), bR = __shfl_down_sync(kFull, b, s);
    const float cR = __shfl_down_sync(kFull, c, s), dR = __shfl_down_sync(kFull, d, s);
    la[i] = a; lb[i] = b; lc[i] = c; ld[i] = d;
    const float k1 = tdiv(a, bL);
    const float k2 = tdiv(c, bR);
    a = -aL * k1;
    b = b - cL * k1 - aR * k2;
    c = -cR * k2;
    d = d - dL * k1 - dR * k2;
  }
  float x = 0.0f;
  if constexpr (L2 == 4) {
    // two rows left (lanes 15 and 31): CR's closing 2x2 solve on the
    // unnormalised rows, so that cr here rounds like every other CR kernel
    const Row<float> r1{__shfl_sync(kFull, a, 15), __shfl_sync(kFull, b, 15), __shfl_sync(kFull, c, 15),
                        __shfl_sync(kFull, d, 15)};
    const Row<float> r2{__shfl_sync(kFull, a, 31), __shfl_sync(kFull, b, 31), __shfl_sync(kFull, c, 31),
                        __shfl_sync(kFull, d, 31)};
    if (lane == 15) x = solve2_upper(r1, r2);
    if (lane == 31) x = solve2_lower(r1, r2);
  } else {
    const float ta[1] = {a}, tb[1] = {b}, tc[1] = {c}, td[1] = {d};
    float xt[1];
    pcr_lanes<1, (1 << L2)>(ta, tb, tc, td, xt, lane);
    if (((lane + 1) & ((1 << L2) - 1)) == 0) x = xt[0];
  }
#pragma unroll
  for (int i = L2 - 1; i >= 0; --i) {
    const int s = 1 << i;
    const float xL = __shfl_up_sync(kFull, x, s), xR = __shfl_down_sync(kFull, x, s);
    if (((lane + 1) & (2 * s - 1)) == s) x = (ld[i] - la[i] * xL - lc[i] * xR) * rcp_approx(lb[i]);
  }
  return x;
}

// LEV CR levels down from the lane's K rows (the levels past K = 1 between
// lanes), the PCR, and the back substitutions up again.  NORM: the in-lane
// levels on normalised even rows (cr_level_norm); else CR's own arithmetic.
template <int K, int LEV, bool NORM>
__device__ __forceinline__ void cr_solve(const float (&a)[K], const float (&b)[K], const float (&c)[K],
                                         const float (&d)[K], float (&x)[K], int lane) {
  float na[K / 2], nb[K / 2], nc[K / 2], nd[K / 2], xo[K / 2];
  if constexpr (NORM) {
    float ea[K / 2], ec[K / 2], ed[K / 2];
    cr_level_norm<K>(a, b, c, d, ea, ec, ed, na, nb, nc, nd);
    if constexpr (LEV == 1) pcr_lanes<K / 2, 1>(na, nb, nc, nd, xo, lane);
    else if constexpr (K == 2) xo[0] = cr_cross<LEV - 1>(na[0], nb[0], nc[0], nd[0], lane);
    else cr_solve<K / 2, LEV - 1, NORM>(na, nb, nc, nd, xo, lane);
    cr_back_norm<K>(ea, ec, ed, xo, x, lane);
  } else {
    cr_level<K>(a, b, c, d, na, nb, nc, nd);
    if constexpr (LEV == 1) pcr_lanes<K / 2, 1>(na, nb, nc, nd, xo, lane);
    else if constexpr (K == 2) xo[0] = cr_cross<LEV - 1>(na[0], nb[0], nc[0], nd[0], lane);
    else cr_solve<K / 2, LEV - 1, NORM>(na, nb, nc, nd, xo, lane);
    cr_back<K>(a, b, c, d, xo, x, lane);
  }
}

}  // namespace pcr2
}  // namespace tridi
