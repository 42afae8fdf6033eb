// Thomas sweeps on the PCR-reduced chains a lane holds in registers, shared by
// the PCR-then-Thomas kernels (pcr_thomas2.cu, pcr_wide.cu).
#pragma once
#include "pcr_twophase.cuh"

namespace tridi {
namespace pcr2 {

// Thomas on the lane's chains: KG chains of R / KG rows, chain s0 in slots
// s0 + KG * k (normalised rows: a x_prev + x + c x_next = d).  emit(s, x)
// takes the unknown of slot s.
template <int R, int KG, class Emit>
__device__ __forceinline__ void thomas_pairs(NR2 (&P)[R / 2], const Emit& emit) {
  constexpr int KP = KG / 2;  // chain pairs (slots 2 j', 2 j' + 1 of pair j')
  constexpr int L = R / KG;   // rows per chain
#pragma unroll
  for (int jp = 0; jp < KP; ++jp) {
    float2 cp = P[jp].c, dp = P[jp].d;
#pragma unroll
    for (int k = 1; k < L; ++k) {
      NR2& r = P[jp + KP * k];
      const float2 na = neg2(r.a);
      const float2 inv = rcp_approx2(__ffma2_rn(na, cp, make_float2(1.0f, 1.0f)));
      cp = __fmul2_rn(r.c, inv);
      dp = __fmul2_rn(__ffma2_rn(na, dp, r.d), inv);
      r.c = cp;
      r.d = dp;
    }
    float2 x = dp;
#pragma unroll
    for (int k = L - 1; k >= 0; --k) {
      const int j = jp + KP * k;
      if (k < L - 1) x = __ffma2_rn(neg2(P[j].c), x, P[j].d);
      emit(2 * j, x.x);
      emit(2 * j + 1, x.y);
    }
  }
}

// One chain a lane: slots 0 .. R-1 in order.
template <int R, class Emit>
__device__ __forceinline__ void thomas_single(NR (&w)[R], const Emit& emit) {
  float cp = w[0].c, dp = w[0].d;
#pragma unroll
  for (int s = 1; s < R; ++s) {
    const float inv = rcp_approx(fmaf(-w[s].a, cp, 1.0f));
    cp = w[s].c * inv;
    dp = fmaf(-w[s].a, dp, w[s].d) * inv;
    w[s].c = cp;
    w[s].d = dp;
  }
  float x = dp;
  emit(R - 1, x);
#pragma unroll
  for (int s = R - 2; s >= 0; --s) {
    x = fmaf(-w[s].c, x, w[s].d);
    emit(s, x);
  }
}

}  // namespace pcr2
}  // namespace tridi
