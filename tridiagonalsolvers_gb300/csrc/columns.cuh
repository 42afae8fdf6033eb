// Interleaved systems (element i of system s at i*m + s) that a CTA holds
// whole, 32 of them: warp w rows [16 w, 16 w + 16), lane l system s0 + l.  Each
// warp has its rows in shared memory (large_tma.cu stages them by tensor
// copies, large.cu by plain loads), eliminates them in place and leaves its
// first-row values beside them; the separators, one a warp, are solved by one
// warp, a lane per system; each warp substitutes back.  20 B a row (FP32) where
// the reduce and back passes move 36, and one launch for their four, or for
// seven with one more level between.  What bounds it for few systems is
// latency: a solve of 32 x 33 .. 448 x 8192 FP32 took 31 to 46 us by the passes,
// 16 to 19 us so (launch and host path included); for many, 448 x 65536, 216
// and 120 us; 65536 x 1024, whose separators end here, 437 and 423 us.
#pragma once
#include "partition.cuh"

namespace tridi {

constexpr int kColChunk = 16;   // rows a warp
constexpr int kColSystems = 32;  // systems a CTA
template <class T>
constexpr int kColWarps = sizeof(T) == 4 ? 28 : 14;  // 224 KB of rows
template <class T>
constexpr int kColRows = kColWarps<T> * kColChunk;
template <class T>
constexpr int kColArray = kColChunk * kColSystems;  // elements per array of a warp's rows
constexpr size_t kColHead = 256;                     // before the rows: a barrier a warp
template <class T>
constexpr size_t columns_smem(int warps) {
  return kColHead + (size_t)warps * 4 * kColArray<T> * sizeof(T);
}
static_assert(columns_smem<float>(kColWarps<float>) <= 232448 && columns_smem<double>(kColWarps<double>) <= 232448);

// From each warp's rows in shared memory (base: the CTA's; a, b, c, d of a warp
// kColArray apart) to x at gx (row 0 of the lane's system; m elements a row).
// ok: this thread's rows are there (false anywhere: nothing is written); live:
// the lane has a system.
template <class T>
__device__ __forceinline__ void columns_solve(T* base, int n, long m, bool ok, bool live, T* gx) {
  constexpr int L = kColChunk, RS = kColSystems, F = kColArray<T>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  T* sa = base + (size_t)warp * 4 * F + lane;
  T *sb = sa + F, *sc = sa + 2 * F, *sd = sa + 3 * F;
  const int r0 = warp * L;
  const int k = n - r0 < L ? n - r0 : L;  // (>= 1)
  ChunkSummary<T> cs;
  chunk_eliminate_smem<T, RS>(cs, k, warp == 0, warp == warps - 1, sa, sb, sc, sd);
  // first-row values into three rows of b that nothing needs any more
  const auto free_row = [](int rows) { return rows >= 4 ? 0 : 4; };
  T* f = sb + free_row(k) * RS;
  f[0] = cs.fD; f[RS] = cs.fC; f[2 * RS] = cs.fA;
  if (!__syncthreads_and(ok)) return;
  T nD = T(0), nC = T(0), nA = T(0);
  if (warp + 1 < warps) {
    const int kn = n - r0 - L < L ? n - r0 - L : L;
    const T* g = sb + 4 * F + free_row(kn) * RS;
    nD = g[0]; nC = g[RS]; nA = g[2 * RS];
  }
  const int last = (k - 1) * RS;  // the separator takes its row's place
  const Row<T> sr = separator_row_s<T>(cs, nD, nC, nA);
  sa[last] = sr.a; sb[last] = sr.b; sc[last] = sr.c; sd[last] = sr.d;
  __syncthreads();
  if (warp == 0) {
    T cp = T(0), dp = T(0);
#pragma unroll 4
    for (int w = 0; w < warps; ++w) {
      T* r = base + (size_t)w * 4 * F + (w == warps - 1 ? n - 1 - w * L : L - 1) * RS + lane;
      tdiv2(r[2 * F], r[3 * F] - r[0] * dp, r[F] - r[0] * cp, cp, dp);
      r[2 * F] = cp;
      r[3 * F] = dp;
    }
    T x = dp;
#pragma unroll 4
    for (int w = warps - 2; w >= 0; --w) {
      T* r = base + (size_t)w * 4 * F + (L - 1) * RS + lane;
      x = r[3 * F] - r[2 * F] * x;
      r[3 * F] = x;
    }
  }
  __syncthreads();
  const T sj = sd[last], sl = warp > 0 ? *(sd - 4 * F + (L - 1) * RS) : T(0);
  T* px = gx + (long)r0 * m;
  auto put = [&](int i, T v) {
    if (live) px[(long)i * m] = v;
  };
  chunk_back_smem<T, RS>(k, sj, sl, sa, sc, sd, put);
}

}  // namespace tridi
