// TMA-tiled passes of the large-system solver for the interleaved FP32
// layout (element i of system s at i*m + s, m a multiple of 32).
//
// The passes of large.cu that read the coefficients as persistent kernels, one
// CTA per SM, on the chunks of its register kernels (16 rows of one system), so
// that the separator system and the recursion are shared with them:
//   * large_reduce_tile_kernel eliminates the chunks and writes the separator
//     system.  A producer warp streams tiles of kTileRows rows x 32 systems of a,
//     b, c, d into a kStages-deep shared-memory ring with
//     cp.async.bulk.tensor.2d (one tensor map per array); 8 consumer warps,
//     warp w rows [w*16, w*16 + 16) of a tile, lane l system s0 + l, eliminate
//     in registers and give the stage back.
//   * large_back_tile_kernel solves each chunk between its separators by a
//     Thomas sweep and writes the unknowns.  Three groups of four warps, each
//     with tiles of its own (64 rows x 32 systems) and a two-stage ring that
//     the group's first thread refills; no producer.
// A lane reads its column of a tile at a row stride of 32 words (lane l always
// on bank l, no conflicts); what it writes goes straight to global memory:
// consecutive lanes, consecutive systems, one 128-byte line per row.
//
// Against the register kernels (one thread per chunk, 64 prefetched values
// and the chunk's eliminated rows in registers, two blocks per SM) the rings
// keep 128 KB and more of loads in flight per SM whatever the compute is doing.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <type_traits>

#include "columns.cuh"
#include "dfloat.cuh"
#include "large_tma.h"
#include "partition.cuh"
#include "runtime.h"

namespace tridi {

namespace {
constexpr int kLtWarps = 8;                  // consumer warps
constexpr int kLtChunk = 16;                 // rows per lane (= the register kernels' chunk)
constexpr int kTileRows = kLtWarps * kLtChunk;  // 128
constexpr int kTileCols = 32;                // systems per tile
constexpr int kStages = 3;
constexpr int kTileFloats = kTileRows * kTileCols;  // per array
constexpr size_t kLtSmem = 128 + (size_t)kStages * 4 * kTileFloats * sizeof(float);  // 192 KB + barriers

struct LtParams {
  long n, m, P, PMp;
  float* red;       // reduce: the separator system, 4 arrays of P*m (stride PMp)
  float* bnd;       // reduce: tile-boundary interface, 10 arrays of row_tiles*m (stride BS)
  long BS;
  const float* sol; // back: separators
  void* x;          // back: solution (FP32, or FP64 in kBackSecond)
  const float* d;   // kBackSecond: the refined system's right-hand side ...
  const float* e0;  // ... and its first solution
  float* r;         // kBackFirst: the residual ...
  float* red_d;     // ... and the right-hand side of its separator system; bnd: lD, fD of each tile (BS apart)
  double* rr;       // kBackFirst, kBackSecond: per-system sums of r^2 ...
  double* dd;       // ... and, kBackFirst, of d^2
  int row_tiles, col_tiles;
  unsigned* status;
};
constexpr int kBndLast = 0;   // bnd arrays 0..6: lD, lC, lA and the separator row of a tile's last chunk
constexpr int kBndFirst = 7;  // bnd arrays 7..9: fD, fC, fA of a tile's first chunk
constexpr size_t kLtExchange = 2 * kLtWarps * 32 * 3 * sizeof(float);  // reduce: fD, fC, fA per lane, two tiles

// Separator row of a chunk (partition.cuh's separator_row_s) from its
// summary and the next chunk's first-row coefficients, into the 4 arrays
// of the separator system at index o.
__device__ __forceinline__ void put_separator(float* red, long S, long o, const Row<float>& sep, float lD, float lC,
                                              float lA, float nD, float nC, float nA) {
  red[0 * S + o] = -sep.a * lA;
  red[1 * S + o] = sep.b - sep.a * lC - sep.c * nA;
  red[2 * S + o] = -sep.c * nC;
  red[3 * S + o] = sep.d - sep.a * lD - sep.c * nD;
}

// Forward elimination of one lane's column (rows 0..k-2 at stride 32 words)
// into registers: the normalised c', a', d' of every interior row.  The
// stage can go back to the producer as soon as this (and the read of the
// separator row) is done.
__device__ __forceinline__ void column_forward(int k, bool first, const float* __restrict__ sa,
                                               const float* __restrict__ sb, const float* __restrict__ sc,
                                               const float* __restrict__ sd, float (&cp)[kLtChunk],
                                               float (&ap)[kLtChunk], float (&dp)[kLtChunk], float& cprev,
                                               float& aprev, float& dprev) {
  cprev = 0.f; aprev = 0.f; dprev = 0.f;
#pragma unroll
  for (int i = 0; i < kLtChunk - 1; ++i) {
    if (i < k - 1) {
      const int o = i * kTileCols;
      const float a = (i == 0 && first) ? 0.f : sa[o];
      const float inv = tdiv(1.f, sb[o] - a * cprev);
      cp[i] = sc[o] * inv;
      ap[i] = (i == 0 ? a : -a * aprev) * inv;
      dp[i] = (sd[o] - a * dprev) * inv;
      cprev = cp[i]; aprev = ap[i]; dprev = dp[i];
    }
  }
}

// The chunk's interface (partition.cuh's Chunk summary) from its eliminated
// rows in registers (last interior row: cl, al, dl).
__device__ __forceinline__ void column_summary(ChunkSummary<float>& cs, int k, const float (&cp)[kLtChunk],
                                               const float (&ap)[kLtChunk], const float (&dp)[kLtChunk], float cl,
                                               float al, float dl) {
  float D = 0.f, C = -1.f, A = 0.f;
#pragma unroll
  for (int i = kLtChunk - 2; i >= 0; --i) {
    if (i <= k - 2) {
      D = dp[i] - cp[i] * D;
      C = -cp[i] * C;
      A = ap[i] - cp[i] * A;
    }
  }
  cs.fD = D; cs.fC = C; cs.fA = A;
  if (k >= 2) {
    cs.lD = dl; cs.lC = cl; cs.lA = al;
  } else {
    cs.lD = 0.f; cs.lC = 0.f; cs.lA = -1.f;
  }
}

__global__ void __launch_bounds__(32 * (kLtWarps + 1), 1)
    large_reduce_tile_kernel(LtParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                      const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + kStages;
  float* ring = reinterpret_cast<float*>(smem + 128);  // stage s, array q at ring + (s*4 + q) * kTileFloats
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ntiles = p.row_tiles * p.col_tiles;
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kLtWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == kLtWarps) {  // ---------------- producer ----------------
    if (lane != 0) return;
    int k = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
      const int s = k % kStages;
      if (k >= kStages && !mbar_wait(&empty[s], ((k / kStages) - 1) & 1, p.status)) return;
      const int x0 = (t % p.col_tiles) * kTileCols, y0 = (t / p.col_tiles) * kTileRows;
      mbar_arrive_expect_tx(&full[s], 4u * kTileFloats * sizeof(float));
      float* st = ring + (size_t)s * 4 * kTileFloats;
      tma_load_2d(st + 0 * kTileFloats, &ma, x0, y0, &full[s]);
      tma_load_2d(st + 1 * kTileFloats, &mb, x0, y0, &full[s]);
      tma_load_2d(st + 2 * kTileFloats, &mc, x0, y0, &full[s]);
      tma_load_2d(st + 3 * kTileFloats, &md, x0, y0, &full[s]);
    }
    return;
  }

  // ---------------- consumers ----------------
  // (the reduce pass exchanges first-row coefficients between its warps
  // through shared memory, so the consumers agree on every wait's outcome
  // and leave together)
  float* exch = reinterpret_cast<float*>(smem + kLtSmem);
  int k = 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
    const int s = k % kStages;
    if (!named_sync_and(1, 32 * kLtWarps, mbar_wait(&full[s], (k / kStages) & 1, p.status))) return;
    const long sys = (long)(t % p.col_tiles) * kTileCols + lane;
    const long r0 = (long)(t / p.col_tiles) * kTileRows + (long)warp * kLtChunk;  // the lane's first row
    const long j = r0 / kLtChunk;                                                 // its chunk
    float* st = ring + (size_t)s * 4 * kTileFloats + warp * kLtChunk * kTileCols + lane;
    float* sa = st;
    float* sb = st + kTileFloats;
    float* sc = st + 2 * kTileFloats;
    float* sd = st + 3 * kTileFloats;
    const long rem = p.n - r0;
    const int kr = rem <= 0 ? 0 : (rem < kLtChunk ? (int)rem : kLtChunk);
    ChunkSummary<float> cs;
    // The eliminated column stays in registers and the stage goes back to
    // the producer right after the elimination (not after the interface
    // exchange).
    float cp[kLtChunk], ap[kLtChunk], dp[kLtChunk];
    float cl = 0.f, al = 0.f, dl = 0.f;
    if (kr > 0) {
      column_forward(kr, j == 0, sa, sb, sc, sd, cp, ap, dp, cl, al, dl);
      const int o = (kr - 1) * kTileCols;
      cs.sep = Row<float>{sa[o], sb[o], sc[o], sd[o]};
      if (kr == 1 && j == 0) cs.sep.a = 0.f;
      if (j == p.P - 1) cs.sep.c = 0.f;
    }
    release_stage(&empty[s]);
    if (kr > 0) column_summary(cs, kr, cp, ap, dp, cl, al, dl);
    // separator rows: warp w < 7 takes the next chunk's first row from warp
    // w + 1 of the same tile; a tile's last chunk and its first chunk go to
    // the boundary arrays, assembled by large_tile_boundary_kernel
    float* ex = exch + (k & 1) * (kLtWarps * 32 * 3);
    float* mine = ex + (warp * 32 + lane) * 3;
    mine[0] = kr > 0 ? cs.fD : 0.f;
    mine[1] = kr > 0 ? cs.fC : 0.f;
    mine[2] = kr > 0 ? cs.fA : 0.f;
    consumer_sync(32 * kLtWarps);
    if (kr > 0) {
      const long tr = t / p.col_tiles;
      if (warp + 1 < kLtWarps) {
        const float* nx = ex + ((warp + 1) * 32 + lane) * 3;
        put_separator(p.red, p.PMp, j * p.m + sys, cs.sep, cs.lD, cs.lC, cs.lA, nx[0], nx[1], nx[2]);
      } else {
        float* b = p.bnd + tr * p.m + sys;
        b[(kBndLast + 0) * p.BS] = cs.lD; b[(kBndLast + 1) * p.BS] = cs.lC; b[(kBndLast + 2) * p.BS] = cs.lA;
        b[(kBndLast + 3) * p.BS] = cs.sep.a; b[(kBndLast + 4) * p.BS] = cs.sep.b;
        b[(kBndLast + 5) * p.BS] = cs.sep.c; b[(kBndLast + 6) * p.BS] = cs.sep.d;
      }
      if (warp == 0) {
        float* b = p.bnd + tr * p.m + sys;
        b[(kBndFirst + 0) * p.BS] = cs.fD; b[(kBndFirst + 1) * p.BS] = cs.fC; b[(kBndFirst + 2) * p.BS] = cs.fA;
      }
    }
  }
}

// The back pass: each lane's column again, between the separators above and
// below it, by a Thomas sweep.  MODE kBackPlain: x.  kBackFirst: x (FP32,
// exact) and the residual r = d - T x in double-float, rounded to FP32, with
// the sums of r^2 and d^2 per system: the first sweep of the refinement without
// reading the system again.  The chunk's elimination is at hand, so r goes
// through it at once, and the correction needs no reduce pass: its separator
// system has the same matrix, and the right-hand side is written here.
// kBackSecond: the solve was of a correction e1 (right-hand side r); x = e0 +
// e1 in FP64 and the sum of its residuals' squares, d and e0 read beside the
// tiles.  A tile's last row needs x of the next tile's first:
// large_tile_edge_kernel adds its share once the pass is done.
//
// Three groups of four warps an SM, each with tiles of its own (64 rows x 32
// systems), a private two-stage ring and its own barrier: a tile goes to
// registers, its stage is refilled at once, and the groups cover one another's
// dependent chains (plain 188 us at 1024 x 65536; eight warps in step on
// 128-row tiles 208 us).  kBackFirst 270 us and kBackSecond 337 us there (94% of
// the copy rate); 282 and 514 us before the full-chunk branch and running
// pointers, when kBackFirst left the correction's elimination to a reduce pass
// of 172 us; a back pass and a pass over the system each 330 and 560 us.  With
// two rows' residuals in paired FP32 instructions 319 and 530 us (the pairs'
// registers).  The norms' squares are summed in two scales (SquareSum): 1024 x
// 65536 refined 963 us with one, 971 us so.
constexpr int kBackGroups = 3, kBackWarps = 4;           // groups a CTA, warps a group
constexpr int kBackRows = kBackWarps * kLtChunk;         // 64
constexpr int kBackFloats = kBackRows * kTileCols;       // per array of a tile
constexpr int kBackThreads = 32 * kBackGroups * kBackWarps;
constexpr size_t kBackSmem = 128 + (size_t)kBackGroups * 2 * 4 * kBackFloats * sizeof(float);
// per group, all for two tiles: x of the warps' first rows (hi, lo), the norms' partial sums (r^2, d^2 in FP64) and fD
constexpr size_t kBackShare = 2 * kBackWarps * 32 * (1 + 2) + 2 * kBackWarps * 32 / 2;
constexpr size_t kBackResidual = kBackGroups * kBackShare * sizeof(float2);
static_assert(kBackSmem + kBackResidual <= 232448, "back pass: shared memory");

template <int MODE>
__global__ void __launch_bounds__(kBackThreads, 1)
    large_back_tile_kernel(LtParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                           const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  constexpr int L = kLtChunk;
  constexpr int GT = 32 * kBackWarps;  // threads a group
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, grp = threadIdx.x / GT, warp = (threadIdx.x % GT) >> 5;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem) + 2 * grp;
  float* ring = reinterpret_cast<float*>(smem + 128) + (size_t)grp * 2 * 4 * kBackFloats;
  float2* exch = reinterpret_cast<float2*>(smem + kBackSmem) + grp * kBackShare;
  double2* norms = reinterpret_cast<double2*>(exch + 2 * kBackWarps * 32);
  float* first_d = reinterpret_cast<float*>(norms + 2 * kBackWarps * 32);
  const int row_tiles = (int)((p.n + kBackRows - 1) / kBackRows);
  const int ntiles = row_tiles * p.col_tiles, step = (int)gridDim.x * kBackGroups;
  const int first = (int)blockIdx.x * kBackGroups + grp;
  const bool leader = threadIdx.x % GT == 0;
  // the t-th tile's first row and system: last tile first, so that what the
  // reduce pass read last comes out of L2 (10000 x 2016: 164 us without, 157 so;
  // 65536 x 1024, much larger than L2: 437 and 435)
  const auto place = [&](int t, int& x0, int& y0) {
    t = ntiles - 1 - t;
    x0 = (t % p.col_tiles) * kTileCols;
    y0 = (t / p.col_tiles) * kBackRows;
  };
  const auto issue = [&](int t, int s) {  // the group's leader
    int x0, y0;
    place(t, x0, y0);
    float* st = ring + (size_t)s * 4 * kBackFloats;
    mbar_arrive_expect_tx(&full[s], 4u * kBackFloats * sizeof(float));
    tma_load_2d(st + 0 * kBackFloats, &ma, x0, y0, &full[s]);
    tma_load_2d(st + 1 * kBackFloats, &mb, x0, y0, &full[s]);
    tma_load_2d(st + 2 * kBackFloats, &mc, x0, y0, &full[s]);
    tma_load_2d(st + 3 * kBackFloats, &md, x0, y0, &full[s]);
  };
  if (leader) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
    if (first < ntiles) issue(first, 0);
    if (first + step < ntiles) issue(first + step, 1);
  }
  __syncthreads();

  // The lane's column of tile t: system, first row; its separators are loaded
  // one tile ahead.
  const auto column = [&](int t, long& sys, long& r0) {
    int x0, y0;
    place(t, x0, y0);
    sys = x0 + lane;
    r0 = (long)y0 + warp * L;
  };
  const auto separators = [&](int t, float& above, float& below) {
    above = below = 0.f;
    if (t >= ntiles) return;
    long sys, r0;
    column(t, sys, r0);
    if (r0 >= p.n) return;
    const long o = (r0 / L) * p.m + sys;
    below = __ldg(p.sol + o);
    if (r0 > 0) above = __ldg(p.sol + o - p.m);
  };
  // sums of tile t's norms (the group's k-th) over its warps, by one of them
  const auto flush = [&](int t, int k) {
    if (warp != (k & (kBackWarps - 1))) return;
    double rs = 0.0, ds = 0.0;
    for (int w = 0; w < kBackWarps; ++w) {
      const double2 v = norms[((k & 1) * kBackWarps + w) * 32 + lane];
      rs += v.x;
      ds += v.y;
    }
    long sys, r0;
    column(t, sys, r0);
    atomicAdd(&p.rr[sys], rs);
    if (MODE == kBackFirst) atomicAdd(&p.dd[sys], ds);
  };
  // kBackFirst: tile t's right-hand sides of the separator system (the group's
  // k-th tile), once every warp's fD is there; a tile's last chunk waits for the
  // tile below (large_tile_edge_kernel)
  float sep_d = 0.f, sep_c = 0.f;
  const auto put_rhs = [&](int t, int k) {
    long sys, r0;
    column(t, sys, r0);
    if (r0 >= p.n || (warp == kBackWarps - 1 && r0 + L < p.n)) return;
    const float nD = warp + 1 < kBackWarps ? first_d[((k & 1) * kBackWarps + warp + 1) * 32 + lane] : 0.f;
    p.red_d[(r0 / L) * p.m + sys] = sep_d - sep_c * nD;
  };
  const long row_bytes = p.m * (long)sizeof(float);
  const auto down = [&](auto* q, long bytes) {  // q one row on
    return reinterpret_cast<decltype(q)>(reinterpret_cast<uintptr_t>(q) + bytes);
  };
  float sl_next, sj_next;
  separators(first, sl_next, sj_next);
  int k = 0;
  bool live = true;
  // One tile; FULL: all L rows of the warp's chunks exist (their bounds checks
  // are a tenth of the pass's instructions).
  const auto tile = [&](auto full_chunk, int t, long sys, long r0, int kr) {
    constexpr bool FULL = decltype(full_chunk)::value;
    const int s = k & 1;
    const float sl = sl_next, sj = sj_next;
    separators(t + step, sl_next, sj_next);
    const long g0 = r0 * p.m + sys;
    [[maybe_unused]] float dv[MODE == kBackSecond ? L : 1], e0[MODE == kBackSecond ? L : 1], e0m = 0.f;
    if constexpr (MODE == kBackSecond) {
      const float *gd = p.d + g0, *ge = p.e0 + g0;
#pragma unroll
      for (int q = 0; q < L; ++q) {
        const bool in = FULL || q < kr;
        dv[q] = in ? __ldg(gd) : 0.f;
        e0[q] = in ? __ldg(ge) : 0.f;
        gd = down(gd, row_bytes);
        ge = down(ge, row_bytes);
      }
      if (kr > 0 && r0 > 0) e0m = __ldg(p.e0 + g0 - p.m);
    }
    const bool ok = mbar_wait(&full[s], (k >> 1) & 1, p.status);
    const float* st = ring + (size_t)s * 4 * kBackFloats + warp * L * kTileCols + lane;
    float a[L], b[L], c[L], d[L];
#pragma unroll
    for (int q = 0; q < L; ++q) {
      a[q] = st[q * kTileCols];
      b[q] = st[kBackFloats + q * kTileCols];
      c[q] = st[2 * kBackFloats + q * kTileCols];
      d[q] = st[3 * kBackFloats + q * kTileCols];
    }
    fence_proxy_async_smem();
    live = named_sync_and(1 + grp, GT, ok);  // every column is read
    if (!live) return;
    if (leader && t + 2 * step < ntiles) issue(t + 2 * step, s);
    if (MODE != kBackPlain && k > 0) flush(t - step, k - 1);
    if (MODE == kBackFirst && k > 0) put_rhs(t - step, k - 1);
    if (r0 == 0) a[0] = 0.f;
    // inv[q] = 1 / pivot (kBackFirst needs it again), or c' = c inv
    float inv[L], x[L], cprev = 0.f, dprev = sl;
#pragma unroll
    for (int q = 0; q < L; ++q) {
      if (q < L - 1 && (FULL || q < kr - 1)) {
        inv[q] = tdiv(1.f, q == 0 ? b[q] : b[q] - a[q] * cprev);
        cprev = c[q] * inv[q];
        x[q] = dprev = (d[q] - a[q] * dprev) * inv[q];
        if (MODE != kBackFirst) inv[q] = cprev;
      }
    }
    const auto cp = [](float ci, float w) { return MODE == kBackFirst ? ci * w : w; };
    float xn = sj;
    if constexpr (MODE == kBackPlain) {
      float* gx = static_cast<float*>(p.x) + g0 + (L - 1) * p.m;
#pragma unroll
      for (int q = L - 1; q >= 0; --q) {
        if (q < L - 1 && (FULL || q <= kr - 2)) xn = x[q] - cp(c[q], inv[q]) * xn;
        if (FULL || q <= kr - 1) *gx = xn;
        gx = down(gx, -row_bytes);
      }
    } else {
#pragma unroll
      for (int q = L - 1; q >= 0; --q) {
        if (q < L - 1 && (FULL || q <= kr - 2)) xn = x[q] - cp(c[q], inv[q]) * xn;
        x[q] = FULL || q <= kr - 1 ? xn : 0.f;
      }
      // x as pairs: the row above, the lane's rows, the row below
      float lo[MODE == kBackSecond ? L : 1] = {};
      float2 xm = make_float2(sl, 0.f);
      if constexpr (MODE == kBackSecond) {
        xm.x = two_sum(e0m, sl, xm.y);
#pragma unroll
        for (int q = 0; q < L; ++q) x[q] = two_sum(e0[q], x[q], lo[q]);
      }
      const auto pair = [&](int q) { return make_float2(x[q], MODE == kBackSecond ? lo[MODE == kBackSecond ? q : 0] : 0.f); };
      float2* ex = exch + (k & 1) * kBackWarps * 32;
      ex[warp * 32 + lane] = pair(0);
      named_sync_and(1 + grp, GT, true);
      // x below the lane's last row: zero past the system's end (that row's c
      // counts as zero); past the tile it is not known here
      const bool open = warp == kBackWarps - 1 && r0 + L < p.n;
      const bool end = kr > 0 && r0 + kr == p.n;
      const float2 below = warp + 1 < kBackWarps && !end ? ex[(warp + 1) * 32 + lane] : make_float2(0.f, 0.f);
      SquareSums rd;  // of r and of d (kBackSecond: rs, of r)
      SquareSum rs;
      [[maybe_unused]] float lD = 0.f;
      float* gx = static_cast<float*>(p.x) + g0;
      double* gx64 = static_cast<double*>(p.x) + g0;
      float* gr = p.r + g0;
#pragma unroll
      for (int q = 0; q < L; ++q) {
        if (FULL || q < kr) {
          const float2 xi = pair(q);
          const bool lastrow = FULL ? q == L - 1 : q == kr - 1;
          if (MODE == kBackFirst) *gx = xi.x;
          else *gx64 = df_to_double(xi.x, xi.y);
          const float2 xp = lastrow ? below : pair(q + 1 < L ? q + 1 : q);
          const float di = MODE == kBackSecond ? dv[MODE == kBackSecond ? q : 0] : d[q];
          const float ci = lastrow && end ? 0.f : c[q];
          const float r = MODE == kBackSecond ? df_residual(a[q], b[q], ci, di, xm, xi, xp)
                                              : f_residual(a[q], b[q], ci, di, xm.x, xi.x, xp.x);
          if (!(lastrow && open)) {
            if (MODE == kBackFirst) *gr = r;
            if (MODE == kBackFirst) rd.add(make_float2(r, di));
            else rs.add(r);
          }
          xm = xi;
          if constexpr (MODE == kBackFirst) {  // r through the elimination, d' in x's place
            if (lastrow) {
              sep_d = r - a[q] * lD;
              sep_c = ci;
            } else {
              lD = (r - a[q] * lD) * inv[q];
              x[q] = lD;
            }
          }
        }
        gx = down(gx, row_bytes);
        gx64 = down(gx64, 2 * row_bytes);
        gr = down(gr, row_bytes);
      }
      if (MODE == kBackFirst) rs = rd.first();
      norms[((k & 1) * kBackWarps + warp) * 32 + lane] =
          make_double2(square_value(rs), MODE == kBackFirst ? square_value(rd.second()) : 0.0);
      if constexpr (MODE == kBackFirst) {
        float fD = 0.f;
#pragma unroll
        for (int q = L - 2; q >= 0; --q)
          if (FULL || q <= kr - 2) fD = x[q] - cp(c[q], inv[q]) * fD;
        first_d[((k & 1) * kBackWarps + warp) * 32 + lane] = fD;
        const long o = (r0 / kBackRows) * p.m + sys;
        if (open) p.bnd[o] = lD;
        if (warp == 0) p.bnd[p.BS + o] = fD;
      }
    }
  };
  for (int t = first; t < ntiles; t += step, ++k) {
    long sys, r0;
    column(t, sys, r0);
    const long rem = p.n - r0;
    if (rem >= L) tile(std::true_type{}, t, sys, r0, L);
    else tile(std::false_type{}, t, sys, r0, rem <= 0 ? 0 : (int)rem);
    if (!live) return;
  }
  if (MODE != kBackPlain && k > 0) {
    named_sync_and(1 + grp, GT, true);
    flush(first + (k - 1) * step, k - 1);
    if (MODE == kBackFirst) put_rhs(first + (k - 1) * step, k - 1);
  }
}

// v as hi + lo, hi its significand's upper 24 bits and lo the next 24, on the
// integer units (three FP64 instructions a value bound the kernel below), by
// one rule over FP32's normal range but its top (lo scaled in two steps: its
// scale alone would leave that range); values outside take those, out of line:
// inline, the compiler issued them for every value and the FP64 pipe was 72% busy).
__device__ __noinline__ float2 double_to_pair_slow(unsigned long long bits) {
  const double v = __longlong_as_double((long long)bits);
  const float hi = __double2float_rn(v);
  return make_float2(hi, __double2float_rn(v - (double)hi));
}
__device__ __forceinline__ float2 double_to_pair(unsigned long long u) {
  const int e = (int)((u >> 52) & 0x7ff) - 1023;  // v = +-1.f * 2^e
  if (e < -126 || e > 119) return double_to_pair_slow(u);
  const unsigned sign = (unsigned)(u >> 32) & 0x80000000u;
  const float hi = __uint_as_float(sign | ((unsigned)(e + 127) << 23) | ((unsigned)(u >> 29) & 0x7fffffu));
  const float part = __uint_as_float(sign | ((unsigned)(e + 127 + 8) << 23));  // 2^(e - 52 + 60)
  return make_float2(hi, (float)((unsigned)u & 0x1fffffffu) * 0x1p-60f * part);
}

// The rows that large_back_tile_kernel leaves open (the last of each tile but
// the system's last row): their residuals, shares of the norms and separator
// rows.  A warp
// takes 32 systems of one tile row, a block eight tile rows.
template <int MODE>
__global__ void __launch_bounds__(256) large_tile_edge_kernel(LtParams p, const float* __restrict__ a,
                                                              const float* __restrict__ b, const float* __restrict__ c,
                                                              const float* __restrict__ d) {
  __shared__ double2 part[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long sys = (long)(blockIdx.x % p.col_tiles) * kTileCols + lane;
  const long i = ((long)(blockIdx.x / p.col_tiles) * 8 + warp + 1) * kBackRows - 1;
  const auto x_at = [&](long o) {
    if constexpr (MODE == kBackFirst) return make_float2(static_cast<const float*>(p.x)[o], 0.f);
    return double_to_pair(static_cast<const unsigned long long*>(p.x)[o]);
  };
  double2 sums = make_double2(0.0, 0.0);
  if (i < p.n - 1) {
    const long o = i * p.m + sys;
    const float di = d[o];
    const float r = df_residual(a[o], b[o], c[o], di, x_at(o - p.m), x_at(o), x_at(o + p.m));
    if (MODE == kBackFirst) {  // and the chunk's separator row
      p.r[o] = r;
      const long t = (i / kBackRows) * p.m + sys;
      p.red_d[(i / kLtChunk) * p.m + sys] = r - a[o] * p.bnd[t] - c[o] * p.bnd[p.BS + t + p.m];
    }
    const double r64 = f2d_exact(r), d64 = f2d_exact(di);
    sums = make_double2(r64 * r64, d64 * d64);
  }
  part[warp][lane] = sums;
  __syncthreads();
  if (warp == 0) {
    double rs = 0.0, ds = 0.0;
    for (int w = 0; w < 8; ++w) {
      rs += part[w][lane].x;
      ds += part[w][lane].y;
    }
    atomicAdd(&p.rr[sys], rs);
    if (MODE == kBackFirst) atomicAdd(&p.dd[sys], ds);
  }
}

// Separator rows of the tiles' last chunks (chunk 8 tr + 7 of every tile row
// tr), whose next chunk opens the next tile row: one thread per (tr, system).
__global__ void __launch_bounds__(256) large_tile_boundary_kernel(LtParams p) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long)p.row_tiles * p.m) return;
  const long tr = gid / p.m, sys = gid - tr * p.m;
  const long j = tr * kLtWarps + kLtWarps - 1;
  if (j >= p.P) return;  // the system's last chunk lies in an earlier warp of this tile
  const float* b = p.bnd + gid;
  const Row<float> sep{b[(kBndLast + 3) * p.BS], b[(kBndLast + 4) * p.BS], b[(kBndLast + 5) * p.BS],
                       b[(kBndLast + 6) * p.BS]};
  float nD = 0.f, nC = 0.f, nA = 0.f;
  if (j + 1 < p.P) {
    const float* f = b + p.m;  // tile row tr + 1, the same system
    nD = f[(kBndFirst + 0) * p.BS]; nC = f[(kBndFirst + 1) * p.BS]; nA = f[(kBndFirst + 2) * p.BS];
  }
  put_separator(p.red, p.PMp, j * p.m + sys, sep, b[(kBndLast + 0) * p.BS], b[(kBndLast + 1) * p.BS],
                b[(kBndLast + 2) * p.BS], nD, nC, nA);
}

// Systems that a CTA holds whole (columns.cuh), staged by tensor copies, each
// warp's rows on a barrier of its own.
__global__ void __launch_bounds__(32 * kColWarps<float>, 1)
    large_columns_kernel(LtParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                         const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int F = kColArray<float>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = (int)blockIdx.x * kColSystems;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* base = reinterpret_cast<float*>(smem + kColHead);
  if (lane == 0) {
    float* st = base + (size_t)warp * 4 * F;
    mbar_init(bar, 1);
    mbar_fence_init();
    mbar_arrive_expect_tx(bar, 4u * F * sizeof(float));
    tma_load_2d(st + 0 * F, &ma, s0, warp * kColChunk, bar);
    tma_load_2d(st + 1 * F, &mb, s0, warp * kColChunk, bar);
    tma_load_2d(st + 2 * F, &mc, s0, warp * kColChunk, bar);
    tma_load_2d(st + 3 * F, &md, s0, warp * kColChunk, bar);
  }
  __syncwarp();
  const bool ok = mbar_wait(bar, 0, p.status);
  columns_solve<float>(base, (int)p.n, p.m, ok, true, static_cast<float*>(p.x) + s0 + lane);
}

bool make_map(CUtensorMap* map, const float* base, long n, long m, int rows) {
  return make_tensor_map_2d(map, base, (uint64_t)m, (uint64_t)n, (uint64_t)m * sizeof(float), kTileCols, rows, false);
}

}  // namespace

// Whether the TMA passes apply: interleaved FP32, m a multiple of 32, 16-byte
// aligned arrays, a chunk count that matches (P = ceil(n / 16)).
bool large_tma_ok(const float* a, const float* b, const float* c, const float* d, long n, long m) {
  return m % kTileCols == 0 && n >= 2 && aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) &&
         n < (1L << 31) && m < (1L << 31);
}

// Bytes of the boundary arrays of a reduce pass (within the 10 * PMp
// interface floats the register kernels use).
long round_up64(long v) { return (v + 63) & ~63L; }
long large_tma_boundary_stride(long n, long m) { return round_up64((n + kTileRows - 1) / kTileRows * m); }

// One TMA pass.  large_tma_reduce: the separator system (with the assembly of
// separator rows fused in; bnd: scratch of 10 boundary arrays).
// large_tma_back: the unknowns, and what f asks for beside them.
namespace {
tridi_status make_maps(CUtensorMap (&tm)[4], const float* a, const float* b, const float* c, const float* d, long n,
                       long m, int rows) {
  const float* src[4] = {a, b, c, d};
  for (int i = 0; i < 4; ++i)
    if (!make_map(&tm[i], src[i], n, m, rows)) return TRIDI_ERROR_INVALID_VALUE;
  return TRIDI_SUCCESS;
}
LtParams tile_params(long n, long m, const DeviceInfo* dev) {
  LtParams p{};
  p.n = n; p.m = m;
  p.BS = large_tma_boundary_stride(n, m);
  p.row_tiles = (int)((n + kTileRows - 1) / kTileRows);
  p.col_tiles = (int)(m / kTileCols);
  p.status = dev->status;
  return p;
}
using TileKernel = void (*)(LtParams, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap);
// `groups` tiles a CTA at a time, one CTA an SM.
cudaError_t launch_tiles(TileKernel kern, int threads, size_t smem, long tiles, int groups, const LtParams& p,
                         const CUtensorMap (&tm)[4], const DeviceInfo& dev, cudaStream_t st) {
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, threads, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  const long ctas = (tiles + groups - 1) / groups;
  return launch_kernel(kern, (unsigned)(dev.sm_count < ctas ? dev.sm_count : ctas), threads, smem, st, p, tm[0], tm[1],
                       tm[2], tm[3]);
}
}  // namespace

tridi_status large_tma_reduce(const float* a, const float* b, const float* c, const float* d, long n, long m, long P,
                              long PMp, float* red, float* bnd, cudaStream_t st) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  constexpr size_t smem = kLtSmem + kLtExchange;
  if ((size_t)dev->max_smem_optin < smem) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  CUtensorMap tm[4];
  const tridi_status ts = make_maps(tm, a, b, c, d, n, m, kTileRows);
  if (ts != TRIDI_SUCCESS) return ts;
  LtParams p = tile_params(n, m, dev);
  p.P = P; p.PMp = PMp; p.red = red; p.bnd = bnd;
  const cudaError_t e = launch_tiles(large_reduce_tile_kernel, 32 * (kLtWarps + 1), smem,
                                     (long)p.row_tiles * p.col_tiles, 1, p, tm, *dev, st);
  if (e != cudaSuccess) return cuda_status(e);
  const long cnt = (long)p.row_tiles * m;
  large_tile_boundary_kernel<<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(p);
  return cuda_status(cudaGetLastError());
}

tridi_status large_tma_back(const float* a, const float* b, const float* c, const float* d, long n, long m,
                            const float* sol, float* x, const LargeFused* f, float* red_d, float* bnd,
                            cudaStream_t st) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  const int mode = f ? f->mode : kBackPlain;
  const size_t smem = mode == kBackPlain ? kBackSmem : kBackSmem + kBackResidual;
  if ((size_t)dev->max_smem_optin < smem) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  CUtensorMap tm[4];
  const tridi_status ts = make_maps(tm, a, b, c, d, n, m, kBackRows);
  if (ts != TRIDI_SUCCESS) return ts;
  LtParams p = tile_params(n, m, dev);
  const int row_tiles = (int)((n + kBackRows - 1) / kBackRows);
  p.sol = sol;
  p.x = x;
  const auto run = [&](TileKernel kern) {
    return launch_tiles(kern, kBackThreads, smem, (long)row_tiles * p.col_tiles, kBackGroups, p, tm, *dev, st);
  };
  if (mode == kBackPlain) return cuda_status(run(large_back_tile_kernel<kBackPlain>));
  p.r = f->r; p.rr = f->rr; p.dd = f->dd; p.d = f->d; p.e0 = f->e0;
  p.red_d = red_d; p.bnd = bnd; p.BS = round_up64((long)row_tiles * m);
  if (mode == kBackSecond) p.x = f->x;
  const cudaError_t e = run(mode == kBackFirst ? large_back_tile_kernel<kBackFirst> : large_back_tile_kernel<kBackSecond>);
  if (e != cudaSuccess) return cuda_status(e);
  if (row_tiles > 1) {
    const unsigned grid = (unsigned)(p.col_tiles * ((row_tiles + 7) / 8));
    if (mode == kBackFirst) large_tile_edge_kernel<kBackFirst><<<grid, 256, 0, st>>>(p, a, b, c, d);
    else large_tile_edge_kernel<kBackSecond><<<grid, 256, 0, st>>>(p, a, b, c, f->d);
  }
  return cuda_status(cudaGetLastError());
}

tridi_status large_columns(const float* a, const float* b, const float* c, const float* d, long n, long m, float* x,
                           cudaStream_t st) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  const int warps = (int)((n + kColChunk - 1) / kColChunk);
  const size_t smem = columns_smem<float>(warps);
  if (n > kColRows<float> || (size_t)dev->max_smem_optin < smem) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  CUtensorMap tm[4];
  const tridi_status ts = make_maps(tm, a, b, c, d, n, m, kColChunk);
  if (ts != TRIDI_SUCCESS) return ts;
  LtParams p = tile_params(n, m, dev);
  p.x = x;
  int per_sm = 0;
  const cudaError_t e = resident_blocks(large_columns_kernel, 32 * warps, smem, *dev, &per_sm);
  if (e != cudaSuccess) return cuda_status(e);
  return cuda_status(launch_kernel(large_columns_kernel, (unsigned)p.col_tiles, 32 * warps, smem, st, p, tm[0], tm[1],
                                   tm[2], tm[3]));
}

}  // namespace tridi
