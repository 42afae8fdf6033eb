// The cyclic-reduction family in FP64 (cr, pcr, crpcr, crNBC, crpcrNBC:
// the reference's algorithms, crpcr_kernel.cu:40-141) and the any-size solve
// in FP64 (cyclic reduction on n rows, whatever n): one kernel.
//
// What bounds it: the FP64 pipe.  The GB300 issues a DFMA of a warp in 16
// cycles of the SM's FP64 pipe, so the kernel is built to issue few of them:
//   * Divisions run on the integer units (div64.cuh).  Every row that
//     divides (an even row of a CR level, every row of a PCR step) is divided
//     by its diagonal once, (a/b, c/b, d/b), and serves both its neighbours
//     and its own back substitution: six FP64 instructions per eliminated
//     row, two per back-substituted one, eight per unknown of the whole CR.
//   * No lane computes a step that another lane repeats: the first log2(K)
//     CR levels run on a thread's K rows in registers, then each level
//     compacts its surviving rows into a dense shared array and only as many
//     threads as it has rows work on it.  (On shuffles, with all lanes
//     computing all levels and four rows a thread, the same CR issued 98 FP64
//     instructions an unknown: 2939 us at 16384 x 1024, 1456 us with the
//     divisions replaced.)
// Measured at 16384 x 1024: 370 us, 8.9 FP64 instructions an unknown, FP64
// pipe 64 % busy; the rest is the latency of the last levels, in which one
// warp of a CTA works.
// Rows are read from global memory as they are (K consecutive rows a thread:
// whole 64-byte segments): the kernel needs no staging, since four resident
// CTAs an SM cover the loads of one another, and so takes any alignment.
//
// Neighbouring systems of a CTA lie side by side in the shared arrays; a row
// at a system's end takes nothing from beyond it (its couplings are not read:
// an infinite or NaN neighbour system stays apart).
#include "runtime.h"
#include "tridi_device.cuh"

namespace tridi {

namespace {

struct Cr64Params {
  const double* a;
  const double* b;
  const double* c;
  const double* d;
  double* x;
  int n, m;
  int tps;     // threads per system, ceil(n / K) <= blockDim.x; G = blockDim.x / tps systems a tile
  int rest;    // rows of the PCR-solved intermediate system (2 = plain CR, n = PCR)
  int ntiles;  // ceil(m / G)
  int vec;     // all five pointers 16-byte aligned and n even
};

// A row divided by its diagonal.
struct N64 {
  double a, c, d;
};
__device__ __forceinline__ N64 normalize64(double a, double b, double c, double d) {
  N64 w;
  div64x3(a, c, d, b, w.a, w.c, w.d);
  return w;
}
// Elimination of a row's left / right neighbour (given normalised).
__device__ __forceinline__ void eliminate_left(Row<double>& r, const N64& L) {
  r.b = fma(-r.a, L.c, r.b);
  r.d = fma(-r.a, L.d, r.d);
  r.a = -r.a * L.a;
}
__device__ __forceinline__ void eliminate_right(Row<double>& r, const N64& R) {
  r.b = fma(-r.c, R.a, r.b);
  r.d = fma(-r.c, R.d, r.d);
  r.c = -r.c * R.c;
}

// The same, r.d's share added to t in place of r.d (t is subtracted from r.d when
// the row is next divided): one rounding of the size of d for several.
__device__ __forceinline__ void eliminate_left(Row<double>& r, const N64& L, double& t, bool first) {
  r.b = fma(-r.a, L.c, r.b);
  t = first ? r.a * L.d : fma(r.a, L.d, t);
  r.a = -r.a * L.a;
}
__device__ __forceinline__ void eliminate_right(Row<double>& r, const N64& R, double& t) {
  r.b = fma(-r.c, R.a, r.b);
  t = fma(r.c, R.d, t);
  r.c = -r.c * R.c;
}

template <int K>
__device__ __forceinline__ void load_rows(const double* p, long at, bool in, bool vec, double other, double (&v)[K]) {
  if (!in) {
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = other;
  } else if (K % 2 == 0 && vec) {
#pragma unroll
    for (int i = 0; i < K / 2; ++i) {
      const double2 q = __ldg(reinterpret_cast<const double2*>(p + at) + i);
      v[2 * i] = q.x;
      v[(2 * i + 1) % K] = q.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = __ldg(p + at + i);
  }
}

// Host memory in place, K = 8: a thread's 64 bytes cross the host link in four
// pieces (1024 x 4096 cr 1190 us a call, pinned arrays), so the tile's rows (all
// of them consecutive) move by consecutive threads and change hands in shared
// memory, a word of padding every 8: STAGED us; 762 us by the kernels before this
// one.  (Four rows a thread would do too, but round differently.)
__device__ __forceinline__ int host_at(int e) { return e + (e >> 3); }
template <int K>
__device__ __forceinline__ void load_rows_host(const double* p, long base, long total, double other, double* s,
                                               double (&v)[K]) {
  const int ct = blockDim.x, tid = threadIdx.x;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const long e = base + j * ct + tid;
    s[host_at(j * ct + tid)] = e < total ? __ldg(p + e) : other;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < K; ++i) v[i] = s[host_at(tid * K + i)];
  __syncthreads();
}

// Shared memory of a CTA of ct threads, in words a thread: the exported rows
// of the in-thread levels (3 words each, up to 3 levels; later the two PCR
// buffers of one row a thread), then the level arrays a, b, c, d of 2 words
// each (the level of `rows` rows at offset 2 * (ct - rows)) or the two
// buffers of a PCR on R rows a thread, then the thread's last unknown.
constexpr int kExportWords = 9;
__host__ __device__ constexpr int cr64_level_words(int pcr_rows) { return 6 * pcr_rows > 8 ? 6 * pcr_rows : 8; }
__host__ __device__ constexpr size_t cr64_smem(int ct, int pcr_rows) {
  return (size_t)(kExportWords + cr64_level_words(pcr_rows) + 1) * ct * sizeof(double);
}

// PCR steps and the closing 2x2 systems on `rows` rows per system, R of them
// (consecutive) in each of the first `work` threads; x into xs.  `sync` is
// the barrier of the threads that take part.
template <int R, class Sync>
__device__ __forceinline__ void pcr64(Row<double> (&y)[R], double (&xs)[R], int tid, int work, int rows, double* buf,
                                      const Sync& sync) {
  // row j of the flat batch of intermediate systems is kept at (j % R) * work
  // + j / R: at a fixed slot consecutive threads touch consecutive words
  const int words = R * work;
  const auto at = [work](int j) { return (j % R) * work + j / R; };
  double* cur = buf;
  double* nxt = buf + 3 * (size_t)words;
  const int j0 = tid * R, in0 = j0 & (rows - 1);  // rows is a power of two
  for (int dl = 1; 4 * dl <= rows; dl *= 2) {
    if (tid < work) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const N64 w = normalize64(y[q].a, y[q].b, y[q].c, y[q].d);
        cur[q * work + tid] = w.a;
        cur[words + q * work + tid] = w.c;
        cur[2 * words + q * work + tid] = w.d;
      }
    }
    sync();
    if (tid < work) {
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int j = (in0 + q) & (rows - 1);  // row within its system
        if (j >= dl) {
          const int o = at(j0 + q - dl);
          eliminate_left(y[q], N64{cur[o], cur[words + o], cur[2 * words + o]});
        }
        if (j + dl < rows) {
          const int o = at(j0 + q + dl);
          eliminate_right(y[q], N64{cur[o], cur[words + o], cur[2 * words + o]});
        }
      }
    }
    double* t = cur;  // the next step writes the other buffer: one barrier a step
    cur = nxt;
    nxt = t;
  }
  // 2x2 systems (j, j + rows/2): x = (d - k d') / (b - k k'), k this row's
  // coupling to the partner, d' and k' the partner's over its diagonal
  const int half = rows / 2;
  if (tid < work) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int j = (in0 + q) & (rows - 1);
      const N64 w = normalize64(y[q].a, y[q].b, y[q].c, y[q].d);
      cur[q * work + tid] = j < half ? w.c : w.a;
      cur[words + q * work + tid] = w.d;
    }
  }
  sync();
  if (tid < work) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int j = (in0 + q) & (rows - 1);
      const int o = at(j < half ? j0 + q + half : j0 + q - half);
      const double k = j < half ? y[q].c : y[q].a;
      xs[q] = tdiv(fma(-k, cur[words + o], y[q].d), fma(-k, cur[o], y[q].b));
    }
  }
}

// Shared arrays of the levels across threads (a, b, c, d; x takes the place
// of b) and the barrier of a step that `items` threads take part in: one
// warp's worth and less stays in the first warp.
struct Levels64 {
  double *A, *B, *C, *D;
};
__device__ __forceinline__ bool level_takes_part(int items) { return items >= 32 || threadIdx.x < 32; }
__device__ __forceinline__ void level_sync(int items) {
  if (items > 32) __syncthreads();
  else __syncwarp();
}

// Cyclic reduction of G systems of `per` rows each (any count), side by side
// in the level arrays, down to one row a system, and back: B[g * per + j]
// ends as x.  Level arrays of decreasing size follow one another; a level of
// `per` rows keeps its floor(per / 2) odd rows.  tid / pairs by the rounded
// reciprocal: exact for these ranges (tid < 1024).
__device__ __forceinline__ void cr_levels_any(const Levels64& v, int G, int per0) {
  const int tid = threadIdx.x;
  int per = per0, o = 0;
  while (per > 1) {
    const int pp = (per + 1) / 2, items = G * pp, on = o + G * per;
    if (level_takes_part(items)) {
      Row<double> me{};
      N64 L{};
      const int g = (int)(((float)tid + 0.5f) * __frcp_rn((float)pp)), p = tid - g * pp, e = o + g * per + 2 * p;
      const bool odd = 2 * p + 1 < per;
      if (tid < items) {
        L = normalize64(v.A[e], v.B[e], v.C[e], v.D[e]);
        if (odd) me = Row<double>{v.A[e + 1], v.B[e + 1], v.C[e + 1], v.D[e + 1]};
        v.A[e] = L.a; v.C[e] = L.c; v.D[e] = L.d;
      }
      level_sync(items);
      if (tid < items && odd) {
        eliminate_left(me, L);
        if (2 * p + 2 < per) eliminate_right(me, N64{v.A[e + 2], v.C[e + 2], v.D[e + 2]});
        const int w = on + g * (per / 2) + p;
        v.A[w] = me.a; v.B[w] = me.b; v.C[w] = me.c; v.D[w] = me.d;
      }
      level_sync(items);
    }
    o = on;
    per /= 2;
  }
  if (level_takes_part(G)) {
    if (tid < G) v.B[o + tid] = tdiv(v.D[o + tid], v.B[o + tid]);
    level_sync(G);
  }
  bool one_warp = G <= 32;
  int depth = 31 - __clz(per0);  // levels above the last: per = per0 >> l
  for (int l = depth - 1; l >= 0; --l) {
    per = per0 >> l;
    const int pp = (per + 1) / 2, items = G * pp, half = per / 2;
    const int on = o;
    o = on - G * per;
    if (items > 32 && one_warp) {  // the first warp's levels are done
      __syncthreads();
      one_warp = false;
    }
    if (level_takes_part(items)) {
      if (tid < items) {
        const int g = (int)(((float)tid + 0.5f) * __frcp_rn((float)pp)), p = tid - g * pp, e = o + g * per + 2 * p;
        const int w = on + g * half + p;
        const double xl = p > 0 ? v.B[w - 1] : 0.0;
        const double xo = 2 * p + 1 < per ? v.B[w] : 0.0;
        const double al = p > 0 ? v.A[e] : 0.0, cr = 2 * p + 1 < per ? v.C[e] : 0.0;
        v.B[e] = fma(-cr, xo, fma(-al, xl, v.D[e]));
        if (2 * p + 1 < per) v.B[e + 1] = xo;
      }
      level_sync(items);
    }
  }
}

// LS = 0: the intermediate system has at most one row a thread (n / rest >=
// K); LS > 0: LS = n / rest < K, K / LS rows a thread; LS = -1: any n, cyclic
// reduction throughout (rows past the system's end are identity rows).
// HOST: the arrays are host memory, moved in whole lines.
template <int K, int LS, int MAXT, int MINB, bool HOST>
__global__ void __launch_bounds__(MAXT, MINB) cr64_kernel(Cr64Params p) {
  constexpr bool ANY = LS < 0;
  static_assert(!HOST || (!ANY && K + 1 <= kExportWords), "cr64: host arrays");
  constexpr int SMAX = LS <= 0 ? K : LS;  // last in-thread CR level
  extern __shared__ __align__(16) double sm[];
  const int ct = blockDim.x, tid = threadIdx.x, tps = p.tps;
  double* ex = sm;  // [3 * level + word][thread]
  double* lv = sm + kExportWords * ct;
  double* xlast = lv + cr64_level_words(LS > 0 ? K / (LS > 0 ? LS : 1) : 1) * ct;
  const int g = tid / tps, t = tid - g * tps;
  const int G = ct / tps;

  for (int tile = blockIdx.x; tile < p.ntiles; tile += gridDim.x) {
    const long sys = (long)tile * G + g;
    const bool in = sys < p.m && (!ANY || g < G);
    const long at = sys * p.n + (long)t * K;
    Row<double> r[K];
    const bool whole = in && (!ANY || (t + 1) * K <= p.n);
    {
      const long base = (long)tile * G * p.n, total = (long)p.m * p.n;
      const auto load = [&](const double* src, double other, double (&v)[K]) {
        if constexpr (HOST) load_rows_host<K>(src, base, total, other, ex, v);
        else load_rows<K>(src, at, whole, p.vec, other, v);
      };
      double v[K];
      load(p.a, 0.0, v);
#pragma unroll
      for (int i = 0; i < K; ++i) r[i].a = v[i];
      load(p.b, 1.0, v);
#pragma unroll
      for (int i = 0; i < K; ++i) r[i].b = v[i];
      load(p.c, 0.0, v);
#pragma unroll
      for (int i = 0; i < K; ++i) r[i].c = v[i];
      load(p.d, 0.0, v);
#pragma unroll
      for (int i = 0; i < K; ++i) r[i].d = v[i];
    }
    if constexpr (ANY) {
      if (in && !whole) {  // the system's last thread
#pragma unroll
        for (int i = 0; i < K; ++i)
          if (t * K + i < p.n) r[i] = Row<double>{p.a[at + i], p.b[at + i], p.c[at + i], p.d[at + i]};
      }
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (t * K + i == p.n - 1) r[i].c = 0.0;
    }
    if (t == 0) r[0].a = 0.0;            // a[0] and c[n-1] are not part of the system
    if (!ANY && t == tps - 1) r[K - 1].c = 0.0;

    // 1. In-thread CR levels; the last row's right neighbours belong to the
    //    next thread and follow below.  Even rows end as (a/b, -, c/b, d/b).
    //    Any n: d's shares are summed apart (dt) and rounded to d once.  With the
    //    last level's even rows below, which add their neighbours' shares before
    //    they touch d, dominant systems of 256 to 4608 rows come out within
    //    1.155e-16 (root mean square, relative), 1.265e-16 without either and 1.18e-16
    //    to 1.30e-16 by the partition method that this kernel took the place of;
    //    4096 x 1000 106 us, 104.5 without.  (CR at 1024 rows, the last level's
    //    form alone: 1.257e-16, 1.269e-16 without; 16384 x 1024 370 and 368 us.)
    [[maybe_unused]] double dt[K];
#pragma unroll
    for (int h = 1; h < SMAX; h *= 2) {
#pragma unroll
      for (int i = h - 1; i < K; i += 2 * h) {
        if (ANY && h > 1) r[i].d -= dt[i];
        const N64 w = normalize64(r[i].a, r[i].b, r[i].c, r[i].d);
        r[i].a = w.a; r[i].c = w.c; r[i].d = w.d;
      }
#pragma unroll
      for (int i = 2 * h - 1; i < K; i += 2 * h) {
        const N64 L{r[i - h].a, r[i - h].c, r[i - h].d}, R{r[(i + h) % K].a, r[(i + h) % K].c, r[(i + h) % K].d};
        if constexpr (ANY) {
          eliminate_left(r[i], L, dt[i], h == 1);
          if (i + h < K) eliminate_right(r[i], R, dt[i]);
        } else {
          eliminate_left(r[i], L);
          if (i + h < K) eliminate_right(r[i], R);
        }
      }
    }
    if constexpr (SMAX > 1) {
#pragma unroll
      for (int h = 1, l = 0; h < SMAX; h *= 2, ++l) {
        ex[(3 * l) * ct + tid] = r[h - 1].a;
        ex[(3 * l + 1) * ct + tid] = r[h - 1].c;
        ex[(3 * l + 2) * ct + tid] = r[h - 1].d;
      }
      __syncthreads();
      if (t < tps - 1) {
#pragma unroll
        for (int h = 1, l = 0; h < SMAX; h *= 2, ++l) {
          const N64 R{ex[(3 * l) * ct + tid + 1], ex[(3 * l + 1) * ct + tid + 1], ex[(3 * l + 2) * ct + tid + 1]};
          if constexpr (ANY) eliminate_right(r[K - 1], R, dt[K - 1]);
          else eliminate_right(r[K - 1], R);
        }
      }
      if (ANY) r[K - 1].d -= dt[K - 1];
    }

    double xr[K];
    double xprev = 0.0;
    if constexpr (LS > 0) {
      // 2a. PCR on K / LS rows a thread
      constexpr int R = K / LS;
      Row<double> y[R];
      double xs[R];
#pragma unroll
      for (int q = 0; q < R; ++q) y[q] = r[LS * q + LS - 1];
      pcr64<R>(y, xs, tid, ct, p.rest, lv, [] { __syncthreads(); });
#pragma unroll
      for (int q = 0; q < R; ++q) xr[LS * q + LS - 1] = xs[q];
      if constexpr (LS > 1) {
        xlast[tid] = xr[K - 1];
        __syncthreads();
        if (t > 0) xprev = xlast[tid - 1];
      }
    } else if constexpr (ANY) {
      // 2b. One row a thread, tps of them a system: cyclic reduction to the end
      const Levels64 v{lv, lv + 2 * ct, lv + 4 * ct, lv + 6 * ct};
      const int w = g * tps + t;  // == tid for the threads of a system
      v.A[w] = r[K - 1].a; v.B[w] = r[K - 1].b; v.C[w] = r[K - 1].c; v.D[w] = r[K - 1].d;
      __syncthreads();
      cr_levels_any(v, G, tps);
      __syncthreads();
      xr[K - 1] = v.B[w];
      if (t > 0) xprev = v.B[w - 1];
    } else {
      // 2c. One row a thread: the CR levels across threads, compacted.  Level
      //     rows / 2 pairs; thread i takes rows 2i (even) and 2i + 1 (odd).
      double* A = lv;
      double* B = lv + 2 * ct;
      double* C = lv + 4 * ct;
      double* D = lv + 6 * ct;
      A[tid] = r[K - 1].a; B[tid] = r[K - 1].b; C[tid] = r[K - 1].c; D[tid] = r[K - 1].d;
      __syncthreads();
      int rows = ct, per = tps;  // rows of the level: in all, per system
      while (per > p.rest) {
        const int pairs = rows / 2, o = 2 * (ct - rows), on = o + rows;
        // one warp's worth of pairs and less stays in the first warp
        if (pairs >= 32 || tid < 32) {
          Row<double> me{};
          N64 L{};
          if (tid < pairs) {
            const int e = o + 2 * tid;
            const double2 va = *reinterpret_cast<const double2*>(A + e), vb = *reinterpret_cast<const double2*>(B + e),
                          vc = *reinterpret_cast<const double2*>(C + e), vd = *reinterpret_cast<const double2*>(D + e);
            L = normalize64(va.x, vb.x, vc.x, vd.x);
            me = Row<double>{va.y, vb.y, vc.y, vd.y};
            A[e] = L.a; C[e] = L.c; D[e] = L.d;
          }
          if (pairs > 32) __syncthreads(); else __syncwarp();
          if (tid < pairs) {
            eliminate_left(me, L);
            if (((tid + 1) & (per / 2 - 1)) != 0) {  // not the system's last row
              const int e = o + 2 * tid + 2;
              eliminate_right(me, N64{A[e], C[e], D[e]});
            }
            A[on + tid] = me.a; B[on + tid] = me.b; C[on + tid] = me.c; D[on + tid] = me.d;
          }
          if (pairs > 32) __syncthreads(); else __syncwarp();
        }
        rows = pairs;
        per /= 2;
      }
      // PCR and the closing 2x2 systems on `rows` rows, its buffers where
      // the exported rows were
      {
        const int o = 2 * (ct - rows);
        const bool one_warp = rows <= 32;
        if (!one_warp || tid < 32) {
          Row<double> y[1];
          double xs[1];
          if (tid < rows) y[0] = Row<double>{A[o + tid], B[o + tid], C[o + tid], D[o + tid]};
          if (one_warp) pcr64<1>(y, xs, tid, rows, per, ex, [] { __syncwarp(); });
          else pcr64<1>(y, xs, tid, rows, per, ex, [] { __syncthreads(); });
          if (tid < rows) B[o + tid] = xs[0];  // x takes the place of b
          if (one_warp) __syncwarp();
        }
        if (!one_warp) __syncthreads();
      }
      // back substitution: x of the level below (B of its rows) to the level
      // above; the first warp alone up to 32 pairs
      while (rows < ct) {
        const int pairs = rows, up = 2 * rows, o = 2 * (ct - up), on = o + up;
        const int perp = per;  // pairs per system
        if (pairs >= 32 || tid < 32) {
          if (pairs == 64) __syncthreads();  // (the first warp's levels are done)
          if (tid < pairs) {
            const int e = o + 2 * tid;
            const double xo = B[on + tid];
            const double xl = (tid & (perp - 1)) != 0 ? B[on + tid - 1] : 0.0;
            const double xe = fma(-C[e], xo, fma(-A[e], xl, D[e]));
            *reinterpret_cast<double2*>(B + e) = make_double2(xe, xo);
          }
          if (pairs > 32) __syncthreads(); else __syncwarp();
        }
        rows = up;
        per *= 2;
      }
      __syncthreads();
      xr[K - 1] = B[tid];
      if (t > 0) xprev = B[tid - 1];
    }

    // 3. In-thread back substitution (the last level's rows: one rounding of the
    //    size of x for two, see above)
#pragma unroll
    for (int h = SMAX / 2; h >= 1; h /= 2) {
#pragma unroll
      for (int i = h - 1; i < K; i += 2 * h) {
        const double xl = i >= h ? xr[(i - h + K) % K] : xprev;
        if (h == SMAX / 2) xr[i] = r[i].d - fma(r[i].a, xl, r[i].c * xr[(i + h) % K]);
        else xr[i] = fma(-r[i].c, xr[(i + h) % K], fma(-r[i].a, xl, r[i].d));
      }
    }
    if constexpr (HOST) {
#pragma unroll
      for (int i = 0; i < K; ++i) ex[host_at(tid * K + i)] = xr[i];
      __syncthreads();
      const long base = (long)tile * G * p.n, total = (long)p.m * p.n;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int e = j * ct + tid;
        if (base + e < total) p.x[base + e] = ex[host_at(e)];
      }
    } else if (ANY && in && !whole) {
#pragma unroll
      for (int i = 0; i < K; ++i)
        if (t * K + i < p.n) p.x[at + i] = xr[i];
    } else if (in) {
      if (K % 2 == 0 && p.vec) {
#pragma unroll
        for (int i = 0; i < K / 2; ++i)
          *(reinterpret_cast<double2*>(p.x + at) + i) = make_double2(xr[2 * i], xr[(2 * i + 1) % K]);
      } else {
#pragma unroll
        for (int i = 0; i < K; ++i) p.x[at + i] = xr[i];
      }
    }
    __syncthreads();  // the shared arrays belong to the next tile
  }
}

template <int K, int LS, int MAXT = 256>
cudaError_t launch_cr64(Cr64Params p, const DeviceInfo& dev, cudaStream_t stream) {
  constexpr int MINB = MAXT > 256 ? 1 : K == 4 ? 3 : 2;
  auto kern = cr64_kernel<K, LS, MAXT, MINB, false>;
  if constexpr (K == 8 && LS == 0) {
    if (g_host_mapped_io) kern = cr64_kernel<K, LS, MAXT, MINB, true>;
  }
  // 128 threads a CTA (a system of 2048 rows takes 256; 256 threads throughout
  // measured 410 us against 371 us at 16384 x 1024, 64 threads no gain), fewer
  // where that would leave SMs without one
  int ct = p.tps > 128 ? (p.tps + 31) / 32 * 32 : 128;
  while (ct > 32 && ct / 2 >= p.tps && (long)p.m * p.tps < 2L * dev.sm_count * ct) ct /= 2;
  const size_t smem = cr64_smem(ct, LS > 0 ? K / (LS > 0 ? LS : 1) : 1);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, ct, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  const int G = ct / p.tps;
  p.ntiles = (int)(((long)p.m + G - 1) / G);
  long grid = (long)per_sm * dev.sm_count;
  if (grid > p.ntiles) grid = p.ntiles;
  return launch_kernel(kern, (unsigned)grid, ct, smem, stream, p);
}

}  // namespace

// n a power of two, 2 <= n <= 2048; stride = n / rest.
tridi_status cr64_solve(const double* a, const double* b, const double* c, const double* d, double* x, int n, int m,
                        int stride, cudaStream_t stream) {
  if (!is_pow2(n) || n < 2 || n > 2048) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  // Rows a thread.  CR: 8 (three levels in registers, 128 registers, 16 warps
  // an SM): 16384 x 1024 371 us, 441 us with 4.  PCR on several rows a thread
  // (stride below 8): 4 rows, 24 warps: crpcr rest 256 of 4096 x 1024 152 and
  // 161 us.  PCR alone up to 512 unknowns: 2 rows (20000 x 512 1081 us, 1139 with
  // 4; one system of 128 11 and 21 us; 1024 unknowns would need 512 threads:
  // 2500 systems 427 us, 332 with 4).  2048 rows need 8 for 256 threads.
  const int K = n <= 8 ? n / 2 : stride == 1 && n <= 512 ? 2 : (stride >= 8 || n == 2048) ? 8 : 4;
  Cr64Params p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m; p.tps = n / K; p.rest = n / stride;
  p.vec = aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && aligned16(x);
  const int ls = stride < K ? stride : 0;
  cudaError_t e = cudaErrorInvalidValue;
  switch (K * 16 + ls) {
    case 1 * 16: e = launch_cr64<1, 0>(p, *dev, stream); break;
    case 2 * 16: e = launch_cr64<2, 0>(p, *dev, stream); break;
    case 2 * 16 + 1: e = launch_cr64<2, 1>(p, *dev, stream); break;
    case 4 * 16: e = launch_cr64<4, 0>(p, *dev, stream); break;
    case 4 * 16 + 1: e = launch_cr64<4, 1>(p, *dev, stream); break;
    case 4 * 16 + 2: e = launch_cr64<4, 2>(p, *dev, stream); break;
    case 8 * 16: e = launch_cr64<8, 0>(p, *dev, stream); break;
    case 8 * 16 + 1: e = launch_cr64<8, 1>(p, *dev, stream); break;
    case 8 * 16 + 2: e = launch_cr64<8, 2>(p, *dev, stream); break;
    case 8 * 16 + 4: e = launch_cr64<8, 4>(p, *dev, stream); break;
    default: break;
  }
  return cuda_status(e);
}

// Any n, 1 <= n <= 4608.  (The partition method that did this before, a chunk
// per lane and PCR on the 32 to 512 separators, issued 90 FP64 instructions a
// row at 1000 rows, 15 of them with the integer division: 4096 x 1000 684 and
// 257 us, cyclic reduction 106 us; 100000 x 20 1571 us, 48 us; 800 x 4608
// 394 us, 152 us.)
tridi_status cr64_solve_any(const double* a, const double* b, const double* c, const double* d, double* x, int n, int m,
                            cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  constexpr int K = 8;
  static_assert(576L * K == partition_max_rows<double>(), "any-size cap");
  if (n < 1 || n > 576 * K) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  Cr64Params p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m; p.tps = (n + K - 1) / K; p.rest = 1;
  p.vec = aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && aligned16(x) && n % 2 == 0;
  return cuda_status(p.tps <= 256   ? launch_cr64<K, -1>(p, *dev, stream)
                     : p.tps <= 512 ? launch_cr64<K, -1, 512>(p, *dev, stream)
                                    : launch_cr64<K, -1, 576>(p, *dev, stream));
}

}  // namespace tridi
