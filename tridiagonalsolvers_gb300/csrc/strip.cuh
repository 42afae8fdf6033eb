// Contiguous rows staged in shared memory, and the partition method on them:
// what the any-size solver (partition.cu) and the contiguous large systems
// (large_rows.cu) share.
//
// Staging.  A tile is a range of consecutive elements [e0, e1) of a, b, c, d.
// It arrives by cp.async.bulk from the 16-byte group that holds e0 on, so any
// n works, not only rows on the 16-byte grid; the elements of the arrays' own
// last group (where n * m is no multiple of four) are read with plain loads,
// and so is everything where an array is not 16-byte aligned.
//
// Block solve.  A CTA of W warps holds up to W * 32 * K consecutive rows of
// one system, K (odd: conflict-free shared reads) a lane.  Three levels of
// the partition method, one CTA barrier:
//   1. each lane eliminates its chunk (partition.cuh): separator = its last row;
//   2. the separators of lanes 0..30 by PCR on shuffles, their couplings to
//      the row before the warp and to lane 31's separator carried along;
//   3. lane 31's separators, one a warp, by PCR on 16 lanes, in every warp;
//      again with the couplings to the row before the block and to the
//      block's last row carried along.
// What is left is one row a block (couplings to the last rows of the blocks
// before and after) and the form of the block's first row.
#pragma once
#include "partition.cuh"

namespace tridi {

// One tile's staging geometry: elements [lo, hi) come by bulk copies (whole
// 16-byte groups within the arrays), [hi, e1) by plain loads; element e is at
// index e - lo of each array's buffer.
template <class T>
struct Strip {
  long e0, e1, lo, hi;
  __device__ __forceinline__ Strip(long first, long end, long total, bool bulk) : e0(first), e1(end) {
    constexpr long Q = 16 / sizeof(T);
    lo = first & ~(Q - 1);
    const long up = (end + Q - 1) & ~(Q - 1), whole = total & ~(Q - 1);
    hi = up < whole ? up : whole;
    if (hi < lo || !bulk) hi = lo;
  }
  __device__ __forceinline__ uint32_t bytes() const { return (uint32_t)((hi - lo) * (long)sizeof(T)); }
};

// Floats (doubles) a buffer needs for `rows` rows at any offset.
template <class T>
__host__ __device__ constexpr long strip_cap(long rows) {
  constexpr long Q = 16 / sizeof(T);
  return (rows + 2 * (Q - 1)) & ~(Q - 1);
}

template <class T>
struct StripIn {
  const T *a, *b, *c, *d;
};

// Issues a tile's bulk copies (one thread; nothing to copy still completes
// the barrier's phase).
template <class T>
__device__ __forceinline__ void strip_issue(const Strip<T>& s, const StripIn<T>& in, T* buf, long cap, uint64_t* bar) {
  const uint32_t bytes = s.bytes();
  mbar_arrive_expect_tx(bar, 4 * bytes);
  if (bytes == 0) return;
  bulk_g2s(buf, in.a + s.lo, bytes, bar);
  bulk_g2s(buf + cap, in.b + s.lo, bytes, bar);
  bulk_g2s(buf + 2 * cap, in.c + s.lo, bytes, bar);
  bulk_g2s(buf + 3 * cap, in.d + s.lo, bytes, bar);
}

// The elements that do not come by bulk copies, by `count` threads.
template <class T>
__device__ __forceinline__ void strip_rest(const Strip<T>& s, const StripIn<T>& in, T* buf, long cap, int tid, int count) {
  for (long e = (s.hi > s.e0 ? s.hi : s.e0) + tid; e < s.e1; e += count) {
    const long i = e - s.lo;
    buf[i] = in.a[e];
    buf[cap + i] = in.b[e];
    buf[2 * cap + i] = in.c[e];
    buf[3 * cap + i] = in.d[e];
  }
}

// Elements [f0, f1) of x from shared memory (xs[e - lo]) to global, by the 32
// lanes of a warp: whole 16-byte groups, the ragged ends element by element.
template <class T>
__device__ __forceinline__ void strip_store(const T* xs, long lo, T* gx, long f0, long f1, bool vec, int lane) {
  constexpr int Q = 16 / sizeof(T);
  if (vec) {
    const long v0 = f0 & ~(long)(Q - 1);
    for (long e = v0 + (long)Q * lane; e < f1; e += 32 * Q) {
      if (e >= f0 && e + Q <= f1) {
        *reinterpret_cast<float4*>(gx + e) = *reinterpret_cast<const float4*>(xs + (e - lo));
      } else {
#pragma unroll
        for (int i = 0; i < Q; ++i)
          if (e + i >= f0 && e + i < f1) gx[e + i] = xs[e + i - lo];
      }
    }
  } else {
    for (long e = f0 + lane; e < f1; e += 32) gx[e] = xs[e - lo];
  }
}

// PCR over the lanes of a group of `width` lanes whose end couplings are zero
// (a lane out of range gets its own row, which contributes exactly nothing).
template <class T>
__device__ __forceinline__ T group_pcr(Row<T> r, int width) {
  for (int dl = 1; dl < width; dl *= 2) {
    const NRow<T> w = normalize_row(r);
    const NRow<T> L = shfl_up(w, dl, width), R = shfl_down(w, dl, width);
    r = reduce_row_nrm(r, L, R);
  }
  return tdiv(r.d, r.b);
}

// PCR over lanes 0 .. count-1 of a warp (count <= 31) with the couplings of
// lane 0 to the row before it and of lane count-1 to the row after it kept:
// afterwards x = d - a (row before) - c (row after) in each of these lanes.
template <class T>
__device__ __forceinline__ NRow<T> open_pcr(Row<T> r, int lane, int count) {
  for (int dl = 1; dl < count; dl *= 2) {
    const NRow<T> w = normalize_row(r);
    const NRow<T> L = shfl_up(w, dl, 32), R = shfl_down(w, dl, 32);
    const bool inl = lane >= dl, inr = lane + dl < count;
    const T ka = inl ? r.a : T(0), kc = inr ? r.c : T(0);
    r.b = r.b - ka * (inl ? L.c : T(0)) - kc * (inr ? R.a : T(0));
    r.d = r.d - ka * (inl ? L.d : T(0)) - kc * (inr ? R.d : T(0));
    if (inl) r.a = -r.a * L.a;
    if (inr) r.c = -r.c * R.c;
  }
  return normalize_row(r);
}

// Words of CTA scratch block_forward needs for W warps.
__host__ __device__ constexpr int block_scratch_words(int W) { return 7 * W; }

template <class T>
struct BlockForward {
  NRow<T> lane;  // lanes 0..30: the lane's separator from (row before the warp, lane 31's separator)
  NRow<T> warp;  // lanes 0..W-2: warp `lane`'s last separator from (row before the block, the block's last row)
  Row<T> last;   // the block's last row: a = coupling to the row before the block, c = to the next block's first row
  NRow<T> first; // the block's first row: x = d - a (row before the block) - c (the block's last row)
};

// Levels 2 and 3 on the lanes' eliminated chunks.  One CTA barrier; the
// scratch may be written again after the caller's next one.  W <= 16.
template <class T, int K>
__device__ __forceinline__ BlockForward<T> block_forward(const Chunk<T, K>& ch, int W, T* scratch) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T nD = __shfl_down_sync(kFull, ch.fD, 1);
  const T nC = __shfl_down_sync(kFull, ch.fC, 1);
  const T nA = __shfl_down_sync(kFull, ch.fA, 1);
  BlockForward<T> o;
  // lanes 0..30: separators as usual; lane 31's right side belongs to the next warp
  o.lane = open_pcr(separator_row<T, K>(ch, nD, nC, nA), lane, 31);
  const T pa = __shfl_up_sync(kFull, o.lane.a, 1), pc = __shfl_up_sync(kFull, o.lane.c, 1),
          pd = __shfl_up_sync(kFull, o.lane.d, 1);
  if (lane == 0) {  // the warp's first row: x = fD - fC s - fA (row before), s = lane 0's separator
    scratch[w] = ch.fD - ch.fC * o.lane.d;             // constant
    scratch[W + w] = ch.fA - ch.fC * o.lane.a;         // times -(row before the warp)
    scratch[2 * W + w] = -ch.fC * o.lane.c;            // times -(lane 31's separator)
  }
  if (lane == 31) {  // its row with the chunk's last interior row, then lane 30's separator, put in
    const Row<T>& s = ch.sep;
    const T a = -s.a * ch.lA, b = s.b - s.a * ch.lC, d = s.d - s.a * ch.lD;
    scratch[3 * W + w] = -a * pa;
    scratch[4 * W + w] = b - a * pc;
    scratch[5 * W + w] = s.c;
    scratch[6 * W + w] = d - a * pd;
  }
  __syncthreads();
  const int v = lane < W ? lane : W - 1, nx = lane + 1 < W ? lane + 1 : W - 1;
  Row<T> r{scratch[3 * W + v], scratch[4 * W + v], scratch[5 * W + v], scratch[6 * W + v]};
  const T c0 = r.c, fd = scratch[nx], fa = scratch[W + nx], fc = scratch[2 * W + nx];
  if (lane < W - 1) {
    r.b -= c0 * fa;
    r.d -= c0 * fd;
    r.c = -c0 * fc;
  }
  o.warp = open_pcr(r, lane, W - 1);
  const T qa = __shfl_sync(kFull, o.warp.a, W - 2), qc = __shfl_sync(kFull, o.warp.c, W - 2),
          qd = __shfl_sync(kFull, o.warp.d, W - 2);
  const T la = __shfl_sync(kFull, r.a, W - 1);
  o.last = Row<T>{-la * qa, __shfl_sync(kFull, r.b, W - 1) - la * qc, __shfl_sync(kFull, r.c, W - 1),
                  __shfl_sync(kFull, r.d, W - 1) - la * qd};
  const T za = __shfl_sync(kFull, o.warp.a, 0), zc = __shfl_sync(kFull, o.warp.c, 0),
          zd = __shfl_sync(kFull, o.warp.d, 0);
  const T f0 = scratch[0], f1 = scratch[W], f2 = scratch[2 * W];
  o.first = NRow<T>{f1 - f2 * za, -f2 * zc, f0 - f2 * zd};
  return o;
}

// The unknowns of the lane's chunk, given those of the row before the block
// and of the block's last row.
template <class T, int K>
__device__ __forceinline__ void block_back(const BlockForward<T>& o, const Chunk<T, K>& ch, int k, int W, T before,
                                           T last, T (&x)[K]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T s = lane < W - 1 ? o.warp.d - o.warp.a * before - o.warp.c * last : last;  // warp `lane`'s last separator
  const T own = __shfl_sync(kFull, s, w);
  const T prev = __shfl_sync(kFull, s, w > 0 ? w - 1 : 0);
  const T wb = w > 0 ? prev : before;
  const T sj = lane < 31 ? o.lane.d - o.lane.a * wb - o.lane.c * own : own;
  const T up = __shfl_up_sync(kFull, sj, 1);
  chunk_back<T, K>(ch, k, sj, lane == 0 ? wb : up, x);
}

// Lanes per system and rows a lane of a warp kernel for a system of n rows:
// the cheapest of the shapes that hold it, by the shared-memory wavefronts and
// instructions of a row slot and of a group's separator solve (their sums
// order the shapes as timed at 20, 61, 100, 250 and 333 rows); lanes of
// different systems n words apart may share banks, which counts.
// max_rows: rows a lane at most; max_tile: rows a warp's tile at most.
inline void strip_warp_shape(int n, int max_rows, long max_tile, int* lps, int* rows) {
  constexpr int kWarpRows[] = {3, 5, 7, 9, 11, 13, 15, 17, 21, 25, 31};
  double best = 1e30;
  for (int l = 1, steps = 0; l <= 32; l *= 2, ++steps) {
    for (int K : kWarpRows) {
      if (K > max_rows || l * K < n || (long)(32 / l) * n > max_tile) continue;
      int hits[32] = {};
      int conflict = 0;
      for (int lane = 0; lane < 32; ++lane) {
        const int g = lane / l, t = lane % l;
        if (t * K >= n) continue;
        const int h = ++hits[(g * n + t * K) % 32];
        conflict = h > conflict ? h : conflict;
      }
      const double slot = 24.0 + 5.0 * (conflict - 1);
      const double cost = ((double)K * slot + 60.0 + 25.0 * steps) / ((double)(32 / l) * n);
      if (cost < best) {
        best = cost;
        *lps = l;
        *rows = K;
      }
    }
  }
}

}  // namespace tridi
