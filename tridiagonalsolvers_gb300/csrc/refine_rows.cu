// One-correction refinement of contiguous systems that a warp or a CTA holds
// (FP32 coefficients, FP64 solution, double-float residual): the whole of
//
//   x0 = solve32(T, d),  r0 = d - T x0,  e = solve32(T, r0),  x = x0 + e,
//   r1 = d - T x,  max over systems of ||r0||^2 / ||d||^2 and ||r1||^2 / ||d||^2
//
// in one kernel.  a, b, c, d are read once, from the staging of strip.cuh, and
// stay in shared memory for the two eliminations and the two residuals; x0, r0
// and x live in the lanes' registers; x leaves once in FP64.  24 B a row, where
// the separate solves and residual passes of refine.cu move 96 B, and a block
// of 256 threads formed the residual of each system, whatever its size.
// What bounds it: issue and dependency latency (about 200 instructions a row).
// 200000 x 64: 4798 -> 210 us; 16000 x 1000: 829 -> 270 us; 2000 x 8000: 590 ->
// 335 us (a call, with its two host round trips before and one now).
//
// Sums of squares are FP32, in two scales (SquareSum: d and r of any size);
// their quotient is formed on the integer units (div64.cuh), so the FP64 pipe
// takes no part.  The first residual's are added over the lanes before the
// second elimination, which needs the registers.  (One scale and double-float
// sums over the lanes: 16000 x 1000 283 us, 269 us so; 2000 x 8000 351 and 334;
// 20000 x 500, whose 17 rows a lane spill, 229 and 240.  Two scales and FP64 sums
// over the lanes: 299, 367 and 232 us.)
#include "dfloat.cuh"
#include "refine_rows.h"
#include "runtime.h"
#include "strip.cuh"

namespace tridi {

namespace {

struct RowsRefine {
  StripIn<float> in;
  double* x;
  int n, m;
  int lps;     // warp kernel: lanes per system
  int bulk;    // inputs staged by bulk copies
  int vec;     // x 16-byte aligned
  long cap;    // elements per array in a staging buffer
  long total;  // n * m
  unsigned long long* rel2;  // bits of the two maxima
  unsigned* status;
};

// The larger of `best` and the bits of ||r||^2 / ||d||^2 (a non-negative
// double: integer order; a NaN's bits lie above every number's).
__device__ __forceinline__ unsigned long long max_rel2(unsigned long long best, const SquareSum& rr, double dd) {
  const unsigned long long u = div64_bits(square_ratio(square_value(rr), dd)) & 0x7fffffffffffffffull;
  return u > best ? u : best;
}
// A warp's maxima into the kernel's, once at its end.
__device__ __forceinline__ void put_rel2(unsigned long long* out, unsigned long long best) {
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_down_sync(kFull, best, o);
    best = v > best ? v : best;
  }
  if ((threadIdx.x & 31) == 0 && best) atomicMax(out, best);
}

// The lane's chunk of rows in shared memory and its place in the system.
struct Rows {
  const float *a, *b, *c, *d;
  int k;        // rows
  bool first;   // holds the system's first row
  bool last;    // holds its last
};

// r_i = d_i - a x_{i-1} - b x_i - c x_{i+1} of the lane's rows for FP32 x, and
// the sums of r^2 and d^2.  above / below: x of the rows around the chunk.
template <int K>
__device__ __forceinline__ void first_residual(const Rows& w, const float (&x)[K], float above, float below,
                                               float (&r)[K], SquareSums& rd) {
#pragma unroll
  for (int i = 0; i < K; ++i) {
    r[i] = 0.f;
    if (i < w.k) {
      const bool end = i == w.k - 1;
      const float a = i == 0 && w.first ? 0.f : w.a[i], c = end && w.last ? 0.f : w.c[i];
      const float d = w.d[i];
      const float xp = end ? below : x[i + 1 < K ? i + 1 : i];
      r[i] = f_residual(a, w.b[i], c, d, i > 0 ? x[i > 0 ? i - 1 : 0] : above, x[i], xp);
      rd.add(make_float2(r[i], d));
    }
  }
}

// The same for x = hi + lo, the sum of r^2 only.
template <int K>
__device__ __forceinline__ SquareSum second_residual(const Rows& w, const float (&hi)[K], const float (&lo)[K],
                                                     float2 above, float2 below) {
  SquareSum rs;
  float2 xm = above;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    if (i < w.k) {
      const bool end = i == w.k - 1;
      const float a = i == 0 && w.first ? 0.f : w.a[i], c = end && w.last ? 0.f : w.c[i];
      const float2 xi = make_float2(hi[i], lo[i]);
      const float2 xp = end ? below : make_float2(hi[i + 1 < K ? i + 1 : i], lo[i + 1 < K ? i + 1 : i]);
      const float r = df_residual(a, w.b[i], c, w.d[i], xm, xi, xp);
      rs.add(r);
      xm = xi;
    }
  }
  return rs;
}

// x + e as pairs, into x (high words) and lo.
template <int K>
__device__ __forceinline__ void add_correction(float (&x)[K], const float (&e)[K], float (&lo)[K]) {
#pragma unroll
  for (int i = 0; i < K; ++i) x[i] = two_sum(x[i], e[i], lo[i]);
}

// One warp per tile of 32 / lps systems, K rows a lane.
template <int K, int MINB>
__global__ void __launch_bounds__(128, MINB) refine_warp_kernel(RowsRefine p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* buf = reinterpret_cast<float*>(smem + 128) + (size_t)warp * 6 * p.cap;
  double* xs = reinterpret_cast<double*>(buf + 4 * p.cap);
  const int lps = p.lps, G = 32 / lps, g = lane / lps, t = lane - g * lps, n = p.n;
  const long tiles = ((long)p.m + G - 1) / G;
  const long first = (long)blockIdx.x * 4 + warp, step = (long)gridDim.x * 4;
  const bool bulk = p.bulk != 0;
  const auto strip = [&](long tile) {
    const long s0 = tile * G, s1 = s0 + G < p.m ? s0 + G : p.m;
    return Strip<float>(s0 * n, s1 * n, p.total, bulk);
  };
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    if (bulk && first < tiles) strip_issue(strip(first), p.in, buf, p.cap, bar);
  }
  __syncwarp();
  unsigned long long best0 = 0, best1 = 0;
  int ph = 0;
  for (long tile = first; tile < tiles; tile += step, ph ^= 1) {
    const Strip<float> s = strip(tile);
    if (bulk && !mbar_wait(bar, ph, p.status)) break;
    if (s.hi < s.e1) strip_rest(s, p.in, buf, p.cap, lane, 32);
    __syncwarp();
    const bool in = tile * G + g < p.m;
    int k = n - t * K;
    k = !in || k < 0 ? 0 : (k > K ? K : k);
    const int off = (int)(s.e0 - s.lo) + g * n + t * K;
    const Rows w{buf + off, buf + p.cap + off, buf + 2 * p.cap + off, buf + 3 * p.cap + off, k, t == 0,
                 k > 0 && t * K + k == n};
    // a solve of the group's system: right-hand side from shared memory or r
    const auto solve = [&](auto eliminate, float (&x)[K], float& above) {
      Chunk<float, K> ch;
      eliminate(ch);
      const float nD = __shfl_down_sync(kFull, ch.fD, 1, lps);
      const float nC = __shfl_down_sync(kFull, ch.fC, 1, lps);
      const float nA = __shfl_down_sync(kFull, ch.fA, 1, lps);
      const float sj = group_pcr(separator_row<float, K>(ch, nD, nC, nA), lps);
      const float up = __shfl_up_sync(kFull, sj, 1, lps);
      above = t == 0 ? 0.f : up;
      chunk_back<float, K>(ch, k, sj, above, x);
    };
    float x[K], r[K], lo[K], above;
    SquareSums rd;
    solve([&](Chunk<float, K>& ch) { chunk_eliminate<float, K>(ch, k, w.first, w.last, w.a, w.b, w.c, w.d); }, x, above);
    const float below = __shfl_down_sync(kFull, x[0], 1, lps);
    first_residual<K>(w, x, above, w.last ? 0.f : below, r, rd);
    const double dd = square_value(square_total(rd.second(), lps));
    const SquareSum r0 = square_total(rd.first(), lps);
    if (t == 0 && in) best0 = max_rel2(best0, r0, dd);
    float e[K], unused;
    solve([&](Chunk<float, K>& ch) { chunk_eliminate_rhs<float, K>(ch, k, w.first, w.last, w.a, w.b, w.c, r); }, e, unused);
    add_correction<K>(x, e, lo);
    const float2 dn = make_float2(__shfl_down_sync(kFull, x[0], 1, lps), __shfl_down_sync(kFull, lo[0], 1, lps));
    const float2 up = make_float2(__shfl_up_sync(kFull, x[K - 1], 1, lps), __shfl_up_sync(kFull, lo[K - 1], 1, lps));
    const float2 zero = make_float2(0.f, 0.f);
    const SquareSum rs1 = second_residual<K>(w, x, lo, t == 0 ? zero : up, w.last ? zero : dn);
    fence_proxy_async_smem();
    __syncwarp();
    if (bulk && lane == 0 && tile + step < tiles) strip_issue(strip(tile + step), p.in, buf, p.cap, bar);
    const SquareSum r1 = square_total(rs1, lps);
    if (t == 0 && in) best1 = max_rel2(best1, r1, dd);
    // (x of the tile at the place its first element has in a 16-byte group)
    const long xlo = s.e0 & ~1L;
    const int xoff = (int)(s.e0 - xlo) + g * n + t * K;
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < k) xs[xoff + i] = df_to_double(x[i], lo[i]);
    __syncwarp();
    strip_store(xs, xlo, p.x, s.e0, s.e1, p.vec != 0, lane);
    __syncwarp();
  }
  put_rel2(p.rel2, best0);
  put_rel2(p.rel2 + 1, best1);
}

// One CTA of W warps per system, K rows a lane.
template <int K, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) refine_cta_kernel(RowsRefine p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = blockDim.x >> 5, n = p.n;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  float* scratch = reinterpret_cast<float*>(smem + 16);         // 7 W
  float2* edge = reinterpret_cast<float2*>(smem + 512);         // per warp: x of its first and of its last row
  SquareSum* sums = reinterpret_cast<SquareSum*>(edge + 2 * 16);  // per warp: r0, r1, d
  float* buf = reinterpret_cast<float*>(smem + 1280);
  double* xs = reinterpret_cast<double*>(buf + 4 * p.cap);
  const bool bulk = p.bulk != 0;
  const auto strip = [&](long sys) { return Strip<float>(sys * n, (sys + 1) * n, p.total, bulk); };
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    if (bulk && (int)blockIdx.x < p.m) strip_issue(strip(blockIdx.x), p.in, buf, p.cap, bar);
  }
  __syncthreads();
  int k = n - tid * K;
  k = k < 0 ? 0 : (k > K ? K : k);
  const bool last = k > 0 && tid * K + k == n;
  unsigned long long best0 = 0, best1 = 0;
  int ph = 0;
  for (long sys = blockIdx.x; sys < p.m; sys += gridDim.x, ph ^= 1) {
    const Strip<float> s = strip(sys);
    bool ok = true;
    if (bulk) ok = mbar_wait(bar, ph, p.status);
    if (s.hi < s.e1) strip_rest(s, p.in, buf, p.cap, tid, blockDim.x);
    if (!__syncthreads_and(ok)) break;
    const int off = (int)(s.e0 - s.lo) + tid * K;
    const Rows w{buf + off, buf + p.cap + off, buf + 2 * p.cap + off, buf + 3 * p.cap + off, k, tid == 0, last};
    // x of the rows around the lane's, across warps through shared memory
    const auto around = [&](float2 mine_first, float2 mine_last, float2& above, float2& below) {
      below = make_float2(__shfl_down_sync(kFull, mine_first.x, 1), __shfl_down_sync(kFull, mine_first.y, 1));
      above = make_float2(__shfl_up_sync(kFull, mine_last.x, 1), __shfl_up_sync(kFull, mine_last.y, 1));
      if (lane == 0) edge[2 * warp] = mine_first;
      if (lane == 31) edge[2 * warp + 1] = mine_last;
      __syncthreads();
      if (lane == 0) above = warp > 0 ? edge[2 * (warp > 0 ? warp - 1 : 0) + 1] : make_float2(0.f, 0.f);
      if (lane == 31) below = warp + 1 < W ? edge[2 * (warp + 1 < W ? warp + 1 : warp)] : make_float2(0.f, 0.f);
      if (last) below = make_float2(0.f, 0.f);
    };
    float x[K], r[K], lo[K], e[K];
    SquareSums rd;
    float2 above, below;
    {
      Chunk<float, K> ch;
      chunk_eliminate<float, K>(ch, k, w.first, last, w.a, w.b, w.c, w.d);
      const BlockForward<float> f = block_forward<float, K>(ch, W, scratch);
      block_back<float, K>(f, ch, k, W, 0.0f, tdiv(f.last.d, f.last.b), x);
    }
    around(make_float2(x[0], 0.f), make_float2(x[K - 1], 0.f), above, below);
    first_residual<K>(w, x, above.x, below.x, r, rd);
    {
      const SquareSum r0 = square_total(rd.first(), 32), dd = square_total(rd.second(), 32);
      if (lane == 0) {
        sums[3 * warp] = r0;
        sums[3 * warp + 2] = dd;
      }
    }
    {
      Chunk<float, K> ch;
      chunk_eliminate_rhs<float, K>(ch, k, w.first, last, w.a, w.b, w.c, r);
      const BlockForward<float> f = block_forward<float, K>(ch, W, scratch);
      block_back<float, K>(f, ch, k, W, 0.0f, tdiv(f.last.d, f.last.b), e);
    }
    add_correction<K>(x, e, lo);
    around(make_float2(x[0], lo[0]), make_float2(x[K - 1], lo[K - 1]), above, below);
    const SquareSum rs1 = second_residual<K>(w, x, lo, above, below);
    const SquareSum r1 = square_total(rs1, 32);
    if (lane == 0) sums[3 * warp + 1] = r1;
    fence_proxy_async_smem();
    __syncthreads();  // every row is read
    if (bulk && tid == 0 && sys + gridDim.x < p.m) strip_issue(strip(sys + gridDim.x), p.in, buf, p.cap, bar);
    if (warp == 1) {
      const auto total = [&](int q) { return square_total(lane < W ? sums[3 * lane + q] : SquareSum{}, 16); };
      const SquareSum r0 = total(0), r1 = total(1), dd = total(2);
      if (lane == 0) {
        const double d2 = square_value(dd);
        best0 = max_rel2(best0, r0, d2);
        best1 = max_rel2(best1, r1, d2);
      }
    }
    const long xlo = s.e0 & ~1L;
    const int xoff = (int)(s.e0 - xlo) + tid * K;
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < k) xs[xoff + i] = df_to_double(x[i], lo[i]);
    __syncwarp();
    const long w0 = s.e0 + (long)warp * 32 * K, w1 = w0 + 32 * K < s.e1 ? w0 + 32 * K : s.e1;
    strip_store(xs, xlo, p.x, w0, w1, p.vec != 0, lane);
    __syncwarp();
  }
  if (warp == 1) {
    put_rel2(p.rel2, best0);
    put_rel2(p.rel2 + 1, best1);
  }
}

template <int K>
cudaError_t launch_warp(RowsRefine p, const DeviceInfo& dev, cudaStream_t stream) {
  constexpr int MINB = K <= 5 ? 5 : K <= 9 ? 4 : 3;
  auto kern = refine_warp_kernel<K, MINB>;
  const int G = 32 / p.lps;
  p.cap = strip_cap<float>((long)G * p.n);
  const size_t smem = 128 + (size_t)4 * 6 * p.cap * sizeof(float);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, 128, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  const long tiles = ((long)p.m + G - 1) / G;
  long grid = (long)per_sm * dev.sm_count;
  if (grid * 4 > tiles) grid = (tiles + 3) / 4;
  return launch_kernel(kern, (unsigned)grid, 128, smem, stream, p);
}

template <int K, int MAXT>
cudaError_t launch_cta(RowsRefine p, const DeviceInfo& dev, cudaStream_t stream) {
  constexpr int REGS = K <= 9 ? 128 : 168;  // a thread
  auto kern = refine_cta_kernel<K, MAXT, (MAXT == 512 ? 1 : 65536 / (REGS * MAXT))>;
  p.cap = strip_cap<float>(p.n);
  const size_t smem = 1280 + (size_t)6 * p.cap * sizeof(float);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, MAXT, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  long grid = (long)per_sm * dev.sm_count;
  if (grid > p.m) grid = p.m;
  return launch_kernel(kern, (unsigned)grid, MAXT, smem, stream, p);
}

}  // namespace

bool refine_rows_applies(long n, long m) { return n <= partition_max_rows<float>() && n * m < (1L << 40) && m < (1L << 31); }

tridi_status refine_rows_device(const float* a, const float* b, const float* c, const float* d, double* x, int n, int m,
                                double* rel2, cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  cudaError_t ce = cudaMemsetAsync(rel2, 0, 2 * sizeof(double), stream);
  if (ce != cudaSuccess) return cuda_status(ce);
  RowsRefine p{};
  p.in = StripIn<float>{a, b, c, d};
  p.x = x;
  p.n = n; p.m = m; p.total = (long)n * m; p.status = dev->status;
  p.bulk = aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && !g_host_mapped_io;
  p.vec = aligned16(x);
  p.rel2 = reinterpret_cast<unsigned long long*>(rel2);
  if (n <= 32 * 17) {
    int K = 17;
    strip_warp_shape(n, 17, 600, &p.lps, &K);
    switch (K) {
      case 3: return cuda_status(launch_warp<3>(p, *dev, stream));
      case 5: return cuda_status(launch_warp<5>(p, *dev, stream));
      case 7: return cuda_status(launch_warp<7>(p, *dev, stream));
      case 9: return cuda_status(launch_warp<9>(p, *dev, stream));
      case 11: return cuda_status(launch_warp<11>(p, *dev, stream));
      case 13: return cuda_status(launch_warp<13>(p, *dev, stream));
      case 15: return cuda_status(launch_warp<15>(p, *dev, stream));
      default: return cuda_status(launch_warp<17>(p, *dev, stream));
    }
  }
  const int warps = n <= 128 * 17 ? 4 : n <= 256 * 17 ? 8 : 16;
  const int rows = (n + warps * 32 - 1) / (warps * 32);
  const auto by_rows = [&](auto maxt) {
    constexpr int MAXT = decltype(maxt)::value;
    if (MAXT == 128 && rows <= 5) return launch_cta<5, 128>(p, *dev, stream);
    if (MAXT == 128 && rows <= 7) return launch_cta<7, 128>(p, *dev, stream);
    if (rows <= 9) return launch_cta<9, MAXT>(p, *dev, stream);
    if (rows <= 11) return launch_cta<11, MAXT>(p, *dev, stream);
    if (rows <= 13) return launch_cta<13, MAXT>(p, *dev, stream);
    if (rows <= 15) return launch_cta<15, MAXT>(p, *dev, stream);
    return launch_cta<17, MAXT>(p, *dev, stream);
  };
  return cuda_status(warps == 4   ? by_rows(std::integral_constant<int, 128>{})
                     : warps == 8 ? by_rows(std::integral_constant<int, 256>{})
                                  : by_rows(std::integral_constant<int, 512>{}));
}

}  // namespace tridi
