// Large systems (any n, contiguous or interleaved layout).  Contiguous
// systems that one CTA holds take the uniform solver (partition.cu), longer
// ones the block passes of large_rows.cu.  Interleaved systems (element i of
// system s at i*m + s): the partition method across the whole GPU, in three
// steps on one stream.
//
//   1. large_reduce: one thread per chunk of L rows of one system.  The chunk
//      is eliminated in registers (partition.cuh) and its interface -- first
//      and last interior row coefficients and the separator row, 10 values --
//      is written out.  A warp covers 32 consecutive systems at the same
//      rows, so every row load is one 128-byte line.
//   2. large_assemble: separator row j of system s from chunk j's interface
//      and chunk j+1's first interior row, in the layout of the data.  The
//      P = ceil(n/L) separators per system form a batch of the same kind,
//      solved by this scheme again, down to a one-thread-per-system Thomas
//      kernel for batches of <= 32 rows.
//   3. large_back: each chunk is read again and solved between the two
//      separators around it, a Thomas sweep (in FP64 3 FP64 instructions a row
//      where the elimination has 8).
// Steps 1 and 3 run in blocks of 128 threads (160 registers in FP64: three
// blocks an SM; one block of 256 there: 128 x 100001 FP64 568 us, 452 us now,
// 850 us before the Thomas sweep and the integer divisions).
// For the interleaved FP32 layout with m a multiple of 32, steps 1 and 3 run
// as TMA-tiled persistent kernels (large_tma.cu) on the same chunks.
// Memory traffic per unknown: inputs read twice (2 x 16 B FP32), x written
// once (4 B), plus ~20/L B of interface data.  No reference kernel
// corresponds; the reference's large-system path is pcrGauss's global-memory
// PCR steps (pcrGauss_kernel.cu:272-386).  Oracle: the gold Thomas solver.
#include "columns.cuh"
#include "large_tma.h"
#include "partition.cuh"
#include "runtime.h"

namespace tridi {

template <class T>
tridi_status partition_solve_device(const T* a, const T* b, const T* c, const T* d, T* x, int n, int m,
                                    tridi_stream_t stream);
template <class T>
tridi_status large_rows_solve(const T* a, const T* b, const T* c, const T* d, T* x, long n, long m, void* ws,
                              cudaStream_t st);
template <class T>
size_t large_rows_bytes(long n, long m);

struct LargeParams {
  const void* a;
  const void* b;
  const void* c;
  const void* d;
  void* x;
  long n, m;
  long P;       // chunks per system
  void* iface;  // 10 arrays of P*m interface values (stride PMp), same layout as the data
  void* red;    // 4 arrays (stride PMp): the separator system, same layout as the data
  long PMp;     // P*m rounded up to 64 elements: keeps each array 256-byte aligned
  void* sol;    // the separator solution (aliases iface), same layout
};

// Thread -> (system, chunk), systems fastest: consecutive threads touch
// consecutive addresses of the data and of the interface and separator
// arrays, whose index is j*m + s.
__device__ __forceinline__ void large_coords(const LargeParams& p, long gid, long* s, long* j) {
  *s = gid % p.m;
  *j = gid / p.m;
}
__device__ __forceinline__ long sep_index(const LargeParams& p, long s, long j) { return j * p.m + s; }

template <class T, int L>
__global__ void __launch_bounds__(128) large_reduce_kernel(LargeParams p) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= p.P * p.m) return;
  long s, j;
  large_coords(p, gid, &s, &j);
  const long r0 = j * L;
  const int k = (int)((p.n - r0) < L ? (p.n - r0) : L);
  const long rs = p.m;
  const long base = r0 * p.m + s;
  Chunk<T, L> ch;
  chunk_eliminate<T, L, true>(ch, k, j == 0, j == p.P - 1, static_cast<const T*>(p.a) + base,
                        static_cast<const T*>(p.b) + base, static_cast<const T*>(p.c) + base,
                        static_cast<const T*>(p.d) + base, rs);
  T* f = static_cast<T*>(p.iface);
  const long S = p.PMp, o = sep_index(p, s, j);
  f[0 * S + o] = ch.fD; f[1 * S + o] = ch.fC; f[2 * S + o] = ch.fA;
  f[3 * S + o] = ch.lD; f[4 * S + o] = ch.lC; f[5 * S + o] = ch.lA;
  f[6 * S + o] = ch.sep.a; f[7 * S + o] = ch.sep.b; f[8 * S + o] = ch.sep.c; f[9 * S + o] = ch.sep.d;
}

template <class T>
__global__ void __launch_bounds__(256) large_assemble_kernel(LargeParams p) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= p.P * p.m) return;
  long s, j;
  large_coords(p, gid, &s, &j);
  const T* f = static_cast<const T*>(p.iface);
  const long S = p.PMp, o = sep_index(p, s, j);
  T nD = T(0), nC = T(0), nA = T(0);
  if (j + 1 < p.P) {
    const long o1 = sep_index(p, s, j + 1);
    nD = f[0 * S + o1]; nC = f[1 * S + o1]; nA = f[2 * S + o1];
  }
  const T lD = f[3 * S + o], lC = f[4 * S + o], lA = f[5 * S + o];
  const T sa = f[6 * S + o], sb = f[7 * S + o], sc = f[8 * S + o], sd = f[9 * S + o];
  T* r = static_cast<T*>(p.red);
  r[0 * S + o] = -sa * lA;
  r[1 * S + o] = sb - sa * lC - sc * nA;
  r[2 * S + o] = -sc * nC;
  r[3 * S + o] = sd - sa * lD - sc * nD;
}

template <class T, int L>
__global__ void __launch_bounds__(128) large_back_kernel(LargeParams p) {
  // last rows first: what the reduce pass read last is still in L2 (FP32 12000 x
  // 1000 134 -> 129 us, FP64 20000 x 500 367 -> 360 us)
  const long gid = p.P * p.m - 1 - ((long)blockIdx.x * blockDim.x + threadIdx.x);
  if (gid < 0) return;
  long s, j;
  large_coords(p, gid, &s, &j);
  const long r0 = j * L;
  const int k = (int)((p.n - r0) < L ? (p.n - r0) : L);
  const long rs = p.m;
  const long base = r0 * p.m + s;
  const T* sol = static_cast<const T*>(p.sol);
  const T sj = sol[sep_index(p, s, j)];
  const T sl = j > 0 ? sol[sep_index(p, s, j - 1)] : T(0);
  T x[L];
  chunk_between<T, L, true>(k, j == 0, sl, sj, static_cast<const T*>(p.a) + base, static_cast<const T*>(p.b) + base,
                            static_cast<const T*>(p.c) + base, static_cast<const T*>(p.d) + base, rs, x);
  T* gx = static_cast<T*>(p.x) + base;
#pragma unroll
  for (int i = 0; i < L; ++i)
    if (i < k) gx[i * rs] = x[i];
}

// Base case for interleaved systems of at most kThomasMax rows: one thread per
// system runs the gold Thomas recurrence (tridiagonal_gold.h:26-44, a[0] and
// c[n-1] ignored) in registers; a warp reads 32 consecutive systems, so every
// row access is coalesced.  The loads of eight rows are issued together: with
// one row at a time the 16-row systems of a 65536-row solve took 12 us of
// memory latency.
constexpr long kThomasMax = 32;
template <class T>
__global__ void __launch_bounds__(32) thomas_interleaved_kernel(const T* __restrict__ a, const T* __restrict__ b,
                                                                const T* __restrict__ c, const T* __restrict__ d,
                                                                T* __restrict__ x, int n, long m) {
  constexpr int N = (int)kThomasMax, B = 8;
  const long s = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= m) return;
  T cp[N], dp[N], cprev = T(0), dprev = T(0);
#pragma unroll
  for (int i0 = 0; i0 < N; i0 += B) {
    if (i0 < n) {
      T ra[B], rb[B], rc[B], rd[B];
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const int i = i0 + q;
        const bool in = i < n;
        const long k = (long)i * m + s;
        ra[q] = in && i > 0 ? a[k] : T(0);
        rb[q] = in ? b[k] : T(1);
        rc[q] = in && i < n - 1 ? c[k] : T(0);
        rd[q] = in ? d[k] : T(0);
      }
#pragma unroll
      for (int q = 0; q < B; ++q) {
        tdiv2(rc[q], rd[q] - ra[q] * dprev, rb[q] - ra[q] * cprev, cprev, dprev);
        cp[i0 + q] = cprev;
        dp[i0 + q] = dprev;
      }
    }
  }
  // (rows past n are identity rows: x = 0, and row n - 1 has c = 0)
  T xn = T(0);
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    if (i < n) {
      xn = dp[i] - cp[i] * xn;
      x[(long)i * m + s] = xn;
    }
  }
}

// Systems that a CTA holds whole (columns.cuh), staged by plain loads: any
// number of them, FP32 or FP64.
template <class T>
__global__ void __launch_bounds__(32 * kColWarps<T>, 1)
    columns_plain_kernel(const T* __restrict__ a, const T* __restrict__ b, const T* __restrict__ c,
                         const T* __restrict__ d, T* __restrict__ x, int n, long m) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int F = kColArray<T>, B = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long s = (long)blockIdx.x * kColSystems + lane;
  const bool live = s < m;
  T* base = reinterpret_cast<T*>(smem + kColHead);
  T* st = base + (size_t)warp * 4 * F + lane;
#pragma unroll
  for (int i0 = 0; i0 < kColChunk; i0 += B) {
    T r[4][B];
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = warp * kColChunk + i0 + q;
      const bool in = live && i < n;
      const long o = (long)i * m + s;
      r[0][q] = in ? a[o] : T(0);
      r[1][q] = in ? b[o] : T(1);
      r[2][q] = in ? c[o] : T(0);
      r[3][q] = in ? d[o] : T(0);
    }
#pragma unroll
    for (int q = 0; q < B; ++q)
#pragma unroll
      for (int v = 0; v < 4; ++v) st[v * F + (i0 + q) * kColSystems] = r[v][q];
  }
  columns_solve<T>(base, n, m, true, live, x + s);
}

namespace {
constexpr int kChunk = 16;

template <class T>
tridi_status large_columns_plain(const T* a, const T* b, const T* c, const T* d, T* x, long n, long m,
                                 cudaStream_t st) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  const int warps = (int)((n + kColChunk - 1) / kColChunk);
  const size_t smem = columns_smem<T>(warps);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(columns_plain_kernel<T>, 32 * warps, smem, *dev, &per_sm);
  if (e != cudaSuccess) return cuda_status(e);
  return cuda_status(launch_kernel(columns_plain_kernel<T>, (unsigned)((m + kColSystems - 1) / kColSystems), 32 * warps,
                                   smem, st, a, b, c, d, x, (int)n, m));
}

long round64(long v) { return (v + 63) & ~63L; }

// Workspace of one level plus the levels below it (for the contiguous layout
// more than its block passes use).
template <class T>
size_t large_ws_bytes(long n, long m, int layout) {
  if (layout == 1 && n <= kThomasMax) return (size_t)2 * round64(n * m) * sizeof(T) + 256;
  const long P = (n + kChunk - 1) / kChunk;
  size_t own = (size_t)14 * round64(P * m) * sizeof(T) + 256;
  if (layout == 1 || P > partition_max_rows<T>()) own += large_ws_bytes<T>(P, m, layout);
  return own;
}
}  // namespace

template <class T>
size_t large_workspace_bytes(long n, long m, int layout) {
  return large_ws_bytes<T>(n, m, layout);
}
template size_t large_workspace_bytes<float>(long, long, int);
template size_t large_workspace_bytes<double>(long, long, int);

bool large_fusable(const float* a, const float* b, const float* c, const float* d, long n, long m) {
  return n > kThomasMax && tunable(TRIDI_TUNE_LARGE_TMA) != 2 && !g_host_mapped_io && large_tma_ok(a, b, c, d, n, m);
}

namespace {
template <class T>
tridi_status large_solve(const T* a, const T* b, const T* c, const T* d, T* x, long n, long m, int layout, void* ws,
                         size_t ws_bytes, const LargeFused* fused, tridi_stream_t stream) {
  if (!a || !b || !c || !d || !x || m <= 0 || n <= 0 || (layout != 0 && layout != 1))
    return TRIDI_ERROR_INVALID_VALUE;
  if (n * m > (1L << 34)) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  if (!ws || ws_bytes < large_ws_bytes<T>(n, m, layout)) return TRIDI_ERROR_WORKSPACE_TOO_SMALL;
  if (!current_device()) return TRIDI_ERROR_CUDA;
  cudaStream_t st = as_stream(stream);
  char* w = static_cast<char*>(ws);
  if (layout == 0) {
    if (n <= partition_max_rows<T>()) return partition_solve_device<T>(a, b, c, d, x, (int)n, (int)m, stream);
    if (ws_bytes < large_rows_bytes<T>(n, m)) return TRIDI_ERROR_WORKSPACE_TOO_SMALL;
    return large_rows_solve<T>(a, b, c, d, x, n, m, ws, st);
  }
  if (n <= kThomasMax) {
    thomas_interleaved_kernel<T><<<(unsigned)((m + 31) / 32), 32, 0, st>>>(a, b, c, d, x, (int)n, m);
    return cuda_status(cudaGetLastError());
  }
  // interleaved FP32 with m a multiple of 32: the TMA-tiled passes (large_tma.cu),
  // or one kernel where a CTA holds 32 systems whole
  bool tma = false;
  if constexpr (sizeof(T) == 4) tma = large_fusable(a, b, c, d, n, m);
  if (!fused && n <= kColRows<T>) {
    if constexpr (sizeof(T) == 4)
      if (tma) return large_columns(a, b, c, d, n, m, x, st);
    return large_columns_plain<T>(a, b, c, d, x, n, m, st);
  }
  LargeParams p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m;
  p.P = (n + kChunk - 1) / kChunk;
  const long PM = p.P * m;
  p.PMp = round64(PM);
  p.iface = w;
  p.red = w + (size_t)10 * p.PMp * sizeof(T);
  p.sol = w;  // the interface is dead once the separator rows are assembled
  void* inner = w + (size_t)14 * p.PMp * sizeof(T) + 256;
  const size_t inner_bytes = ws_bytes - ((size_t)14 * p.PMp * sizeof(T) + 256);
  const unsigned blocks = (unsigned)((PM + 255) / 256);
  if (fused && fused->mode == kBackSecond) {
    // the separator system is there: the first sweep's matrix, and its right-
    // hand side from that sweep's back pass
  } else if (tma) {
    // the separator rows assembled in the pass (the interface area holds the
    // tile-boundary arrays only)
    const tridi_status t = large_tma_reduce(
        reinterpret_cast<const float*>(a), reinterpret_cast<const float*>(b), reinterpret_cast<const float*>(c),
        reinterpret_cast<const float*>(d), n, m, p.P, p.PMp, static_cast<float*>(p.red), static_cast<float*>(p.iface), st);
    if (t != TRIDI_SUCCESS) return t;
  } else {
    large_reduce_kernel<T, kChunk><<<(unsigned)((PM + 127) / 128), 128, 0, st>>>(p);
    large_assemble_kernel<T><<<blocks, 256, 0, st>>>(p);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e);
  const T* r = static_cast<const T*>(p.red);
  const tridi_status ts = large_solve<T>(r, r + p.PMp, r + 2 * p.PMp, r + 3 * p.PMp, static_cast<T*>(p.sol), p.P, m,
                                         layout, inner, inner_bytes, nullptr, stream);
  if (ts != TRIDI_SUCCESS) return ts;
  if (tma)  // (a first sweep's boundary values: beside the separator solution, P m / 2 elements)
    return large_tma_back(reinterpret_cast<const float*>(a), reinterpret_cast<const float*>(b),
                          reinterpret_cast<const float*>(c), reinterpret_cast<const float*>(d), n, m,
                          static_cast<const float*>(p.sol), reinterpret_cast<float*>(x), fused,
                          static_cast<float*>(p.red) + 3 * p.PMp, static_cast<float*>(p.iface) + 2 * p.PMp, st);
  large_back_kernel<T, kChunk><<<(unsigned)((PM + 127) / 128), 128, 0, st>>>(p);
  return cuda_status(cudaGetLastError());
}

}  // namespace

template <class T>
tridi_status large_solve_device(const T* a, const T* b, const T* c, const T* d, T* x, long n, long m, int layout,
                                void* ws, size_t ws_bytes, tridi_stream_t stream) {
  return large_solve<T>(a, b, c, d, x, n, m, layout, ws, ws_bytes, nullptr, stream);
}
tridi_status large_solve_fused(const float* a, const float* b, const float* c, const float* rhs, float* x, long n,
                               long m, void* ws, size_t ws_bytes, const LargeFused& f, tridi_stream_t stream) {
  return large_solve<float>(a, b, c, rhs, x, n, m, TRIDI_LAYOUT_INTERLEAVED, ws, ws_bytes, &f, stream);
}

template tridi_status large_solve_device<float>(const float*, const float*, const float*, const float*, float*, long,
                                                long, int, void*, size_t, tridi_stream_t);
template tridi_status large_solve_device<double>(const double*, const double*, const double*, const double*,
                                                 double*, long, long, int, void*, size_t, tridi_stream_t);

}  // namespace tridi

extern "C" {

size_t tridi_large_workspace_bytes(long n, long num_systems, int elem_size) {
  // the larger of the two layouts' needs, so one query serves both
  const size_t c0 = elem_size == 8 ? tridi::large_ws_bytes<double>(n, num_systems, 0)
                                   : tridi::large_ws_bytes<float>(n, num_systems, 0);
  const size_t c1 = elem_size == 8 ? tridi::large_ws_bytes<double>(n, num_systems, 1)
                                   : tridi::large_ws_bytes<float>(n, num_systems, 1);
  return c0 > c1 ? c0 : c1;
}
tridi_status tridi_solve_large_f32(const float* a, const float* b, const float* c, const float* d, float* x, long n,
                                   long m, int layout, void* ws, size_t ws_bytes, tridi_stream_t s) {
  return tridi::large_solve_device<float>(a, b, c, d, x, n, m, layout, ws, ws_bytes, s);
}
tridi_status tridi_solve_large_f64(const double* a, const double* b, const double* c, const double* d, double* x,
                                   long n, long m, int layout, void* ws, size_t ws_bytes, tridi_stream_t s) {
  return tridi::large_solve_device<double>(a, b, c, d, x, n, m, layout, ws, ws_bytes, s);
}

}  // extern "C"
