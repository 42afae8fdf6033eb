// Large systems in the contiguous layout (element i of system s at s*n + i):
// two passes over blocks of 128 * K consecutive rows, staged and solved as in
// strip.cuh, around one small system of block rows.
//
//   1. rows_kernel<BACK = 0>: a CTA per block; what is left of it is its last
//      row (coupled to the last row of the block before and to the first row
//      of the block after) and the form of its first row: seven values.  Each
//      lane's and each warp's separator is kept as a function of its
//      neighbours, three values each.
//   2. The system of its ceil(n / 128 K) block rows: rows_sep_kernel, a warp per
//      system, or for long systems rows_assemble_kernel and the contiguous
//      solvers again (the any-size solver, beyond its range these passes).
//   3. rows_kernel<BACK = 1>: the separators from what pass 1 kept, then every
//      lane's chunk again, between two known rows: a plain Thomas sweep.
// The blocks of pass 3 run in reverse, so that the rows pass 1 read last are
// still in L2 (129 MB).  What bounds it is HBM in FP32 (two reads of the
// inputs, one write of x: 257 x 100001 156 us, 91 % of what those bytes take;
// one thread per 16 rows, each reading its chunk from global memory, took 494
// us) and the FP64 pipe in FP64 (15 FP64 instructions a row in pass 1, 3 in
// pass 3: 128 x 100001 539 us, 1139 us before).
#include "runtime.h"
#include "strip.cuh"

namespace tridi {

template <class T>
tridi_status partition_solve_device(const T* a, const T* b, const T* c, const T* d, T* x, int n, int m,
                                    tridi_stream_t stream);

namespace {

constexpr int kWarps = 4;

template <class T>
struct RowsParams {
  StripIn<T> in;
  T* x;
  long n, m;
  long NB;      // blocks per system
  T* form;      // 7 arrays of NB * m values (stride FS), system-major
  long FS;
  T* sep;       // x of each block's last row
  T* lanes;     // 3 arrays of 128 values a block (stride 128 FS): the lanes' separators
  T* warps;     // 3 arrays of 4 values a block (stride 4 FS): the warps' last separators
  int bulk, vec;
  unsigned* status;
};

template <class T, int K>
struct RowsShape {
  static constexpr long B = 32 * kWarps * K;
  static constexpr long CAP = strip_cap<T>(B);
  static constexpr size_t HEAD = (16 + block_scratch_words(kWarps) * sizeof(T) + 127) & ~(size_t)127;
  static constexpr size_t smem(bool back) { return HEAD + (back ? 5 : 4) * CAP * sizeof(T); }
};

template <class T, int K, bool BACK, int MINB>
__global__ void __launch_bounds__(32 * kWarps, MINB) rows_kernel(RowsParams<T> p) {
  using S = RowsShape<T, K>;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  T* scratch = reinterpret_cast<T*>(smem + 16);
  T* buf = reinterpret_cast<T*>(smem + S::HEAD);
  const long total = p.n * p.m, blocks = p.NB * p.m;
  const bool bulk = p.bulk != 0;
  // block i of this pass
  const auto block = [&](long i) { return BACK ? blocks - 1 - i : i; };
  const auto strip = [&](long b) {
    const long s = b / p.NB, r0 = (b - s * p.NB) * S::B;
    return Strip<T>(s * p.n + r0, s * p.n + (r0 + S::B < p.n ? r0 + S::B : p.n), total, bulk);
  };
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    if (bulk && blockIdx.x < blocks) strip_issue(strip(block(blockIdx.x)), p.in, buf, S::CAP, bar);
  }
  __syncthreads();
  int ph = 0;
  for (long i = blockIdx.x; i < blocks; i += gridDim.x, ph ^= 1) {
    const long b = block(i), J = b % p.NB;
    const Strip<T> s = strip(b);
    T sl = T(0), sj = T(0);  // back: the rows around the lane's interior ones
    if constexpr (BACK) {
      const T before = J > 0 ? p.sep[b - 1] : T(0), last = p.sep[b];
      const T* wr = p.warps + 4 * b;
      const long WS = 4 * p.FS, LS = 128 * p.FS;
      const T own = warp < kWarps - 1 ? wr[2 * WS + warp] - wr[warp] * before - wr[WS + warp] * last : last;
      const T wb = warp > 0 ? wr[2 * WS + warp - 1] - wr[warp - 1] * before - wr[WS + warp - 1] * last : before;
      const T* lr = p.lanes + 128 * b + tid;
      sj = lane < 31 ? lr[2 * LS] - lr[0] * wb - lr[LS] * own : own;
      const T up = __shfl_up_sync(kFull, sj, 1);
      sl = lane == 0 ? wb : up;
    }
    bool ok = true;
    if (bulk) ok = mbar_wait(bar, ph, p.status);
    if (s.hi < s.e1) strip_rest(s, p.in, buf, S::CAP, tid, 32 * kWarps);
    if (!__syncthreads_and(ok)) break;
    const int rows = (int)(s.e1 - s.e0);
    int k = rows - tid * K;
    k = k < 0 ? 0 : (k > K ? K : k);
    const int off = (int)(s.e0 - s.lo) + tid * K;
    const bool head = J == 0 && tid == 0;
    if constexpr (BACK) {
      T* xs = buf + 4 * S::CAP;
      T x[K];
      chunk_between<T, K>(k, head, sl, sj, buf + off, buf + S::CAP + off, buf + 2 * S::CAP + off,
                          buf + 3 * S::CAP + off, 1, x);
      fence_proxy_async_smem();
      __syncthreads();  // every row is read
      if (bulk && tid == 0 && i + gridDim.x < blocks) strip_issue(strip(block(i + gridDim.x)), p.in, buf, S::CAP, bar);
#pragma unroll
      for (int q = 0; q < K; ++q)
        if (q < k) xs[off + q] = x[q];
      __syncwarp();
      const long w0 = s.e0 + (long)warp * 32 * K, w1 = w0 + 32 * K < s.e1 ? w0 + 32 * K : s.e1;
      strip_store(xs, s.lo, p.x, w0, w1, p.vec != 0, lane);
      __syncwarp();
    } else {
      Chunk<T, K> ch;
      chunk_eliminate<T, K>(ch, k, head, J == p.NB - 1 && k > 0 && tid * K + k == rows, buf + off, buf + S::CAP + off,
                            buf + 2 * S::CAP + off, buf + 3 * S::CAP + off);
      fence_proxy_async_smem();
      const BlockForward<T> f = block_forward<T, K>(ch, kWarps, scratch);  // (its barrier: every row is read)
      if (bulk && tid == 0 && i + gridDim.x < blocks) strip_issue(strip(block(i + gridDim.x)), p.in, buf, S::CAP, bar);
      T* lr = p.lanes + 128 * b + tid;
      const long LS = 128 * p.FS;
      lr[0] = f.lane.a;
      lr[LS] = f.lane.c;
      lr[2 * LS] = f.lane.d;
      if (warp == 0 && lane < kWarps - 1) {
        T* wr = p.warps + 4 * b + lane;
        wr[0] = f.warp.a;
        wr[4 * p.FS] = f.warp.c;
        wr[8 * p.FS] = f.warp.d;
      }
      if (tid == 0) {
        p.form[b] = f.last.a;
        p.form[p.FS + b] = f.last.b;
        p.form[2 * p.FS + b] = f.last.c;
        p.form[3 * p.FS + b] = f.last.d;
        p.form[4 * p.FS + b] = f.first.a;
        p.form[5 * p.FS + b] = f.first.c;
        p.form[6 * p.FS + b] = f.first.d;
      }
    }
  }
}

// A block row's coupling to the next block's first row replaced by that row's
// form (f: the row's a; j < NB - 1).
template <class T>
__device__ __forceinline__ void join_blocks(T* f, long FS) {
  const T c = f[2 * FS];
  f[FS] -= c * f[4 * FS + 1];
  f[3 * FS] -= c * f[6 * FS + 1];
  f[2 * FS] = -c * f[5 * FS + 1];
}
template <class T>
__global__ void __launch_bounds__(256) rows_assemble_kernel(RowsParams<T> p) {
  const long i = (long)blockIdx.x * 256 + threadIdx.x;
  if (i < p.NB * p.m && i % p.NB < p.NB - 1) join_blocks(p.form + i, p.FS);
}

// The block rows of one system by one warp: joined, then the partition method
// with ceil(NB / 32) rows a lane, in place.
template <class T>
__global__ void __launch_bounds__(128) rows_sep_kernel(RowsParams<T> p) {
  const int lane = threadIdx.x & 31;
  const long s = (long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (s >= p.m) return;
  const long NB = p.NB, base = s * NB, FS = p.FS;
  T* fa = p.form + base;
  T* fb = fa + FS;
  T* fc = fa + 2 * FS;
  T* fd = fa + 3 * FS;
  for (long j = lane; j + 1 < NB; j += 32) join_blocks(fa + j, FS);
  __syncwarp();
  const long kk = (NB + 31) / 32, r0 = lane * kk;
  long k = NB - r0;
  k = k < 0 ? 0 : (k > kk ? kk : k);
  ChunkSummary<T> cs;
  chunk_eliminate_smem<T>(cs, (int)k, lane == 0, k > 0 && r0 + k == NB, fa + r0, fb + r0, fc + r0, fd + r0);
  const T nD = __shfl_down_sync(kFull, cs.fD, 1);
  const T nC = __shfl_down_sync(kFull, cs.fC, 1);
  const T nA = __shfl_down_sync(kFull, cs.fA, 1);
  const T sj = group_pcr(separator_row_s<T>(cs, nD, nC, nA), 32);
  const T up = __shfl_up_sync(kFull, sj, 1);
  T* out = p.sep + base + r0;
  const auto emit = [&](long q, T v) { out[q] = v; };
  chunk_back_smem<T>((int)k, sj, lane == 0 ? T(0) : up, fa + r0, fc + r0, fd + r0, emit);
}

template <class T, int K, bool BACK, int MINB>
cudaError_t launch_rows(const RowsParams<T>& p, const DeviceInfo& dev, cudaStream_t st) {
  using S = RowsShape<T, K>;
  auto kern = rows_kernel<T, K, BACK, MINB>;
  const size_t smem = S::smem(BACK);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, 32 * kWarps, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  long grid = (long)per_sm * dev.sm_count;
  if (grid > p.NB * p.m) grid = p.NB * p.m;
  return launch_kernel(kern, (unsigned)grid, 32 * kWarps, smem, st, p);
}

template <class T>
constexpr int kRows = sizeof(T) == 4 ? 17 : 13;  // rows a lane

}  // namespace

// Block rows a system up to which a warp solves them, a serial chain of NB / 32
// rows from global memory; the two launches of the other way cost 3 to 5 us.
// Level at 128 block rows (FP32, one system 23.5 us by the warp and 22.9, 64
// systems 118 and 115; FP64 42.9 and 40.5, 559 and 557), at 64 20.0 and 24.4, at
// 1024 69 and 28.  One FP32 system of 1e8 rows: 3330 us by the warp, 569 us.
constexpr long kWarpBlocks = 128;

// Stride of the form arrays: whole 16-byte groups, for the solvers that read them.
inline long rows_stride(long blocks) { return (blocks + 3) & ~3L; }

// Bytes of workspace: 8 + 3 * 128 + 3 * 4 values a block, at most a quarter of
// a value a row and one block more, and the same for the block rows where they
// take these passes; tridi_large_workspace_bytes() asks for 14 / 16 of a value a
// row.
template <class T>
size_t large_rows_bytes(long n, long m) {
  constexpr long B = RowsShape<T, kRows<T>>::B;
  const long NB = (n + B - 1) / B;
  return (size_t)(8 + 3 * 128 + 3 * 4) * rows_stride(NB * m) * sizeof(T) +
         (NB > partition_max_rows<T>() ? large_rows_bytes<T>(NB, m) : 0);
}

template <class T>
tridi_status large_rows_solve(const T* a, const T* b, const T* c, const T* d, T* x, long n, long m, void* ws,
                              cudaStream_t st) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  constexpr int K = kRows<T>;
  constexpr long B = RowsShape<T, K>::B;
  RowsParams<T> p{};
  p.in = StripIn<T>{a, b, c, d};
  p.x = x;
  p.n = n; p.m = m; p.status = dev->status;
  p.NB = (n + B - 1) / B;
  p.FS = rows_stride(p.NB * m);
  p.form = static_cast<T*>(ws);
  p.sep = p.form + 7 * p.FS;
  p.warps = p.sep + p.FS;
  p.lanes = p.warps + 3 * 4 * p.FS;
  p.bulk = aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && !g_host_mapped_io;
  p.vec = aligned16(x);
  constexpr int MR = sizeof(T) == 4 ? 5 : 3, MB = sizeof(T) == 4 ? 5 : 3;  // CTAs an SM
  cudaError_t e = launch_rows<T, K, false, MR>(p, *dev, st);
  if (e != cudaSuccess) return cuda_status(e);
  if (p.NB <= kWarpBlocks) {
    rows_sep_kernel<T><<<(unsigned)((m + 3) / 4), 128, 0, st>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
  } else {
    rows_assemble_kernel<T><<<(unsigned)((p.NB * m + 255) / 256), 256, 0, st>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_status(e);
    const T* f = p.form;
    const tridi_status ts =
        p.NB <= partition_max_rows<T>()
            ? partition_solve_device<T>(f, f + p.FS, f + 2 * p.FS, f + 3 * p.FS, p.sep, (int)p.NB, (int)m,
                                        reinterpret_cast<tridi_stream_t>(st))
            : large_rows_solve<T>(f, f + p.FS, f + 2 * p.FS, f + 3 * p.FS, p.sep, p.NB, m, p.lanes + 3 * 128 * p.FS, st);
    if (ts != TRIDI_SUCCESS) return ts;
  }
  return cuda_status(launch_rows<T, K, true, MB>(p, *dev, st));
}

template size_t large_rows_bytes<float>(long, long);
template size_t large_rows_bytes<double>(long, long);
template tridi_status large_rows_solve<float>(const float*, const float*, const float*, const float*, float*, long,
                                              long, void*, cudaStream_t);
template tridi_status large_rows_solve<double>(const double*, const double*, const double*, const double*, double*,
                                               long, long, void*, cudaStream_t);

}  // namespace tridi
