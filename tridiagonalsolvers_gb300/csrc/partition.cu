// Uniform-size batched solve of any n (partition.cuh, strip.cuh): tridi_solve_*.
// FP32: the partition method.  Up to 992 rows a system is solved by 4 to 32
// lanes of a warp (part_warp_kernel), above by a CTA (part_cta_kernel), up to
// 8704 rows.  FP64 runs the cyclic reduction of cr64.cu instead.
//
// Both kernels stream: while a tile is solved in registers, the bulk copies
// of the next one fill the staging buffer it came from; x leaves through a
// shared buffer of its own in whole 16-byte groups.  Tiles start at any
// element (strip.cuh), so an n that is no multiple of four is staged like the
// others.  What bounds them is HBM: 55-56 us at 65536 x 250, 32768 x 500 and
// 8192 x 2000 (86-88 % of the copy rate), 62 us at 4096 x 4000; 82 us at 2048 x
// 8000, where one CTA fills an SM's shared memory and its loads wait for its
// eliminations.  The kernels before these (a producer warp and PCR over a
// CTA's separators in shared memory, one system a warp, rows off the grid read
// by each lane from global memory): 72, 171, 168, 162 and 131 us; 500000 x 20
// 239 us (37 us here, four systems and more a warp).
#include "runtime.h"
#include "strip.cuh"

namespace tridi {

namespace {

struct PartParams {
  StripIn<float> in;
  float* x;
  int n, m;
  int lps;     // warp kernel: lanes per system (a power of two)
  int bulk;    // inputs staged by bulk copies
  int vec;     // x 16-byte aligned
  long cap;    // floats per array in a staging buffer
  long total;  // n * m
  unsigned* status;
};

// One warp per tile of 32 / lps systems, K rows a lane.
template <int K, int MINB>
__global__ void __launch_bounds__(128, MINB) part_warp_kernel(PartParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* buf = reinterpret_cast<float*>(smem + 128) + (size_t)warp * 5 * p.cap;
  float* xs = buf + 4 * p.cap;
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
    Chunk<float, K> ch;
    chunk_eliminate<float, K>(ch, k, t == 0, k > 0 && t * K + k == n, buf + off, buf + p.cap + off,
                              buf + 2 * p.cap + off, buf + 3 * p.cap + off);
    fence_proxy_async_smem();
    __syncwarp();
    if (bulk && lane == 0 && tile + step < tiles) strip_issue(strip(tile + step), p.in, buf, p.cap, bar);
    const float nD = __shfl_down_sync(kFull, ch.fD, 1, lps);
    const float nC = __shfl_down_sync(kFull, ch.fC, 1, lps);
    const float nA = __shfl_down_sync(kFull, ch.fA, 1, lps);
    const float sj = group_pcr(separator_row<float, K>(ch, nD, nC, nA), lps);
    const float up = __shfl_up_sync(kFull, sj, 1, lps);
    float x[K];
    chunk_back<float, K>(ch, k, sj, t == 0 ? 0.0f : up, x);
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < k) xs[off + i] = x[i];
    __syncwarp();
    strip_store(xs, s.lo, p.x, s.e0, s.e1, p.vec != 0, lane);
    __syncwarp();
  }
}

// One CTA of W warps per system, K rows a lane.
template <int K, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) part_cta_kernel(PartParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, W = blockDim.x >> 5, n = p.n;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  float* scratch = reinterpret_cast<float*>(smem + 16);
  float* buf = reinterpret_cast<float*>(smem + 512);
  float* xs = buf + 4 * p.cap;
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
  int ph = 0;
  for (long sys = blockIdx.x; sys < p.m; sys += gridDim.x, ph ^= 1) {
    const Strip<float> s = strip(sys);
    bool ok = true;
    if (bulk) ok = mbar_wait(bar, ph, p.status);
    if (s.hi < s.e1) strip_rest(s, p.in, buf, p.cap, tid, blockDim.x);
    if (!__syncthreads_and(ok)) break;
    const int off = (int)(s.e0 - s.lo) + tid * K;
    Chunk<float, K> ch;
    chunk_eliminate<float, K>(ch, k, tid == 0, k > 0 && tid * K + k == n, buf + off, buf + p.cap + off,
                              buf + 2 * p.cap + off, buf + 3 * p.cap + off);
    fence_proxy_async_smem();
    const BlockForward<float> f = block_forward<float, K>(ch, W, scratch);  // (its barrier: every row is read)
    if (bulk && tid == 0 && sys + gridDim.x < p.m) strip_issue(strip(sys + gridDim.x), p.in, buf, p.cap, bar);
    float x[K];
    block_back<float, K>(f, ch, k, W, 0.0f, tdiv(f.last.d, f.last.b), x);
#pragma unroll
    for (int i = 0; i < K; ++i)
      if (i < k) xs[off + i] = x[i];
    __syncwarp();
    const long w0 = s.e0 + (long)warp * 32 * K, w1 = w0 + 32 * K < s.e1 ? w0 + 32 * K : s.e1;
    strip_store(xs, s.lo, p.x, w0, w1, p.vec != 0, lane);
    __syncwarp();
  }
}

template <int K>
cudaError_t launch_warp(PartParams p, const DeviceInfo& dev, cudaStream_t stream) {
  constexpr int MINB = K <= 9 ? 5 : K <= 15 ? 4 : K <= 21 ? 3 : 2;
  auto kern = part_warp_kernel<K, MINB>;
  const int G = 32 / p.lps;
  p.cap = strip_cap<float>((long)G * p.n);
  const size_t smem = 128 + (size_t)4 * 5 * p.cap * sizeof(float);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, 128, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  const long tiles = ((long)p.m + G - 1) / G;
  long grid = (long)per_sm * dev.sm_count;
  if (grid * 4 > tiles) grid = (tiles + 3) / 4;
  return launch_kernel(kern, (unsigned)grid, 128, smem, stream, p);
}

template <int K, int MAXT>
cudaError_t launch_cta(PartParams p, int threads, const DeviceInfo& dev, cudaStream_t stream) {
  auto kern = part_cta_kernel<K, MAXT, 512 / MAXT>;  // 128 registers a thread
  p.cap = strip_cap<float>(p.n);
  const size_t smem = 512 + (size_t)5 * p.cap * sizeof(float);
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, threads, smem, dev, &per_sm);
  if (e != cudaSuccess) return e;
  long grid = (long)per_sm * dev.sm_count;
  if (grid > p.m) grid = p.m;
  return launch_kernel(kern, (unsigned)grid, threads, smem, stream, p);
}

tridi_status solve_f32(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                       cudaStream_t s) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  PartParams p{};
  p.in = StripIn<float>{a, b, c, d};
  p.x = x;
  p.n = n; p.m = m; p.total = (long)n * m; p.status = dev->status;
  p.bulk = aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) && !g_host_mapped_io;
  p.vec = aligned16(x);
  if (n <= 32 * 31) {
    int K = 31;
    strip_warp_shape(n, 31, 1100, &p.lps, &K);
    switch (K) {
      case 3: return cuda_status(launch_warp<3>(p, *dev, s));
      case 5: return cuda_status(launch_warp<5>(p, *dev, s));
      case 7: return cuda_status(launch_warp<7>(p, *dev, s));
      case 9: return cuda_status(launch_warp<9>(p, *dev, s));
      case 11: return cuda_status(launch_warp<11>(p, *dev, s));
      case 13: return cuda_status(launch_warp<13>(p, *dev, s));
      case 15: return cuda_status(launch_warp<15>(p, *dev, s));
      case 17: return cuda_status(launch_warp<17>(p, *dev, s));
      case 21: return cuda_status(launch_warp<21>(p, *dev, s));
      case 25: return cuda_status(launch_warp<25>(p, *dev, s));
      default: return cuda_status(launch_warp<31>(p, *dev, s));
    }
  }
  // the smallest of 4, 8 or 16 warps that hold the system at 17 rows a lane,
  // then as few rows a lane as that takes
  const int warps = n <= 128 * 17 ? 4 : n <= 256 * 17 ? 8 : 16;
  const int rows = (n + warps * 32 - 1) / (warps * 32);
  const auto by_rows = [&](auto maxt) {
    constexpr int MAXT = decltype(maxt)::value;
    if (rows <= 9) return launch_cta<9, MAXT>(p, warps * 32, *dev, s);
    if (rows <= 11) return launch_cta<11, MAXT>(p, warps * 32, *dev, s);
    if (rows <= 13) return launch_cta<13, MAXT>(p, warps * 32, *dev, s);
    if (rows <= 15) return launch_cta<15, MAXT>(p, warps * 32, *dev, s);
    return launch_cta<17, MAXT>(p, warps * 32, *dev, s);
  };
  return cuda_status(warps == 4   ? by_rows(std::integral_constant<int, 128>{})
                     : warps == 8 ? by_rows(std::integral_constant<int, 256>{})
                                  : by_rows(std::integral_constant<int, 512>{}));
}

}  // namespace

template <class T>
tridi_status partition_solve_device(const T* a, const T* b, const T* c, const T* d, T* x, int n, int m,
                                    tridi_stream_t stream) {
  if (!a || !b || !c || !d || !x || m <= 0) return TRIDI_ERROR_INVALID_VALUE;
  if (n < 1 || n > partition_max_rows<T>()) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  static_assert(partition_max_rows<float>() == 512L * 17, "partition size cap");
  if constexpr (sizeof(T) == 8) return cr64_solve_any(a, b, c, d, x, n, m, as_stream(stream));
  else return solve_f32(a, b, c, d, x, n, m, as_stream(stream));
}

template tridi_status partition_solve_device<float>(const float*, const float*, const float*, const float*, float*,
                                                    int, int, tridi_stream_t);
template tridi_status partition_solve_device<double>(const double*, const double*, const double*, const double*,
                                                     double*, int, int, tridi_stream_t);

}  // namespace tridi

extern "C" {

tridi_status tridi_solve_f32(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                             tridi_stream_t s) {
  return tridi::partition_solve_device<float>(a, b, c, d, x, n, m, s);
}
tridi_status tridi_solve_f64(const double* a, const double* b, const double* c, const double* d, double* x, int n,
                             int m, tridi_stream_t s) {
  return tridi::partition_solve_device<double>(a, b, c, d, x, n, m, s);
}

}  // extern "C"
