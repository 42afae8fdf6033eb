// CR and CR-PCR for FP32 systems of 2048 and 4096 unknowns in registers: the
// scheme of crpcr2.cu across the warps of a CTA.  The switch level is the
// caller's up to rest = n / 32, where a lane still holds one row; a larger
// rest would leave the PCR on rows spread over the CTA, so it switches there
// too (the extra CR levels leave the same solution, and round less than the
// PCR steps they stand in for: 0.73e-7 against 0.83e-7 at rest n / 2).
//
// One CTA of M = n / 1024 warps per system, warp w rows 1024 w .. 1024 w +
// 1023, 32 contiguous rows a lane (TMA tiles, one staging buffer a warp,
// refilled while the warp solves).  The first five CR levels run inside the
// lane for every row but its last, whose right neighbours are the next lane's
// rows 2^j - 1, final once that lane's levels are done: over shuffles, and for
// lane 31 from the rows the next warp's lane 0 left in shared memory.  Then a
// lane holds one row; the 32 M rows of the system go to the CTA's first warp,
// M consecutive rows a lane, which runs the remaining CR levels, the PCR and
// their back substitution (crpcr2.cuh), and hands x back.  The in-lane back
// substitution follows, and the lane's 32 unknowns leave in 16-byte stores.
// Every CR level keeps CR's own divisions and operand order, so that rest 2
// (cr) is bit for bit the result of the other CR kernels.  (On normalised even
// rows, as crpcr2.cu's levels above rest 2, it took 60 us where this takes
// 57 and 58 us, and its error was 1 to 5 % larger.)
//
// What bounds it: HBM, and the three barriers of a system around the first
// warp's solve, which the SM's other CTAs cover.  16.8 M unknowns: cr 57 us at
// 2048 and 58 us at 4096 (86 and 84 % of the copy rate; the hybrid kernel, CR
// levels between warps through shared memory, 80 and 151 us), crpcr the same at
// every rest (79 to 161 and 147 to 327 us; above n / 32 the hybrid kernel's times
// are with PCR steps that are CR levels here).
#include "crpcr2.cuh"
#include "hybrid.cuh"
#include "runtime.h"

namespace tridi {

namespace {

using namespace pcr2;

constexpr int kR = 32;     // rows a lane
constexpr int kTF = 1024;  // values of one array in a warp's tile

template <int M>
struct CrWideShape {
  static constexpr int N = M * 1024;
  static constexpr int ROWS = 32 * M;                    // rows left after the in-lane levels
  static constexpr int EXPORT = M * 5 * 4;               // lane 0's even rows of the five levels, per warp
  static constexpr int WORDS = EXPORT + 4 * ROWS + ROWS; // then the rows left (a, b, c, d) and their x
  static constexpr size_t HEAD = (128 + WORDS * sizeof(float) + 127) & ~(size_t)127;
  static constexpr size_t SMEM = HEAD + 1024 + (size_t)M * 4 * kTF * sizeof(float);
};

// The CR levels h = 1, 2, 4, 8, 16 of a lane's rows but its last.  Even rows
// end with the reciprocal of their diagonal in b.
__device__ __forceinline__ void lane_levels(float (&a)[kR], float (&b)[kR], float (&c)[kR], float (&d)[kR]) {
#pragma unroll
  for (int h = 1; h < kR; h *= 2) {
#pragma unroll
    for (int i = h - 1; i < kR; i += 2 * h) b[i] = rcp_approx(b[i]);
#pragma unroll
    for (int i = 2 * h - 1; i + h < kR; i += 2 * h) {
      const int l = i - h, r = i + h;
      const float k1 = a[i] * b[l], k2 = c[i] * b[r];
      b[i] = b[i] - c[l] * k1 - a[r] * k2;
      d[i] = d[i] - d[l] * k1 - d[r] * k2;
      a[i] = -a[l] * k1;
      c[i] = -c[r] * k2;
    }
  }
}

// One level of the lane's last row: left neighbour row l, right neighbour (ra,
// rb, rc, rd), both as lane_levels leaves them.
__device__ __forceinline__ void last_row_level(float (&a)[kR], float (&b)[kR], float (&c)[kR], float (&d)[kR], int l,
                                               float ra, float rb, float rc, float rd) {
  constexpr int i = kR - 1;
  const float k1 = a[i] * b[l], k2 = c[i] * rb;
  b[i] = b[i] - c[l] * k1 - ra * k2;
  d[i] = d[i] - d[l] * k1 - rd * k2;
  a[i] = -a[l] * k1;
  c[i] = -rc * k2;
}

// The 32 M rows left of a system, M consecutive ones a lane: CR down to
// 32 M / 2^LEV rows, PCR, back.
template <int M, int LEV>
__device__ __forceinline__ void rows_left(const float (&a)[M], const float (&b)[M], const float (&c)[M],
                                          const float (&d)[M], float (&x)[M], int lane) {
  if constexpr (LEV == 0) pcr_lanes<M, 1>(a, b, c, d, x, lane);
  else cr_solve<M, LEV, false>(a, b, c, d, x, lane);
}

// levels: CR levels past the five in the lane, log2(32 M / rest).
template <int M>
__global__ void __launch_bounds__(M * 32, 8 / M)
    crpcr_wide_kernel(HybridParams p, int levels, const __grid_constant__ CUtensorMap ma,
                      const __grid_constant__ CUtensorMap mb, const __grid_constant__ CUtensorMap mc,
                      const __grid_constant__ CUtensorMap md) {
  using S = CrWideShape<M>;
  static_assert(M == 2 || M == 4, "crpcr_wide: 2048 or 4096 rows");
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* ex = reinterpret_cast<float*>(smem + 128);
  float* left = ex + S::EXPORT;  // a, b, c, d of the rows left
  float* xl = left + 4 * S::ROWS;
  const uint32_t base = smem_addr(smem);
  const uint32_t ring = (base + (uint32_t)S::HEAD + 1023) & ~1023u;
  float* buf = reinterpret_cast<float*>(smem + (ring - base)) + (size_t)warp * 4 * kTF;
  float* gx = static_cast<float*>(p.x);
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  const auto issue = [&](long sys) {  // lane 0
    const int row = (int)((sys * M + warp) * (kTF / 32));
    mbar_arrive_expect_tx(bar, 4 * kTF * sizeof(float));
    tma_load_2d(buf + 0 * kTF, &ma, 0, row, bar);
    tma_load_2d(buf + 1 * kTF, &mb, 0, row, bar);
    tma_load_2d(buf + 2 * kTF, &mc, 0, row, bar);
    tma_load_2d(buf + 3 * kTF, &md, 0, row, bar);
  };
  if (lane == 0 && (int)blockIdx.x < p.m) issue(blockIdx.x);
  int chunk[kR / 4];
#pragma unroll
  for (int q = 0; q < kR / 4; ++q) {
    const int c = lane * (kR / 4) + q, row = c >> 3;
    chunk[q] = row * 32 + (((c & 7) ^ (row & 7)) << 2);
  }
  const int g = warp * 32 + lane;  // the lane's row among the rows left
  int k = 0;
  for (long sys = blockIdx.x; sys < p.m; sys += gridDim.x, ++k) {
    const bool ok = mbar_wait(bar, k & 1, p.status);
    float v[4][kR];
#pragma unroll
    for (int arr = 0; arr < 4; ++arr)
#pragma unroll
      for (int q = 0; q < kR / 4; ++q) {
        const float4 f = *reinterpret_cast<const float4*>(buf + arr * kTF + chunk[q]);
        v[arr][4 * q] = f.x; v[arr][4 * q + 1] = f.y; v[arr][4 * q + 2] = f.z; v[arr][4 * q + 3] = f.w;
      }
    fence_proxy_async_smem();
    __syncwarp();
    if (ok && lane == 0 && sys + gridDim.x < p.m) issue(sys + gridDim.x);
    if (g == 0) v[0][0] = 0.0f;                  // a[0] is not part of the system
    if (g == S::ROWS - 1) v[2][kR - 1] = 0.0f;   // nor is c[n-1]
    lane_levels(v[0], v[1], v[2], v[3]);
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < 5; ++j)
#pragma unroll
        for (int w = 0; w < 4; ++w) ex[(warp * 5 + j) * 4 + w] = v[w][(1 << j) - 1];
    }
    if (!__syncthreads_and(ok)) break;
    // the last row's levels (the system's last lane gets its own rows from the
    // shuffles: its c is zero)
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      float r[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        r[w] = __shfl_down_sync(kFull, v[w][(1 << j) - 1], 1);
        if (lane == 31 && warp < M - 1) r[w] = ex[((warp + 1) * 5 + j) * 4 + w];
      }
      last_row_level(v[0], v[1], v[2], v[3], kR - 1 - (1 << j), r[0], r[1], r[2], r[3]);
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) left[w * S::ROWS + g] = v[w][kR - 1];
    __syncthreads();
    if (warp == 0) {
      float ra[M], rb[M], rc[M], rd[M], rx[M];
#pragma unroll
      for (int q = 0; q < M; ++q) {
        ra[q] = left[M * lane + q];
        rb[q] = left[S::ROWS + M * lane + q];
        rc[q] = left[2 * S::ROWS + M * lane + q];
        rd[q] = left[3 * S::ROWS + M * lane + q];
      }
      constexpr int FULL = M == 2 ? 5 : 6;  // down to two rows (cr)
      switch (levels) {
        case 0: rows_left<M, 0>(ra, rb, rc, rd, rx, lane); break;
        case 1: rows_left<M, 1>(ra, rb, rc, rd, rx, lane); break;
        case 2: rows_left<M, 2>(ra, rb, rc, rd, rx, lane); break;
        case 3: rows_left<M, 3>(ra, rb, rc, rd, rx, lane); break;
        case 4: rows_left<M, 4>(ra, rb, rc, rd, rx, lane); break;
        case FULL: rows_left<M, FULL>(ra, rb, rc, rd, rx, lane); break;
        default: rows_left<M, FULL - 1>(ra, rb, rc, rd, rx, lane); break;
      }
#pragma unroll
      for (int q = 0; q < M; ++q) xl[M * lane + q] = rx[q];
    }
    __syncthreads();
    float x[kR];
    x[kR - 1] = xl[g];
    const float xprev = g > 0 ? xl[g - 1] : 0.0f;
#pragma unroll
    for (int h = kR / 2; h >= 1; h /= 2) {
#pragma unroll
      for (int i = h - 1; i < kR; i += 2 * h) {
        const float l = i >= h ? x[i >= h ? i - h : 0] : xprev, r = x[i + h];
        x[i] = (v[3][i] - v[0][i] * l - v[2][i] * r) * v[1][i];
      }
    }
    float4* dst = reinterpret_cast<float4*>(gx + sys * S::N + kR * g);
#pragma unroll
    for (int q = 0; q < kR / 4; ++q) dst[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
  }
}

template <int M>
cudaError_t launch_wide(const HybridParams& p, int levels, const DeviceInfo& dev, cudaStream_t stream) {
  using S = CrWideShape<M>;
  auto kern = crpcr_wide_kernel<M>;
  const uint64_t rows = (uint64_t)p.m * S::N / 32;
  CUtensorMap ma, mb, mc, md;
  if (!make_tensor_map_2d(&ma, static_cast<const float*>(p.a), 32, rows, 128, 32, kR, true) ||
      !make_tensor_map_2d(&mb, static_cast<const float*>(p.b), 32, rows, 128, 32, kR, true) ||
      !make_tensor_map_2d(&mc, static_cast<const float*>(p.c), 32, rows, 128, 32, kR, true) ||
      !make_tensor_map_2d(&md, static_cast<const float*>(p.d), 32, rows, 128, 32, kR, true))
    return cudaErrorInvalidValue;
  if (S::SMEM > (size_t)dev.max_smem_optin) return cudaErrorInvalidConfiguration;
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, M * 32, S::SMEM, dev, &per_sm);
  if (e != cudaSuccess) return e;
  long grid = (long)per_sm * dev.sm_count;
  if (grid > p.m) grid = p.m;
  return launch_kernel(kern, (unsigned)grid, M * 32, S::SMEM, stream, p, levels, ma, mb, mc, md);
}

}  // namespace

// cr, and crpcr at any stride = n / rest >= 2, at n = 2048 or 4096 (FP32,
// 16-byte aligned a..d and x, the batch within the tensor maps' 32-bit row
// count).
bool crpcr_wide_applies(const void* a, const void* b, const void* c, const void* d, const void* x, int n, long m,
                        int stride) {
  return (n == 2048 || n == 4096) && stride >= 2 && stride <= n / 2 && is_pow2(stride) && aligned16(a) &&
         aligned16(b) && aligned16(c) && aligned16(d) && aligned16(x) && m * n / 32 < (1L << 31) &&
         tunable(TRIDI_TUNE_PCR_KERNEL) != 2 && !g_host_mapped_io;
}

tridi_status crpcr_wide_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                              int stride, cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  HybridParams p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m; p.stride = stride;
  p.status = dev->status;
  const int levels = stride > 32 ? ilog2(stride) - 5 : 0;
  return cuda_status(n == 2048 ? launch_wide<2>(p, levels, *dev, stream) : launch_wide<4>(p, levels, *dev, stream));
}

}  // namespace tridi
