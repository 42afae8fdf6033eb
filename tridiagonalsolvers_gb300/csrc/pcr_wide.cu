// PCR and PCR-then-Thomas for FP32 systems of 2048 and 4096 unknowns, on the
// two-phase kernels of 1024 (pcr_twophase.cuh, pcr_thomas2.cu).
//
// One CTA of M = n / 1024 warps per system.  Warp w loads rows 1024 w ..
// 1024 w + 1023, 32 contiguous rows a lane, exactly as a warp of the
// 1024-unknown kernel loads a system.  The first log2(M) PCR steps (distances
// 1 .. M/2) run there; the rows at a warp's ends cross through shared memory.
// They leave M independent systems of 1024 rows each, the rows of equal
// residue mod M, and the normalised rows move once through shared memory so
// that warp w holds residue w, again 32 consecutive rows a lane.  From there
// on each warp runs the 1024-unknown kernel's steps unchanged: PCR to the end
// (G = 0), or PCR steps of distance 1 .. G/2 and Thomas on the G chains (M * G
// chains of the whole system).  x goes out through shared memory, consecutive
// unknowns by consecutive lanes.
//
// What bounds it: latency, at 8 warps of 255 registers an SM, and the barriers of
// a system, six at 2048 rows and seven at 4096 (the other CTAs of the SM run in
// their shadow).  16.8 M
// unknowns: pcr 99 us at 2048 and 106 us at 4096 (the hybrid kernel, PCR steps
// through shared memory with two barriers each: 352 and 630 us), pcrGauss g = 8
// 84 and 91 us (pcr_thomas.cu: 1085 and 1097 us).
//
// A split into fewer than 32 M chains would leave chains spread over lanes, so
// it takes 32 M; the solution stays exact (any number of PCR steps leaves
// systems with the same solution) and only the rounding differs.
#include "hybrid.cuh"
#include "pcr_thomas2.cuh"
#include "pcr_twophase.cuh"
#include "runtime.h"

namespace tridi {

namespace {

using namespace pcr2;

constexpr int kR = 32;     // rows a lane
constexpr int kTF = 1024;  // values of one array in a warp's tile

template <int M>
struct WideShape {
  static constexpr int N = M * 1024;
  // Row r of a word array sits at r + r/32 + r/(32 M): the 4-byte stores of
  // lanes 32 rows apart and the loads of lanes 32 M rows apart fall on
  // distinct banks (but for a few of the stores).
  static constexpr int WORDS = N + N / 32 + 32;
  static constexpr int EDGES = M * 2 * 9;  // first and last row (3 words), first and last pair (6 words) per warp
  static constexpr size_t HEAD = (128 + EDGES * sizeof(float) + 127) & ~(size_t)127;
  static constexpr size_t SMEM = HEAD + 2 * (size_t)WORDS * sizeof(float) + 1024 + (size_t)M * 4 * kTF * sizeof(float);
  static_assert(WORDS % 4 == 0 && (1024 + 32) % 4 == 0 && M * (1024 + 32) <= WORDS && N <= WORDS &&
                    (N - 1) + (N - 1) / 32 + (N - 1) / (32 * M) < WORDS && HEAD % 16 == 0,
                "pcr_wide: shared arrays");
  static __device__ __forceinline__ int at(int r) { return r + (r >> 5) + r / (32 * M); }
};

// x of row r before it leaves: the low bits by r / 32, so that the stores of
// lanes M rows apart fall on distinct banks.
template <int M>
__device__ __forceinline__ int x_at(int r) {
  return r ^ ((r >> 5) & (M - 1));
}

// PCR steps of distance 1 and 2 with the neighbours beyond the warp given; the
// first three steps of a system in the finer form (fine_step): error against
// FP64 at 4096 rows 0.91e-7 (1.23e-7 without, 1.01e-7 for the shared-memory
// kernels, which keep the diagonals; in every step it cost 15 % more time).
template <int R>
__device__ __forceinline__ void step1_edges(NR2 (&P)[R / 2], const NR& fromL, const NR& fromR) {
  constexpr int NP = R / 2;
  NR2 o[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) {
    const NR lo = fine_step(row_x(P[j]), j > 0 ? row_y(P[j > 0 ? j - 1 : 0]) : fromL, row_y(P[j]));
    const NR hi = fine_step(row_y(P[j]), row_x(P[j]), j + 1 < NP ? row_x(P[j + 1 < NP ? j + 1 : j]) : fromR);
    o[j] = pair_of(lo, hi);
  }
#pragma unroll
  for (int j = 0; j < NP; ++j) P[j] = o[j];
}
template <int R>
__device__ __forceinline__ void step2_edges(NR2 (&P)[R / 2], const NR2& fromL, const NR2& fromR) {
  constexpr int NP = R / 2;
  NR2 o[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j)
    o[j] = fine_step2(P[j], j > 0 ? P[j > 0 ? j - 1 : 0] : fromL, j + 1 < NP ? P[j + 1 < NP ? j + 1 : j] : fromR);
#pragma unroll
  for (int j = 0; j < NP; ++j) P[j] = o[j];
}

__device__ __forceinline__ void put_row(float* e, const NR& v) { e[0] = v.a; e[1] = v.c; e[2] = v.d; }
__device__ __forceinline__ NR get_row(const float* e) { return {e[0], e[1], e[2]}; }

template <int M, int G>
__global__ void __launch_bounds__(M * 32, 8 / M)
    pcr_wide_kernel(HybridParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                    const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  using S = WideShape<M>;
  static_assert(M == 2 || M == 4, "pcr_wide: 2048 or 4096 rows");
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* edges = reinterpret_cast<float*>(smem + 128);
  float* w1 = reinterpret_cast<float*>(smem + S::HEAD);
  float* w2 = w1 + S::WORDS;
  const uint32_t base = smem_addr(smem);
  const uint32_t ring = (base + (uint32_t)S::HEAD + 2u * S::WORDS * (uint32_t)sizeof(float) + 1023) & ~1023u;
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
  int k = 0;
  for (long sys = blockIdx.x; sys < p.m; sys += gridDim.x, ++k) {
    const bool ok = mbar_wait(bar, k & 1, p.status);
    NR2 P[kR / 2];
    {
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
      if (warp == 0 && lane == 0) v[0][0] = 0.0f;             // a[0] is not part of the system
      if (warp == M - 1 && lane == 31) v[2][kR - 1] = 0.0f;   // nor is c[n-1]
#pragma unroll
      for (int j = 0; j < kR / 2; ++j) {
        const float2 ib = rcp_approx2(make_float2(v[1][2 * j], v[1][2 * j + 1]));
        P[j] = NR2{__fmul2_rn(make_float2(v[0][2 * j], v[0][2 * j + 1]), ib),
                   __fmul2_rn(make_float2(v[2][2 * j], v[2][2 * j + 1]), ib),
                   __fmul2_rn(make_float2(v[3][2 * j], v[3][2 * j + 1]), ib)};
      }
    }
    // ---- distances 1 .. M/2 on contiguous rows; the edge rows of a warp from
    //      its neighbours (at the system's ends the lane's own row stands in:
    //      its coupling there is exactly zero) ----
    {
      if (lane == 0) put_row(edges + warp * 6, row_x(P[0]));
      if (lane == 31) put_row(edges + warp * 6 + 3, row_y(P[kR / 2 - 1]));
      NR fromL = shfl_up_nr(row_y(P[kR / 2 - 1]), 32), fromR = shfl_down_nr(row_x(P[0]), 32);
      if (!__syncthreads_and(ok)) break;
      if (lane == 0 && warp > 0) fromL = get_row(edges + (warp - 1) * 6 + 3);
      if (lane == 31 && warp < M - 1) fromR = get_row(edges + (warp + 1) * 6);
      step1_edges<kR>(P, fromL, fromR);
    }
    if constexpr (M == 4) {
      float* e2 = edges + 6 * M;
      if (lane == 0) { put_row(e2 + warp * 12, row_x(P[0])); put_row(e2 + warp * 12 + 3, row_y(P[0])); }
      if (lane == 31) {
        put_row(e2 + warp * 12 + 6, row_x(P[kR / 2 - 1]));
        put_row(e2 + warp * 12 + 9, row_y(P[kR / 2 - 1]));
      }
      NR2 fromL = shfl_up_nr2(P[kR / 2 - 1], 32), fromR = shfl_down_nr2(P[0], 32);
      __syncthreads();
      if (lane == 0 && warp > 0)
        fromL = pair_of(get_row(e2 + (warp - 1) * 12 + 6), get_row(e2 + (warp - 1) * 12 + 9));
      if (lane == 31 && warp < M - 1)
        fromR = pair_of(get_row(e2 + (warp + 1) * 12), get_row(e2 + (warp + 1) * 12 + 3));
      step2_edges<kR>(P, fromL, fromR);
    }
    // ---- to residues: warp w takes rows M u + w, lane t u = 32 t .. 32 t + 31 ----
    const int r0 = 1024 * warp + 32 * lane;
    const auto put = [&](float* dst, auto word) {
#pragma unroll
      for (int j = 0; j < kR / 2; ++j) {
        const float2 v = word(j);
        dst[S::at(r0 + 2 * j)] = v.x;
        dst[S::at(r0 + 2 * j + 1)] = v.y;
      }
    };
    const auto get = [&](const float* src, auto word) {
#pragma unroll
      for (int j = 0; j < kR / 2; ++j)
        word(j) = make_float2(src[S::at(M * (32 * lane + 2 * j) + warp)], src[S::at(M * (32 * lane + 2 * j + 1) + warp)]);
    };
    put(w1, [&](int j) -> float2& { return P[j].a; });
    __syncthreads();
    get(w1, [&](int j) -> float2& { return P[j].a; });
    put(w2, [&](int j) -> float2& { return P[j].c; });
    __syncthreads();
    get(w2, [&](int j) -> float2& { return P[j].c; });
    put(w1, [&](int j) -> float2& { return P[j].d; });
    __syncthreads();
    get(w1, [&](int j) -> float2& { return P[j].d; });
    // ---- the 1024-unknown kernel on the warp's residue ----
    float* sw = w2 + (size_t)warp * (1024 + 32);  // (every warp has read c)
    const int rb = 32 * lane;
    phase_a_step1_pairs<32, kR, true>(P);
    phase_a_step_pairs<1, 32, kR, M == 2>(P);
    phase_a_step_pairs<2, 32, kR>(P);
    phase_a_step_pairs<4, 32, kR>(P);
    phase_a_step_pairs<8, 32, kR>(P);
    transpose_word<kR, 32>(sw, rb, lane, [&](int j) -> float2& { return P[j].a; });
    transpose_word<kR, 32>(sw, rb, lane, [&](int j) -> float2& { return P[j].c; });
    transpose_word<kR, 32>(sw, rb, lane, [&](int j) -> float2& { return P[j].d; });
    __syncthreads();  // every warp has read d: x takes its place
    const auto emit = [&](int s, float v) { w1[x_at<M>(M * (lane + 32 * s) + warp)] = v; };
    if constexpr (G == 0) {
      phase_b_pairs<1, kR>(P);
      phase_b_pairs<2, kR>(P);
      phase_b_pairs<4, kR>(P);
      phase_b_pairs<8, kR>(P);
#pragma unroll
      for (int j = 0; j < kR / 4; ++j) {  // 2x2 systems (s, s + R/2), two at a time
        const NR2& u = P[j];
        const NR2& l = P[j + kR / 4];
        const float2 den = __ffma2_rn(neg2(u.c), l.a, make_float2(1.0f, 1.0f));
        const float2 num = __ffma2_rn(neg2(u.c), l.d, u.d);
        const float2 xu = __fmul2_rn(num, rcp_approx2(den));
        const float2 xl = __ffma2_rn(neg2(l.a), xu, l.d);
        emit(2 * j, xu.x);
        emit(2 * j + 1, xu.y);
        emit(2 * j + kR / 2, xl.x);
        emit(2 * j + 1 + kR / 2, xl.y);
      }
    } else {
      constexpr int KG = G / 32;  // chains a lane
      if constexpr (G >= 64) phase_b_pairs<1, kR>(P);
      if constexpr (G >= 128) phase_b_pairs<2, kR>(P);
      if constexpr (G >= 256) phase_b_pairs<4, kR>(P);
      if constexpr (KG == 1) {
        NR w[kR];
#pragma unroll
        for (int j = 0; j < kR / 2; ++j) {
          w[2 * j] = row_x(P[j]);
          w[2 * j + 1] = row_y(P[j]);
        }
        thomas_single<kR>(w, emit);
      } else {
        thomas_pairs<kR, KG>(P, emit);
      }
    }
    __syncthreads();
    float* dst = gx + sys * S::N;
#pragma unroll 8
    for (int i = threadIdx.x; i < S::N; i += M * 32) dst[i] = w1[x_at<M>(i)];
  }
}

template <int M, int G>
cudaError_t launch_wide(const HybridParams& p, const DeviceInfo& dev, cudaStream_t stream) {
  using S = WideShape<M>;
  auto kern = pcr_wide_kernel<M, G>;
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
  return launch_kernel(kern, (unsigned)grid, M * 32, S::SMEM, stream, p, ma, mb, mc, md);
}

template <int M>
cudaError_t launch_split(const HybridParams& p, int g, const DeviceInfo& dev, cudaStream_t stream) {
  if (g >= M * 512) return launch_wide<M, 0>(p, dev, stream);
  if (g >= M * 256) return launch_wide<M, 256>(p, dev, stream);
  if (g >= M * 128) return launch_wide<M, 128>(p, dev, stream);
  if (g >= M * 64) return launch_wide<M, 64>(p, dev, stream);
  return launch_wide<M, 32>(p, dev, stream);
}

}  // namespace

// FP32, n = 2048 or 4096, contiguous 16-byte aligned device arrays, the batch
// within the tensor maps' 32-bit row count; at least four chains: with one or
// two the shared-memory kernel's Thomas on unreduced rows rounds less (0.60e-7
// and 0.76e-7 against 0.91e-7).
bool pcr_wide_applies(const void* a, const void* b, const void* c, const void* d, int n, long m, int g) {
  return (n == 2048 || n == 4096) && g >= 4 && aligned16(a) && aligned16(b) && aligned16(c) && aligned16(d) &&
         m * n / 32 < (1L << 31) && tunable(TRIDI_TUNE_PCR_KERNEL) != 2 && !g_host_mapped_io;
}

// g chains (a power of two); g >= n/2 is PCR to the end.
tridi_status pcr_wide_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                            int g, cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  HybridParams p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m; p.stride = 1;
  p.status = dev->status;
  return cuda_status(n == 2048 ? launch_split<2>(p, g, *dev, stream) : launch_split<4>(p, g, *dev, stream));
}

}  // namespace tridi
