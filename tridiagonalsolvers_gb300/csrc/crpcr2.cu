// CR-PCR for FP32 systems of 1024 (and, in large batches, 512) unknowns in
// registers, one system a warp (n / 32 contiguous rows a lane, loaded by TMA
// into the warp's buffer): every switch level of "crpcr" (restSystemSize
// 2 .. n/2, crpcr_kernel.cu:1-148, crpcr_app.cu:5) and, at rest 2, "cr"
// (cr_kernel.cu, cr_app.cu:4).
//
// crpcr_lanes_kernel<N, LEV> (rest = N / 2^LEV): the first log2(N/32) CR
// levels run inside the lane (32 -> 16 -> 8 -> 4 -> 2 -> 1 rows at N = 1024; each level's
// last odd row takes its right neighbour from the next lane over one
// shuffle), the levels past five between lanes (lane strides 1, 2, 4, 8).
// PCR on the rows left: distances below the rows a lane holds inside the
// lane, the others between lanes (the neighbour at distance K2 ld is lane
// t -/+ ld, same slot), the closing 2x2 systems between lanes t and t ^ 16.
// The back substitutions retrace the levels from the coefficients each lane
// kept in registers; the lane's 32 unknowns leave in 16-byte stores.  No
// shared memory but the TMA buffer.  At rest 2 the levels and the closing
// solve are CR's own (divisions, unnormalised rows), so cr here rounds
// exactly like every other CR kernel of the library; above rest 2 the
// in-lane levels divide each even row by its diagonal once and eliminate
// against those normalised rows (cr_level_norm).
//
// crpcr512_kernel (rest 512): one CR level inside the lane (on normalised even
// rows, as above) leaves lane t the
// intermediate rows 16t .. 16t+15 as normalised 3-word rows -- exactly the
// 512-row layout of the two-phase PCR (pcr_twophase.cuh, 16 rows a lane, one
// system a warp), so its phase A, transpose, phase B and closing 2x2 systems
// run unchanged and leave x of intermediate row t + 32s in lane t.  Those
// 512 values go through the warp's scratch once (padded so the
// lane-contiguous reads hit distinct banks), each lane forms its 16 even
// rows' x from its own coefficients, and writes its 32 unknowns.  (The lanes
// design at rest 512 -- 16 rows a lane, four PCR steps between lanes with 16
// rows each -- measured 64 % of HBM against this kernel's 80 %, 87 % since
// its level works on normalised even rows.)
#include "crpcr2.cuh"
#include "hybrid.cuh"
#include "pcr_twophase.cuh"
#include "runtime.h"

namespace tridi {

namespace {

using namespace pcr2;

constexpr int kN = 1024;
constexpr int kR = 32;          // original rows a lane
constexpr int kRR = 16;         // intermediate rows a lane
constexpr int kLPS = 32;        // lanes per system
constexpr int kTF = kN;         // values of one array in a warp tile (one system)
constexpr int kWarps = 2;       // warps per CTA
constexpr int kScratch = 512 + 32;  // one word array of the 512-row transpose, then x of the 512 rows (padded)
constexpr size_t kSmem = 128 + (size_t)kWarps * kScratch * sizeof(float) + 1024 + (size_t)kWarps * 4 * kTF * 4;

__device__ __forceinline__ int xr_index(int r) { return r + (r >> 4); }  // one pad word per 16

__global__ void __launch_bounds__(kWarps * 32, 3)
    crpcr512_kernel(HybridParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                    const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  float* sw = reinterpret_cast<float*>(smem + 128) + (size_t)warp * kScratch;
  const uint32_t base = smem_addr(smem);
  const uint32_t ring = (base + 128 + kWarps * kScratch * (uint32_t)sizeof(float) + 1023) & ~1023u;
  float* buf = reinterpret_cast<float*>(smem + (ring - base)) + (size_t)warp * 4 * kTF;
  float* gx = static_cast<float*>(p.x);
  const long tiles = p.m;  // one system a tile
  const long first = (long)blockIdx.x * kWarps + warp;
  const long step = (long)gridDim.x * kWarps;
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  const auto issue = [&](long tile) {  // lane 0
    const int row = (int)(tile * (kTF / 32));
    mbar_arrive_expect_tx(bar, 4 * kTF * sizeof(float));
    tma_load_2d(buf + 0 * kTF, &ma, 0, row, bar);
    tma_load_2d(buf + 1 * kTF, &mb, 0, row, bar);
    tma_load_2d(buf + 2 * kTF, &mc, 0, row, bar);
    tma_load_2d(buf + 3 * kTF, &md, 0, row, bar);
  };
  if (lane == 0 && first < tiles) issue(first);
  int chunk[kR / 4];
#pragma unroll
  for (int q = 0; q < kR / 4; ++q) {
    const int c = lane * (kR / 4) + q, row = c >> 3;
    chunk[q] = row * 32 + (((c & 7) ^ (row & 7)) << 2);
  }
  int k = 0;
  for (long tile = first; tile < tiles; tile += step, ++k) {
    if (!mbar_wait(bar, k & 1, p.status)) break;
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
    if (lane == 0 && tile + step < tiles) issue(tile + step);
    if (lane == 0) v[0][0] = 0.0f;          // a[0] is not part of the system
    if (lane == 31) v[2][kR - 1] = 0.0f;    // nor is c[n-1]
    // ---- CR level: odd rows 2j+1 against their even neighbours, which are
    //      normalised once (one reciprocal per even row; the back
    //      substitution reuses them) ----
    // (lane 31's last odd row has c = 0, so the shuffled-in neighbour, its
    // own first row, contributes nothing)
    NR e[kRR];  // even row 2j / its diagonal
#pragma unroll
    for (int j = 0; j < kRR; ++j) {
      const float ib = rcp_approx(v[1][2 * j]);
      e[j] = NR{v[0][2 * j] * ib, v[2][2 * j] * ib, v[3][2 * j] * ib};
    }
    const NR eR = shfl_down_nr(e[0], 32);  // the next lane's row 0
    NR2 P[kRR / 2];
#pragma unroll
    for (int j = 0; j < kRR; ++j) {
      const int q = 2 * j + 1;
      const NR& L = e[j];
      const NR& Rn = j + 1 < kRR ? e[j + 1] : eR;
      const float aq = v[0][q], cq = v[2][q];
      const float an = -aq * L.a;
      const float bn = v[1][q] - aq * L.c - cq * Rn.a;
      const float cn = -cq * Rn.c;
      const float dn = v[3][q] - aq * L.d - cq * Rn.d;
      const float ib = rcp_approx(bn);
      const NR r{an * ib, cn * ib, dn * ib};
      if (j & 1) {
        P[j / 2].a.y = r.a; P[j / 2].c.y = r.c; P[j / 2].d.y = r.d;
      } else {
        P[j / 2].a.x = r.a; P[j / 2].c.x = r.c; P[j / 2].d.x = r.d;
      }
    }
    // ---- PCR on the 512 intermediate rows (the two-phase kernel's n = 512 path) ----
    phase_a_pairs<kLPS, kRR>(P);
    transpose_word<kRR, kLPS>(sw, kRR * lane, lane, [&](int j) -> float2& { return P[j].a; });
    transpose_word<kRR, kLPS>(sw, kRR * lane, lane, [&](int j) -> float2& { return P[j].c; });
    transpose_word<kRR, kLPS>(sw, kRR * lane, lane, [&](int j) -> float2& { return P[j].d; });
    {
      NR w[kRR];
#pragma unroll
      for (int j = 0; j < kRR / 2; ++j) {
        w[2 * j] = row_x(P[j]);
        w[2 * j + 1] = row_y(P[j]);
      }
      phase_b_xor16<kRR>(w, lane);
      phase_b_step<1, kRR>(w);
#pragma unroll
      for (int j = 0; j < kRR / 2; ++j) P[j] = pair_of(w[2 * j], w[2 * j + 1]);
    }
    phase_b_pairs<2, kRR>(P);
    phase_b_pairs<4, kRR>(P);
    // ---- closing 2x2 systems (slots s, s + 8): x of intermediate row lane + 32 s ----
#pragma unroll
    for (int j = 0; j < kRR / 4; ++j) {
      const NR2& u = P[j];
      const NR2& l = P[j + kRR / 4];
      const float2 den = __ffma2_rn(neg2(u.c), l.a, make_float2(1.0f, 1.0f));
      const float2 num = __ffma2_rn(neg2(u.c), l.d, u.d);
      const float2 xu = __fmul2_rn(num, rcp_approx2(den));
      const float2 xl = __ffma2_rn(neg2(l.a), xu, l.d);
      sw[xr_index(lane + 32 * (2 * j))] = xu.x;
      sw[xr_index(lane + 32 * (2 * j + 1))] = xu.y;
      sw[xr_index(lane + 32 * (2 * j + kRR / 2))] = xl.x;
      sw[xr_index(lane + 32 * (2 * j + 1 + kRR / 2))] = xl.y;
    }
    __syncwarp();
    // ---- CR back substitution of the even rows; the lane's 32 unknowns out ----
    float xo[kR];
    float xprev = lane > 0 ? sw[xr_index(kRR * lane - 1)] : 0.0f;  // (row 0's a is zero)
#pragma unroll
    for (int j = 0; j < kRR; ++j) {
      const float xodd = sw[xr_index(kRR * lane + j)];
      const int q = 2 * j;
      xo[q] = e[j].d - e[j].a * xprev - e[j].c * xodd;
      xo[q + 1] = xodd;
      xprev = xodd;
    }
    __syncwarp();  // the scratch is the next tile's transpose scratch
    if (tile < p.m) {
      float4* dst = reinterpret_cast<float4*>(gx + tile * kN + kR * lane);
#pragma unroll
      for (int q = 0; q < kR / 4; ++q) dst[q] = make_float4(xo[4 * q], xo[4 * q + 1], xo[4 * q + 2], xo[4 * q + 3]);
    }
  }
}

// Shared memory of a lanes-kernel CTA for n unknowns: barriers, then the two
// warps' TMA buffers (1024-byte aligned for the 128-byte swizzle).
constexpr size_t lanes_smem(int n) { return 128 + 1024 + (size_t)kWarps * 4 * n * 4; }

// CR-PCR with the switch at N / 2^LEV for N = 512 or 1024 unknowns (R = N / 32
// rows a lane), in registers and shuffles (the file header gives the scheme).
// At 1024 unknowns four CTAs of two warps an SM (at most 255 registers: none
// spill; three or five to six measured the same or slower), at 512 eight (the
// same bytes of tiles in flight an SM).
template <int N, int LEV>
__global__ void __launch_bounds__(kWarps * 32, N == 512 ? 8 : 4)
    crpcr_lanes_kernel(HybridParams p, const __grid_constant__ CUtensorMap ma, const __grid_constant__ CUtensorMap mb,
                       const __grid_constant__ CUtensorMap mc, const __grid_constant__ CUtensorMap md) {
  constexpr int R = N / 32, TF = N;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem) + warp;
  const uint32_t base = smem_addr(smem);
  const uint32_t ring = (base + 128 + 1023) & ~1023u;
  float* buf = reinterpret_cast<float*>(smem + (ring - base)) + (size_t)warp * 4 * TF;
  float* gx = static_cast<float*>(p.x);
  const long tiles = p.m;
  const long first = (long)blockIdx.x * kWarps + warp;
  const long step = (long)gridDim.x * kWarps;
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  const auto issue = [&](long tile) {
    const int row = (int)(tile * (TF / 32));
    mbar_arrive_expect_tx(bar, 4 * TF * sizeof(float));
    tma_load_2d(buf + 0 * TF, &ma, 0, row, bar);
    tma_load_2d(buf + 1 * TF, &mb, 0, row, bar);
    tma_load_2d(buf + 2 * TF, &mc, 0, row, bar);
    tma_load_2d(buf + 3 * TF, &md, 0, row, bar);
  };
  if (lane == 0 && first < tiles) issue(first);
  int chunk[R / 4];
#pragma unroll
  for (int q = 0; q < R / 4; ++q) {
    const int c = lane * (R / 4) + q, row = c >> 3;
    chunk[q] = row * 32 + (((c & 7) ^ (row & 7)) << 2);
  }
  int k = 0;
  for (long tile = first; tile < tiles; tile += step, ++k) {
    if (!mbar_wait(bar, k & 1, p.status)) break;
    float v[4][R];
#pragma unroll
    for (int arr = 0; arr < 4; ++arr)
#pragma unroll
      for (int q = 0; q < R / 4; ++q) {
        const float4 f = *reinterpret_cast<const float4*>(buf + arr * TF + chunk[q]);
        v[arr][4 * q] = f.x; v[arr][4 * q + 1] = f.y; v[arr][4 * q + 2] = f.z; v[arr][4 * q + 3] = f.w;
      }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && tile + step < tiles) issue(tile + step);
    if (lane == 0) v[0][0] = 0.0f;
    if (lane == 31) v[2][R - 1] = 0.0f;
    float x[R];
    // rest 2 is cr: CR's own arithmetic, bit for bit that of the other CR kernels
    cr_solve<R, LEV, ((N >> LEV) > 2)>(v[0], v[1], v[2], v[3], x, lane);
    float4* dst = reinterpret_cast<float4*>(gx + tile * N + R * lane);
#pragma unroll
    for (int q = 0; q < R / 4; ++q) dst[q] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
  }
}

using TileKernel = void (*)(HybridParams, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap);

// One warp a system, as many CTAs of two warps as fit on every SM up to
// max_per_sm (the warps then loop over the batch).  At 1024 unknowns five or
// six CTAs an SM, where the registers allow it, measured 5 % slower than four:
// more warps contend for the shared-memory pipe without hiding more DRAM
// latency.
tridi_status launch_tiles(TileKernel kern, size_t smem, int max_per_sm, const HybridParams& p,
                          const CUtensorMap* tm, const DeviceInfo* dev, cudaStream_t stream) {
  if (smem > (size_t)dev->max_smem_optin) return TRIDI_ERROR_UNSUPPORTED_SIZE;
  int per_sm = 0;
  const cudaError_t e = resident_blocks(kern, kWarps * 32, smem, *dev, &per_sm);
  if (e != cudaSuccess) return cuda_status(e);
  if (per_sm > max_per_sm) per_sm = max_per_sm;
  long grid = (long)per_sm * dev->sm_count;
  if (grid * kWarps > p.m) grid = (p.m + kWarps - 1) / kWarps;
  return cuda_status(launch_kernel(kern, (unsigned)grid, kWarps * 32, smem, stream, p, tm[0], tm[1], tm[2], tm[3]));
}

template <int N>
tridi_status launch_lanes(int stride, const HybridParams& p, const CUtensorMap* tm, const DeviceInfo* dev,
                          cudaStream_t stream) {
  constexpr int M = N == 512 ? 8 : 4;
  constexpr size_t S = lanes_smem(N);
  switch (stride) {
    case 2: if constexpr (N == 512) return launch_tiles(crpcr_lanes_kernel<N, 1>, S, M, p, tm, dev, stream);
            break;
    case 4: return launch_tiles(crpcr_lanes_kernel<N, 2>, S, M, p, tm, dev, stream);
    case 8: return launch_tiles(crpcr_lanes_kernel<N, 3>, S, M, p, tm, dev, stream);
    case 16: return launch_tiles(crpcr_lanes_kernel<N, 4>, S, M, p, tm, dev, stream);
    case 32: return launch_tiles(crpcr_lanes_kernel<N, 5>, S, M, p, tm, dev, stream);
    case 64: return launch_tiles(crpcr_lanes_kernel<N, 6>, S, M, p, tm, dev, stream);
    case 128: return launch_tiles(crpcr_lanes_kernel<N, 7>, S, M, p, tm, dev, stream);
    case 256: return launch_tiles(crpcr_lanes_kernel<N, 8>, S, M, p, tm, dev, stream);
    case 512: if constexpr (N == 1024) return launch_tiles(crpcr_lanes_kernel<N, 9>, S, M, p, tm, dev, stream);
              break;
    default: break;
  }
  return TRIDI_ERROR_UNSUPPORTED_SIZE;
}

}  // namespace

// True when a register kernel takes this FP32 call: cr, or crpcr at any
// switch level (stride = n / rest = 2 .. n/2), at n = 1024, or at n = 512 from
// 4096 systems up (on a small batch one warp a system leaves the GPU short of
// threads: 512 x 512 cr 6.1 us against 4.7 us for the block kernel, which
// gives a system two warps; 32768 x 512 cr 54.6 against 58.0 us, crpcr rest
// 256 55.9 against 117.2 us), 16-byte aligned a..d and x, the batch within
// the tensor maps' 32-bit row count.
bool crpcr_regs_applies(const void* a, const void* b, const void* c, const void* d, const void* x, int n, long m,
                        int stride) {
  return (n == 1024 || (n == 512 && m >= 4096)) && stride >= 2 && stride <= n / 2 && is_pow2(stride) &&
         aligned16(a) &&
         aligned16(b) && aligned16(c) && aligned16(d) && aligned16(x) && m * n / 32 < (1L << 31) &&
         tunable(TRIDI_TUNE_PCR_KERNEL) != 2 && !g_host_mapped_io;
}

tridi_status crpcr_regs_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n,
                              int m, int stride, cudaStream_t stream) {
  const DeviceInfo* dev = current_device();
  if (!dev) return TRIDI_ERROR_CUDA;
  HybridParams p{};
  p.a = a; p.b = b; p.c = c; p.d = d; p.x = x;
  p.n = n; p.m = m; p.stride = stride;
  p.status = dev->status;
  const uint64_t rows = (uint64_t)m * n / 32;
  const uint32_t box = (uint32_t)(n / 32);  // a system: n / 32 rows of 32 values
  CUtensorMap tma, tmb, tmc, tmd;
  if (!make_tensor_map_2d(&tma, a, 32, rows, 128, 32, box, true) ||
      !make_tensor_map_2d(&tmb, b, 32, rows, 128, 32, box, true) ||
      !make_tensor_map_2d(&tmc, c, 32, rows, 128, 32, box, true) ||
      !make_tensor_map_2d(&tmd, d, 32, rows, 128, 32, box, true))
    return cuda_status(cudaErrorInvalidValue);
  const CUtensorMap tm[4] = {tma, tmb, tmc, tmd};
  if (n == 512) return launch_lanes<512>(stride, p, tm, dev, stream);
  if (stride == 2) return launch_tiles(crpcr512_kernel, kSmem, 4, p, tm, dev, stream);
  return launch_lanes<1024>(stride, p, tm, dev, stream);
}

}  // namespace tridi
