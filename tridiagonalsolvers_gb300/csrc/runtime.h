// Host-side runtime shared by every entry point: per-device facts (SM count,
// shared-memory limit), the per-device status word that bounded device waits
// report into, CUDA error capture, and the stream type conversion.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tridi.h"

namespace tridi {

struct DeviceInfo {
  int device = -1;
  int sm_count = 0;
  int max_smem_optin = 0;   // bytes of dynamic shared memory a CTA may opt into
  unsigned* status = nullptr;  // device status word (TRIDI_DEVERR_* bits)
};

// Facts about the current device; allocates its status word on first use.
// Returns nullptr and sets the thread's CUDA error if the device cannot be
// queried.
const DeviceInfo* current_device();

// Records a CUDA error for tridi_last_cuda_error() and returns TRIDI_ERROR_CUDA
// (or TRIDI_SUCCESS for cudaSuccess).
tridi_status cuda_status(cudaError_t e);

inline cudaStream_t as_stream(tridi_stream_t s) { return reinterpret_cast<cudaStream_t>(s); }

// CTAs of `threads` threads and `smem` bytes of dynamic shared memory that one
// SM holds of the kernel (at least 1).  The first call of a thread for a shape
// raises the kernel's shared-memory limit to the device's and asks the
// runtime; later ones find the answer in a table of the thread (the two calls
// took 1 to 2 us of each launch).
cudaError_t resident_blocks(const void* kern, int threads, size_t smem, const DeviceInfo& dev, int* per_sm);
template <class... P>
cudaError_t resident_blocks(void (*kern)(P...), int threads, size_t smem, const DeviceInfo& dev, int* per_sm) {
  return resident_blocks(reinterpret_cast<const void*>(kern), threads, smem, dev, per_sm);
}
// Raises the kernel's dynamic shared-memory limit to what the device leaves
// beside its static shared memory.
cudaError_t raise_smem_limit(const void* kern, const DeviceInfo& dev);

// Whether the kernel may be launched with `smem` bytes of dynamic shared memory.
bool smem_allowed(const void* kern, size_t smem);

// A launch with `smem` bytes of dynamic shared memory.  A device reset drops a
// raised limit; the launch then fails and is repeated with the limit set.  Only
// then: the same error may be one that the thread had not read, which is
// returned, as after every other launch here, and is no reason to launch again.
template <class Launch>
cudaError_t checked_launch(const Launch& launch, const void* kern, size_t smem) {
  launch();
  cudaError_t e = cudaGetLastError();
  if (e == cudaErrorInvalidValue && smem > 48 * 1024 && !smem_allowed(kern, smem)) {
    const DeviceInfo* dev = current_device();
    if (!dev || raise_smem_limit(kern, *dev) != cudaSuccess) return e;
    launch();
    e = cudaGetLastError();
  }
  return e;
}

#ifdef __CUDACC__
// Launch of a kernel that resident_blocks() has seen.
template <class... P, class... A>
cudaError_t launch_kernel(void (*kern)(P...), unsigned grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  return checked_launch([&] { kern<<<grid, threads, smem, stream>>>(args...); }, reinterpret_cast<const void*>(kern), smem);
}
#endif

// Launch-shape tunables (tridi_set_tunable); 0 means "choose automatically".
int tunable(int key);

// Set, on the calling thread, while a host-pointer launcher runs its kernels
// on host memory that the device maps (pinned, mapped arrays): the launches
// then read their inputs with plain loads, never with bulk or tensor copies.
extern thread_local bool g_host_mapped_io;

// Table written by the autotuner (tridi_autotune): per table (TRIDI_AUTOTUNE_*)
// and key (log2 of the system size, or of the size bucket), the chosen value;
// 0 where nothing was tuned.
int tuned(int table, int log2key);
// Ragged plans: the largest padded row count a warp or team item may hold
// (larger systems always take a whole CTA, whatever the threads table says).
long ragged_team_max_rows();
// PCR-then-Thomas in registers (pcr_thomas2.cu): whether it takes an FP32
// call, and the launch.
bool pcr_thomas2_applies(const void* a, const void* b, const void* c, const void* d, int n, long m, int g);
tridi_status pcr_thomas2_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n,
                               int m, int g, cudaStream_t stream);
// PCR (g >= n/2) and PCR-then-Thomas at 2048 and 4096 unknowns (pcr_wide.cu).
bool pcr_wide_applies(const void* a, const void* b, const void* c, const void* d, int n, long m, int g);
tridi_status pcr_wide_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                            int g, cudaStream_t stream);
// cr and crpcr at every switch level for 512 and 1024 unknowns, in registers
// (crpcr2.cu); stride = n / rest.
bool crpcr_regs_applies(const void* a, const void* b, const void* c, const void* d, const void* x, int n, long m,
                        int stride);
tridi_status crpcr_regs_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n,
                              int m, int stride, cudaStream_t stream);

// cr and crpcr for 2048 and 4096 unknowns in registers (crpcr_wide.cu).
bool crpcr_wide_applies(const void* a, const void* b, const void* c, const void* d, const void* x, int n, long m,
                        int stride);
tridi_status crpcr_wide_solve(const float* a, const float* b, const float* c, const float* d, float* x, int n, int m,
                              int stride, cudaStream_t stream);
// cr, pcr and crpcr at every switch level in FP64 (cr64.cu); stride = n / rest.
tridi_status cr64_solve(const double* a, const double* b, const double* c, const double* d, double* x, int n, int m,
                        int stride, cudaStream_t stream);
// The any-size solve in FP64 (cr64.cu).
tridi_status cr64_solve_any(const double* a, const double* b, const double* c, const double* d, double* x, int n, int m,
                            cudaStream_t stream);

inline int ilog2(long v) {
  int k = 0;
  while (v > 1) {
    v >>= 1;
    ++k;
  }
  return k;
}

// Pipeline depth for a tiled kernel: the tunable if set, else `fallback`,
// reduced until the shared memory fits the device.
int pick_stages(size_t fixed_bytes, size_t stage_bytes, int fallback, const DeviceInfo& dev);

// A 2-D FP32 tensor map for cp.async.bulk.tensor: `outer` rows of `inner`
// elements, consecutive rows `row_bytes` apart, copied in boxes of
// box_inner x box_outer elements; swizzle128 selects the 128-byte swizzle
// (16-byte chunk c of box row r lands at chunk c ^ (r mod 8); the shared
// destination must then be 1024-byte aligned).  Out-of-range box elements
// read as zero.  False if the driver's encoder is unavailable or refuses the
// arguments.
bool make_tensor_map_2d(CUtensorMap* map, const float* base, uint64_t inner, uint64_t outer, uint64_t row_bytes,
                        uint32_t box_inner, uint32_t box_outer, bool swizzle128);

// Largest system the uniform partition solver (tridi_solve_*) takes: 512
// threads of 17 rows (FP32) or 9 rows (FP64) each.
template <class T>
constexpr long partition_max_rows() {
  return sizeof(T) == 4 ? 512L * 17 : 512L * 9;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool is_pow2(long v) { return v > 0 && (v & (v - 1)) == 0; }

}  // namespace tridi
