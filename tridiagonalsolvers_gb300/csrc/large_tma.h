// The TMA-tiled passes of the interleaved large systems (large_tma.cu) and
// what the refinement has them do beside the solve.
#pragma once
#include <cuda_runtime.h>

#include "tridi.h"

namespace tridi {

// What the back pass does with a chunk's unknowns.
enum { kBackPlain = 0, kBackFirst = 1, kBackSecond = 2 };

// A solve that is a sweep of the refinement (double-float residual).
// kBackFirst: x is the first solution (FP32); r, rr and dd are written, and r's
// share of the separator system.  kBackSecond: the solve is of the correction
// to e0, with the separator system that kBackFirst left in the workspace (the
// next call on it); x receives e0 + correction in FP64, rr the squares of
// d - T x.  rr and dd are added to.
struct LargeFused {
  int mode;
  const float* d;   // kBackSecond
  const float* e0;  // kBackSecond
  double* x;        // kBackSecond
  float* r;         // kBackFirst
  double* rr;
  double* dd;       // kBackFirst
};

bool large_tma_ok(const float* a, const float* b, const float* c, const float* d, long n, long m);
tridi_status large_tma_reduce(const float* a, const float* b, const float* c, const float* d, long n, long m, long P,
                              long PMp, float* red, float* bnd, cudaStream_t st);
tridi_status large_tma_back(const float* a, const float* b, const float* c, const float* d, long n, long m,
                            const float* sol, float* x, const LargeFused* f, float* red_d, float* bnd,
                            cudaStream_t st);
// Systems of at most kColRows<float> rows (large_tma_ok() holds) in one kernel.
tridi_status large_columns(const float* a, const float* b, const float* c, const float* d, long n, long m, float* x,
                           cudaStream_t st);

// Whether a solve of this interleaved system takes the TMA passes (and so can
// be fused with a sweep).
bool large_fusable(const float* a, const float* b, const float* c, const float* d, long n, long m);
// The interleaved solve with the sweep f in its back pass (large_fusable()
// holds); x: kBackFirst's solution, unused by kBackSecond.
tridi_status large_solve_fused(const float* a, const float* b, const float* c, const float* rhs, float* x, long n,
                               long m, void* ws, size_t ws_bytes, const LargeFused& f, tridi_stream_t stream);

}  // namespace tridi
