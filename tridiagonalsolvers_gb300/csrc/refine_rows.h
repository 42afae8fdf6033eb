// One-correction refinement of contiguous systems in one kernel
// (refine_rows.cu).
#pragma once
#include <cuda_runtime.h>

#include "tridi.h"

namespace tridi {

// Contiguous systems of at most 8704 rows.
bool refine_rows_applies(long n, long m);
// x = x0 + e (FP64) with e the correction of the FP32 solution x0; rel2[0],
// rel2[1] (device): the maxima over systems of ||d - T x||^2 / ||d||^2 before
// and after the correction.
tridi_status refine_rows_device(const float* a, const float* b, const float* c, const float* d, double* x, int n, int m,
                                double* rel2, cudaStream_t stream);

}  // namespace tridi
