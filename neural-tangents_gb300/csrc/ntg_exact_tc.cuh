// Residuals of many right-hand sides by exact sums on the tensor cores (ntg_exact_tc.cu).
#pragma once

#include <climits>

#include "ntg_common.cuh"

namespace ntg {

// Whether n x n times n x m products are worth the digits, from 2^26 on: there the six
// launches take 71 us (n 512, m 256) and 103 us (n 1024, m 64) against 158 and 302 us of the
// double-float kernel, at 2^30 113 - 358 us against 513 - 1330. Below, the digits and the
// launches take more and more of the time.
bool exact_residual_pays(int64_t n, int64_t m);
size_t exact_residual_bytes(int64_t n, int64_t m);
// R = B (B64 when given) - (A + lambda[0] I) X, X float64, rounded to float32; rnorm receives
// max |R| (zeroed by the caller). same_a: the workspace holds A's digits from the last call.
int exact_residual(cudaStream_t s, const float* A, int64_t n, const double* lambda, const float* B,
                   const double* B64, const double* X, int64_t m, float* R, double* rnorm,
                   void* workspace, bool same_a);

}  // namespace ntg
