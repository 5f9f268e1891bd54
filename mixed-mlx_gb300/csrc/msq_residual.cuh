// The float-float residual on the tensor cores (msq_residual.cu).  Internal.
#pragma once

#include "msq_internal.cuh"

namespace msq {

// Orders from which the residual runs on the tensor cores: the first that
// takes more than one 64 x 64 tile of the CUDA-core kernel (1500 matrices of
// order 80: 424 us against 731; 2000 of order 64 take 280 on the CUDA cores,
// one tile each, and a 128 x 64 tile would be half padding).
constexpr int kResidualMmaOrder = 65;
bool residualOnTensorCores(int n);
// Bytes of a matrix's digits, and how many of them are kept at a time: a batch
// with more runs in several passes over one arena (152 of
// order 512 have 0.64 GB; three more launches per pass).
int64_t residualDigitBytes(int n);
constexpr int64_t kResidualDigits = int64_t{2} << 30;
// R = (a + a_lo) - X^T X, X = x_hi + x_lo (x_lo, a_lo and r may be null), and
// ||R||^2, ||A||^2 added to `norms` (2 per matrix), for the matrices of the
// batch whose order residualOnTensorCores accepts.  May return kNoScratch.
int residualMma(msq_ctx *ctx, const DeviceBatch *b, const float *a, const float *x_hi,
                const float *x_lo, float *r, double *norms, const float *a_lo);

}  // namespace msq
