// FP32 products on the tensor cores in BF16 pieces (msq_gemm_sliced.cu).
// Internal.
#pragma once

#include "msq_internal.cuh"

namespace msq {

// True if the FP32 reconstruction and correction of the batch's larger
// matrices, those that slicedMatrix accepts, run as sliced products.
bool slicedProducts(const DeviceBatch *b);
bool slicedMatrix(int n);
// Bytes of the pieces of a matrix's four operands, and how many of them are kept
// at a time: a batch with more runs in several passes over one arena (152 of
// order 512 have 0.95 GB).
int64_t slicedBytes(int n);
constexpr int64_t kSlicedBytes = int64_t{2} << 30;
// The functions below do those matrices only, and may return kNoScratch.
// X = F^T F.
int slicedReconstruct(msq_ctx *ctx, const DeviceBatch *b, const float *f, float *x);
// E of one Sylvester sweep, G = R^T V, C = (V^T G) o H, E = V C V^T.
// basis_packed: the pieces of V are still those of the previous call on the
// same V and batch.
int slicedSylvester(msq_ctx *ctx, const DeviceBatch *b, const float *v, const float *lam,
                    const float *r, float *ws, float *e, bool basis_packed);

}  // namespace msq
