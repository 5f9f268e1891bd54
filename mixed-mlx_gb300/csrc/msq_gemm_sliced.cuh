// FP32 products on the tensor cores in BF16 pieces (msq_gemm_sliced.cu).
// Internal.
#pragma once

#include "msq_internal.cuh"

namespace msq {

// True if the FP32 reconstruction and correction of the batch's larger
// matrices, those that slicedMatrix accepts, run as sliced products.
bool slicedProducts(const DeviceBatch *b);
bool slicedMatrix(int n);
// The functions below do those matrices only.  X = F^T F.
int slicedReconstruct(msq_ctx *ctx, const DeviceBatch *b, const float *f, float *x);
// E of one Sylvester sweep, G = R^T V, C = (V^T G) o H, E = V C V^T.
// basis_packed: the pieces of V are still those of the previous call on the
// same V and batch.
int slicedSylvester(msq_ctx *ctx, const DeviceBatch *b, const float *v, const float *lam,
                    const float *r, float *ws, float *e, bool basis_packed);

}  // namespace msq
