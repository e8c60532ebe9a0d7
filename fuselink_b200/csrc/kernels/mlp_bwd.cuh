// Gradient of bias + ReLU of a linear layer (see mlp_bwd.cu).
#pragma once
#include <cuda_runtime.h>

#ifdef __cplusplus
extern "C" {
#endif
// how many rows of partial sums fl_relu_bias_bwd needs: part is [that][cols] fp32
int fl_relu_bias_parts(long long rows, int cols);
// dz = y <= 0 ? 0 : dy, db[c] = sum over the rows of dz; dy, y, dz: [rows, cols] fp32, contiguous (dz may be dy).  No alignment beyond
// the type's is asked for.  Returns 0, a cudaError or < 0 for arguments it does not take.
int fl_relu_bias_bwd(const float* dy, const float* y, float* dz, float* part, float* db, long long rows, int cols, cudaStream_t stream);
#ifdef __cplusplus
}
#endif
