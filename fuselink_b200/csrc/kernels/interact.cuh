// Pairwise-dot feature interaction of a recommendation model, forward and backward (see interact.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

struct FlInteractArgs {
  const float* x;         // [batch, dim]: vector 0 of every sample (the dense features' vector)
  const float* pooled;    // [batch, vectors - 1, dim]: the other vectors
  long long batch;
  int vectors;            // 2 .. 28
  int dim;                // a multiple of 128
  // forward: [batch, ld]: x, then z_i . z_j for all i < j (row by row), then zeros up to ld; backward: the gradient of that
  float* out;
  const float* dout;
  long long ld;           // >= dim + vectors * (vectors - 1) / 2, a multiple of 4
  float* dx;              // backward: [batch, dim]
  float* dpooled;         // backward: [batch, vectors - 1, dim], times `scale`
  float scale;
};

#ifdef __cplusplus
extern "C" {
#endif
// the products have tf32 inputs (to nearest) and fp32 sums
int fl_interact_fwd(const FlInteractArgs* a, cudaStream_t stream);
int fl_interact_bwd(const FlInteractArgs* a, cudaStream_t stream);
#ifdef __cplusplus
}
#endif
