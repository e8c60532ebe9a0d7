// Products of a few rows with a large matrix (see thin_gemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "decoder.cuh"

// What becomes of the sums.  The first three are FlDecAct's; every intermediate value is rounded to the type, as separate
// operations would round it.
enum FlThinEpi : int {
  FL_THIN_SILU_GATED = 0,   // w [2 n, k]: gate rows, then up rows; y [rows, n] = silu(gate) * up; takes no bias
  FL_THIN_RELU = 1,         // relu(x w^T + bias)
  FL_THIN_GELU_TANH = 2,    // gelu(x w^T + bias), tanh form
  FL_THIN_STORE = 3,        // x w^T + bias
  FL_THIN_QKV = 4,          // fl_thin_qkv's
};

constexpr int FL_THIN_MAX_ROWS = 16;

// y [rows, n] = f(x [rows, k] w [n, k]^T + bias), rows 1 .. FL_THIN_MAX_ROWS, k a multiple of 8; x, w and y contiguous, of one type
// (FlDecDtype), x and w from a multiple of 16 bytes on, y from a multiple of 4.
// early: the kernel starts while the one before it in the stream still runs and reads w ahead of its end.  For callers who know
// that w was complete before that kernel started.
// status: FL_DEC_STALLED is written there (null: nowhere) if the kernel gave up waiting for its operands.
// Returns 0, a cudaError, or < 0 for arguments it does not take; nothing is launched then.
#ifdef __cplusplus
extern "C"
#endif
int fl_thin_gemm(int dtype, const void* x, int rows, const void* w, long long n, int k, const void* bias, int epilogue, void* y, int early,
                 int* status, cudaStream_t stream);

// The product of a decoding step whose sums are queries, keys and values: bias, rotation and page write as fl_dec_qkv does them behind
// it.  y [rows, n], n = (heads + 2 kv.heads) * dim: the queries; keys and values go to their pages, what y has there is unwritten.
struct FlThinQkv {
  const float* rope; long long rope_rows;   // from a multiple of 16 bytes on; null: no rotation
  const long long* pos;                     // [rows]
  int heads, dim;                           // dim divides 128
  FlPagedKv kv;
};
#ifdef __cplusplus
extern "C"
#endif
int fl_thin_qkv(int dtype, const void* x, int rows, const void* w, long long n, int k, const void* bias, const FlThinQkv* qkv, void* y, int early,
                int* status, cudaStream_t stream);
