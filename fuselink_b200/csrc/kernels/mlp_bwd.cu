// The backward pass between two linear layers of an MLP: the ReLU's gradient and the bias gradient in one trip through memory.
//
// Bound by memory: dy and y are read once and dz is written once.  As framework operations the masked gradient is written by one
// kernel and read again by another, which sums it up at a third of the memory's rate (65536 rows, 512 + 256 + 128 + 1024 + 1024 +
// 512 + 256 columns: 386 + 557 us; here 475 + 29, 6.1 TB/s).  A warp takes 128 columns (16 bytes per lane) of four rows at a time, so
// that 16 KB per CTA are on the way; the sums stay in registers until the CTA's rows are done, and a second small kernel adds the CTAs'
// parts up, always in the same order.
#include "mlp_bwd.cuh"
#include <stdint.h>

namespace fl {

constexpr int RB_WARPS = 8, RB_ROWS = 4;
constexpr int RB_MAX_COLS = 0x7fffffff - 127;      // the columns of the last CTA still count in 32 bits

template <int VEC> struct RbVec;
template <> struct RbVec<4> { using type = float4; };
template <> struct RbVec<1> { using type = float; };

template <int VEC>
__global__ void __launch_bounds__(RB_WARPS * 32) relu_bias_bwd_kernel(const float* dy, const float* y, float* dz, float* part, long long rows, int cols) {
  using V = typename RbVec<VEC>::type;
  __shared__ float sums[RB_WARPS][32 * VEC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.x * 32 + lane) * VEC;
  float acc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) acc[e] = 0.f;
  if (c < cols) {
    const long long step = (long long)gridDim.y * RB_WARPS * RB_ROWS;
    for (long long r0 = ((long long)blockIdx.y * RB_WARPS + warp) * RB_ROWS; r0 < rows; r0 += step) {
      __align__(16) float g[RB_ROWS][VEC], a[RB_ROWS][VEC];
#pragma unroll
      for (int i = 0; i < RB_ROWS; ++i) {
        if (r0 + i < rows) {
          *reinterpret_cast<V*>(g[i]) = *reinterpret_cast<const V*>(dy + (r0 + i) * cols + c);
          *reinterpret_cast<V*>(a[i]) = *reinterpret_cast<const V*>(y + (r0 + i) * cols + c);
        }
      }
#pragma unroll
      for (int i = 0; i < RB_ROWS; ++i) {
        if (r0 + i < rows) {
#pragma unroll
          for (int e = 0; e < VEC; ++e) {
            if (a[i][e] <= 0.f) g[i][e] = 0.f;           // a NaN passes the gradient on, as the framework's ReLU does
            acc[e] += g[i][e];
          }
          *reinterpret_cast<V*>(dz + (r0 + i) * cols + c) = *reinterpret_cast<V*>(g[i]);
        }
      }
    }
  }
#pragma unroll
  for (int e = 0; e < VEC; ++e) sums[warp][lane * VEC + e] = acc[e];
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * VEC; i += RB_WARPS * 32) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < RB_WARPS; ++w) s += sums[w][i];
    const int col = blockIdx.x * 32 * VEC + i;
    if (col < cols) part[(long long)blockIdx.y * cols + col] = s;
  }
}

__global__ void __launch_bounds__(256) sum_parts_kernel(const float* part, float* db, int parts, int cols) {
  __shared__ float sums[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < cols) {
#pragma unroll 8
    for (int p = warp; p < parts; p += 8) s += part[(long long)p * cols + c];
  }
  sums[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += sums[w][lane];
    db[c] = t;
  }
}

}  // namespace fl

// about four CTAs per SM over all column blocks, but no CTA without a few rows for each of its warps
extern "C" int fl_relu_bias_parts(long long rows, int cols) {
  if (rows < 1 || cols < 1 || cols > fl::RB_MAX_COLS) return 0;
  const long long blocks = (cols + 127) / 128, most = (rows + fl::RB_WARPS * fl::RB_ROWS - 1) / (fl::RB_WARPS * fl::RB_ROWS);
  long long n = (4 * 148 + blocks - 1) / blocks;
  if (n > most) n = most;
  return (int)n;
}

extern "C" int fl_relu_bias_bwd(const float* dy, const float* y, float* dz, float* part, float* db, long long rows, int cols, cudaStream_t stream) {
  if (rows < 1 || cols < 1 || cols > fl::RB_MAX_COLS) return -1;
  const int parts = fl_relu_bias_parts(rows, cols);
  const uintptr_t at = (uintptr_t)dy | (uintptr_t)y | (uintptr_t)dz;
  if (cols % 4 == 0 && (at & 15) == 0)
    fl::relu_bias_bwd_kernel<4><<<dim3((cols + 127) / 128, parts), fl::RB_WARPS * 32, 0, stream>>>(dy, y, dz, part, rows, cols);
  else
    fl::relu_bias_bwd_kernel<1><<<dim3((cols + 31) / 32, parts), fl::RB_WARPS * 32, 0, stream>>>(dy, y, dz, part, rows, cols);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  fl::sum_parts_kernel<<<(cols + 31) / 32, 256, 0, stream>>>(part, db, parts, cols);
  return (int)cudaGetLastError();
}
