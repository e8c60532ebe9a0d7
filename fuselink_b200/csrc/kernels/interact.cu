// Feature interaction of a recommendation model: the dot products of all pairs of a sample's vectors, and their gradient.
//
// As framework operations this is a concatenation of the vectors, a batched product, a gather of its upper triangle and a
// second concatenation; the gradient of the gather sorts one index per output element, and the products have 27 rows.  At
// 65536 samples of 27 x 128 that took 1.7 ms forward and 8 ms backward (now 0.18 and 0.53 ms).  The vectors are 0.9 GB, so one
// read of them is 0.14 ms and a read and a write 0.28 ms: here both directions are one kernel that touches every vector once.
//
// The gradient's products run on the fp32 pipes, as they did as library products: 27 x 28 x 128 multiply-adds per sample are
// about 760 cycles per SM, and the memory takes about 1250 to deliver the sample.  The forward products have tf32 inputs, and
// the kernel is for callers that allow those.  The ReLUs behind it pass a gradient or not depending on the sign of values
// next to zero, so it keeps the order of the sums of the library's m16n8k8 products: the results are the library's bits (CUDA
// 12.8; tests/test_interact_gpu.py) at 4, 8, 12 and 16 to 28 vectors, which are the counts that models/dlrm.py sends here.
//
// Reference parity: the reference runs this workload through an external DLRM checkout (.gitmodules:5-7).
#include "interact.cuh"
#include "../common/fl_ptx.cuh"

namespace fl {

constexpr int IA_WARPS = 4;            // samples in flight per CTA, one per warp
constexpr int IA_COLS = 128;           // columns of the vectors handled at a time: 4 per lane
constexpr int IA_LD = IA_COLS + 4;     // floats per row in shared memory: rows r and r + 1 are 4 banks apart

__device__ __forceinline__ void cp_async16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ const float* ia_row(const FlInteractArgs& a, long long b, int i) {
  return i == 0 ? a.x + b * a.dim : a.pooled + (b * (a.vectors - 1) + i - 1) * a.dim;
}
__device__ __forceinline__ int ia_pair(int n, int i, int j) { return i * (2 * n - i - 1) / 2 + j - i - 1; }   // i < j

// tf32 inputs (rounded to nearest) and m16n8k8 products: the rows of z are both operands.  Rows are 4 banks apart, so
// the fragments' loads (lane = 4 g + t reads row g, column t) have no conflicts.  BLK: groups of 8 rows; only products of groups
// on or above the diagonal are computed.
__device__ __forceinline__ uint32_t to_tf32(float v) {
  uint32_t r;
  asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return r;
}
template <int BLK>
__global__ void __launch_bounds__(IA_WARPS * 32) interact_fwd_kernel(const FlInteractArgs a) {
  constexpr int R = 8 * BLK, MT = (BLK + 1) / 2, PAIRS = R * (R - 1) / 2;
  extern __shared__ __align__(16) float ia_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  float* z = ia_smem + warp * (R * IA_LD + PAIRS);
  float* tri = z + R * IA_LD;
  const int n = a.vectors, pairs = n * (n - 1) / 2;
  for (int e = lane; e < (R - n) * IA_LD; e += 32) z[n * IA_LD + e] = 0.f;
  for (long long b = (long long)blockIdx.x * IA_WARPS + warp; b < a.batch; b += (long long)gridDim.x * IA_WARPS) {
    float acc[MT][BLK][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int k = 0; k < BLK; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][k][e] = 0.f;
    float* out = a.out + b * a.ld;
    for (int c0 = 0; c0 < a.dim; c0 += IA_COLS) {
#pragma unroll 4
      for (int i = 0; i < n; ++i) cp_async16(z + i * IA_LD + lane * 4, ia_row(a, b, i) + c0 + lane * 4);
      cp_async_wait_all();
      __syncwarp();
      *reinterpret_cast<float4*>(out + c0 + lane * 4) = *reinterpret_cast<const float4*>(z + lane * 4);
#pragma unroll 4
      for (int k = 0; k < IA_COLS; k += 8) {
        uint32_t f[2 * MT][2];
#pragma unroll
        for (int i = 0; i < 2 * MT; ++i) {
          f[i][0] = i < BLK ? to_tf32(z[(8 * i + g) * IA_LD + k + t]) : 0u;
          f[i][1] = i < BLK ? to_tf32(z[(8 * i + g) * IA_LD + k + t + 4]) : 0u;
        }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int j = 2 * m; j < BLK; ++j)
            asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                         : "+f"(acc[m][j][0]), "+f"(acc[m][j][1]), "+f"(acc[m][j][2]), "+f"(acc[m][j][3])
                         : "r"(f[2 * m][0]), "r"(f[2 * m + 1][0]), "r"(f[2 * m][1]), "r"(f[2 * m + 1][1]), "r"(f[j][0]), "r"(f[j][1]));
      }
      __syncwarp();
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 2 * m; j < BLK; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = 16 * m + g + 8 * (e >> 1), c = 8 * j + 2 * t + (e & 1);
          if (r < c && c < n) tri[ia_pair(n, r, c)] = acc[m][j][e];
        }
    __syncwarp();
    for (int e = lane; e < a.ld - a.dim; e += 32) out[a.dim + e] = e < pairs ? tri[e] : 0.f;
    __syncwarp();
  }
}

// dz_i = sum_j S_ij z_j with S the symmetric matrix of the products' gradients (zero diagonal).  A lane owns 4 columns of every
// dz_i; the rows z_j come straight from memory, four ahead, S from shared memory (every lane reads the same 16 bytes).  65536 x
// 27 x 128: 497 us; the shared-memory loads are what bounds it (7 for 112 multiply-adds): with 2 columns per lane and twice the
// warps it takes 555 us.
template <int C>
__global__ void __launch_bounds__(IA_WARPS * 32, 3) interact_bwd_kernel(const FlInteractArgs a) {
  constexpr int R = 4 * C;
  __shared__ __align__(16) float s_all[IA_WARPS][R * R];
  __shared__ uint16_t s_at[R * (R - 1) / 2 + 1];            // where pair e goes: i * R + j
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = a.vectors, pairs = n * (n - 1) / 2, parts = a.dim / IA_COLS;
  float* S = s_all[warp];
  for (int e = threadIdx.x; e < IA_WARPS * R * R; e += blockDim.x) (&s_all[0][0])[e] = 0.f;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e - i * n;
    if (i < j) s_at[ia_pair(n, i, j)] = (uint16_t)(i * R + j);
  }
  __syncthreads();
  for (long long u = (long long)blockIdx.x * IA_WARPS + warp; u < a.batch * parts; u += (long long)gridDim.x * IA_WARPS) {
    const long long b = u / parts;
    const int c0 = (int)(u - b * parts) * IA_COLS + lane * 4;
    const float* dout = a.dout + b * a.ld;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 z[4], nz[4], acc[R];
#pragma unroll
    for (int t = 0; t < 4; ++t) z[t] = t < n ? *reinterpret_cast<const float4*>(ia_row(a, b, t) + c0) : none;
    for (int e = lane; e < pairs; e += 32) {
      const float v = dout[a.dim + e];
      const int at = s_at[e], i = at / R, j = at - i * R;
      S[at] = v;
      S[j * R + i] = v;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = none;
#pragma unroll 1
    for (int j0 = 0; j0 < R; j0 += 4) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int j = j0 + 4 + t;
        nz[t] = j < n ? *reinterpret_cast<const float4*>(ia_row(a, b, j) + c0) : none;
      }
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int i = 0; i < R; i += 4) {
          const float4 s = *reinterpret_cast<const float4*>(S + (j0 + t) * R + i);
          const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            acc[i + k].x = fmaf(sv[k], z[t].x, acc[i + k].x);
            acc[i + k].y = fmaf(sv[k], z[t].y, acc[i + k].y);
            acc[i + k].z = fmaf(sv[k], z[t].z, acc[i + k].z);
            acc[i + k].w = fmaf(sv[k], z[t].w, acc[i + k].w);
          }
        }
#pragma unroll
      for (int t = 0; t < 4; ++t) z[t] = nz[t];
    }
    const float4 d = *reinterpret_cast<const float4*>(dout + c0);      // x reaches the output directly as well
    *reinterpret_cast<float4*>(a.dx + b * a.dim + c0) = make_float4(acc[0].x + d.x, acc[0].y + d.y, acc[0].z + d.z, acc[0].w + d.w);
#pragma unroll
    for (int i = 1; i < R; ++i)
      if (i < n)
        *reinterpret_cast<float4*>(a.dpooled + (b * (n - 1) + i - 1) * a.dim + c0) =
            make_float4(acc[i].x * a.scale, acc[i].y * a.scale, acc[i].z * a.scale, acc[i].w * a.scale);
    __syncwarp();
  }
}

}  // namespace fl

static int ia_check(const FlInteractArgs* a) {
  if (a->vectors < 2 || a->vectors > 28 || a->dim < 128 || a->dim % 128 || a->batch < 0) return -1;
  if (a->ld % 4 || a->ld < a->dim + a->vectors * (a->vectors - 1) / 2) return -2;
  const uintptr_t at = (uintptr_t)a->x | (uintptr_t)a->pooled | (uintptr_t)a->out | (uintptr_t)a->dout | (uintptr_t)a->dx | (uintptr_t)a->dpooled;
  return at & 15 ? -3 : 0;
}

template <int BLK>
static int ia_launch_fwd(const FlInteractArgs* a, cudaStream_t stream) {
  constexpr int R = 8 * BLK;
  const long long ctas = (a->batch + fl::IA_WARPS - 1) / fl::IA_WARPS;
  const int smem = fl::IA_WARPS * (R * fl::IA_LD + R * (R - 1) / 2) * (int)sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(fl::interact_fwd_kernel<BLK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  fl::interact_fwd_kernel<BLK><<<(unsigned)(ctas < 148 * 12 ? ctas : 148 * 12), fl::IA_WARPS * 32, smem, stream>>>(*a);
  return (int)cudaGetLastError();
}

extern "C" int fl_interact_fwd(const FlInteractArgs* a, cudaStream_t stream) {
  const int rc = ia_check(a);
  if (rc || a->batch == 0) return rc;
  switch ((a->vectors + 7) / 8) {
    case 1: return ia_launch_fwd<1>(a, stream);
    case 2: return ia_launch_fwd<2>(a, stream);
    case 3: return ia_launch_fwd<3>(a, stream);
    default: return ia_launch_fwd<4>(a, stream);
  }
}

extern "C" int fl_interact_bwd(const FlInteractArgs* a, cudaStream_t stream) {
  const int rc = ia_check(a);
  if (rc || a->batch == 0) return rc;
  const long long ctas = (a->batch * (a->dim / fl::IA_COLS) + fl::IA_WARPS - 1) / fl::IA_WARPS;
  const unsigned grid = (unsigned)(ctas < 148 * 12 ? ctas : 148 * 12);
#define FL_IA(C) case C: fl::interact_bwd_kernel<C><<<grid, fl::IA_WARPS * 32, 0, stream>>>(*a); break
  switch ((a->vectors + 3) / 4) { FL_IA(1); FL_IA(2); FL_IA(3); FL_IA(4); FL_IA(5); FL_IA(6); FL_IA(7); }
#undef FL_IA
  return (int)cudaGetLastError();
}
