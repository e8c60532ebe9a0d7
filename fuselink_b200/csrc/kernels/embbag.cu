// DLRM sparse side, table-wise sharded: embedding-bag sum pooling fused with the pooled-embedding
// all-to-all (forward) and its mirror fused with the sparse SGD update (backward).
//
//   forward : the GPU that owns table t pools the rows of every sample b of the GLOBAL batch and stores
//             the pooled vector straight into the sample owner's [B_local, T_total, D] buffer over NVLink.
//             No [B_global, T_local, D] send buffer and no separate all-to-all exist.
//   backward: the table owner reads d(pooled)[b, t, :] from the sample owner's gradient buffer over
//             NVLink and applies  W[idx] -= lr * g  for every index of the bag with vector reductions.
//
// One warp handles one (table, sample) bag; D = 32 * 4 * VEC floats (D = 128 -> one float4 per lane).
// Reference parity: the reference runs this workload through an external DLRM checkout
// (.gitmodules:5-7) that uses a framework EmbeddingBag followed by an NCCL all-to-all.
#include "embbag.cuh"
#include <stdlib.h>
#include "../common/fl_ptx.cuh"

namespace fl {

__device__ __forceinline__ float4 ld_f4(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_f4_coherent(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_f4(float* p, float4 v) {
  asm volatile("st.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void red_add_f4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}

// grid: persistent; each warp walks bags  w, w + nwarps, ...   bag id = t_local * B_global + b
// Bound by the latency of rows that are anywhere in memory: what counts is how many are on the way.  Rows are requested EB_ROWS
// at a time (32 warps of 64 registers per SM, 160 KB on the way) and the next bag's indices before this bag's rows.  With a
// bag's 20 rows at once, 16 warps per SM and the indices waited for first, 26 tables x 65536 bags of 20 took 2276 us (DRAM at
// 28 % of its peak, L2 at 21 %); with 32 warps 1950 us, its issue slots 65 % busy: indices broadcast as 64 bits, addresses from 64-bit
// products, every row behind a select.  Now 1169 us: 32-bit places, and no selects for batches of good indices.
constexpr int EB_ROWS = 10;

template <typename Place>     // of a row in its table, in units of 16 bytes: 32 bits, or 64 for tables beyond 64 GB
__global__ void __launch_bounds__(256, 4) embbag_fwd_kernel(const FlEmbBagArgs a) {
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long nbags = (long long)a.t_local * a.b_global;
  long long bag = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  long long next_idx = bag < nbags && lane < a.pooling ? a.indices[bag * a.pooling + lane] : 0;
  const Place vecs = (Place)(a.dim / 4), none = ~(Place)0;
  for (; bag < nbags; bag += nwarps) {
    const int t = (int)(bag / a.b_global);
    const int b = (int)(bag - (long long)t * a.b_global);
    // lanes load the bag's indices once, then broadcast the rows' places
    const long long my_idx = next_idx;
    const bool bad = my_idx < 0 || my_idx >= a.rows;       // bounds check: skip the access, record it
    if (bad) report(a.status, kBadIndex, 900);
    const Place my_at = bad ? none : (Place)my_idx * vecs;
    const bool all_good = __all_sync(0xffffffffu, !bad);
    next_idx = bag + nwarps < nbags && lane < a.pooling ? a.indices[(bag + nwarps) * a.pooling + lane] : 0;
    const float* table = a.weights + (long long)t * a.rows * a.dim + lane * 4;
    const int owner = b / a.b_local;
    const int bl = b - owner * a.b_local;
    float* out = reinterpret_cast<float*>(a.out_peers.p[owner]) + ((long long)bl * a.t_total + (a.t_first + t)) * a.dim + lane * 4;
    for (int c = 0; c < a.dim; c += 128) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int j0 = 0; j0 < a.pooling; j0 += EB_ROWS) {
        float4 r[EB_ROWS];
        if (all_good && j0 + EB_ROWS <= a.pooling) {
#pragma unroll
          for (int j = 0; j < EB_ROWS; ++j) r[j] = ld_f4(table + c + 4ull * (unsigned long long)__shfl_sync(0xffffffffu, my_at, j0 + j));
        } else {
#pragma unroll
          for (int j = 0; j < EB_ROWS; ++j) {
            const Place at = __shfl_sync(0xffffffffu, my_at, (j0 + j) & 31);
            r[j] = (j0 + j < a.pooling && at != none) ? ld_f4(table + c + 4ull * (unsigned long long)at) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
#pragma unroll
        for (int j = 0; j < EB_ROWS; ++j) {
          acc.x += r[j].x; acc.y += r[j].y; acc.z += r[j].z; acc.w += r[j].w;
        }
      }
      st_f4(out + c, acc);
    }
  }
}

template <int MAXL>
__global__ void __launch_bounds__(256) embbag_bwd_kernel(const FlEmbBagArgs a) {
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long nbags = (long long)a.t_local * a.b_global;
  const int vec_per_lane = a.dim / 128;
  for (long long bag = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); bag < nbags; bag += nwarps) {
    const int t = (int)(bag / a.b_global);
    const int b = (int)(bag - (long long)t * a.b_global);
    const long long* idx = a.indices + bag * a.pooling;
    long long my_idx = -1;
    if (lane < a.pooling) {
      my_idx = idx[lane];
      if (my_idx < 0 || my_idx >= a.rows) {
        report(a.status, kBadIndex, 901);
        my_idx = -1;
      }
    }
    float* table = a.weights_rw + (long long)t * a.rows * a.dim;
    const int owner = b / a.b_local;
    const int bl = b - owner * a.b_local;
    const float* g = reinterpret_cast<const float*>(a.out_peers.p[owner]) +
                     ((long long)bl * a.t_total + (a.t_first + t)) * a.dim;
    for (int v = 0; v < vec_per_lane; ++v) {
      float4 gv = ld_f4_coherent(g + v * 128 + lane * 4);  // peer memory written this step: no .nc
      gv.x *= -a.lr; gv.y *= -a.lr; gv.z *= -a.lr; gv.w *= -a.lr;
#pragma unroll
      for (int j = 0; j < MAXL; ++j) {
        const long long ij = __shfl_sync(0xffffffffu, my_idx, j);
        if (j < a.pooling && ij >= 0) red_add_f4(table + ij * a.dim + v * 128 + lane * 4, gv);
      }
    }
  }
}

// Backward with accumulators for the first `hot` rows of the table.  With ids ordered by frequency a handful of rows take a
// large share of all updates (Zipf(1.05) over 1M rows: the first 24 rows get 30 %, row 0 alone 7 %), and every one of them is a
// vector reduction on the same few L2 lines, one after the other.  Here a CTA works on ONE table (blockIdx.y), and each warp
// sums the updates of those rows in shared memory of its own, which takes no atomics; a row is sent to global memory once per
// warp, at the end.  The next bag's indices and gradient are fetched a bag ahead, and a bag's updates of other rows leave one
// after the other before its hot ones.  26 tables x 65536 bags of 20: 5177 us without accumulators, 3785 us with 64 rows shared
// by eight warps (atomics on shared memory are compare-and-swap loops, and the warps retry against each other on the hottest
// rows); here 3370 us with 8 rows, 3122 with 16, 3021 with 24 (48 KB, 16 warps per SM).
constexpr int EB_WARPS = 4;

__global__ void __launch_bounds__(EB_WARPS * 32) embbag_bwd_hot_kernel(const FlEmbBagArgs a, const int hot) {
  extern __shared__ __align__(16) float hot_acc[];            // [warp][hot][dim]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.y;
  float* acc = hot_acc + warp * hot * a.dim;
  for (int i = lane * 4; i < hot * a.dim; i += 128) *reinterpret_cast<float4*>(acc + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  float* table = a.weights_rw + (long long)t * a.rows * a.dim;
  const long long* indices = a.indices + (long long)t * a.b_global * a.pooling;
  auto grad_at = [&](int b) -> const float* {
    const int owner = b / a.b_local, bl = b - owner * a.b_local;
    return reinterpret_cast<const float*>(a.out_peers.p[owner]) + ((long long)bl * a.t_total + (a.t_first + t)) * a.dim + lane * 4;
  };
  const int nwarps = gridDim.x * EB_WARPS;
  int b = blockIdx.x * EB_WARPS + warp;
  long long next_idx = b < a.b_global && lane < a.pooling ? indices[(long long)b * a.pooling + lane] : 0;
  float4 next_g = b < a.b_global ? ld_f4_coherent(grad_at(b)) : make_float4(0.f, 0.f, 0.f, 0.f);   // peers wrote it this step: no .nc
  while (b < a.b_global) {
    const long long my_idx = next_idx;
    float4 gv = next_g;
    const int nb = a.b_global - b > nwarps ? b + nwarps : a.b_global;
    if (nb < a.b_global) {
      next_idx = lane < a.pooling ? indices[(long long)nb * a.pooling + lane] : 0;
      next_g = ld_f4_coherent(grad_at(nb));
    }
    const bool bad = my_idx < 0 || my_idx >= a.rows;
    if (bad) report(a.status, kBadIndex, 902);
    const bool mine = lane < a.pooling && !bad;
    const unsigned cold = __ballot_sync(0xffffffffu, mine && my_idx >= hot), warm = __ballot_sync(0xffffffffu, mine && my_idx < hot);
    for (int c = 0; c < a.dim; c += 128) {
      if (c) gv = ld_f4_coherent(grad_at(b) + c);
      gv.x *= -a.lr; gv.y *= -a.lr; gv.z *= -a.lr; gv.w *= -a.lr;
      for (unsigned m = cold; m; m &= m - 1)
        red_add_f4(table + __shfl_sync(0xffffffffu, my_idx, __ffs(m) - 1) * a.dim + c + lane * 4, gv);
      for (unsigned m = warm; m; m &= m - 1) {
        float4* s = reinterpret_cast<float4*>(acc + __shfl_sync(0xffffffffu, (int)my_idx, __ffs(m) - 1) * a.dim + c + lane * 4);
        float4 x = *s;
        x.x += gv.x; x.y += gv.y; x.z += gv.z; x.w += gv.w;
        *s = x;
      }
    }
    b = nb;
  }
  for (int r = 0; r < hot; ++r)
    for (int c = lane * 4; c < a.dim; c += 128) {
      const float4 x = *reinterpret_cast<const float4*>(acc + r * a.dim + c);
      const bool nz = x.x != 0.f || x.y != 0.f || x.z != 0.f || x.w != 0.f;
      if (__any_sync(0xffffffffu, nz)) red_add_f4(table + (long long)r * a.dim + c, x);
    }
}

}  // namespace fl

static int check(const FlEmbBagArgs* a) {
  if (a->dim <= 0 || a->dim % 128) return -1;   // one float4 per lane per 128 columns
  if (a->pooling < 1 || a->pooling > 32) return -2;
  if (a->b_local <= 0 || a->b_global % a->b_local) return -3;
  if (a->b_global / a->b_local > 8) return -4;
  return 0;
}

extern "C" int fl_embbag_a2a_fwd(const FlEmbBagArgs* a, int num_ctas, cudaStream_t stream) {
  int rc = check(a);
  if (rc) return rc;
  if (num_ctas <= 0) num_ctas = 148 * 8;
  if ((unsigned long long)a->rows * (a->dim / 4) < 0xffffffffull) fl::embbag_fwd_kernel<unsigned><<<num_ctas, 256, 0, stream>>>(*a);
  else fl::embbag_fwd_kernel<unsigned long long><<<num_ctas, 256, 0, stream>>>(*a);
  return (int)cudaGetLastError();
}

extern "C" int fl_embbag_hot_rows(int asked, long long rows, int dim) {
  const long long fit = 48 * 1024 / ((long long)dim * sizeof(float) * fl::EB_WARPS);     // the default shared-memory limit
  const long long hot = asked < rows ? asked : rows;
  return (int)(hot < fit ? hot : fit);
}

extern "C" int fl_embbag_a2a_bwd_sgd(const FlEmbBagArgs* a, int num_ctas, cudaStream_t stream) {
  int rc = check(a);
  if (rc) return rc;
  if (num_ctas <= 0) num_ctas = 148 * 8;
  int hot = a->hot_rows;
  if (hot == 0) {
    static int dflt = -2;
    if (dflt == -2) { const char* e = getenv("FUSELINK_EMBBAG_HOT_ROWS"); dflt = e ? atoi(e) : 24; }
    hot = dflt;
  }
  hot = fl_embbag_hot_rows(hot, a->rows, a->dim);
  if (hot > 0 && a->t_local > 0) {
    // at least about 8 bags per warp: below that its accumulator is cleared and flushed for a handful of updates
    const int most = (a->b_global + 8 * fl::EB_WARPS - 1) / (8 * fl::EB_WARPS), want = 2 * num_ctas / a->t_local;
    dim3 grid(want < 1 ? 1 : want < most ? want : most, a->t_local);
    fl::embbag_bwd_hot_kernel<<<grid, fl::EB_WARPS * 32, (size_t)hot * a->dim * sizeof(float) * fl::EB_WARPS, stream>>>(*a, hot);
    return (int)cudaGetLastError();
  }
  if (a->pooling <= 20) fl::embbag_bwd_kernel<20><<<num_ctas, 256, 0, stream>>>(*a);
  else fl::embbag_bwd_kernel<32><<<num_ctas, 256, 0, stream>>>(*a);
  return (int)cudaGetLastError();
}
