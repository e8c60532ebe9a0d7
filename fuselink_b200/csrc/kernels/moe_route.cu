// What a mixture-of-experts layer does with the router's logits: softmax, the k largest, their weights, the load-balancing
// term; and the gradient of all of it.
//
// The arrays are small (tokens x experts), so every framework operation on them is a launch and little else: 13 forward and 17
// backward, 60 and 90 us of a layer whose smallest batches take 1.2 ms in all.  Here it is one kernel each, and one that adds up
// the blocks' sums for the load-balancing term.  A token is one thread's: its probabilities stay in registers, and a block of
// 64 keeps 8192 tokens on all SMs.  Sums run in a fixed order.
//
// Reference parity: the reference's MoE workload routes in an external Megatron-DeepSpeed checkout (.gitmodules:11-13).
#include "moe_route.cuh"
#include <cuda_bf16.h>
#include <math.h>
#include "../common/fl_ptx.cuh"

namespace fl {

constexpr int RT_THREADS = 64;
constexpr int RT_TOPK = 8;

template <int E>   // at least the number of experts
__global__ void __launch_bounds__(RT_THREADS) moe_route_kernel(const FlMoeRouteArgs a) {
  __shared__ float red[RT_THREADS / 32][2][E];
  const int n = a.experts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tok = blockIdx.x * RT_THREADS + threadIdx.x;
  const bool live = tok < a.tokens;
  float p[E];
  int first = -1;
  if (live) {
    const __nv_bfloat16* l = reinterpret_cast<const __nv_bfloat16*>(a.logits) + (long long)tok * n;
    float mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      p[e] = e < n ? __bfloat162float(l[e]) + a.bias[e] : -INFINITY;
      mx = fmaxf(mx, p[e]);
    }
    float sum = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (e < n) sum += p[e] = expf(p[e] - mx);
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (e < n) a.probs[(long long)tok * n + e] = p[e] = p[e] / sum;
    float pw[RT_TOPK], total = 0.f;
    unsigned long long taken = 0;
#pragma unroll
    for (int k = 0; k < RT_TOPK; ++k) {
      if (k >= a.topk) break;
      int at = -1;
      float best = 0.f;
#pragma unroll
      for (int e = 0; e < E; ++e)      // a value that is no number counts as largest
        if (e < n && !(taken >> e & 1) && (at < 0 || p[e] > best || (p[e] != p[e] && best == best))) { best = p[e]; at = e; }
      taken |= 1ull << at;
      if (k == 0) first = at;
      pw[k] = best;
      total += best;
      a.idx[(long long)tok * a.topk + k] = at;
      a.idx64[(long long)tok * a.topk + k] = at;
    }
#pragma unroll
    for (int k = 0; k < RT_TOPK; ++k)
      if (k < a.topk) a.w[(long long)tok * a.topk + k] = pw[k] / total;
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    if (e >= n) break;
    float s = live ? p[e] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const unsigned c = __popc(__ballot_sync(0xffffffffu, first == e));
    if (lane == 0) { red[warp][0][e] = s; red[warp][1][e] = (float)c; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * n; i += RT_THREADS) {
    const int k = i / n, e = i - k * n;
    float s = 0.f;
#pragma unroll
    for (int x = 0; x < RT_THREADS / 32; ++x) s += red[x][k][e];
    a.part[(long long)blockIdx.x * 2 * n + i] = s;
  }
}

// one warp per expert
__global__ void __launch_bounds__(1024) moe_route_sum_kernel(const FlMoeRouteArgs a, int blocks) {
  __shared__ float term[64];
  const int lane = threadIdx.x & 31;
  for (int e = threadIdx.x >> 5; e < a.experts; e += blockDim.x >> 5) {
    float s = 0.f, c = 0.f;
    for (int b = lane; b < blocks; b += 32) {
      s += a.part[((long long)b * 2 + 0) * a.experts + e];
      c += a.part[((long long)b * 2 + 1) * a.experts + e];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
      const float share = c / a.tokens;
      a.share[e] = share;
      term[e] = s / a.tokens * share;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int e = 0; e < a.experts; ++e) t += term[e];
    a.aux[0] = t * a.experts;
  }
}

template <int E>
__global__ void __launch_bounds__(RT_THREADS) moe_route_bwd_kernel(const FlMoeRouteArgs a) {
  const int n = a.experts, tok = blockIdx.x * RT_THREADS + threadIdx.x;
  if (tok >= a.tokens) return;
  const float each = a.daux != nullptr ? a.daux[0] * n / a.tokens : 0.f;      // to the mean probability, and from it to each
  float p[E], d[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    p[e] = e < n ? a.probs[(long long)tok * n + e] : 0.f;
    d[e] = e < n && a.daux != nullptr ? each * a.share[e] : 0.f;
  }
  if (a.dw != nullptr) {
    const float* dw = a.dw + (long long)tok * a.topk;
    const float* w = a.w + (long long)tok * a.topk;
    float dot = 0.f, total = 0.f;
    for (int k = 0; k < a.topk; ++k) {
      dot += dw[k] * w[k];
      total += a.probs[(long long)tok * n + a.idx[(long long)tok * a.topk + k]];
    }
    for (int k = 0; k < a.topk; ++k) {
      const int at = a.idx[(long long)tok * a.topk + k];
      const float v = (dw[k] - dot) / total;
#pragma unroll
      for (int e = 0; e < E; ++e) d[e] += e == at ? v : 0.f;
    }
  }
  float dot = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) dot += p[e] * d[e];
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(a.dlogits) + (long long)tok * n;
#pragma unroll
  for (int e = 0; e < E; ++e)
    if (e < n) out[e] = __float2bfloat16_rn(p[e] * (d[e] - dot));
}

}  // namespace fl

static int rt_check(const FlMoeRouteArgs* a) {
  return a->tokens < 1 || a->experts < 1 || a->experts > 64 || a->topk < 1 || a->topk > fl::RT_TOPK || a->topk > a->experts ? -1 : 0;
}
extern "C" int fl_moe_route_blocks(int tokens) { return (tokens + fl::RT_THREADS - 1) / fl::RT_THREADS; }

extern "C" int fl_moe_route(const FlMoeRouteArgs* a, cudaStream_t stream) {
  if (rt_check(a)) return -1;
  const int blocks = fl_moe_route_blocks(a->tokens);
  if (a->experts <= 8) fl::moe_route_kernel<8><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else if (a->experts <= 16) fl::moe_route_kernel<16><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else if (a->experts <= 32) fl::moe_route_kernel<32><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else fl::moe_route_kernel<64><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  const int warps = a->experts < 32 ? a->experts : 32;
  fl::moe_route_sum_kernel<<<1, warps * 32, 0, stream>>>(*a, blocks);
  return (int)cudaGetLastError();
}

extern "C" int fl_moe_route_bwd(const FlMoeRouteArgs* a, cudaStream_t stream) {
  if (rt_check(a)) return -1;
  const int blocks = fl_moe_route_blocks(a->tokens);
  if (a->experts <= 8) fl::moe_route_bwd_kernel<8><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else if (a->experts <= 16) fl::moe_route_bwd_kernel<16><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else if (a->experts <= 32) fl::moe_route_bwd_kernel<32><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  else fl::moe_route_bwd_kernel<64><<<blocks, fl::RT_THREADS, 0, stream>>>(*a);
  return (int)cudaGetLastError();
}
