// The passes of a decoder layer between its matrix products, one launch each.
//
// Written as separate framework operations these passes were half of a prefill's time (16 x 2048 tokens of an 8B model:
// 300 of 590 ms in elementwise kernels, every one of them a trip through memory) and nearly all of a decoding step's
// launches (72 kernels per layer, of which four are matrix products, at 1 to 4 us each whatever they do).  Here a layer is
// norm | QKV product | bias + rotation + page write | attention | output product | residual + norm | MLP products and
// activation.  Intermediate values are rounded to the model's type at the same places as in the operation-by-operation
// formulation (models/llama.py), so the two agree to the rounding of the attention itself.
//
// Reference parity: the reference's serving experiment links an external engine for all of this
// (experiments/serving/model.hh:165-177).
#include "decoder.cuh"
#include "kv_pack.cuh"
#include "thin_gemm.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>
#include <type_traits>
#include <initializer_list>
#include "../common/fl_ptx.cuh"
#include "tile_map.cuh"

namespace fl {

template <typename T> struct Num;
template <> struct Num<__nv_bfloat16> {
  using two = __nv_bfloat162;
  static __device__ __forceinline__ float2 f2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<two*>(&w)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    two h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float round(float a) { return __bfloat162float(__float2bfloat16_rn(a)); }
  static __device__ __forceinline__ float f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    [[maybe_unused]] float d2, d3;   // rows 8..15 of the tile: zero in, not used
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%9,%9};"
                 : "+f"(c[0]), "+f"(c[1]), "=f"(d2), "=f"(d3)
                 : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
  }
};
template <> struct Num<__half> {
  using two = __half2;
  static __device__ __forceinline__ float2 f2(uint32_t w) { return __half22float2(*reinterpret_cast<two*>(&w)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    two h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float round(float a) { return __half2float(__float2half_rn(a)); }
  static __device__ __forceinline__ float f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ void mma(float* c, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
    [[maybe_unused]] float d2, d3;
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%9,%9};"
                 : "+f"(c[0]), "+f"(c[1]), "=f"(d2), "=f"(d3)
                 : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
  }
};

template <typename T>
__device__ __forceinline__ void unpack8(uint4 u, float* v) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = Num<T>::f2(w[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float* v) {
  return make_uint4(Num<T>::pack(v[0], v[1]), Num<T>::pack(v[2], v[3]), Num<T>::pack(v[4], v[5]), Num<T>::pack(v[6], v[7]));
}
template <typename T>
__device__ __forceinline__ void load8(const T* p, float* v) { unpack8<T>(ld_v4(p), v); }

// An index that framework indexing would refuse: the access is skipped and the status word says which it was.  A plain store, since
// the word may be in host memory and any one of the values will do.
__device__ __forceinline__ void note(int* status, int what) {
  if (status != nullptr) *reinterpret_cast<volatile int*>(status) = what;
}

// ---- embedding --------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) dec_embed_kernel(const long long* tokens, const long long* pos, const T* embed, const T* pos_embed,
                                                        T* x, long long rows, int vecs, int seq, int offset, long long vocab,
                                                        long long pos_rows, int* status) {
  grid_dep_launch();
  const long long total = rows * vecs;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / vecs;
    const int c = (int)(i - n * vecs);
    long long tok = tokens[n];
    if (tok < 0) tok += vocab;                      // as indexing does
    uint4 u = make_uint4(0, 0, 0, 0);
    if (tok >= 0 && tok < vocab) u = ld_v4(embed + (tok * vecs + c) * 8);
    else note(status, FL_DEC_BAD_TOKEN);
    if (pos_embed != nullptr) {
      long long p = (pos ? pos[n] : n % seq) + offset;
      if (p < 0) p += pos_rows;
      if (p < 0 || p >= pos_rows) {
        note(status, FL_DEC_BAD_POSITION);
      } else {
        float a[8], b[8];
        unpack8<T>(u, a);
        load8<T>(pos_embed + (p * vecs + c) * 8, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += b[j];
        u = pack8<T>(a);
      }
    }
    st_v4(x + i * 8, u);
  }
}

// ---- residual add + norm ----------------------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum(float v, float* red, int threads) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.f;
  for (int i = 0; i < threads / 32; ++i) s += red[i];
  __syncthreads();
  return s;
}

// One CTA per row, VPT 16-byte vectors per thread, the row in registers between the two passes of the norm: x, y and w are
// read once, x and h written once.  Bound by memory in prefill, by the latency of one row in decoding; wide rows take more
// threads and not more work per thread, which is what the latency of the small case depends on.
template <typename T, int VPT>
__global__ void __launch_bounds__(1024) dec_add_norm_kernel(T* x, const T* y, const T* y_bias, const T* w, const T* b, T* h, int hidden,
                                                            float eps) {
  __shared__ float red[32];
  grid_dep_launch();
  const int vecs = hidden >> 3;
  if (gridDim.x <= FL_THIN_MAX_ROWS && threadIdx.x < vecs) {     // a step's parameters come from memory: on their way before the wait
    prefetch_l2(w + threadIdx.x * 8);
    if (b) prefetch_l2(b + threadIdx.x * 8);
    if (y_bias) prefetch_l2(y_bias + threadIdx.x * 8);
  }
  grid_dep_wait();
  const long long row = blockIdx.x;
  T* xr = x + row * hidden;
  const T* yr = y ? y + row * hidden : nullptr;
  float v[VPT][8];
  float sum = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int c = threadIdx.x + k * blockDim.x;
    if (c < vecs) {
      load8<T>(xr + c * 8, v[k]);
      if (yr) {
        float d[8];
        load8<T>(yr + c * 8, d);
        if (y_bias) {
          float e[8];
          load8<T>(y_bias + c * 8, e);
#pragma unroll
          for (int j = 0; j < 8; ++j) d[j] = Num<T>::round(d[j] + e[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) v[k][j] = Num<T>::round(v[k][j] + d[j]);
        st_v4(xr + c * 8, pack8<T>(v[k]));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[k][j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += b ? v[k][j] : v[k][j] * v[k][j];
  }
  float mean = 0.f, var = block_sum(sum, red, blockDim.x) / hidden;
  if (b) {
    mean = var;
    float s2 = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      if (threadIdx.x + k * blockDim.x < vecs) {
#pragma unroll
        for (int j = 0; j < 8; ++j) s2 += (v[k][j] - mean) * (v[k][j] - mean);
      }
    }
    var = block_sum(s2, red, blockDim.x) / hidden;
  }
  const float r = rsqrtf(var + eps);
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int c = threadIdx.x + k * blockDim.x;
    if (c < vecs) {
      float g[8];
      load8<T>(w + c * 8, g);
      if (b) {
        float e[8];
        load8<T>(b + c * 8, e);
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = (v[k][j] - mean) * r * g[j] + e[j];
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = Num<T>::round(v[k][j] * r) * g[j];
      }
      st_v4(h + row * hidden + c * 8, pack8<T>(g));
    }
  }
}

// ---- bias + rotation + page write ---------------------------------------------------------------------------------------
// A thread owns 8 columns of the first half of a head and the matching 8 of the second (the pairs the rotation mixes).
template <typename T>
__global__ void __launch_bounds__(256) dec_qkv_kernel(T* qkv, const T* bias, const float* rope, long long rope_rows, const long long* pos,
                                                      long long rows, int seq, int heads, int dim, const FlPagedKv kv) {
  grid_dep_launch();
  if (bias != nullptr && rows <= FL_THIN_MAX_ROWS) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c < (heads + 2 * kv.heads) * dim) prefetch_l2(bias + c);
  }
  grid_dep_wait();
  const int total_heads = heads + 2 * kv.heads, chunks = dim / 16, half = dim / 2;
  const int per_row = total_heads * chunks;
  const long long total = rows * per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / per_row;
    const int r = (int)(i - n * per_row);
    const int hd = r / chunks, c = (r - hd * chunks) * 8;
    T* p = qkv + (n * total_heads + hd) * dim + c;
    const bool is_q = hd < heads, is_v = hd >= heads + kv.heads;
    const bool rotate = rope != nullptr && !is_v;
    if (is_q && !rotate && bias == nullptr) continue;
    const long long at = pos ? pos[n] : n % seq;
    float a[8], b[8];
    load8<T>(p, a);
    load8<T>(p + half, b);
    if (bias) {
      float e[8];
      load8<T>(bias + hd * dim + c, e);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = Num<T>::round(a[j] + e[j]);
      load8<T>(bias + hd * dim + c + half, e);
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = Num<T>::round(b[j] + e[j]);
    }
    const long long turn = at < 0 ? -at : at;
    if (rotate && turn < rope_rows) {
      const float* cs = rope + turn * dim + c;        // row: half cosines, half sines
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float co = cs[j], si = at < 0 ? -cs[half + j] : cs[half + j], x1 = a[j], x2 = b[j];
        a[j] = x1 * co - x2 * si;
        b[j] = x2 * co + x1 * si;
      }
    }
    const uint4 lo = pack8<T>(a), hi = pack8<T>(b);
    if (rotate || bias) {
      st_v4(p, lo);
      st_v4(p + half, hi);
    }
    if (is_q) continue;
    const long long req = pos ? n : n / seq;
    const int kh = hd - heads - (is_v ? kv.heads : 0);
    const int at32 = (int)at;                         // 64-bit divisions are slow; a position beyond 32 bits is in no table
    int page = at32 / kv.block_size, slot = at32 - page * kv.block_size;
    if (slot < 0) { slot += kv.block_size; page -= 1; }
    if (page < 0) page += kv.table_stride;            // negative positions and page ids count from the end, as indexing does
    if (at32 != at || page < 0 || page >= kv.table_stride) { note(kv.status, FL_DEC_BAD_POSITION); continue; }
    int blk = kv.block_table[req * kv.table_stride + page];
    if (blk < 0) blk += kv.num_blocks;
    if (blk < 0 || blk >= kv.num_blocks) { note(kv.status, FL_DEC_BAD_PAGE); continue; }
    const long long row = kv.layout == FL_KV_BLHSD
                              ? (((long long)blk * kv.layers + kv.layer) * kv.heads + kh) * kv.block_size + slot
                              : (((long long)kv.layer * kv.num_blocks + blk) * kv.block_size + slot) * kv.heads + kh;
    T* dst = reinterpret_cast<T*>(is_v ? kv.v : kv.k) + row * dim + c;
    st_v4(dst, lo);
    st_v4(dst + half, hi);
  }
}

// ---- activation -----------------------------------------------------------------------------------------------------------
// Bound by memory, where its arithmetic lets it be: an exponential and an IEEE division per element took 573 us for 32768 x 14336 in
// bf16 (2.8 GB, 436 us at the rate of a copy), with the hardware's 443.  The result is rounded to bf16 before it is used, and of every
// bf16 gate that gives the bits of expf and an IEEE division, though __expf's error grows to some 2^-17 at |x| = 87.  fp16 has three bits
// more, behind which it shows, so fp16 keeps the others.  Both sides of the quotient are a sixteenth: __fdividef gives 0 for divisors
// beyond 2^126, which 1 + e^-x is below x = -87.3.
template <typename T>
__device__ __forceinline__ float silu_of(float x) {
  if constexpr (std::is_same_v<T, __nv_bfloat16>) return __fdividef(0.0625f * x, fmaf(__expf(-x), 0.0625f, 0.0625f));
  else return x / (1.f + expf(-x));
}

template <typename T, int KIND>
__global__ void __launch_bounds__(256) dec_act_kernel(const T* h, const T* bias, T* out, long long rows, int ffn) {
  grid_dep_launch();
  grid_dep_wait();
  const int vecs = ffn / 8;
  const long long total = rows * vecs;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / vecs;
    const int c = (int)(i - n * vecs) * 8;
    float a[8];
    if (KIND == FL_ACT_SILU_GATED) {
      float u[8];
      const T* p = h + n * 2 * ffn + c;
      unpack8<T>(ld_stream_v4(p), a);
      unpack8<T>(ld_stream_v4(p + ffn), u);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = Num<T>::round(silu_of<T>(a[j])) * u[j];
    } else {
      unpack8<T>(ld_stream_v4(h + n * ffn + c), a);
      if (bias) {
        float e[8];
        load8<T>(bias + c, e);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = Num<T>::round(a[j] + e[j]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (KIND == FL_ACT_RELU) a[j] = a[j] < 0.f ? 0.f : a[j];     // keeps NaN
        else a[j] = 0.5f * a[j] * (1.f + tanhf(0.7978845608028654f * (a[j] + 0.044715f * a[j] * a[j] * a[j])));
      }
    }
    st_v4(out + n * ffn + c, pack8<T>(a));
  }
}

// ---- attention of one new token over its pages --------------------------------------------------------------------------
// Bound by reading every cached key and value once.  A warp takes 16 tokens of one KV head at a time and reads them straight
// from the pool into the fragments of m16n8k16 products, 16 bytes per lane and load; nothing is staged in shared memory and
// no page is gathered first.  Two orders that the products do not fix make that possible: the contraction index of q.k may
// run over the head dimension in any order, so lane t of a quad takes columns 8 t .. 8 t + 7 of each 32; the output columns
// of p.v may be dealt out in any order, so lane group g takes columns 8 g .. 8 g + 7 of each 64.  The rows of a product are
// the query heads that share the KV head (8 at most per CTA; the other eight rows are zero).  The values of a step are
// requested before its scores are computed and the next step's keys right after them, so a warp always has 4 to 8 KB on the
// way.  The warps of a CTA walk different tokens; the context is cut further over the CTAs of a cluster, which merge their
// (max, sum, output) through distributed shared memory.  16 x 2048 tokens, 8 KV heads of 128: 64 us per layer with one CTA of
// eight warps per (request, head) and all of a step's loads waited for at once; now 38 us (20 us of bytes).  3 x 400 tokens, 32
// heads of 64: 7.5 us, of which 0.3 us are the looks at page ids and at sums that are not finite.
constexpr int ATT_G = 8;          // query heads per CTA

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// scores of 16 tokens: s[p][e] is token 2 t + e + 8 p of the step, -inf where bit 2 p + e of `there` is off
template <typename T, int KJ>
__device__ __forceinline__ void att_scores(const uint32_t (&qa)[KJ][4], const uint4 (&kr)[2][KJ], unsigned there, float scale_log2, float (&s)[2][2]) {
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    s[p][0] = s[p][1] = 0.f;
#pragma unroll
    for (int j = 0; j < KJ; ++j) {
      Num<T>::mma(s[p], qa[j][0], qa[j][1], kr[p][j].x, kr[p][j].y);
      Num<T>::mma(s[p], qa[j][2], qa[j][3], kr[p][j].z, kr[p][j].w);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) s[p][e] = there >> (2 * p + e) & 1 ? s[p][e] * scale_log2 : -INFINITY;
  }
}

// the step's part of the softmax and of the output; m, l: running maximum and this lane's sum
template <typename T, int VC>
__device__ __forceinline__ void att_values(float (&s)[2][2], const uint4 (&vr)[4][VC], float& m, float& l, float (&o)[VC][8][2]) {
  const float m_old = m;
  float mx = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  // A score may be -inf (an infinite key): 0 stands in for a maximum of -inf, so that a step of nothing else adds nothing.
  // One that is NaN or +inf makes the sums NaN, and NaN they stay.
  m = fmaxf(m, mx);
  const float mn = m == -INFINITY ? 0.f : m;
  const float f = exp2f(m_old - mn);
  float add = 0.f;
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      s[p][e] = exp2f(s[p][e] - mn);
      add += s[p][e];
    }
  l = l * f + add;                               // this lane's tokens only; summed over the quad at the end
  const uint32_t p0 = Num<T>::pack(s[0][0], s[0][1]), p1 = Num<T>::pack(s[1][0], s[1][1]);
#pragma unroll
  for (int c = 0; c < VC; ++c) {
    const uint32_t v0[4] = {vr[0][c].x, vr[0][c].y, vr[0][c].z, vr[0][c].w};
    const uint32_t v1[4] = {vr[1][c].x, vr[1][c].y, vr[1][c].z, vr[1][c].w};
    const uint32_t v2[4] = {vr[2][c].x, vr[2][c].y, vr[2][c].z, vr[2][c].w};
    const uint32_t v3[4] = {vr[3][c].x, vr[3][c].y, vr[3][c].z, vr[3][c].w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[c][j][0] *= f;
      o[c][j][1] *= f;
      const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
      Num<T>::mma(o[c][j], p0, p1, __byte_perm(v0[j >> 1], v1[j >> 1], sel), __byte_perm(v2[j >> 1], v3[j >> 1], sel));
    }
  }
}

template <int W> struct AttParts { float m[W][ATT_G], l[W][ATT_G], cm[ATT_G], cl[ATT_G]; };

// Merges the parts of the warps, and those of the CTAs of the cluster, into res [nh][dim].  so: W parts of [ATT_G][DP + 4] in shared
// memory, so_stride floats apart.
template <typename T, int DP, int W>
__device__ __forceinline__ void att_finish(AttParts<W>& parts, float* so, int so_stride, float m, float l, const float (&o)[DP / 64][8][2], int nh,
                                           int dim, int len, int split, int splits, T* res) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  auto part = [&](int w, int hg, int d) -> float* { return so + w * so_stride + hg * (DP + 4) + d; };
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t == 0) { parts.m[warp][g] = m; parts.l[warp][g] = l; }
#pragma unroll
  for (int c = 0; c < DP / 64; ++c)
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      *reinterpret_cast<float4*>(part(warp, g, 64 * c + 16 * t + j)) = make_float4(o[c][j][0], o[c][j + 1][0], o[c][j + 2][0], o[c][j + 3][0]);
      *reinterpret_cast<float4*>(part(warp, g, 64 * c + 16 * t + 8 + j)) = make_float4(o[c][j][1], o[c][j + 1][1], o[c][j + 2][1], o[c][j + 3][1]);
    }
  __syncthreads();
  // merge the warps: with one split this is the result, otherwise it replaces the first warp's part
  const int cells = nh * dim;
  for (int i = threadIdx.x; i < cells; i += W * 32) {
    const int hg = i / dim, d = i - hg * dim;
    float mm = -INFINITY;
#pragma unroll
    for (int x = 0; x < W; ++x) mm = fmaxf(mm, parts.m[x][hg]);
    float acc = 0.f, ll = 0.f;
#pragma unroll
    for (int x = 0; x < W; ++x) {
      const float e = parts.l[x][hg] == 0.f ? 0.f : exp2f(parts.m[x][hg] - mm);       // a part without weight; not one whose sum is NaN
      acc += e * *part(x, hg, d);
      ll += e * parts.l[x][hg];
    }
    if (splits == 1) {
      res[i] = T(len > 0 ? acc / ll : 0.f);
    } else {
      *part(0, hg, d) = acc;
      if (d == 0) { parts.cm[hg] = mm; parts.cl[hg] = ll; }
    }
  }
  if (splits == 1) return;
  cluster_sync_all();
  for (int i = split * W * 32 + threadIdx.x; i < cells; i += splits * W * 32) {
    const int hg = i / dim, d = i - hg * dim;
    const uint32_t am = smem_u32(&parts.cm[hg]), al = smem_u32(&parts.cl[hg]), ao = smem_u32(part(0, hg, d));
    float mm = -INFINITY;
    for (int x = 0; x < splits; ++x) mm = fmaxf(mm, ld_cluster_f32(map_to_cta(am, x)));
    float acc = 0.f, ll = 0.f;
    for (int x = 0; x < splits; ++x) {
      const float pm = ld_cluster_f32(map_to_cta(am, x)), pl = ld_cluster_f32(map_to_cta(al, x)), po = ld_cluster_f32(map_to_cta(ao, x));
      const float e = pl == 0.f ? 0.f : exp2f(pm - mm);      // all three on the way before the first is needed
      acc += e * po;
      ll += e * pl;
    }
    res[i] = T(len > 0 ? acc / ll : 0.f);
  }
  cluster_sync_all();                            // nobody leaves while its part is being read
}

template <typename T, int DP, int W, bool PAGE16>   // DP: head dimension rounded up to a multiple of 64; PAGE16: pages of whole 16s
__global__ void __launch_bounds__(W * 32, 16 / W) dec_attention_kernel(const T* q, long long q_stride, const long long* pos, const FlPagedKv kv,
                                                                        T* out, int heads, int dim, int group, int gparts, float scale_log2) {
  constexpr int KJ = DP / 32, VC = DP / 64;
  __shared__ AttParts<W> parts;
  __shared__ float s_o[W][ATT_G][DP + 4];
  grid_dep_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int kh = blockIdx.x / gparts, gp = blockIdx.x - kh * gparts, b = blockIdx.y, split = blockIdx.z, splits = gridDim.z;
  const int h0 = kh * group + gp * ATT_G, nh = min(ATT_G, group - gp * ATT_G);
  const int bs = kv.block_size;
  const long long cap = (long long)kv.table_stride * bs;
  const int* table = kv.block_table + (long long)b * kv.table_stride;
  const long long tok_stride = (long long)kv.heads * dim;
  if (gridDim.y <= FL_THIN_MAX_ROWS) {
    // a look ahead, before the wait for the kernel that writes q and the new token's page: the keys and values of this warp's first
    // steps (lanes 0 to 15 and 16 to 31) asked into L2; whatever it finds only says what is worth having there
    const int units = (int)((min(max(__ldcg(pos + b) + 1, 0ll), cap) + 15) / 16), nw = splits * W, w = split * W + warp;
    const int from = w * (units / nw) + min(w, units % nw), to = from + units / nw + (w < units % nw ? 1 : 0);
    for (int u = from; u < min(to, from + 4); ++u) {
      const int tok = u * 16 + (lane & 15), page = tok / bs;
      if (page < kv.table_stride) {
        int id = __ldcg(table + page);
        if (id < 0) id += kv.num_blocks;
        if (id >= 0 && id < kv.num_blocks) {
          const T* r = reinterpret_cast<const T*>(lane < 16 ? kv.k : kv.v) + (((long long)kv.layer * kv.num_blocks + id) * bs + tok % bs) * tok_stride + kh * dim;
          prefetch_l2(r);
          if (dim > 64) prefetch_l2(r + dim - 8);
        }
      }
    }
  }
  grid_dep_wait();

  // this warp's tokens: whole groups of 16, dealt out evenly over the warps of all splits
  const int len = (int)min(max(pos[b] + 1, 0ll), cap);
  const int units = (len + 15) / 16, nw = splits * W, w = split * W + warp;
  const int per = units / nw, extra = units % nw;
  const int first = (w * per + min(w, extra)) * 16;
  const int last = min(len, first + (per + (w < extra ? 1 : 0)) * 16);

  // page ids: with PAGE16 one per step, fetched a step ahead; otherwise looked up token by token
  auto page_of = [&](int base) -> int { return PAGE16 && base < last ? table[base / bs] : -1; };
  auto row_of = [&](const void* pool, int blk, int base, int tok) -> const T* {
    int slot;
    if (PAGE16) {
      slot = base % bs + (tok - base);
    } else {
      blk = tok < last ? table[tok / bs] : -1;
      slot = tok % bs;
    }
    if (blk < 0) blk += kv.num_blocks;
    if (tok >= last || blk < 0 || blk >= kv.num_blocks) return nullptr;
    return reinterpret_cast<const T*>(pool) + (((long long)kv.layer * kv.num_blocks + blk) * bs + slot) * tok_stride + kh * dim;
  };
  uint4 kr[2][KJ];
  auto load_keys = [&](int base, int blk) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const T* r = row_of(kv.k, blk, base, base + 8 * p + g);
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const int d = 32 * j + 8 * t;
        kr[p][j] = make_uint4(0, 0, 0, 0);
        if (r != nullptr && d < dim) kr[p][j] = ld_stream_v4(r + d);
      }
    }
  };
  int blk = page_of(first), blk_next = page_of(first + 16);
  load_keys(first, blk);

  uint32_t qa[KJ][4];
#pragma unroll
  for (int j = 0; j < KJ; ++j) {
    const int d = 32 * j + 8 * t;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (g < nh && d < dim) u = ld_v4(q + (long long)b * q_stride + (long long)(h0 + g) * dim + d);
    qa[j][0] = u.x; qa[j][1] = u.y; qa[j][2] = u.z; qa[j][3] = u.w;
  }
  float o[VC][8][2];
#pragma unroll
  for (int c = 0; c < VC; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) o[c][j][0] = o[c][j][1] = 0.f;
  float m = -INFINITY, l = 0.f;

  for (int base = first; base < last; base += 16) {
    uint4 vr[4][VC];
    unsigned there = 0;                            // bit 2 p + e: the token of s[p][e] is in the context and its page in the pool
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tok = base + 2 * t + (i & 1) + 8 * (i >> 1);
      const T* r = row_of(kv.v, blk, base, tok);
      if (r != nullptr) there |= 1u << i;
      else if (tok < last) note(kv.status, FL_DEC_BAD_PAGE);
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        const int d = 64 * c + 8 * g;
        vr[i][c] = make_uint4(0, 0, 0, 0);
        if (r != nullptr && d < dim) vr[i][c] = ld_stream_v4(r + d);
      }
    }
    float s[2][2];
    att_scores<T, KJ>(qa, kr, there, scale_log2, s);
    blk = blk_next;
    blk_next = page_of(base + 32);
    load_keys(base + 16, blk);
    att_values<T, VC>(s, vr, m, l, o);
  }
  att_finish<T, DP, W>(parts, &s_o[0][0][0], ATT_G * (DP + 4), m, l, o, nh, dim, len, split, splits,
                       out + (long long)b * heads * dim + (long long)h0 * dim);
}

// The same for heads of whole 64 columns in pages of whole 16 tokens, with the pages on the way through shared memory: a warp has a
// ring of its own, filled by TMA loads of 16 tokens x 64 columns (2 KB, 128-byte swizzle) that its first lane issues.  Through
// registers a warp has 4 to 8 KB on the way and waits for the values of every step; here it is three steps ahead (24 KB, of 8 warps
// per SM).  Nor does it ask for the L1 cache, which has no room beside the products' shared memory (thin_gemm.cu): next to those the
// loads through registers took 57 us a layer for 16 x 2048 tokens, 8 KV heads of 128; these take 25 (20 us of bytes).  The lanes of a
// quad take chunks 2 t and 2 t + 1 of a row's eight, so that the reads of two rows meet different banks.  Before the wait for the
// kernel that writes q and the new token's page, the first steps' pages are asked into L2.
template <int DP> struct AttRing {
  static constexpr int kHalf = 16 * 128;                       // one box: 16 tokens x 64 columns
  static constexpr int kStage = 2 * (DP / 64) * kHalf;         // keys, then values
  static constexpr int kStages = 3 * (128 / DP);
  static constexpr int kBytes = kStages * kStage;              // per warp
};

__device__ __forceinline__ void tma_prefetch_2d(const void* tmap, int x, int y) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(tmap), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

template <typename T, int DP, int W>
__global__ void __launch_bounds__(W * 32, 8 / W) dec_attention_ring_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                                                                            const T* q, long long q_stride, const long long* pos, const FlPagedKv kv,
                                                                            T* out, int heads, int group, int gparts, float scale_log2) {
  using Ring = AttRing<DP>;
  constexpr int KJ = DP / 32, VC = DP / 64, ST = Ring::kStages;
  extern __shared__ uint8_t att_smem[];
  __shared__ AttParts<W> parts;
  __shared__ uint64_t full[W][ST];
  __shared__ int abort_flag;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int kh = blockIdx.x / gparts, gp = blockIdx.x - kh * gparts, b = blockIdx.y, split = blockIdx.z, splits = gridDim.z;
  const int h0 = kh * group + gp * ATT_G, nh = min(ATT_G, group - gp * ATT_G);
  const int bs = kv.block_size;
  const long long cap = (long long)kv.table_stride * bs;
  uint8_t* rings = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(att_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* ring = rings + warp * Ring::kBytes;
  const int* table = kv.block_table + (long long)b * kv.table_stride;
  const int rows = kv.layers * kv.num_blocks * bs;               // rows of the tensor maps: a box from here on reads zeros

  if (lane == 0) {
    for (int s = 0; s < ST; ++s) mbar_init(&full[warp][s], 1);
    mbar_fence_init();
  }
  if (threadIdx.x == 0) abort_flag = 0;
  __syncthreads();
  grid_dep_launch();

  // this warp's tokens: whole groups of 16, dealt out evenly over the warps of all splits
  int len, first, last, ids;
  auto plan = [&]() {
    len = (int)min(max(__ldcg(pos + b) + 1, 0ll), cap);
    const int units = (len + 15) / 16, nw = splits * W, w = split * W + warp;
    const int per = units / nw, extra = units % nw;
    first = w * per + min(w, extra);
    last = first + per + (w < extra ? 1 : 0);
  };
  // the row of a group of 16 tokens in the pools, `rows` if its page is not there; ids: what the lanes hold of the block table
  auto page_ids = [&](int u0) { ids = u0 + lane < last ? __ldcg(table + (long long)(u0 + lane) * 16 / bs) : -1; };
  auto row_of = [&](int u, int id) -> int {
    if (id < 0) id += kv.num_blocks;
    if (id < 0 || id >= kv.num_blocks) return rows;
    return (kv.layer * kv.num_blocks + id) * bs + u * 16 % bs;
  };
  if (lane == 0) {
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  // a look ahead, before the wait: whatever it finds only says what is worth having in L2
  plan();
  page_ids(first);
  if (lane < min(last - first, 2 * ST)) {
    const int row = row_of(first + lane, ids);
    if (row < rows) {
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        tma_prefetch_2d(&tm_k, kh * DP + 64 * c, row);
        tma_prefetch_2d(&tm_v, kh * DP + 64 * c, row);
      }
    }
  }
  grid_dep_wait();
  plan();
  page_ids(first);

  int ids_at = first;                                            // lane i holds the page of unit ids_at + i
  auto fetch = [&](int u) {                                      // every lane calls it
    if (u >= ids_at + 32) { ids_at += 32; page_ids(ids_at); }
    const int id = __shfl_sync(0xffffffffu, ids, u - ids_at);
    const int row = row_of(u, id);
    if (lane == 0) {
      const int s = (u - first) % ST;
      uint8_t* dst = ring + s * Ring::kStage;
      mbar_arrive_expect_tx(&full[warp][s], Ring::kStage);
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        tma_load_2d(dst + c * Ring::kHalf, &tm_k, &full[warp][s], kh * DP + 64 * c, row);
        tma_load_2d(dst + (VC + c) * Ring::kHalf, &tm_v, &full[warp][s], kh * DP + 64 * c, row);
      }
    }
    return row < rows;
  };
  unsigned present = 0;                                          // bit s: the page in stage s is one of the pool
  for (int u = first; u < min(last, first + ST); ++u) present |= (fetch(u) ? 1u : 0u) << (u - first);

  uint32_t qa[KJ][4];
#pragma unroll
  for (int j = 0; j < KJ; ++j) {
    const int d = 64 * (j >> 1) + 16 * t + 8 * (j & 1);
    uint4 u = make_uint4(0, 0, 0, 0);
    if (g < nh) u = ld_v4(q + (long long)b * q_stride + (long long)(h0 + g) * DP + d);
    qa[j][0] = u.x; qa[j][1] = u.y; qa[j][2] = u.z; qa[j][3] = u.w;
  }
  float o[VC][8][2];
#pragma unroll
  for (int c = 0; c < VC; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) o[c][j][0] = o[c][j][1] = 0.f;
  float m = -INFINITY, l = 0.f;

  for (int u = first; u < last; ++u) {
    const int s = (u - first) % ST;
    if (!mbar_wait_warp(&full[warp][s], ((u - first) / ST) & 1, &abort_flag, nullptr, kTimeoutMbarFull, 0)) {
      note(kv.status, FL_DEC_STALLED);
      let_copies_land();                                         // before shared memory goes away
      break;
    }
    const uint32_t at = smem_u32(ring + s * Ring::kStage);
    uint4 kr[2][KJ], vr[4][VC];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int j = 0; j < KJ; ++j)
        kr[p][j] = lds_v4(at + (j >> 1) * Ring::kHalf + (8 * p + g) * 128 + (((2 * t + (j & 1)) ^ g) << 4));
    unsigned there = 0;
    const bool page = present >> s & 1;
    if (!page) note(kv.status, FL_DEC_BAD_PAGE);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tok = 2 * t + (i & 1) + 8 * (i >> 1);
      const bool in = page && u * 16 + tok < len;
      there |= (in ? 1u : 0u) << i;
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        vr[i][c] = lds_v4(at + (VC + c) * Ring::kHalf + tok * 128 + ((g ^ (tok & 7)) << 4));
        if (!in) vr[i][c] = make_uint4(0, 0, 0, 0);              // what a page holds behind the context may be anything
      }
    }
    float sc[2][2];
    att_scores<T, KJ>(qa, kr, there, scale_log2, sc);
    __syncwarp();                                                // the stage has been read
    if (u + ST < last) present = (present & ~(1u << s)) | ((fetch(u + ST) ? 1u : 0u) << s);
    att_values<T, VC>(sc, vr, m, l, o);
  }
  att_finish<T, DP, W>(parts, reinterpret_cast<float*>(rings), Ring::kBytes / 4, m, l, o, nh, DP, len, split, splits,
                       out + (long long)b * heads * DP + (long long)h0 * DP);
}

// ---- greedy choice ----------------------------------------------------------------------------------------------------------
// A cluster per row, whose CTAs take stretches of it and whose first one compares what they found.  With one CTA per row, 16 loads of
// 16 bytes per thread and their comparisons one after the other, a row of 128256 entries took 22 us.
template <typename T>
__global__ void __launch_bounds__(1024) dec_argmax_kernel(const T* logits, long long* out, long long vocab) {
  __shared__ float sv[32], cv[8];
  __shared__ long long si[32], ci[8];
  const int parts = gridDim.x, part = blockIdx.x;           // of the row; a cluster is the CTAs of one row
  if (parts > 1) cluster_sync_all();                        // all of them are there before one writes into the first
  grid_dep_launch();
  grid_dep_wait();
  const T* row = logits + blockIdx.y * vocab;
  float best = -INFINITY;
  long long at = vocab;                                   // vocab: nothing seen yet
  auto better = [](float v, long long i, float w, long long j) {      // (v, i) before (w, j)
    const bool vn = v != v, wn = w != w;
    if (vn != wn) return vn;
    if (!vn && v != w) return v > w;
    return i < j;
  };
  const bool wide = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const long long vecs = wide ? vocab / 8 : 0, first = part * (long long)blockDim.x + threadIdx.x, step = parts * (long long)blockDim.x;
  for (long long i = first; i < vecs; i += step) {
    float v[8];
    unpack8<T>(ld_stream_v4(row + i * 8), v);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (better(v[j], i * 8 + j, best, at)) { best = v[j]; at = i * 8 + j; }
  }
  for (long long i = vecs * 8 + first; i < vocab; i += step) {
    const float v = Num<T>::f(row[i]);
    if (better(v, i, best, at)) { best = v; at = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float v = __shfl_xor_sync(0xffffffffu, best, o);
    const long long i = __shfl_xor_sync(0xffffffffu, at, o);
    if (better(v, i, best, at)) { best = v; at = i; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = at; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)blockDim.x / 32; ++k)
      if (better(sv[k], si[k], best, at)) { best = sv[k]; at = si[k]; }
    if (parts == 1) {
      out[blockIdx.y] = at < vocab ? at : 0;
    } else {
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_u32(&cv[part]), 0)), "f"(best) : "memory");
      asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(map_to_cta(smem_u32(&ci[part]), 0)), "l"(at) : "memory");
    }
  }
  if (parts == 1) return;
  __syncwarp();
  cluster_sync_all();
  if (part == 0 && threadIdx.x == 0) {
    for (int k = 1; k < parts; ++k)
      if (better(cv[k], ci[k], best, at)) { best = cv[k]; at = ci[k]; }
    out[blockIdx.y] = at < vocab ? at : 0;
  }
}

__global__ void __launch_bounds__(256) dec_advance_kernel(const long long* next, long long* tokens, long long* pos, long long* history,
                                                          long long* step, int batch, int rows) {
  grid_dep_wait();
  const long long k = *step;
  for (int b = threadIdx.x; b < batch; b += blockDim.x) {
    if (k >= 0 && k < rows) history[k * batch + b] = next[b];
    tokens[b] = next[b];
    pos[b] += 1;
  }
  __syncthreads();                          // every thread has read the step
  if (threadIdx.x == 0) *step = k + 1;
}

}  // namespace fl

// --------------------------------------------------------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------------------------------------------------------
static unsigned grid_for(long long items) {
  const long long ctas = (items + 255) / 256;
  return (unsigned)(ctas < 1 ? 1 : ctas > 148ll * 64 ? 148 * 64 : ctas);
}

// every access is 16 bytes wide; a null pointer is an argument that is not given
static bool aligned(std::initializer_list<const void*> pointers) {
  uintptr_t all = 0;
  for (const void* p : pointers) all |= reinterpret_cast<uintptr_t>(p);
  return (all & 15) == 0;
}

// Whether a kernel over so many rows may start while the one before it in the stream ends (before grid_dep_wait it touches nothing that
// decides a result: the attention looks at positions and page ids, for what to ask into L2, and reads them again behind it): the launch
// itself, 2 to 3 us in a chain of kernels that take no longer, is then out of the way.  Only as far as the products are thin_gemm.cu's,
// which take part in it; between library products it costs (23 requests, 8B model: 15.1 ms without, 15.3 with).  dec_embed_kernel is
// launched without: it begins a chain, in which weights written by whatever came before are complete.
static bool chained(long long rows) { return rows <= FL_THIN_MAX_ROWS; }

template <typename... P, typename... A>
static int launch_chained(void (*kernel)(P...), long long rows, unsigned grid, unsigned threads, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained(rows) ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

#define FL_DEC_TYPES(dtype, ...)                                             \
  do {                                                                       \
    if ((dtype) == FL_DEC_BF16) { using T = __nv_bfloat16; __VA_ARGS__; }    \
    else if ((dtype) == FL_DEC_FP16) { using T = __half; __VA_ARGS__; }      \
    else return -1;                                                          \
  } while (0)

extern "C" int fl_dec_embed(int dtype, const long long* tokens, const long long* pos, const void* embed, const void* pos_embed, void* x,
                            long long rows, int hidden, int seq, int offset, long long vocab, long long pos_rows, int* status,
                            cudaStream_t stream) {
  if (hidden % 8 || hidden < 8 || rows < 0 || (pos == nullptr && pos_embed != nullptr && seq < 1)) return -2;
  if (!aligned({embed, pos_embed, x})) return -4;
  if (rows == 0) return 0;
  FL_DEC_TYPES(dtype, (fl::dec_embed_kernel<T><<<grid_for(rows * (hidden / 8)), 256, 0, stream>>>(
                          tokens, pos, (const T*)embed, (const T*)pos_embed, (T*)x, rows, hidden / 8, seq < 1 ? 1 : seq, offset, vocab, pos_rows,
                          status)));
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_add_norm(int dtype, void* x, const void* y, const void* y_bias, const void* w, const void* b, void* h, long long rows,
                               int hidden, float eps, cudaStream_t stream) {
  if (hidden % 8 || hidden < 8 || hidden > 8 * 4 * 1024 || rows < 0 || rows > 0x7fffffffll) return -2;
  if (!aligned({x, y, y_bias, w, b, h})) return -4;
  if (rows == 0) return 0;
  const int vecs = hidden / 8;
  // few rows: one vector per thread, as many threads as that takes; many rows: two per thread keeps more CTAs resident
  const int vpt = vecs > 2048 ? 4 : (vecs > 1024 || (rows > 148 && vecs > 128)) ? 2 : 1;
  const int threads = ((vecs + vpt - 1) / vpt + 31) / 32 * 32;
#define FL_NORM(V) return launch_chained(fl::dec_add_norm_kernel<T, V>, rows, (unsigned)rows, threads, stream, (T*)x, (const T*)y, (const T*)y_bias, (const T*)w, (const T*)b, (T*)h, hidden, eps)
  FL_DEC_TYPES(dtype, { if (vpt == 4) FL_NORM(4); else if (vpt == 2) FL_NORM(2); else FL_NORM(1); });
#undef FL_NORM
}

extern "C" int fl_dec_qkv(int dtype, void* qkv, const void* bias, const float* rope, long long rope_rows, const long long* pos,
                          long long rows, int seq, int heads, int dim, const FlPagedKv* kv, cudaStream_t stream) {
  if (dim % 16 || dim < 16 || heads < 1 || kv->heads < 1 || kv->block_size < 1 || rows < 0 || (pos == nullptr && seq < 1)) return -2;
  if (!aligned({qkv, bias, kv->k, kv->v})) return -4;
  if (rows == 0) return 0;
  FL_DEC_TYPES(dtype, return launch_chained(fl::dec_qkv_kernel<T>, rows, grid_for(rows * (heads + 2 * kv->heads) * (dim / 16)), 256, stream, (T*)qkv,
                                            (const T*)bias, rope, rope_rows, pos, rows, seq, heads, dim, *kv));
}

extern "C" int fl_dec_act(int dtype, int kind, const void* h, const void* bias, void* out, long long rows, int ffn, cudaStream_t stream) {
  if (ffn % 8 || ffn < 8 || rows < 0) return -2;
  if (!aligned({h, bias, out})) return -4;
  if (rows == 0) return 0;
  const unsigned grid = grid_for(rows * (ffn / 8));
#define FL_ACT(K) return launch_chained(fl::dec_act_kernel<T, K>, rows, grid, 256, stream, (const T*)h, (const T*)bias, (T*)out, rows, ffn)
  FL_DEC_TYPES(dtype, {
    if (kind == FL_ACT_SILU_GATED) FL_ACT(FL_ACT_SILU_GATED);
    else if (kind == FL_ACT_RELU) FL_ACT(FL_ACT_RELU);
    else if (kind == FL_ACT_GELU_TANH) FL_ACT(FL_ACT_GELU_TANH);
    else return -3;
  });
#undef FL_ACT
}

template <typename T, int DP, int W>
static int launch_attention(const void* q, long long q_stride, const long long* pos, const FlPagedKv* kv, void* out, int batch, int heads,
                            int dim, int group, int gparts, int splits, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kv->heads * gparts, batch, splits);
  cfg.blockDim = dim3(W * 32, 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = splits;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained(batch) ? 2 : 1;
  const float scale = 1.4426950408889634f / sqrtf((float)dim);
  auto kernel = kv->block_size % 16 == 0 ? fl::dec_attention_kernel<T, DP, W, true> : fl::dec_attention_kernel<T, DP, W, false>;
  return (int)cudaLaunchKernelEx(&cfg, kernel, (const T*)q, q_stride, pos, *kv, (T*)out, heads, dim, group, gparts, scale);
}

template <typename T, int DP, int W>
static int launch_attention_ring(const CUtensorMap& tm_k, const CUtensorMap& tm_v, const void* q, long long q_stride, const long long* pos,
                                 const FlPagedKv* kv, void* out, int batch, int heads, int group, int gparts, int splits, cudaStream_t stream) {
  constexpr int smem = W * fl::AttRing<DP>::kBytes + 1024;
  static bool set_on[64];                          // per device: a process may drive several GPUs
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return -3;
  if (!set_on[dev]) {
    e = cudaFuncSetAttribute(fl::dec_attention_ring_kernel<T, DP, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    set_on[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kv->heads * gparts, batch, splits);
  cfg.blockDim = dim3(W * 32, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = splits;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained(batch) ? 2 : 1;
  const float scale = 1.4426950408889634f / sqrtf((float)DP);
  return (int)cudaLaunchKernelEx(&cfg, fl::dec_attention_ring_kernel<T, DP, W>, tm_k, tm_v, (const T*)q, q_stride, pos, *kv, (T*)out, heads, group,
                                 gparts, scale);
}

// How the context is cut: enough CTAs for sixteen warps per SM (a warp keeps 4 to 8 KB on the way, and that many saturate
// the memory), but no warp below 32 tokens of a full context and at most 8 CTAs per cluster.  Where even that leaves SMs
// idle (a few requests with long contexts) the CTAs get eight warps instead of four.
extern "C" int fl_dec_attention(int dtype, const void* q, long long q_stride, const long long* pos, const FlPagedKv* kv, void* out,
                                int batch, int heads, int dim, cudaStream_t stream) {
  if (batch < 1 || batch > 65535 || kv->heads < 1 || heads % kv->heads || dim < 8 || dim % 8 || dim > 128 || kv->layout != FL_KV_LBSHD ||
      q_stride % 8)
    return -2;
  if (!aligned({q, kv->k, kv->v})) return -4;
  const int group = heads / kv->heads, gparts = (group + fl::ATT_G - 1) / fl::ATT_G;
  const long long units = (long long)batch * kv->heads * gparts, cap = (long long)kv->table_stride * kv->block_size;
  // Heads of 64 or 128 in pages of whole 16 tokens, of a pool whose rows 32 bits count: through the ring, two CTAs of four warps per
  // SM, if that is three steps for each of them.  Below, its start (descriptors, barriers) costs more than it hides: 3 x 400 tokens,
  // 32 heads of 64, take 13 us through it and 9 without.
  const long long rows = (long long)kv->layers * kv->num_blocks * kv->block_size;
  const bool ring = (dim == 64 || dim == 128) && kv->block_size % 16 == 0 && rows > 0 && rows < 0x7fffffffll && units * (cap / 16) >= 3 * 8 * 148;
  long long splits = (ring ? 2 : 4) * 148 / units;
  if (splits > (cap + 127) / 128) splits = (cap + 127) / 128;
  if (splits > 8) splits = 8;
  if (splits < 1) splits = 1;
  const bool wide = units * splits <= (ring ? 1 : 2) * 148 && cap >= splits * 8 * 32;
  if (ring) {
    if (dtype != FL_DEC_BF16 && dtype != FL_DEC_FP16) return -1;
    const int type = dtype == FL_DEC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap tm_k, tm_v;
    int rc = fl::tile_map(&tm_k, type, kv->k, (long long)kv->heads * dim, rows, 16);
    if (rc == 0) rc = fl::tile_map(&tm_v, type, kv->v, (long long)kv->heads * dim, rows, 16);
    if (rc != 0) return rc;
#define FL_ATT(D, W) return launch_attention_ring<T, D, W>(tm_k, tm_v, q, q_stride, pos, kv, out, batch, heads, group, gparts, (int)splits, stream)
    FL_DEC_TYPES(dtype, {
      if (dim == 64) { if (wide) FL_ATT(64, 8); else FL_ATT(64, 4); }
      else { if (wide) FL_ATT(128, 8); else FL_ATT(128, 4); }
    });
#undef FL_ATT
  }
#define FL_ATT(D, W) return launch_attention<T, D, W>(q, q_stride, pos, kv, out, batch, heads, dim, group, gparts, (int)splits, stream)
  FL_DEC_TYPES(dtype, {
    if (dim <= 64) { if (wide) FL_ATT(64, 8); else FL_ATT(64, 4); }
    else { if (wide) FL_ATT(128, 8); else FL_ATT(128, 4); }
  });
#undef FL_ATT
  return 0;
}

extern "C" int fl_dec_argmax(int dtype, const void* logits, long long* out, int rows, long long vocab, cudaStream_t stream) {
  if (rows < 0 || vocab < 1) return -2;
  if (rows == 0) return 0;
  // Eight CTAs for rows that have a vector for each of their threads, where all of them find room at once (one CTA | eight, us: 32768
  // entries, 4 rows 10.4 | 5.5, 37 rows 10.3 | 8.3; 128256, 37 rows 22.7 | 12.5, 64 rows 24.1 | 16.5; 50272, 100 rows 12.8 | 14.4).  More
  // rows than a grid's second dimension takes go in several launches.
  const int parts = vocab >= 8ll * 8 * 512 && rows <= 148 / 4 ? 8 : 1;
  for (int r = 0; r < rows; r += 65535) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(parts, rows - r < 65535 ? rows - r : 65535, 1);
    cfg.blockDim = dim3(parts > 1 ? 512 : 1024, 1, 1);
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = parts; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chained(rows) ? 2 : 1;
    int rc = 0;
    FL_DEC_TYPES(dtype, rc = (int)cudaLaunchKernelEx(&cfg, fl::dec_argmax_kernel<T>, (const T*)logits + (long long)r * vocab, out + r, vocab));
    if (rc != 0) return rc;
  }
  return 0;
}

extern "C" int fl_dec_advance(const long long* next, long long* tokens, long long* pos, long long* history, long long* step, int batch,
                              int rows, cudaStream_t stream) {
  if (batch < 1) return -2;
  return launch_chained(fl::dec_advance_kernel, batch, 1, 256, stream, next, tokens, pos, history, step, batch, rows);
}
