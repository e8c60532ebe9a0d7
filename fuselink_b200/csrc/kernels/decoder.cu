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
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>
#include "../common/fl_ptx.cuh"

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

// ---- embedding --------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) dec_embed_kernel(const long long* tokens, const long long* pos, const T* embed, const T* pos_embed,
                                                        T* x, long long rows, int vecs, int seq, int offset, long long vocab,
                                                        long long pos_rows) {
  const long long total = rows * vecs;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / vecs;
    const int c = (int)(i - n * vecs);
    long long tok = tokens[n];
    if (tok < 0) tok += vocab;                      // as indexing does
    uint4 u = make_uint4(0, 0, 0, 0);
    if (tok >= 0 && tok < vocab) u = ld_v4(embed + (tok * vecs + c) * 8);
    if (pos_embed != nullptr) {
      const long long p = (pos ? pos[n] : n % seq) + offset;
      if (p >= 0 && p < pos_rows) {
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
  const long long row = blockIdx.x;
  const int vecs = hidden >> 3;
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
    if (rotate && at >= 0 && at < rope_rows) {
      const float* cs = rope + at * dim + c;          // row: half cosines, half sines
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float co = cs[j], si = cs[half + j], x1 = a[j], x2 = b[j];
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
    const long long page = at / kv.block_size;
    if (at < 0 || page >= kv.table_stride) continue;
    const int slot = (int)(at - page * kv.block_size);
    const int blk = kv.block_table[req * kv.table_stride + page];
    if (blk < 0 || blk >= kv.num_blocks) continue;
    const long long row = kv.layout == FL_KV_BLHSD
                              ? (((long long)blk * kv.layers + kv.layer) * kv.heads + kh) * kv.block_size + slot
                              : (((long long)kv.layer * kv.num_blocks + blk) * kv.block_size + slot) * kv.heads + kh;
    T* dst = reinterpret_cast<T*>(is_v ? kv.v : kv.k) + row * dim + c;
    st_v4(dst, lo);
    st_v4(dst + half, hi);
  }
}

// ---- activation -----------------------------------------------------------------------------------------------------------
template <typename T, int KIND>
__global__ void __launch_bounds__(256) dec_act_kernel(const T* h, const T* bias, T* out, long long rows, int ffn) {
  const int vecs = ffn / 8;
  const long long total = rows * vecs;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / vecs;
    const int c = (int)(i - n * vecs) * 8;
    float a[8];
    if (KIND == FL_ACT_SILU_GATED) {
      float u[8];
      const T* p = h + n * 2 * ffn + c;
      unpack8<T>(ld_nc_v4(p), a);
      unpack8<T>(ld_nc_v4(p + ffn), u);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = Num<T>::round(a[j] / (1.f + expf(-a[j]))) * u[j];
    } else {
      unpack8<T>(ld_nc_v4(h + n * ffn + c), a);
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
// from the pool into the fragments of m16n8k16 products, 16 bytes per lane and load, all of a step's loads issued before its
// first product; nothing is staged in shared memory and no page is gathered first.  Two orders that the products do not fix
// make that possible: the contraction index of q.k may run over the head dimension in any order, so lane t of a quad takes
// columns 8 t .. 8 t + 7 of each 32; the output columns of p.v may be dealt out in any order, so lane group g takes columns
// 8 g .. 8 g + 7 of each 64.  The rows of a product are the query heads that share the KV head (8 at most per CTA; the other
// eight rows are zero).  The eight warps of a CTA walk different tokens and merge their (max, sum, output) in shared memory;
// where batch x KV heads leaves SMs idle the context is cut into `splits` more parts, merged by the last CTA to finish.
constexpr int ATT_WARPS = 8;
constexpr int ATT_G = 8;          // query heads per CTA

template <typename T, int DP>     // DP: head dimension rounded up to a multiple of 64
__global__ void __launch_bounds__(ATT_WARPS * 32) dec_attention_kernel(const T* q, long long q_stride, const long long* pos,
                                                                        const FlPagedKv kv, T* out, int heads, int dim, int group,
                                                                        int gparts, float scale_log2, float* ws, int* tickets) {
  constexpr int KJ = DP / 32, VC = DP / 64;
  __shared__ float s_m[ATT_WARPS][ATT_G], s_l[ATT_WARPS][ATT_G];
  __shared__ float s_o[ATT_WARPS][ATT_G][DP];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int kh = blockIdx.x / gparts, gp = blockIdx.x - kh * gparts, b = blockIdx.y, split = blockIdx.z, splits = gridDim.z;
  const int h0 = kh * group + gp * ATT_G, nh = min(ATT_G, group - gp * ATT_G);
  const int bs = kv.block_size;
  const long long cap = (long long)kv.table_stride * bs;
  const int len = (int)min(max(pos[b] + 1, 0ll), cap);
  const int* table = kv.block_table + (long long)b * kv.table_stride;

  // this warp's tokens: whole groups of 16, dealt out evenly over the warps of all splits
  const int units = (len + 15) / 16, nw = splits * ATT_WARPS, w = split * ATT_WARPS + warp;
  const int per = units / nw, extra = units % nw;
  const int first = (w * per + min(w, extra)) * 16;
  const int last = min(len, first + (per + (w < extra ? 1 : 0)) * 16);

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

  // address of token `tok`'s row of this head in the key (or value) pool, 0 if its page id is bad
  auto row_of = [&](const void* pool, int tok) -> const T* {
    const int pg = tok / bs;
    const int blk = table[pg];
    if (blk < 0 || blk >= kv.num_blocks) return nullptr;
    return reinterpret_cast<const T*>(pool) +
           ((((long long)kv.layer * kv.num_blocks + blk) * bs + (tok - pg * bs)) * kv.heads + kh) * dim;
  };

  for (int base = first; base < last; base += 16) {
    uint4 kr[2][KJ], vr[4][VC];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const int tok = base + 8 * p + g;
      const T* r = tok < last ? row_of(kv.k, tok) : nullptr;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const int d = 32 * j + 8 * t;
        kr[p][j] = make_uint4(0, 0, 0, 0);
        if (r != nullptr && d < dim) kr[p][j] = ld_nc_v4(r + d);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int tok = base + 2 * t + (i & 1) + 8 * (i >> 1);
      const T* r = tok < last ? row_of(kv.v, tok) : nullptr;
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        const int d = 64 * c + 8 * g;
        vr[i][c] = make_uint4(0, 0, 0, 0);
        if (r != nullptr && d < dim) vr[i][c] = ld_nc_v4(r + d);
      }
    }
    float s[2][2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      s[p][0] = s[p][1] = 0.f;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        Num<T>::mma(s[p], qa[j][0], qa[j][1], kr[p][j].x, kr[p][j].y);
        Num<T>::mma(s[p], qa[j][2], qa[j][3], kr[p][j].z, kr[p][j].w);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) s[p][e] = base + 8 * p + 2 * t + e < last ? s[p][e] * scale_log2 : -INFINITY;
    }
    float mx = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);               // finite: at least one token of the step is in range
    const float f = exp2f(m - mn);
    m = mn;
    float add = 0.f;
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[p][e] = exp2f(s[p][e] - mn);
        add += s[p][e];
      }
    l = l * f + add;                             // this lane's tokens only; summed over the quad at the end
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
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (t == 0) { s_m[warp][g] = m; s_l[warp][g] = l; }
#pragma unroll
  for (int c = 0; c < VC; ++c)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s_o[warp][g][64 * c + 16 * t + j] = o[c][j][0];
      s_o[warp][g][64 * c + 16 * t + 8 + j] = o[c][j][1];
    }
  __syncthreads();
  // merge the warps; with one split this is the result
  const int cells = nh * dim;
  const long long unit = ((long long)b * gridDim.x + blockIdx.x);
  float* part = ws + (unit * splits + split) * (ATT_G * (DP + 2));
  for (int i = threadIdx.x; i < cells; i += blockDim.x) {
    const int hg = i / dim, d = i - hg * dim;
    float mm = -INFINITY;
#pragma unroll
    for (int x = 0; x < ATT_WARPS; ++x) mm = fmaxf(mm, s_m[x][hg]);
    float acc = 0.f, ll = 0.f;
#pragma unroll
    for (int x = 0; x < ATT_WARPS; ++x) {
      const float e = s_m[x][hg] == -INFINITY ? 0.f : exp2f(s_m[x][hg] - mm);
      acc += e * s_o[x][hg][d];
      ll += e * s_l[x][hg];
    }
    if (splits == 1) {
      out[(long long)b * heads * dim + (long long)(h0 + hg) * dim + d] = T(ll > 0.f ? acc / ll : 0.f);
    } else {
      part[hg * (DP + 2) + d] = acc;
      if (d == 0) { part[hg * (DP + 2) + DP] = mm; part[hg * (DP + 2) + DP + 1] = ll; }
    }
  }
  if (splits == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(tickets + unit, 1) == splits - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const float* all = ws + unit * splits * (ATT_G * (DP + 2));
  for (int i = threadIdx.x; i < cells; i += blockDim.x) {
    const int hg = i / dim, d = i - hg * dim;
    float mm = -INFINITY;
    for (int x = 0; x < splits; ++x) mm = fmaxf(mm, __ldcg(all + (x * ATT_G + hg) * (DP + 2) + DP));
    float acc = 0.f, ll = 0.f;
    for (int x = 0; x < splits; ++x) {
      const float* r = all + (x * ATT_G + hg) * (DP + 2);
      const float pm = __ldcg(r + DP), e = pm == -INFINITY ? 0.f : exp2f(pm - mm);
      acc += e * __ldcg(r + d);
      ll += e * __ldcg(r + DP + 1);
    }
    out[(long long)b * heads * dim + (long long)(h0 + hg) * dim + d] = T(ll > 0.f ? acc / ll : 0.f);
  }
  if (threadIdx.x == 0) tickets[unit] = 0;
}

// ---- greedy choice ----------------------------------------------------------------------------------------------------------
// One CTA per row; a vocabulary row (256 KB at 128256 entries) is 16 loads of 16 bytes per thread, read once.
template <typename T>
__global__ void __launch_bounds__(1024) dec_argmax_kernel(const T* logits, long long* out, long long vocab) {
  __shared__ float sv[32];
  __shared__ long long si[32];
  const T* row = logits + blockIdx.x * vocab;
  float best = -INFINITY;
  long long at = vocab;                                   // vocab: nothing seen yet
  auto better = [](float v, long long i, float w, long long j) {      // (v, i) before (w, j)
    const bool vn = v != v, wn = w != w;
    if (vn != wn) return vn;
    if (!vn && v != w) return v > w;
    return i < j;
  };
  const bool wide = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  const long long vecs = wide ? vocab / 8 : 0;
  for (long long i = threadIdx.x; i < vecs; i += blockDim.x) {
    float v[8];
    unpack8<T>(ld_nc_v4(row + i * 8), v);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (better(v[j], i * 8 + j, best, at)) { best = v[j]; at = i * 8 + j; }
  }
  for (long long i = vecs * 8 + threadIdx.x; i < vocab; i += blockDim.x) {
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
    out[blockIdx.x] = at < vocab ? at : 0;
  }
}

__global__ void dec_advance_kernel(const long long* next, long long* tokens, long long* pos, long long* history, long long pos0, int batch,
                                   int steps) {
  for (int b = threadIdx.x; b < batch; b += blockDim.x) {
    const long long k = pos[b] - pos0;
    if (k >= 0 && k < steps) history[k * batch + b] = next[b];
    tokens[b] = next[b];
    pos[b] += 1;
  }
}

}  // namespace fl

// --------------------------------------------------------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------------------------------------------------------
static unsigned grid_for(long long items) {
  const long long ctas = (items + 255) / 256;
  return (unsigned)(ctas < 1 ? 1 : ctas > 148ll * 64 ? 148 * 64 : ctas);
}

#define FL_DEC_TYPES(dtype, ...)                                             \
  do {                                                                       \
    if ((dtype) == FL_DEC_BF16) { using T = __nv_bfloat16; __VA_ARGS__; }    \
    else if ((dtype) == FL_DEC_FP16) { using T = __half; __VA_ARGS__; }      \
    else return -1;                                                          \
  } while (0)

extern "C" int fl_dec_embed(int dtype, const long long* tokens, const long long* pos, const void* embed, const void* pos_embed, void* x,
                            long long rows, int hidden, int seq, int offset, long long vocab, long long pos_rows, cudaStream_t stream) {
  if (hidden % 8 || hidden < 8 || rows < 0 || (pos == nullptr && pos_embed != nullptr && seq < 1)) return -2;
  if (rows == 0) return 0;
  FL_DEC_TYPES(dtype, (fl::dec_embed_kernel<T><<<grid_for(rows * (hidden / 8)), 256, 0, stream>>>(
                          tokens, pos, (const T*)embed, (const T*)pos_embed, (T*)x, rows, hidden / 8, seq < 1 ? 1 : seq, offset, vocab, pos_rows)));
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_add_norm(int dtype, void* x, const void* y, const void* y_bias, const void* w, const void* b, void* h, long long rows,
                               int hidden, float eps, cudaStream_t stream) {
  if (hidden % 8 || hidden < 8 || hidden > 8 * 4 * 1024 || rows < 0 || rows > 0x7fffffffll) return -2;
  if (rows == 0) return 0;
  const int vecs = hidden / 8;
  // few rows: one vector per thread, as many threads as that takes; many rows: two per thread keeps more CTAs resident
  const int vpt = vecs > 2048 ? 4 : (vecs > 1024 || (rows > 148 && vecs > 128)) ? 2 : 1;
  const int threads = ((vecs + vpt - 1) / vpt + 31) / 32 * 32;
#define FL_NORM(V) fl::dec_add_norm_kernel<T, V><<<(unsigned)rows, threads, 0, stream>>>((T*)x, (const T*)y, (const T*)y_bias, (const T*)w, (const T*)b, (T*)h, hidden, eps)
  FL_DEC_TYPES(dtype, { if (vpt == 4) FL_NORM(4); else if (vpt == 2) FL_NORM(2); else FL_NORM(1); });
#undef FL_NORM
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_qkv(int dtype, void* qkv, const void* bias, const float* rope, long long rope_rows, const long long* pos,
                          long long rows, int seq, int heads, int dim, const FlPagedKv* kv, cudaStream_t stream) {
  if (dim % 16 || dim < 16 || heads < 1 || kv->heads < 1 || kv->block_size < 1 || rows < 0 || (pos == nullptr && seq < 1)) return -2;
  if (rows == 0) return 0;
  FL_DEC_TYPES(dtype, (fl::dec_qkv_kernel<T><<<grid_for(rows * (heads + 2 * kv->heads) * (dim / 16)), 256, 0, stream>>>(
                          (T*)qkv, (const T*)bias, rope, rope_rows, pos, rows, seq, heads, dim, *kv)));
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_act(int dtype, int kind, const void* h, const void* bias, void* out, long long rows, int ffn, cudaStream_t stream) {
  if (ffn % 8 || ffn < 8 || rows < 0) return -2;
  if (rows == 0) return 0;
  const unsigned grid = grid_for(rows * (ffn / 8));
#define FL_ACT(K) fl::dec_act_kernel<T, K><<<grid, 256, 0, stream>>>((const T*)h, (const T*)bias, (T*)out, rows, ffn)
  FL_DEC_TYPES(dtype, {
    if (kind == FL_ACT_SILU_GATED) FL_ACT(FL_ACT_SILU_GATED);
    else if (kind == FL_ACT_RELU) FL_ACT(FL_ACT_RELU);
    else if (kind == FL_ACT_GELU_TANH) FL_ACT(FL_ACT_GELU_TANH);
    else return -3;
  });
#undef FL_ACT
  return (int)cudaGetLastError();
}

// Two CTAs' worth of work per SM, as long as every warp still gets about 64 tokens of a full context.
extern "C" int fl_dec_attention_plan(int batch, int heads, int kv_heads, int dim, int capacity, long long* ws_floats, int* tickets,
                                     int* splits) {
  if (batch < 1 || kv_heads < 1 || heads < kv_heads || heads % kv_heads || dim < 8 || dim % 8 || dim > 128) return -2;
  const int group = heads / kv_heads, gparts = (group + fl::ATT_G - 1) / fl::ATT_G, units = batch * kv_heads * gparts;
  int s = (2 * 148 + units - 1) / units;
  const int most = (capacity + 64 * fl::ATT_WARPS - 1) / (64 * fl::ATT_WARPS);
  if (s > most) s = most;
  if (s < 1) s = 1;
  const int dp = dim <= 64 ? 64 : 128;
  *splits = s;
  *tickets = units;
  *ws_floats = s > 1 ? (long long)units * s * fl::ATT_G * (dp + 2) : 0;
  return 0;
}

extern "C" int fl_dec_attention(int dtype, const void* q, long long q_stride, const long long* pos, const FlPagedKv* kv, void* out,
                                int batch, int heads, int dim, int splits, float* ws, int* tickets, cudaStream_t stream) {
  if (batch < 1 || batch > 65535 || kv->heads < 1 || heads % kv->heads || dim < 8 || dim % 8 || dim > 128 || kv->layout != FL_KV_LBSHD)
    return -2;
  if (splits < 1 || splits > 65535 || (splits > 1 && (ws == nullptr || tickets == nullptr))) return -3;
  const int group = heads / kv->heads, gparts = (group + fl::ATT_G - 1) / fl::ATT_G;
  const dim3 grid(kv->heads * gparts, batch, splits);
  const float scale = 1.4426950408889634f / sqrtf((float)dim);
  FL_DEC_TYPES(dtype, {
    if (dim <= 64)
      fl::dec_attention_kernel<T, 64><<<grid, fl::ATT_WARPS * 32, 0, stream>>>((const T*)q, q_stride, pos, *kv, (T*)out, heads, dim, group, gparts, scale, ws, tickets);
    else
      fl::dec_attention_kernel<T, 128><<<grid, fl::ATT_WARPS * 32, 0, stream>>>((const T*)q, q_stride, pos, *kv, (T*)out, heads, dim, group, gparts, scale, ws, tickets);
  });
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_argmax(int dtype, const void* logits, long long* out, int rows, long long vocab, cudaStream_t stream) {
  if (rows < 0 || vocab < 1) return -2;
  if (rows == 0) return 0;
  FL_DEC_TYPES(dtype, (fl::dec_argmax_kernel<T><<<rows, 1024, 0, stream>>>((const T*)logits, out, vocab)));
  return (int)cudaGetLastError();
}

extern "C" int fl_dec_advance(const long long* next, long long* tokens, long long* pos, long long* history, long long pos0, int batch,
                              int steps, cudaStream_t stream) {
  if (batch < 1) return -2;
  fl::dec_advance_kernel<<<1, 256, 0, stream>>>(next, tokens, pos, history, pos0, batch, steps);
  return (int)cudaGetLastError();
}
