// y = f(x w^T + bias) for a handful of rows x: the matrix products of a decoding step.
//
// Bound by reading w once.  A CTA streams 128 rows of w through shared memory, 64 columns (16 KB) per TMA load, and multiplies them
// with the same columns of x on the tensor cores (tcgen05, M = 128 rows of w, N = 16 rows of x); the sums stay in TMEM until the last
// block.  Two CTAs of about 100 KB share an SM, so 160 KB of w per SM are on the way.  Matrices with fewer than 148 x 2 such tiles are
// cut along k over a cluster of up to eight CTAs.  Each stores its sums straight from TMEM into the shared memory of the CTA that owns
// the row of x, which adds them up, always in the same order: no workspace, no atomics, and the same bits on every run.  (Blocks dealt
// out evenly over all CTAs, with shared tiles summed through global memory, were tried: the last CTA's trip for the others' sums costs
// 8 us, more than the uneven grids, 6144 x 4096 and 16 rows: 21 us against 13.)
//
// A step is a chain of seven or eight short kernels per layer.  Launched one after the other, each fills its pipeline from an idle
// memory and drains it into one.  With `early` a kernel starts as soon as the one before it has started and the SMs have room, and
// requests its first blocks of w, which do not depend on that kernel; it waits (griddepcontrol.wait) before it reads x.
//
// 16 rows, one product after another with w from memory: 6144 x 4096 13.1 us (library 11.7), 4096 x 4096 9.4 (9.3), 2 x 14336 x 4096
// with the activation 39.8 (40.9 without it), 4096 x 14336 22.3 (23.0); 3 rows: 2048 x 8192 9.4 (17.9), 2048 x 2048 4.3 (6.4).  What
// counts is the chain: with library products a layer of an 8B model at 16 rows and 2048 tokens took 143 us, with these and the
// attention's ring (decoder.cu) 121.  The output head is the last of them and gains least: 128256 x 4096 takes 167 us alone (library
// 157), a step with it here or there the same within 0.5 % (16 x 2048 tokens 4049 | 4030 us, 1.3B model 16 x 1000 1937 | 1927, 8B
// 1 x 500 3301 | 3304), GPT-2's less (16 x 500: 486 | 529).
//
// The line is at 16 rows, one tile's N.  From 17 on the tile would be of 32 rows, with four stages.  As measured with it, own | library:
// 17 rows 6144 x 4096 14.0 | 10.9 us, 4096 x 14336 23.3 | 23.7; 24 rows 14.4 | 10.9, 24.1 | 23.7; a step of an 8B model 3794 | 3804 us
// at 17 requests, 3928 | 3884 at 24, 4040 | 3994 at 31, of a 1.3B model 1608 | 1602 and 1790 | 1745 at 17 and 24; only GPT-2 gains (503 |
// 526 at 17, 603 | 647 at 28).
#include "thin_gemm.cuh"
#include "decoder.cuh"
#include "kv_pack.cuh"
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "../common/fl_ptx.cuh"
#include "tile_map.cuh"

namespace fl {

constexpr int TG_M = 128;                          // rows of w per tile
constexpr int TG_N = FL_THIN_MAX_ROWS;             // rows of x, padded
constexpr int TG_K = 64;                           // columns per block: one 128-byte swizzle row
constexpr int TG_W_BYTES = TG_M * TG_K * 2;
constexpr int TG_STAGE_BYTES = TG_W_BYTES + TG_N * TG_K * 2;
constexpr int TG_STAGES = 5;
constexpr int TG_PART_BYTES = TG_N * TG_M * 4;     // what the cluster's CTAs send this one: [CTA][row of x][row of w] fp32
constexpr int TG_SMEM = TG_STAGES * TG_STAGE_BYTES + TG_PART_BYTES + 1024 /*alignment*/;
constexpr int TG_TMEM_COLS = 32;
constexpr int TG_THREADS = 128;

template <typename T> struct ThinNum;
template <> struct ThinNum<__nv_bfloat16> {
  static constexpr uint32_t kFmt = 1;
  using two = __nv_bfloat162;
  static __device__ __forceinline__ float2 f2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<two*>(&w)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    two h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float round(float a) { return __bfloat162float(__float2bfloat16_rn(a)); }
};
template <> struct ThinNum<__half> {
  static constexpr uint32_t kFmt = 0;
  using two = __half2;
  static __device__ __forceinline__ float2 f2(uint32_t w) { return __half22float2(*reinterpret_cast<two*>(&w)); }
  static __device__ __forceinline__ uint32_t pack(float a, float b) {
    two h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float round(float a) { return __half2float(__float2half_rn(a)); }
};

__device__ __forceinline__ void st_cluster_float(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void cluster_arrive_all() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_all() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// OUT: what becomes of the sums, FL_THIN_QKV by itself, the others (FL_THIN_STORE here) by `epilogue`.  For FL_THIN_QKV a fifth warp looks
// up where the keys and values go while the products run.  As a kernel of its own between product and attention the pass was one more link
// of the chain: 1.2 us per layer of a 1.3B model at 3 requests (16 steps 17.35 ms, now 16.89), nothing that shows beside the bytes of an 8B
// model at 16.  (The norms in the products on both sides of them were tried as well: normalised on its way in, x comes 2.8 us later, and
// the norm's own kernel costs 1 to 2.)
template <typename T, int OUT>
__global__ void __launch_bounds__(OUT == FL_THIN_QKV ? TG_THREADS + 32 : TG_THREADS, 2)
thin_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const T* bias, T* y, const int rows,
                 const long long n, const int k, const int splits, const int epilogue, const int early, int* status,
                 const __grid_constant__ FlThinQkv qk) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[TG_STAGES], empty[TG_STAGES], done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % splits;                        // = rank in the cluster
  const long long tile = blockIdx.x / splits;
  const bool gated = OUT == FL_THIN_STORE && epilogue == FL_THIN_SILU_GATED;
  const long long n0 = tile * (gated ? TG_M / 2 : TG_M);        // first output column
  const int blocks = (k + TG_K - 1) / TG_K;
  const int first = (int)((long long)split * blocks / splits), last = (int)((long long)(split + 1) * blocks / splits);
  using R = ThinNum<T>;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TG_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(&done, 1);
    abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TG_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (splits > 1) cluster_arrive_all();                         // waited for before the first store into another CTA
  grid_dep_launch();
  if (bias != nullptr && threadIdx.x < TG_THREADS && n0 + threadIdx.x < n) prefetch_l2(bias + n0 + threadIdx.x);
  const uint32_t tmem_base = tmem_base_s;

  // FL_THIN_QKV: of this CTA's rows, the row of the page (before layer and head; -1: none) and the angles (0: not turned)
  __shared__ int qk_page[OUT == FL_THIN_QKV ? TG_N : 1], qk_slot[OUT == FL_THIN_QKV ? TG_N : 1], qk_turn[OUT == FL_THIN_QKV ? TG_N : 1];
  __shared__ __align__(16) float qk_angle[OUT == FL_THIN_QKV ? TG_N * TG_M : 1];

  if (warp == 0 && lane == 0) {
    // ---- loads: w of the first stages before the wait for the kernel that makes x, where w may be read that early
    auto load_w = [&](int b) {
      const int s = (b - first) % TG_STAGES;
      uint8_t* dst = smem + s * TG_STAGE_BYTES;
      mbar_arrive_expect_tx(&full[s], TG_STAGE_BYTES);
      if (gated) {                                              // 64 gate rows and the 64 up rows that belong to them
        tma_load_2d(dst, &tm_w, &full[s], b * TG_K, (int)n0);
        tma_load_2d(dst + TG_W_BYTES / 2, &tm_w, &full[s], b * TG_K, (int)(n + n0));
      } else {
        tma_load_2d(dst, &tm_w, &full[s], b * TG_K, (int)n0);
      }
    };
    auto load_x = [&](int b) {
      const int s = (b - first) % TG_STAGES;
      tma_load_2d(smem + s * TG_STAGE_BYTES + TG_W_BYTES, &tm_x, &full[s], b * TG_K, 0);
    };
    const int ahead = min(last, first + TG_STAGES);
    if (!early) grid_dep_wait();
    for (int b = first; b < ahead; ++b) load_w(b);
    if (early) grid_dep_wait();
    for (int b = first; b < ahead; ++b) load_x(b);
    for (int b = ahead; b < last; ++b) {
      const int i = b - first;
      if (!mbar_wait(&empty[i % TG_STAGES], ((i / TG_STAGES) & 1) ^ 1, &abort_flag, nullptr, kTimeoutMbarEmpty, 0)) break;
      load_w(b);
      load_x(b);
    }
  } else if (warp == 1 && lane == 0) {
    // ---- products
    constexpr uint32_t idesc = make_idesc(ThinNum<T>::kFmt, ThinNum<T>::kFmt, 0, 0, TG_M, TG_N);
    bool ok = true;
    grid_dep_wait();                                            // x comes behind it: the limit of the waits counts from there
    for (int b = first; b < last && ok; ++b) {
      const int i = b - first, s = i % TG_STAGES;
      ok = mbar_wait(&full[s], (i / TG_STAGES) & 1, &abort_flag, nullptr, kTimeoutMbarFull, 0);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t w_base = smem_u32(smem + s * TG_STAGE_BYTES), x_base = w_base + TG_W_BYTES;
#pragma unroll
      for (int kk = 0; kk < TG_K / 16; ++kk)
        umma_f16(tmem_base, make_smem_desc(w_base + kk * 32, 16, 1024), make_smem_desc(x_base + kk * 32, 16, 1024), idesc, (i | kk) != 0);
      umma_commit(&empty[s]);
    }
    if (ok) umma_commit(&done);
  } else if (OUT == FL_THIN_QKV && warp == 4) {
    // ---- this CTA's rows: page and slot of the position, and its angles
    grid_dep_wait();
    const int own_rows = (rows - split + splits - 1) / splits;
    int turn = -1;
    if (lane < own_rows) {
      const int r = split + lane * splits;
      const long long at = __ldcg(qk.pos + r);
      const int at32 = (int)at;                                 // a position beyond 32 bits is in no table
      int page = at32 / qk.kv.block_size, slot = at32 - page * qk.kv.block_size, blk = -1;
      if (slot < 0) { slot += qk.kv.block_size; page -= 1; }
      if (page < 0) page += qk.kv.table_stride;                 // negative positions and page ids count from the end, as indexing does
      int what = 0;
      if (at32 != at || page < 0 || page >= qk.kv.table_stride) {
        what = FL_DEC_BAD_POSITION;
      } else {
        blk = __ldcg(qk.kv.block_table + (long long)r * qk.kv.table_stride + page);
        if (blk < 0) blk += qk.kv.num_blocks;
        if (blk < 0 || blk >= qk.kv.num_blocks) { what = FL_DEC_BAD_PAGE; blk = -1; }
      }
      if (what != 0 && qk.kv.status != nullptr) *reinterpret_cast<volatile int*>(qk.kv.status) = what;
      const long long t = at < 0 ? -at : at;
      turn = qk.rope != nullptr && t < qk.rope_rows ? (int)t : -1;
      qk_page[lane] = blk;
      qk_slot[lane] = slot;
      qk_turn[lane] = turn < 0 ? 0 : at < 0 ? -1 : 1;
    }
    if (qk.rope != nullptr) {
#pragma unroll 4
      for (int j = 0; j < own_rows; ++j) {
        const int t = __shfl_sync(0xffffffffu, turn, j);
        if (t >= 0)
          for (int c = lane * 4; c < qk.dim; c += 128)
            *reinterpret_cast<float4*>(qk_angle + j * TG_M + c) = __ldcg(reinterpret_cast<const float4*>(qk.rope + (long long)t * qk.dim + c));
      }
    }
  }
  __syncwarp();
  grid_dep_wait();                                              // y may still be read by kernels before this one
  const bool have = mbar_wait_warp(&done, 0, &abort_flag, nullptr, kTimeoutTmemFull, 0);
  tc_fence_after_sync();
  if (!have && status != nullptr) *reinterpret_cast<volatile int*>(status) = FL_DEC_STALLED;

  // ---- sums to the CTAs that own the rows of x: row r belongs to CTA r % splits, as its row r / splits
  float* part = reinterpret_cast<float*>(smem + TG_STAGES * TG_STAGE_BYTES);
  const int own = (rows + splits - 1) / splits;                 // rows per CTA; rows <= TG_N and splits divides TG_N: own * splits <= TG_N
  if (splits > 1) cluster_wait_all();
  if (have && (OUT != FL_THIN_QKV || warp < 4)) {
    uint32_t v[32];                                             // the second half: columns that the products do not write
    tmem_ld_32x32(tmem_base + ((uint32_t)(warp * 32) << 16), v);
    tmem_ld_wait();
    const uint32_t at = smem_u32(part + split * own * TG_M + threadIdx.x);
#pragma unroll
    for (int r = 0; r < TG_N; ++r) {
      if (r < rows) {
        if (splits == 1) part[r * TG_M + threadIdx.x] = __uint_as_float(v[r]);
        else st_cluster_float(map_to_cta(at + (uint32_t)(r / splits) * TG_M * 4, r % splits), __uint_as_float(v[r]));
      }
    }
  }
  tc_fence_before_sync();
  if (splits > 1) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    // whoever gave up, the loader may have copies on the way: they land before TMEM and, with this warp, the CTA's shared memory go away
    if (*reinterpret_cast<volatile int*>(&abort_flag)) let_copies_land();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TG_TMEM_COLS);
  }

  // ---- this CTA's rows: two neighbouring columns per lane, the CTAs' sums in their order
  auto sums = [&](int r, int c) -> float2 {
    const float* p = part + r / splits * TG_M + c;
    float2 t = *reinterpret_cast<const float2*>(p);
    for (int s = 1; s < splits; ++s) {
      const float2 v = *reinterpret_cast<const float2*>(p + s * own * TG_M);
      t.x += v.x; t.y += v.y;
    }
    return t;
  };
  auto store = [&](int r, long long col, float a, float b) {
    T* p = y + (long long)r * n + col;
    if (col + 1 < n && (n & 1) == 0) {
      T two[2] = {T(a), T(b)};
      *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(two);
    } else {
      if (col < n) p[0] = T(a);
      if (col + 1 < n) p[1] = T(b);
    }
  };
  const int c2 = 2 * (threadIdx.x & 63);
  const long long col = n0 + c2;
  if (OUT == FL_THIN_QKV) {
    // Whole heads: dim divides the tile.  Bias, rotation of q and k by the position's angles, q to y, k and v to their pages.
    const int dim = qk.dim, half = dim / 2, in = c2 % dim;      // even, as half is: a thread's two columns turn alike
    const long long head = col / dim;
    const bool is_q = head < qk.heads, is_v = head >= qk.heads + qk.kv.heads, low = in < half;
    const int other = low ? c2 + half : c2 - half;
    if (threadIdx.x < TG_THREADS && col < n) {
      const long long oc = n0 + other;
      float ba[2] = {0.f, 0.f}, bo[2] = {0.f, 0.f};
      if (bias != nullptr) { ba[0] = (float)bias[col]; ba[1] = (float)bias[col + 1]; bo[0] = (float)bias[oc]; bo[1] = (float)bias[oc + 1]; }
      for (int r = split + splits * (threadIdx.x >> 6); r < rows; r += 2 * splits) {
        const int j = r / splits, turn = is_v ? 0 : qk_turn[j];
        const float2 t = sums(r, c2);
        float a[2] = {R::round(t.x), R::round(t.y)};
        if (bias != nullptr) { a[0] = R::round(a[0] + ba[0]); a[1] = R::round(a[1] + ba[1]); }
        if (turn != 0) {
          const float2 u = sums(r, other);
          float o[2] = {R::round(u.x), R::round(u.y)};
          if (bias != nullptr) { o[0] = R::round(o[0] + bo[0]); o[1] = R::round(o[1] + bo[1]); }
          const float* cs = qk_angle + j * TG_M + (low ? in : in - half);      // half cosines, half sines
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            // the products of the second half's value are rounded by themselves, as dec_qkv_kernel's are
            const float co = cs[e], si = turn < 0 ? -cs[half + e] : cs[half + e];
            a[e] = low ? fmaf(a[e], co, -__fmul_rn(o[e], si)) : fmaf(o[e], si, __fmul_rn(a[e], co));
          }
        }
        const uint32_t two = R::pack(a[0], a[1]);
        if (is_q) {
          *reinterpret_cast<uint32_t*>(y + (long long)r * n + col) = two;
        } else if (qk_page[j] >= 0) {
          const long long blk = qk_page[j], slot = qk_slot[j];
          const int kh = (int)(head - qk.heads - (is_v ? qk.kv.heads : 0));
          const long long at = qk.kv.layout == FL_KV_BLHSD ? ((blk * qk.kv.layers + qk.kv.layer) * qk.kv.heads + kh) * qk.kv.block_size + slot
                                                           : (((long long)qk.kv.layer * qk.kv.num_blocks + blk) * qk.kv.block_size + slot) * qk.kv.heads + kh;
          *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(is_v ? qk.kv.v : qk.kv.k) + at * dim + in) = two;
        }
      }
    }
  } else if (gated) {
    const int c = 2 * lane;
    for (int r = split + splits * warp; r < rows; r += 4 * splits) {
      const float2 g = sums(r, c), u = sums(r, 64 + c);
      const float g0 = R::round(g.x), g1 = R::round(g.y);
      store(r, n0 + c, R::round(g0 / (1.f + expf(-g0))) * R::round(u.x), R::round(g1 / (1.f + expf(-g1))) * R::round(u.y));
    }
  } else {
    const float b0 = bias != nullptr && col < n ? (float)bias[col] : 0.f, b1 = bias != nullptr && col + 1 < n ? (float)bias[col + 1] : 0.f;
    for (int r = split + splits * (threadIdx.x >> 6); r < rows; r += 2 * splits) {
      const float2 t = sums(r, c2);
      float a[2] = {R::round(t.x), R::round(t.y)};
      if (bias != nullptr) { a[0] = R::round(a[0] + b0); a[1] = R::round(a[1] + b1); }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (epilogue == FL_THIN_RELU) a[j] = a[j] < 0.f ? 0.f : a[j];      // keeps NaN
        else if (epilogue == FL_THIN_GELU_TANH) a[j] = 0.5f * a[j] * (1.f + tanhf(0.7978845608028654f * (a[j] + 0.044715f * a[j] * a[j] * a[j])));
      }
      store(r, col, a[0], a[1]);
    }
  }
}

// --------------------------------------------------------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------------------------------------------------------
struct FlThinStep {
  int dtype; const void* x; int rows; const void* w; long long n; int k; const void* bias; int epilogue; void* y; int early; int* status;
  FlThinQkv qkv;
};

template <typename T, int OUT>
static int launch_thin(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const FlThinStep& a, long long tiles, int splits, cudaStream_t stream) {
  static bool set_on[64];                          // per device: a process may drive several GPUs
  const auto kernel = thin_gemm_kernel<T, OUT>;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return -3;
  if (!set_on[dev]) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TG_SMEM);
    if (e != cudaSuccess) return (int)e;
    set_on[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * splits), 1, 1);
  cfg.blockDim = dim3(OUT == FL_THIN_QKV ? TG_THREADS + 32 : TG_THREADS, 1, 1);
  cfg.dynamicSmemBytes = TG_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = a.early ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, tm_w, tm_x, (const T*)a.bias, (T*)a.y, a.rows, a.n, a.k, splits, a.epilogue, a.early, a.status, a.qkv);
}

}  // namespace fl

static int thin_step(const fl::FlThinStep* a, cudaStream_t stream) {
  using namespace fl;
  const bool gated = a->epilogue == FL_THIN_SILU_GATED, qkv = a->epilogue == FL_THIN_QKV;
  if (a->dtype != FL_DEC_BF16 && a->dtype != FL_DEC_FP16) return -1;
  if (a->rows < 1 || a->rows > FL_THIN_MAX_ROWS || a->n < 1 || a->n > 0x3fffff00ll || a->k < 8 || a->k % 8) return -2;
  if (a->epilogue < FL_THIN_SILU_GATED || a->epilogue > FL_THIN_QKV || (gated && a->bias != nullptr)) return -3;
  if (((uintptr_t)a->x | (uintptr_t)a->w) & 15 || (uintptr_t)a->y & 3) return -4;
  if (qkv) {
    const FlThinQkv& q = a->qkv;
    if (q.pos == nullptr || q.dim < 16 || q.dim % 16 || TG_M % q.dim || q.heads < 1 || q.kv.heads < 1 || q.kv.block_size < 1 || q.kv.table_stride < 1 ||
        (long long)(q.heads + 2ll * q.kv.heads) * q.dim != a->n || ((uintptr_t)q.kv.k | (uintptr_t)q.kv.v) & 3 || (uintptr_t)q.rope & 15)
      return -5;
  }
  const int per_tile = gated ? TG_M / 2 : TG_M, blocks = (a->k + TG_K - 1) / TG_K;
  const long long tiles = (a->n + per_tile - 1) / per_tile;
  // As many CTAs as fit at two per SM, so that all of them run from start to end at an equal share of the memory's rate; clusters of
  // 1, 2, 4 or 8, since others leave SMs over (6144 x 4096, 16 rows: 17.2 us in clusters of 6, 13.1 in clusters of 4).
  int splits = 1;
  while (splits < 8 && 2 * splits * tiles <= 2 * 148 && 2 * splits <= blocks) splits *= 2;
  const int type = a->dtype == FL_DEC_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm_w, tm_x;
  int rc = tile_map(&tm_w, type, a->w, a->k, gated ? 2 * a->n : a->n, per_tile);
  if (rc == 0) rc = tile_map(&tm_x, type, a->x, a->k, a->rows, TG_N);
  if (rc != 0) return rc;
  if (a->dtype == FL_DEC_BF16) return qkv ? launch_thin<__nv_bfloat16, FL_THIN_QKV>(tm_w, tm_x, *a, tiles, splits, stream)
                                          : launch_thin<__nv_bfloat16, FL_THIN_STORE>(tm_w, tm_x, *a, tiles, splits, stream);
  return qkv ? launch_thin<__half, FL_THIN_QKV>(tm_w, tm_x, *a, tiles, splits, stream) : launch_thin<__half, FL_THIN_STORE>(tm_w, tm_x, *a, tiles, splits, stream);
}

extern "C" int fl_thin_gemm(int dtype, const void* x, int rows, const void* w, long long n, int k, const void* bias, int epilogue, void* y, int early,
                            int* status, cudaStream_t stream) {
  if (epilogue == FL_THIN_QKV) return -3;
  const fl::FlThinStep a = {dtype, x, rows, w, n, k, bias, epilogue, y, early, status, {}};
  return thin_step(&a, stream);
}

extern "C" int fl_thin_qkv(int dtype, const void* x, int rows, const void* w, long long n, int k, const void* bias, const FlThinQkv* qkv, void* y,
                           int early, int* status, cudaStream_t stream) {
  const fl::FlThinStep a = {dtype, x, rows, w, n, k, bias, FL_THIN_QKV, y, early, status, *qkv};
  return thin_step(&a, stream);
}
