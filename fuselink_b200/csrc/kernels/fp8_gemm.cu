// Block-scaled fp8 grouped GEMM (see fp8_gemm.cuh for the scheme).
//
//   warp 0      : TMA producer (e4m3 tiles, 128-byte swizzle, never multicast)
//   warp 1      : MMA issuer   (tcgen05.mma kind::f8f6f4; one 128-deep block per TMEM partial buffer)
//   warps 2, 3  : the operands' scales, from memory to shared memory, several blocks ahead
//   warps 4..11 : promotion + epilogue (tcgen05.ld partial -> scale -> fp32 registers -> fused epilogue); two warps
//                 share each TMEM lane quadrant and split the tile's columns
//
// Bound by the promotion: every partial sum makes a trip from TMEM and takes an fp32 FMA, in a chain that the next multiplication
// into the same buffer waits for.  So nothing else is in that chain: the scales come through shared memory (read from global
// memory by the promotion threads, one 4-byte load per row 4 K / 128 bytes apart, they cost a fifth of the kernel's time), a chunk of
// a partial is on its way while the one before it is added, also from one block to the next, and two FMAs are one instruction.
// 8 experts, 1024 rows each, hidden 4096, ffn 14336, before and now: second product forward (K = 14336, N = 4096) 582 (scales from
// global memory, the rest as now) -> 524 us, gradient of the first (K = 28672) 1204 -> 1043; without the FMAs it is 902, without the
// trips to TMEM 760 (multiplications and loads).  In a training step of 4096 tokens the four products took 4950 us with the loads of
// the scales, the trips and the FMAs one after the other, now 4230.  Sixteen promotion warps with half the columns each: 1060.
// The epilogues run between two tiles of a CTA and are not hidden: they store whole sectors through shared memory and ask for the saved
// gate and up rows a tile ahead.  Their quotients are IEEE divisions: __fdividef takes 1228 instead of 1423 us (SWIGLU in that step) and
// 872 instead of 1020 (DSWIGLU), but rounds more results to the wrong bf16 neighbour (74 of 8388608 for 60) and gives 0 for gates below -87.3.
//
// Reference parity: none in the reference (it has no kernels); this is the fp8 arm of the MoE expert GEMMs.
#include "fp8_gemm.cuh"
#include "../common/fl_ptx.cuh"
#include "staged_store.cuh"
#include "tile_map.cuh"
#include <cuda.h>
#include <cuda_fp8.h>
#include <stdio.h>
#include <string.h>

namespace fl8 {
using namespace fl;

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BKB = 128;                      // bytes (= e4m3 elements) of contraction per stage = one scale block
constexpr int STAGES = 4;
constexpr int A_STAGE = BM * BKB;             // 16 KiB
constexpr int B_STAGE = BN * BKB;             // 32 KiB
constexpr int STAGE = A_STAGE + B_STAGE;
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 128 + 32 * EPI_WARPS;
// Registers: 384 threads start with 168 each (64512).  The first four warps give 112 each back, the others take 56 more: 128 x 56 +
// 256 x 224 = 64512.  A promotion thread holds 128 sums, 32 values being added and 32 on their way from TMEM.
constexpr int PRODUCER_REGS = 56, EPI_REGS = 224;
constexpr int TMEM_COLS = 512;                // two partial buffers of 256 columns
constexpr int SC_BLOCKS = 8;                  // blocks of contraction whose scales travel together (a 32-byte sector per row)
constexpr int SC_STAGES = 2;
struct ScaleStage {
  float a[SC_BLOCKS][BM];
  float b[SC_BLOCKS][2];
};
constexpr int SHARED_BYTES = 1024;            // barriers, counts
constexpr int SMEM_BYTES = STAGES * STAGE + 1024 /*align*/ + SHARED_BYTES + EPI_WARPS * EPI_STAGE_BYTES + SC_STAGES * (int)sizeof(ScaleStage);

struct KParams {
  int num_groups, cap, N, K;
  const int* counts;
  const float* a_scale;
  const float* b_scale;
  int b_mn;
  int epilogue;
  __nv_bfloat16* C; long long ldc;
  __nv_bfloat16* gu; long long ldgu;
  __nv_bfloat16* dgu;
  const int* row_info;
  FlPeerPtrs peers;
  int num_peers; long long peer_rows;
  int zero_tail;
  int group_m;
  int* status;
};

struct Shared {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t pfull[2];
  uint64_t pempty[2];
  uint64_t sfull[SC_STAGES];
  uint64_t sempty[SC_STAGES];
  uint32_t tmem_base;
  int abort_flag;
  int counts[FL_GEMM_MAX_GROUPS];
};

static_assert(sizeof(Shared) <= SHARED_BYTES, "barriers and counts");

struct Tile {
  int g, m0, n0, rows, cnt;
};

__device__ __forceinline__ bool map_tile(const KParams& p, const int* counts, int id, Tile& t) {
  const int NT = (p.N + BN - 1) / BN;
  int acc = 0;
  for (int g = 0; g < p.num_groups; ++g) {
    const int cnt = counts[g];
    const int mt = (cnt + BM - 1) / BM;
    const int tiles = mt * NT;
    if (id < acc + tiles) {
      const int l = id - acc;
      const int per_sg = p.group_m * NT;
      const int sg = l / per_sg;
      const int first_m = sg * p.group_m;
      const int gsz = min(p.group_m, mt - first_m);
      const int r = l - sg * per_sg;
      t.g = g; t.m0 = (first_m + r % gsz) * BM; t.n0 = (r / gsz) * BN;
      t.rows = min(BM, cnt - t.m0);
      t.cnt = cnt;
      return true;
    }
    acc += tiles;
  }
  return false;
}

// 8 neighbouring values; WIDE: the address is a multiple of 16 bytes (otherwise of 8)
template <bool WIDE>
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) {
  if (WIDE) return ld_nc_v4(p);
  const uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 4);
  return make_uint4(a.x, a.y, b.x, b.y);
}
template <bool WIDE>
__device__ __forceinline__ void store8(__nv_fp8_storage_t* p, uint2 v) {
  if (WIDE) { *reinterpret_cast<uint2*>(p) = v; return; }
  reinterpret_cast<uint32_t*>(p)[0] = v.x;
  reinterpret_cast<uint32_t*>(p)[1] = v.y;
}
// 8 bf16 values times inv as 8 e4m3 values; the largest absolute value of 8 bf16 values
__device__ __forceinline__ uint2 quantize8(uint4 raw, float inv) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    p[i] = __nv_cvt_float2_to_fp8x2(make_float2(f.x * inv, f.y * inv), __NV_SATFINITE, __NV_E4M3);
  }
  return make_uint2(p[0] | p[1] << 16, p[2] | p[3] << 16);
}
__device__ __forceinline__ float amax8(uint4 raw) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
  return m;
}

// One scale per 1 x 128 block.  Bound by memory: a half warp takes a block (16 bytes per lane), a warp eight neighbouring blocks
// of a row, all requested before the first is used.  The buffers are sized for the worst case and mostly empty, so the warps
// walk the rows that hold tokens (up to a whole tile) group by group, each group starting with the warp at which the one
// before it stopped: one visit per block of the whole buffer, with a division and one small load, took 1439 us of a training
// step of 4096 tokens (32768 rows of capacity, 8192 in use), these 232 us; the used rows' bytes take 190 us.
constexpr int QR_BLOCKS = 8;
template <bool WIDE>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const __nv_bfloat16* x, __nv_fp8_storage_t* q, float* scale,
                                                            long long rows, int K, const int* counts, int cap) {
  const int lane = threadIdx.x & 31, half = lane >> 4, l16 = lane & 15;
  const unsigned kblocks = K / 128, per_row = (kblocks + QR_BLOCKS - 1) / QR_BLOCKS;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const int groups = counts != nullptr ? (int)((rows + cap - 1) / cap) : 1;
  long long u = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (int g = 0; g < groups; ++g) {
    const long long row0 = counts != nullptr ? (long long)g * cap : 0;
    long long used = rows - row0;
    if (counts != nullptr) used = min(used, (long long)min(cap, (min(counts[g], cap) + 127) / 128 * 128));
    const long long units = max(used, 0ll) * per_row;
    for (; u < units; u += nwarps) {
      const unsigned r = (unsigned)u / per_row;               // units of 1024 values: their number fits 32 bits on any GPU
      const long long row = row0 + r;
      const unsigned kb0 = ((unsigned)u - r * per_row) * QR_BLOCKS + half;
      const long long at = row * K + kb0 * 128 + l16 * 8;
      uint4 raw[QR_BLOCKS / 2];
#pragma unroll
      for (int j = 0; j < QR_BLOCKS / 2; ++j)
        raw[j] = kb0 + 2 * j < kblocks ? load8<WIDE>(x + at + j * 256) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < QR_BLOCKS / 2; ++j) {
        float amax = amax8(raw[j]);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        const float s = amax > 0.f ? amax / 448.f : 1.f;
        if (kb0 + 2 * j < kblocks) {
          store8<WIDE>(q + at + j * 256, quantize8(raw[j], 1.f / s));
          if (l16 == 0) scale[row * kblocks + kb0 + 2 * j] = s;
        }
      }
    }
    u -= units;
  }
}

// One CTA (256 threads) per 128 x 128 block of a [G, R, C] weight, 64 values per thread in registers between the maximum and
// the conversion (16-byte loads, 8-byte stores).  Read twice with 8-byte loads: 1078 us for both weights of 8 experts (3 x 4096 x
// 14336 values each, 4.2 GB read and written); now 620 us, 6.8 TB/s.  One 8 x 4096 x 14336 weight: 212 us, 6.65 TB/s; a plain copy
// reaches 6.46 TB/s, but it writes a byte for each one read and this half of one.
template <bool WIDE>
__global__ void __launch_bounds__(256) quantize_blocks_kernel(const __nv_bfloat16* w, __nv_fp8_storage_t* q, float* scale,
                                                              int R, int C) {
  const int cb = blockIdx.x, rb = blockIdx.y, g = blockIdx.z;
  const long long at = (long long)g * R * C + (long long)(rb * 128 + (threadIdx.x >> 4)) * C + cb * 128 + (threadIdx.x & 15) * 8;
  __shared__ float red[8];
  uint4 raw[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) raw[i] = load8<WIDE>(w + at + (long long)i * 16 * C);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, amax8(raw[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const float s = amax > 0.f ? amax / 448.f : 1.f;
  const float inv = 1.f / s;
  if (threadIdx.x == 0) scale[((long long)g * (R / 128) + rb) * (C / 128) + cb] = s;
#pragma unroll
  for (int i = 0; i < 8; ++i) store8<WIDE>(q + at + (long long)i * 16 * C, quantize8(raw[i], inv));
}

// ------------------------------------------------------------------------------------------------
// GEMM
// ------------------------------------------------------------------------------------------------
// Columns a promotion thread owns inside the 256-wide tile: chunks 0,1 in the first 128-column block, chunks 2,3 in
// the second, 64 columns per warp-half in each.  With the gate|up interleaved weight this gives every thread the gate
// and the up value of the same 64 activation columns, and every chunk pair exactly one weight scale block.
__device__ __forceinline__ int chunk_col(int half, int c) { return (c < 2 ? 0 : 128) + 64 * half + 32 * (c & 1); }

// two fp32 accumulators: acc += v * s, each rounded as fmaf does
__device__ __forceinline__ void fma2(float2& acc, uint32_t v0, uint32_t v1, float s) {
  asm volatile("{\n\t.reg .b64 a, v, s;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 v, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\t"
      "fma.rn.f32x2 a, v, s, a;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "+f"(acc.x), "+f"(acc.y) : "r"(v0), "r"(v1), "f"(s));
}

template <int EPI>
__global__ void __launch_bounds__(NUM_THREADS, 1)
fp8_grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const KParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Shared* sh = reinterpret_cast<Shared*>(smem + STAGES * STAGE);
  ScaleStage* sc_ring = reinterpret_cast<ScaleStage*>(smem + STAGES * STAGE + SHARED_BYTES + EPI_WARPS * EPI_STAGE_BYTES);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int KB = p.K / 128;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->pfull[b], 1);
      mbar_init(&sh->pempty[b], EPI_WARPS);
    }
    for (int i = 0; i < SC_STAGES; ++i) {
      mbar_init(&sh->sfull[i], 2);
      mbar_init(&sh->sempty[i], EPI_WARPS);
    }
    sh->abort_flag = 0;
    mbar_fence_init();
  }
  for (int g = threadIdx.x; g < p.num_groups; g += NUM_THREADS)
    sh->counts[g] = p.counts ? min(p.counts[g], p.cap) : p.cap;
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = sh->tmem_base;
  volatile int* abort_flag = &sh->abort_flag;
  const int* counts = sh->counts;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    if (warp == 0) {
      if (lane == 0) {
        uint32_t it = 0;
        bool ok = true;
        Tile t;
        for (int id = blockIdx.x; ok && map_tile(p, counts, id, t); id += gridDim.x) {
          for (int kb = 0; kb < KB && ok; ++kb, ++it) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1;
            ok = mbar_wait(&sh->empty[s], ph ^ 1, abort_flag, p.status, kTimeoutMbarEmpty, 2100 + s);
            if (!ok) break;
            uint8_t* a_dst = smem + s * STAGE;
            uint8_t* b_dst = a_dst + A_STAGE;
            mbar_arrive_expect_tx(&sh->full[s], STAGE);
            const int k0 = kb * 128;
            tma_load_3d(a_dst, &tmA, &sh->full[s], k0, t.m0, t.g);
            if (!p.b_mn) {
              tma_load_3d(b_dst, &tmB, &sh->full[s], k0, t.n0, t.g);
            } else {
#pragma unroll
              for (int j = 0; j < BN / 128; ++j)
                tma_load_3d(b_dst + j * (128 * BKB), &tmB, &sh->full[s], t.n0 + 128 * j, k0, t.g);
            }
          }
        }
      }
    } else if (warp == 1) {
      if (lane == 0) {
        const uint32_t idesc = make_idesc(0, 0, 0u, p.b_mn ? 1u : 0u, BM, BN);   // e4m3 x e4m3 -> fp32
        uint32_t it = 0;
        bool ok = true;
        Tile t;
        for (int id = blockIdx.x; ok && map_tile(p, counts, id, t); id += gridDim.x) {
          for (int kb = 0; kb < KB && ok; ++kb, ++it) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1;
            const int b = it & 1;
            const uint32_t bph = (it >> 1) & 1;
            ok = mbar_wait(&sh->pempty[b], bph ^ 1, abort_flag, p.status, kTimeoutTmemEmpty, 2200 + b);
            if (!ok) break;
            ok = mbar_wait(&sh->full[s], ph, abort_flag, p.status, kTimeoutMbarFull, 2300 + s);
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t a_base = smem_u32(smem + s * STAGE);
            const uint32_t b_base = a_base + A_STAGE;
            const uint32_t d_tmem = tmem_base + b * BN;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {   // 4 x (K = 32) per 128-deep block
              const uint64_t da = make_smem_desc(a_base + kk * 32, 16, 1024);
              const uint64_t db = p.b_mn ? make_smem_desc(b_base + kk * 4096, 128 * BKB, 1024)
                                         : make_smem_desc(b_base + kk * 32, 16, 1024);
              umma_f8(d_tmem, da, db, idesc, kk != 0 ? 1u : 0u);
            }
            umma_commit(&sh->empty[s]);
            umma_commit(&sh->pfull[b]);
          }
        }
      }
    } else {
      const int i = (warp - 2) * 32 + lane;
      const int NB = p.N / 128;
      uint32_t it = 0;
      bool ok = true;
      Tile t;
      for (int id = blockIdx.x; ok && map_tile(p, counts, id, t); id += gridDim.x) {
        const float* a0 = p.a_scale + ((long long)t.g * p.cap + t.m0 + i) * KB;
        // of block kb: b0[kb * next_k] and b0[kb * next_k + next_n]
        const long long nb = t.n0 / 128, next_n = p.b_mn ? 1 : KB, next_k = p.b_mn ? NB : 1;
        const float* b0 = p.b_scale + (p.b_mn ? (long long)t.g * KB * NB + nb : ((long long)t.g * NB + nb) * KB);
        for (int kb = 0; kb < KB; kb += SC_BLOCKS, ++it) {
          const int n = min(SC_BLOCKS, KB - kb);
          float v[2][SC_BLOCKS], w = 0.f;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < SC_BLOCKS; ++k) v[h][k] = k < n && i + 64 * h < t.rows ? a0[64ll * h * KB + kb + k] : 0.f;
          if (i < 2 * n) w = b0[(kb + (i >> 1)) * next_k + (i & 1) * next_n];
          const int s = it % SC_STAGES;
          ok = mbar_wait_warp(&sh->sempty[s], ((it / SC_STAGES) & 1) ^ 1, abort_flag, p.status, kTimeoutMbarEmpty, 2600 + s);
          if (!ok) break;
          ScaleStage& st = sc_ring[s];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < SC_BLOCKS; ++k) st.a[k][i + 64 * h] = v[h][k];
          if (i < 2 * n) st.b[i >> 1][i & 1] = w;
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->sfull[s]);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(EPI_REGS));
    const int q = warp & 3;
    const int half = (warp - 4) >> 2;
    uint8_t* stg = smem + STAGES * STAGE + SHARED_BYTES + (warp - 4) * EPI_STAGE_BYTES;
    const int r_in_tile = q * 32 + lane;
    uint32_t it = 0, sit = 0;                     // blocks and stages of scales so far
    bool ok = true;
    Tile t;
    for (int id = blockIdx.x; ok && map_tile(p, counts, id, t); id += gridDim.x) {
      const int row = t.m0 + r_in_tile;
      const long long grow = (long long)t.g * p.cap + row;
      const bool valid = r_in_tile < t.rows;
      if (EPI == FL_EPI_DSWIGLU && half == 0 && valid)      // the saved gate/up of this row: in L2 by the time they are wanted
        bulk_prefetch_l2(p.gu + grow * p.ldgu + 2ll * t.n0, BN * 2 * 2);
      float2 acc[64];                                                 // chunk c: acc[16 c .. 16 c + 15]
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = make_float2(0.f, 0.f);
      // A chunk is on its way from TMEM while the one before it is added, over the ends of blocks as well: what bounds this loop is
      // the chain of trips to TMEM, not their number of bytes or the additions.
      auto t_addr = [&](int c) { return tmem_base + (it & 1) * BN + ((uint32_t)(q * 32) << 16) + chunk_col(half, c); };
      auto partial = [&]() {                      // block `it` has been multiplied
        ok = mbar_wait_warp(&sh->pfull[it & 1], (it >> 1) & 1, abort_flag, p.status, kTimeoutTmemFull, 2400 + (it & 1));
        tc_fence_after_sync();
      };
      uint32_t r[2][32];
      partial();
      if (!ok) break;
      tmem_ld_32x32(t_addr(0), r[0]);
      for (int kb = 0; kb < KB; ++kb) {
        const int k = kb % SC_BLOCKS, s = sit % SC_STAGES;
        if (k == 0) ok = mbar_wait_warp(&sh->sfull[s], (sit / SC_STAGES) & 1, abort_flag, p.status, kTimeoutMbarFull, 2700 + s);
        if (!ok) break;
        const float sa = sc_ring[s].a[k][r_in_tile];
        const float sc[2] = {sa * sc_ring[s].b[k][0], sa * sc_ring[s].b[k][1]};
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (c < 3) {
            tmem_ld_32x32(t_addr(c + 1), r[(c + 1) & 1]);
          } else {                                // everything of this block is in registers
            tc_fence_before_sync();
            __syncwarp();
            const bool scales_done = k == SC_BLOCKS - 1 || kb == KB - 1;
            if (lane == 0) {
              mbar_arrive(&sh->pempty[it & 1]);
              if (scales_done) mbar_arrive(&sh->sempty[s]);
            }
            sit += scales_done;
            ++it;
            if (kb + 1 < KB) {
              partial();
              if (ok) tmem_ld_32x32(t_addr(0), r[0]);
            }
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) fma2(acc[c * 16 + i], r[c & 1][2 * i], r[c & 1][2 * i + 1], sc[c >> 1]);
          if (c < 3) tmem_ld_wait();
        }
        if (!ok) break;
      }
      if (!ok) break;
      // ---- fused epilogue from registers ----------------------------------------------------------
      const bool zero_row = !valid && p.zero_tail && row < min(p.cap, (t.cnt + 127) / 128 * 128);
      auto at = [](__nv_bfloat16* d) { return reinterpret_cast<unsigned long long>(d); };
      if (EPI == FL_EPI_STORE || EPI == FL_EPI_SCATTER) {
        __nv_bfloat16* dst = nullptr;
        if (EPI == FL_EPI_STORE) {
          if (valid || zero_row) dst = p.C + grow * p.ldc;
        } else if (valid) {
          const int info = p.row_info[grow];
          const int rk = (info >> 28) & 0xF;
          const long long slot = info & 0x0FFFFFFF;
          if (rk < p.num_peers && (p.peer_rows <= 0 || slot < p.peer_rows))
            dst = reinterpret_cast<__nv_bfloat16*>(p.peers.p[rk]) + slot * p.ldc;
          else
            report(p.status, kBadIndex, 2500);   // names no rank / no slot of the receive buffer: not stored
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = valid ? pack_bf16(acc[c * 16 + i].x, acc[c * 16 + i].y) : 0u;
          staged_store_packed(stg, lane, pk, dst != nullptr ? at(dst + t.n0 + chunk_col(half, c)) : 0ull);
        }
      } else if (EPI == FL_EPI_SWIGLU) {
        const bool st = valid || zero_row;
        __nv_bfloat16* act = p.C + grow * p.ldc + t.n0 / 2 + 64 * half;
        __nv_bfloat16* gu = p.gu ? p.gu + grow * p.ldgu + t.n0 : nullptr;
        uint32_t pk[16];
#pragma unroll
        for (int c = 0; c < 2; ++c) {                                 // gate in chunk c, up in chunk c + 2
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 g = valid ? acc[c * 16 + i] : make_float2(0.f, 0.f), u = valid ? acc[32 + c * 16 + i] : make_float2(0.f, 0.f);
            pk[i] = pack_bf16(g.x / (1.f + __expf(-g.x)) * u.x, g.y / (1.f + __expf(-g.y)) * u.y);
          }
          staged_store_packed(stg, lane, pk, st ? at(act + 32 * c) : 0ull);
        }
        if (gu) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = valid ? pack_bf16(acc[c * 16 + i].x, acc[c * 16 + i].y) : 0u;
            staged_store_packed(stg, lane, pk, st ? at(gu + chunk_col(half, c)) : 0ull);
          }
        }
      } else {  // FL_EPI_DSWIGLU: acc = dAct over 256 activation columns
        const bool st = valid || zero_row;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int a_col = t.n0 + chunk_col(half, c);
          const long long gcol = (long long)(a_col >> 7) * 256 + (a_col & 127);
          uint32_t pdg[16], pdu[16];
#pragma unroll
          for (int h = 0; h < 4; ++h) {                               // 8 columns at a time
            uint4 g8 = make_uint4(0, 0, 0, 0), u8 = make_uint4(0, 0, 0, 0);
            if (valid) {
              g8 = ld_v4(p.gu + grow * p.ldgu + gcol + 8 * h);
              u8 = ld_v4(p.gu + grow * p.ldgu + gcol + 128 + 8 * h);
            }
            const uint32_t gw[4] = {g8.x, g8.y, g8.z, g8.w}, uw[4] = {u8.x, u8.y, u8.z, u8.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float g[2], u[2], dg[2], du[2];
              unpack_bf16(gw[i], g[0], g[1]);
              unpack_bf16(uw[i], u[0], u[1]);
              const float2 d2 = acc[c * 16 + 4 * h + i];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float da = e ? d2.y : d2.x;
                const float sg = 1.f / (1.f + __expf(-g[e]));
                dg[e] = da * u[e] * (sg * (1.f + g[e] * (1.f - sg)));
                du[e] = da * g[e] * sg;
              }
              pdg[4 * h + i] = valid ? pack_bf16(dg[0], dg[1]) : 0u;
              pdu[4 * h + i] = valid ? pack_bf16(du[0], du[1]) : 0u;
            }
          }
          __nv_bfloat16* dst = p.dgu + grow * p.ldgu + gcol;
          staged_store_packed(stg, lane, pdg, st ? at(dst) : 0ull);
          staged_store_packed(stg, lane, pdu, st ? at(dst + 128) : 0ull);
        }
      }
    }
    if (!ok) tmem_ld_wait();                      // a chunk may be on its way
    if (EPI == FL_EPI_SCATTER) fence_sys();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    // whoever gave up, copies may be on the way and products running: they end before TMEM and, with this warp, the CTA's shared memory go away
    if (*abort_flag) let_copies_land();
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------
// host
// ------------------------------------------------------------------------------------------------
static thread_local char g_err[256] = "";

static int make_map(CUtensorMap* m, const void* base, long long inner, long long outer, long long groups, int box_inner,
                    int box_outer) {
  const fl::TileEncodeFn enc = fl::tile_encode();
  if (!enc) { snprintf(g_err, sizeof g_err, "cuTensorMapEncodeTiled entry point not available"); return -10; }
  cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)groups};
  cuuint64_t strides[2] = {(cuuint64_t)inner, (cuuint64_t)inner * (cuuint64_t)outer};   // bytes: 1 per element
  cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (strides[0] & 15)) {
    snprintf(g_err, sizeof g_err, "fp8 operand base and row pitch must be 16-byte aligned");
    return -11;
  }
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { snprintf(g_err, sizeof g_err, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r); return -12; }
  return 0;
}

template <int EPI>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const KParams& p, int max_ctas, cudaStream_t stream) {
  static int sms_of[64];                       // per device: the shared-memory attribute belongs to the device's copy of the kernel
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) { snprintf(g_err, sizeof g_err, "device ordinal out of range"); return -1; }
  int& num_sms = sms_of[dev];
  if (!num_sms) {
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
    cudaError_t e = cudaFuncSetAttribute(fp8_grouped_gemm_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) { num_sms = 0; return (int)e; }
  }
  int grid = num_sms;
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  fp8_grouped_gemm_kernel<EPI><<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(tmA, tmB, p);
  return (int)cudaGetLastError();
}

}  // namespace fl8

extern "C" const char* fl_fp8_last_error(void) { return fl8::g_err; }

extern "C" int fl_fp8_grouped_gemm(const FlFp8GemmDesc* d, cudaStream_t stream) {
  using namespace fl8;
  g_err[0] = 0;
  auto bad = [](const char* why) { snprintf(g_err, sizeof g_err, "%s", why); return -1; };
  if (d->num_groups < 1 || d->num_groups > FL_GEMM_MAX_GROUPS) return bad("num_groups out of range");
  if (d->cap <= 0 || d->cap % 128) return bad("cap must be a positive multiple of 128");
  if (d->N % 256) return bad("N must be a multiple of 256");
  if (d->K % 128) return bad("K must be a multiple of 128 (one scale block per stage)");
  if (d->epilogue != FL_EPI_STORE && d->epilogue != FL_EPI_SWIGLU && d->epilogue != FL_EPI_SCATTER && d->epilogue != FL_EPI_DSWIGLU)
    return bad("unsupported epilogue for the fp8 kernel");
  KParams p;
  memset(&p, 0, sizeof p);
  p.num_groups = d->num_groups; p.cap = d->cap; p.N = d->N; p.K = d->K; p.counts = d->counts;
  p.a_scale = d->a_scale; p.b_scale = d->b_scale; p.b_mn = d->b_mn_major; p.epilogue = d->epilogue;
  p.C = (__nv_bfloat16*)d->C; p.ldc = d->ldc; p.gu = (__nv_bfloat16*)d->gu; p.ldgu = d->ldgu; p.dgu = (__nv_bfloat16*)d->dgu;
  p.row_info = d->row_info; p.peers = d->peers; p.zero_tail = d->zero_tail;
  p.num_peers = d->num_peers; p.peer_rows = d->peer_rows;
  if (d->epilogue == FL_EPI_SCATTER) {
    if (d->num_peers < 1 || d->num_peers > FL_MAX_PEERS) return bad("SCATTER needs 1..8 receive buffers (num_peers)");
    if (d->row_info == nullptr) return bad("SCATTER needs row_info");
    for (int i = 0; i < d->num_peers; ++i)
      if (d->peers.p[i] == nullptr) return bad("SCATTER: a receive buffer is null");
  }
  p.group_m = d->group_m > 0 ? d->group_m : 16; p.status = d->status;
  CUtensorMap tmA, tmB;
  int rc = make_map(&tmA, d->A, d->K, d->cap, d->num_groups, 128, BM);
  if (rc) return rc;
  rc = d->b_mn_major ? make_map(&tmB, d->B, d->N, d->K, d->num_groups, 128, 128)
                     : make_map(&tmB, d->B, d->K, d->N, d->num_groups, 128, BN);
  if (rc) return rc;
  switch (d->epilogue) {
    case FL_EPI_STORE: return launch<FL_EPI_STORE>(tmA, tmB, p, d->max_ctas, stream);
    case FL_EPI_SWIGLU: return launch<FL_EPI_SWIGLU>(tmA, tmB, p, d->max_ctas, stream);
    case FL_EPI_SCATTER: return launch<FL_EPI_SCATTER>(tmA, tmB, p, d->max_ctas, stream);
    default: return launch<FL_EPI_DSWIGLU>(tmA, tmB, p, d->max_ctas, stream);
  }
}

extern "C" int fl_fp8_quantize_rows(const void* x, void* q, float* scale, long long rows, int K, const int* counts, int cap,
                                    cudaStream_t stream) {
  if (K % 128 || rows <= 0) return -1;
  if (counts != nullptr && cap < 1) return -1;
  const long long warps = rows * ((K / 128 + fl8::QR_BLOCKS - 1) / fl8::QR_BLOCKS);
  const int ctas = (int)((warps + 7) / 8 < 148 * 8 ? (warps + 7) / 8 : 148 * 8);
  const bool wide = (((uintptr_t)x & 15) | ((uintptr_t)q & 7)) == 0;
  auto kernel = wide ? fl8::quantize_rows_kernel<true> : fl8::quantize_rows_kernel<false>;
  kernel<<<ctas, 256, 0, stream>>>((const __nv_bfloat16*)x, (__nv_fp8_storage_t*)q, scale, rows, K, counts, cap);
  return (int)cudaGetLastError();
}

extern "C" int fl_fp8_quantize_blocks(const void* w, void* q, float* scale, int G, int R, int C, cudaStream_t stream) {
  if (R % 128 || C % 128 || G < 1) return -1;
  dim3 grid(C / 128, R / 128, G);
  const bool wide = (((uintptr_t)w & 15) | ((uintptr_t)q & 7)) == 0;
  auto kernel = wide ? fl8::quantize_blocks_kernel<true> : fl8::quantize_blocks_kernel<false>;
  kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)w, (__nv_fp8_storage_t*)q, scale, R, C);
  return (int)cudaGetLastError();
}
