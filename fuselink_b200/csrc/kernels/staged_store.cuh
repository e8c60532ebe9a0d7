// Stores of bf16 blocks from the layout that TMEM hands out (one row per thread), for the GEMMs' epilogues.
#pragma once
#include <cuda_bf16.h>
#include "../common/fl_ptx.cuh"

namespace fl {

constexpr int EPI_STAGE_BYTES = 32 * 64;   // per epilogue warp: 32 rows x 32 bf16, the transposition buffer of its stores

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack_bf16(uint32_t u, float& a, float& b) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  a = __bfloat162float(v.x);
  b = __bfloat162float(v.y);
}

// Coalesced store of a 32-row x 32-column bf16 block that the warp holds row-per-thread (thread t = row t, as TMEM hands
// it out).  Written straight from the registers, every store instruction would touch 32 rows x 16 bytes: 32 half-used
// sectors.  Instead every thread parks its row (64 bytes) in the warp's shared-memory buffer and the warp writes the block
// back out with four lanes per row: one instruction covers 8 rows x 64 contiguous bytes, whole sectors only.
//   pk       the thread's 32 values as 16 packed bf16 pairs
//   row_dst  global address of the first of these 32 columns in the thread's OWN row, 0 if the row is not to be stored
// The 16-byte pieces of a row are XOR-swizzled by the row number so that neither the row-wise writes nor the
// four-lanes-per-row reads conflict on shared-memory banks.
__device__ __forceinline__ void staged_store_packed(uint8_t* stg, int lane, const uint32_t* pk, unsigned long long row_dst) {
  const uint32_t base = smem_u32(stg);
  const uint32_t wsw = (uint32_t)((lane >> 1) & 3);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t a = base + lane * 64 + (((uint32_t)j ^ wsw) << 4);
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(pk[4 * j + 0]), "r"(pk[4 * j + 1]), "r"(pk[4 * j + 2]),
                 "r"(pk[4 * j + 3])
                 : "memory");
  }
  __syncwarp();
  const int piece = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (lane >> 2) + 8 * i;
    const unsigned long long d = __shfl_sync(0xffffffffu, row_dst, r);
    const uint32_t a = base + r * 64 + (((uint32_t)piece ^ (uint32_t)((r >> 1) & 3)) << 4);
    uint4 x;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(a) : "memory");
    if (d != 0) st_v4(reinterpret_cast<void*>(d + 16ull * piece), x);
  }
  __syncwarp();
}

}  // namespace fl
