// kv_pack_send: the KV hand-off of disaggregated serving as one kernel.
//
// Reference behaviour being replaced (experiments/serving/model.hh:253-337): after the whole prefill,
// five ncclSend calls in one group ship the first tokens, the entire K pool, the entire V pool, the
// block table and the block counts to rank + world/2; the decoder mirrors them with ncclRecv
// (model.hh:420-426).  Here only the pages a request owns are moved, they are re-laid-out on the fly for
// the decode side, the metadata rides along as a header, and completion is one release-store per launch,
// so layer l can be in flight while layer l+1 is still being computed.
#include "kv_pack.cuh"
#include "../common/fl_ptx.cuh"

namespace fl {

__device__ __forceinline__ long long page_base(int layout, int nblocks, int layers, long long page_elems, int blk,
                                               int layer) {
  return layout == FL_KV_BLHSD ? ((long long)blk * layers + layer) * page_elems
                               : ((long long)layer * nblocks + blk) * page_elems;
}

// v / d for v, d < 2^16, with m = ceil(2^32 / d): the error m d - 2^32 is below d, so v times it stays below 2^32
__device__ __forceinline__ unsigned div16(unsigned v, unsigned m, unsigned d) { return d == 1 ? v : __umulhi(v, m); }

// Bound by memory: a page at a time per CTA, four 16-byte copies per thread requested before the first is stored, six CTAs per
// SM.  The page's request comes from a table of running totals in shared memory, and the next page's ids are fetched while this
// one is copied; with a walk over the requests' counts and two divisions per 16 bytes 16 x 2048 tokens of 32 layers took
// 1968 us, now 1540 (8.6 GB of bytes: 1310 us).  ORDER: the order inside a page differs.
constexpr int KV_BATCH = 1024;      // requests whose running totals are kept; larger batches walk the counts

template <bool ORDER, bool SMALL>   // SMALL: a page of fewer than 2^16 vectors
__global__ void __launch_bounds__(256, 6) kv_pack_send_kernel(const FlKvSendArgs a) {
  const int H = a.heads, S = a.block_size, D = a.head_dim;
  const unsigned vec_per_row = D / 8;                  // 16-byte vectors per (head, slot) row
  const unsigned vec_per_page = (unsigned)H * S * vec_per_row;
  const long long page_elems = (long long)H * S * D;
  const int nl = a.layer_end - a.layer_begin;
  const bool dst_shd = a.dst_layout == FL_KV_LBSHD;
  const unsigned inner = dst_shd ? H : S;              // rows run over (outer, inner) in the destination, the other way in the source
  const unsigned outer = dst_shd ? S : H;
  const unsigned mrow = SMALL ? 0xffffffffu / vec_per_row + 1 : 0, minner = SMALL ? 0xffffffffu / inner + 1 : 0;

  __shared__ int s_end[KV_BATCH];
  __shared__ int s_total;
  if (a.batch <= KV_BATCH)
    for (int b = threadIdx.x; b < a.batch; b += blockDim.x) s_end[b] = max(0, min(a.num_blocks[b], a.max_blocks));
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0;
    for (int b = 0; b < a.batch; ++b) {
      tot += a.batch <= KV_BATCH ? s_end[b] : max(0, min(a.num_blocks[b], a.max_blocks));
      if (a.batch <= KV_BATCH) s_end[b] = tot;
    }
    s_total = tot;
  }
  __syncthreads();
  const long long units = (long long)s_total * nl * 2;

  auto page_ids = [&](long long u) -> int2 {
    if (u >= units) return make_int2(-1, -1);
    int pg = (int)((u >> 1) / nl), b = 0;
    if (a.batch <= KV_BATCH) {
      for (int hi = a.batch - 1; b < hi;) {              // the first request that ends behind pg
        const int mid = (b + hi) / 2;
        if (s_end[mid] <= pg) b = mid + 1; else hi = mid;
      }
      if (b > 0) pg -= s_end[b - 1];
    } else {
      for (; b < a.batch; ++b) {
        const int nb = max(0, min(a.num_blocks[b], a.max_blocks));
        if (pg < nb) break;
        pg -= nb;
      }
    }
    const long long at = (long long)b * a.max_blocks + pg;
    return make_int2(a.src_block_table[at], a.dst_block_table[at]);
  };
  int2 next = page_ids(blockIdx.x);
  for (long long u = blockIdx.x; u < units; u += gridDim.x) {
    const int sblk = next.x, dblk = next.y;
    next = page_ids(u + gridDim.x);
    const int kv = (int)(u & 1);
    const int layer = a.layer_begin + (int)((u >> 1) % nl);
    if (sblk < 0 || sblk >= a.src_num_blocks || dblk < 0 || dblk >= a.dst_num_blocks) {
      if (threadIdx.x == 0) report(a.status, kBadIndex, 1000);
      continue;  // skip the access, keep going
    }
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(kv ? a.src_v : a.src_k) +
                               page_base(a.src_layout, a.src_num_blocks, a.layers, page_elems, sblk, layer);
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(kv ? a.dst_v : a.dst_k) +
                         page_base(a.dst_layout, a.dst_num_blocks, a.layers, page_elems, dblk, layer);
    auto source_of = [&](unsigned v) -> unsigned {       // iterates in destination order
      if (!ORDER) return v;
      const unsigned rw = SMALL ? div16(v, mrow, vec_per_row) : v / vec_per_row;
      const unsigned o = SMALL ? div16(rw, minner, inner) : rw / inner;
      return ((rw - o * inner) * outer + o) * vec_per_row + (v - rw * vec_per_row);
    };
    for (unsigned v = threadIdx.x; v < vec_per_page; v += 4 * 256) {
      uint4 r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (v + i * 256 < vec_per_page) r[i] = ld_nc_v4(reinterpret_cast<const uint4*>(src) + source_of(v + i * 256));
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (v + i * 256 < vec_per_page) st_v4(reinterpret_cast<uint4*>(dst) + v + i * 256, r[i]);
    }
  }

  // completion: the last CTA to finish copies the header and publishes the flag
  __syncthreads();
  __shared__ int s_last;
  if (threadIdx.x == 0) {
    fence_sys();
    const unsigned int prev = atomicAdd(a.cta_counter, 1u);
    s_last = (prev == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (s_last) {
    if (a.hdr_bytes > 0 && a.hdr_src && a.hdr_dst) {
      for (int i = threadIdx.x; i < a.hdr_bytes; i += blockDim.x)
        reinterpret_cast<uint8_t*>(a.hdr_dst)[i] = reinterpret_cast<const uint8_t*>(a.hdr_src)[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      *a.cta_counter = 0;
      fence_sys();
      if (a.done_flag) st_release_sys(a.done_flag, a.seq);
    }
  }
}

}  // namespace fl

extern "C" int fl_kv_pack_send(const FlKvSendArgs* a, int num_ctas, cudaStream_t stream) {
  if (a->head_dim % 8) return -1;
  if (a->layer_begin < 0 || a->layer_end > a->layers || a->layer_begin >= a->layer_end) return -2;
  if (a->batch < 1 || a->max_blocks < 1) return -3;
  if (!a->cta_counter) return -4;
  if (num_ctas <= 0) num_ctas = 148 * 6;
  const bool order = a->src_layout != a->dst_layout, small = (long long)a->heads * a->block_size * (a->head_dim / 8) < 65536;
  auto kernel = order ? (small ? fl::kv_pack_send_kernel<true, true> : fl::kv_pack_send_kernel<true, false>)
                      : fl::kv_pack_send_kernel<false, true>;
  kernel<<<num_ctas, 256, 0, stream>>>(*a);
  return (int)cudaGetLastError();
}
