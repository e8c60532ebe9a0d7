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
#include "tile_map.cuh"

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

// The same through the copy engine: a unit is a few heads of a page (up to 32 KiB), contiguous in the source, brought into shared memory by
// one bulk load and stored by one TMA store, whose tensor map walks the destination in the source's order of head, slot and column.
// Bound by memory.  A warp per CTA and two CTAs per SM, three slots each (192 KB per SM on the way): the lanes look up the pages of 32
// units at a time, the first lane feeds the engine.  Through registers | here, us: 16 x 2048 tokens of 32 layers, 8 heads of 128 (8.6 GB of
// bytes, 1330 us at the rate of a copy) 1540 | 1391; 13 x 816 of 12 layers, 12 heads of 64 178 | 144; 4 x 1808 of 24 layers, 16 of 64 286 |
// 243; 13 x 1280 of one layer, 32 of 64 77 | 60.  Units of 16 KiB in six slots: 1506, 146, 258, 64; of 8 KiB in twelve: 2420 (a store costs
// the engine over a microsecond whatever its size), so pages of less than 16 KiB stay with the other kernel (4 x 1584 of 32 layers, 2 heads
// of 128: 100 | 113).
constexpr int KVB_SLOTS = 3, KVB_SLOT_BYTES = 32 * 1024, KVB_LEAST = 16 * 1024, KVB_LEAST_CALL = 16 << 20;

__global__ void __launch_bounds__(32) kv_pack_bulk_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                                                          const FlKvSendArgs a, const int group /* heads per unit */) {
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ uint64_t full[KVB_SLOTS];
  __shared__ int s_end[KV_BATCH];
  __shared__ int abort_flag;
  const int lane = threadIdx.x;
  if (lane == 0) {
    for (int s = 0; s < KVB_SLOTS; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
    abort_flag = 0;
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  int total = 0;                                       // running totals of the requests' pages
  for (int b0 = 0; b0 < a.batch; b0 += 32) {
    int n = b0 + lane < a.batch ? max(0, min(a.num_blocks[b0 + lane], a.max_blocks)) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int m = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += m;
    }
    if (b0 + lane < a.batch) s_end[b0 + lane] = total + n;
    total += __shfl_sync(0xffffffffu, n, 31);
  }
  __syncwarp();
  const int H = a.heads, chunks = (H + group - 1) / group, nl = a.layer_end - a.layer_begin;
  const unsigned head_bytes = (unsigned)a.block_size * a.head_dim * 2;
  const long long units = (long long)total * nl * 2 * chunks, mine = units > blockIdx.x ? (units - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  auto unit = [&](long long i) { return blockIdx.x + i * gridDim.x; };
  // where a unit comes from (bytes) and goes to (page of the destination map); -1: not this CTA's, or a page id outside its pool
  struct Place { long long from; int to; int what; };     // what: chunk * 2 + (0: keys, 1: values)
  auto look_up = [&](long long i) -> Place {
    Place p = {-1, -1, 0};
    if (i >= mine) return p;
    const long long u = unit(i), w = u / (2 * chunks);
    const int rest = (int)(u - w * (2 * chunks)), layer = a.layer_begin + (int)(w % nl);
    int pg = (int)(w / nl), b = 0;
    for (int hi = a.batch - 1; b < hi;) {                 // the first request that ends behind pg
      const int mid = (b + hi) / 2;
      if (s_end[mid] <= pg) b = mid + 1; else hi = mid;
    }
    if (b > 0) pg -= s_end[b - 1];
    const long long at = (long long)b * a.max_blocks + pg;
    const int sblk = a.src_block_table[at], dblk = a.dst_block_table[at];
    if (sblk < 0 || sblk >= a.src_num_blocks || dblk < 0 || dblk >= a.dst_num_blocks) {
      report(a.status, kBadIndex, 1000);
      return p;                                           // skipped
    }
    p.what = rest;                                        // chunk outermost, keys and values of it next to one another
    p.from = page_base(a.src_layout, a.src_num_blocks, a.layers, (long long)H * head_bytes, sblk, layer) + (long long)(rest >> 1) * group * head_bytes;
    p.to = (int)page_base(a.dst_layout, a.dst_num_blocks, a.layers, 1, dblk, layer);
    return p;
  };
  Place here = look_up(lane), next = look_up(32 + lane);  // of units [32 w, 32 w + 32) and the 32 behind them, w of the unit being loaded
  uint32_t phases = 0;
  bool ok = true;
  long long loaded = 0, window = 0;
  int held_to[KVB_SLOTS], held_what[KVB_SLOTS];           // lane 0: what the slots hold (-1: nothing)
#pragma unroll
  for (int s = 0; s < KVB_SLOTS; ++s) { held_to[s] = -1; held_what[s] = 0; }
  auto load = [&](int s) {                                // every lane; unit `loaded` into slot s
    if (loaded - window == 32) {
      window += 32;
      here = next;
      next = look_up(window + 32 + lane);
    }
    const int l = (int)(loaded - window);
    const long long from = __shfl_sync(0xffffffffu, here.from, l);
    const int to = __shfl_sync(0xffffffffu, here.to, l), what = __shfl_sync(0xffffffffu, here.what, l);
    held_to[s] = from < 0 ? -1 : to;
    held_what[s] = what;
    if (lane == 0 && from >= 0) {
      const unsigned bytes = (unsigned)min(group, H - (what >> 1) * group) * head_bytes;
      mbar_arrive_expect_tx(&full[s], bytes);
      bulk_load(ring + s * KVB_SLOT_BYTES, reinterpret_cast<const uint8_t*>(what & 1 ? a.src_v : a.src_k) + from, bytes, &full[s]);
    }
    ++loaded;
  };
#pragma unroll
  for (int s = 0; s < KVB_SLOTS - 1; ++s)
    if (loaded < mine) load(s);
  for (long long i0 = 0; i0 < mine && ok; i0 += KVB_SLOTS) {
#pragma unroll
    for (int s = 0; s < KVB_SLOTS; ++s) {
      if (i0 + s < mine && ok) {
        if (held_to[s] >= 0) {
          ok = mbar_wait_warp(&full[s], (phases >> s) & 1, &abort_flag, a.status, kTimeoutMbarFull, 1010 + s);
          if (!ok) break;
          phases ^= 1u << s;
          if (lane == 0) {
            fence_proxy_async_smem();
            tma_store_4d(held_what[s] & 1 ? &tm_v : &tm_k, ring + s * KVB_SLOT_BYTES, 0, 0, (held_what[s] >> 1) * group, held_to[s]);
          }
        }
        if (lane == 0) {
          tma_store_commit();
          tma_store_wait_read<1>();                       // the store before this one has left its slot
        }
        __syncwarp();
        if (loaded < mine) load((s + KVB_SLOTS - 1) % KVB_SLOTS);
      }
    }
  }
  if (lane == 0) {
    if (!ok) let_copies_land();
    tma_store_wait<0>();
    fence_proxy_async_all();
    fence_sys();
  }
  unsigned before = 0;
  if (lane == 0) before = atomicAdd(a.cta_counter, fl_kv_ticket(ok));
  const FlKvEnd end = fl_kv_end(__shfl_sync(0xffffffffu, before, 0), ok, gridDim.x);
  if (!end.last) return;
  if (end.publish && a.hdr_bytes > 0 && a.hdr_src && a.hdr_dst) {
    // by a single warp: a launch with a header of 8 KiB and no pages takes 47 us byte after byte, 11 as vectors (the other kernel's 13)
    const uint8_t* from = reinterpret_cast<const uint8_t*>(a.hdr_src);
    uint8_t* to = reinterpret_cast<uint8_t*>(a.hdr_dst);
    const int whole = (((uintptr_t)from | (uintptr_t)to) & 15) ? 0 : a.hdr_bytes / 16 * 16;
#pragma unroll 4
    for (int i = 16 * lane; i < whole; i += 16 * 32) st_v4(to + i, ld_v4(from + i));
    for (int i = whole + lane; i < a.hdr_bytes; i += 32) to[i] = from[i];
  }
  __syncwarp();
  if (lane == 0) {
    *a.cta_counter = 0;
    fence_sys();
    if (end.publish && a.done_flag) st_release_sys(a.done_flag, a.seq);
  }
}

// The destination's pages in the source's order: columns, slots, heads, pages.
static int kv_map(CUtensorMap* m, void* base, const FlKvSendArgs* a, int group) {
  const TileEncodeFn enc = tile_encode();
  if (enc == nullptr) return -10;
  const cuuint64_t D = a->head_dim, H = a->heads, S = a->block_size;
  const bool shd = a->dst_layout == FL_KV_LBSHD;
  const cuuint64_t dims[4] = {D, S, H, (cuuint64_t)a->dst_num_blocks * a->layers};
  const cuuint64_t strides[3] = {shd ? H * D * 2 : D * 2, shd ? D * 2 : S * D * 2, H * S * D * 2};
  const cuuint32_t box[4] = {(cuuint32_t)D, (cuuint32_t)S, (cuuint32_t)group, 1}, step[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, base, dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -12;
}

// Heads per unit of the bulk kernel, 0 if it does not take the call: heads of at most 256 columns and pages of at most 256 slots (a
// box's sides), contiguous in the source, units of 16 to 32 KiB, pools from a multiple of 16 bytes on.  Not where the block tables have
// room for less than 16 MiB of pages (how many are used only the GPU knows): a prefill of small models sends layer by layer, and a launch
// costs more than the other kernel's (GPT-2, 4 x 64 tokens: 2106 us, 2163 here).  The launch that ends a hand-off, a header and no pages, takes
// this kernel with the rest.
static int kv_group(const FlKvSendArgs* a) {
  const long long head = (long long)a->block_size * a->head_dim * 2;
  if (a->src_layout != FL_KV_BLHSD || a->batch > KV_BATCH || a->head_dim < 8 || a->head_dim > 256 || a->block_size < 1 || a->block_size > 256 ||
      a->heads < 1 || a->dst_num_blocks < 1 || (long long)a->dst_num_blocks * a->layers > 0x7fffffffll)
    return 0;
  if (((uintptr_t)a->src_k | (uintptr_t)a->src_v | (uintptr_t)a->dst_k | (uintptr_t)a->dst_v) & 15) return 0;
  long long g = KVB_SLOT_BYTES / head;
  if (g > a->heads) g = a->heads;
  if (g > 256) g = 256;
  const double bytes = 2. * a->batch * a->max_blocks * (a->layer_end - a->layer_begin) * (double)a->heads * (double)head;
  return g * head >= KVB_LEAST && bytes >= KVB_LEAST_CALL ? (int)g : 0;
}

}  // namespace fl

extern "C" int fl_kv_pack_send(const FlKvSendArgs* a, int num_ctas, cudaStream_t stream) {
  if (a->head_dim % 8) return -1;
  if (a->layer_begin < 0 || a->layer_end > a->layers || a->layer_begin >= a->layer_end) return -2;
  if (a->batch < 1 || a->max_blocks < 1) return -3;
  if (!a->cta_counter) return -4;
  const int group = fl::kv_group(a);
  if (group > 0) {
    CUtensorMap tm_k, tm_v;
    int rc = fl::kv_map(&tm_k, a->dst_k, a, group);
    if (rc == 0) rc = fl::kv_map(&tm_v, a->dst_v, a, group);
    if (rc != 0) return rc;
    constexpr int smem = fl::KVB_SLOTS * fl::KVB_SLOT_BYTES, most = 2 * 148;
    static bool set_on[64];                 // per device: a process may drive several GPUs
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -5;
    if (!set_on[dev]) {
      cudaError_t e = cudaFuncSetAttribute(fl::kv_pack_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fl::kv_pack_bulk_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return (int)e;
      set_on[dev] = true;
    }
    fl::kv_pack_bulk_kernel<<<num_ctas > 0 && num_ctas < most ? num_ctas : most, 32, smem, stream>>>(tm_k, tm_v, *a, group);
    return (int)cudaGetLastError();
  }
  if (num_ctas <= 0) num_ctas = 148 * 6;
  const bool order = a->src_layout != a->dst_layout, small = (long long)a->heads * a->block_size * (a->head_dim / 8) < 65536;
  auto kernel = order ? (small ? fl::kv_pack_send_kernel<true, true> : fl::kv_pack_send_kernel<true, false>)
                      : fl::kv_pack_send_kernel<false, true>;
  kernel<<<num_ctas, 256, 0, stream>>>(*a);
  return (int)cudaGetLastError();
}
