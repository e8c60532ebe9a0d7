// Chunked multi-segment put, flag wait and flag barrier (see comm_kernels.cuh for the protocol).
//
// Reference parity: the reference moves bytes between GPUs only implicitly (NCCL's copy kernel writes
// through a remapped VA, src/fuselink.cc:43-56) and stripes one transfer over NCCL channels in 512 KiB
// chunks with 8 steps in flight (experiments/bw_test/run_bw_test.sbatch:34-46, src/fuselink.h:14).  Here
// the stripes are explicit: one launch copies any number of (src, dst) segments chunk by chunk and
// publishes a flag per chunk, so a relay GPU can forward chunk c while chunk c+1 is still in flight.
#include "comm_kernels.cuh"
#include "../common/fl_ptx.cuh"
#include <string.h>

namespace fl {

// Bound by memory (or the link): every byte is read once and written once, and small launches by their start and end.  One thread per
// CTA streams through a ring of 16 KiB slots in shared memory with the bulk-copy engine.  A launch is split evenly, in slots, over two
// CTAs per SM, which drain their ring once per segment; dealt out in chunks, each drained before the next was asked for, 320 chunks
// left some SMs with three and some with two.  In chunks | evenly, us: 8 exchanges of 8 x 2.6 MB in a row 137 | 117, of 8 x 131 KB 91 | 70, 4 of
// 4 x 8.4 MB 86 | 75, 2 of 2 x 67 MB 111 | 107; a put and its wait of 64 KiB 8.3 | 6.4, 4 MiB 9.7 | 9.4, 16 MiB 12.9 | 13.3, 64 MiB 27.7 | 27.9, 256 MiB
// 102 | 98.  One CTA per SM with 12 slots: 131, 70, 72, 105; 6.4, 9.4, 10.9, 26, 96; three with 4: 131, 71, 79, 108; 6.4, 9.4, 13.2, 27.4, 99.
constexpr int BULK_SLOT_BYTES = 16 * 1024;
constexpr int BULK_MAX_SLOTS = 6;

__device__ __forceinline__ void copy_bytes(const uint8_t* src, uint8_t* dst, unsigned long long bytes) {
  for (unsigned long long b = threadIdx.x; b < bytes; b += blockDim.x) dst[b] = src[b];
}

// src and dst at the same distance from a multiple of 16, by all threads of the CTA
__device__ __forceinline__ void copy_vec(const uint8_t* src, uint8_t* dst, unsigned long long bytes) {
  const unsigned long long to16 = (16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15, head = to16 < bytes ? to16 : bytes;
  copy_bytes(src, dst, head);
  const int tid = threadIdx.x, nt = blockDim.x;
  const unsigned long long n16 = (bytes - head) >> 4;
  const uint4* s = reinterpret_cast<const uint4*>(src + head);
  uint4* d = reinterpret_cast<uint4*>(dst + head);
  unsigned long long i = tid;
  // 4 independent 16-byte loads in flight per thread before the first store
  for (; i + 3ull * nt < n16; i += 4ull * nt) {
    uint4 a = ld_stream_v4(s + i), b = ld_stream_v4(s + i + nt), c = ld_stream_v4(s + i + 2 * nt), e = ld_stream_v4(s + i + 3 * nt);
    st_v4(d + i, a); st_v4(d + i + nt, b); st_v4(d + i + 2 * nt, c); st_v4(d + i + 3 * nt, e);
  }
  for (; i < n16; i += nt) st_v4(d + i, ld_stream_v4(s + i));
  copy_bytes(src + head + (n16 << 4), dst + head + (n16 << 4), bytes - head - (n16 << 4));
}

// 16 bytes from `sh` bytes (1 to 15) into the 32 that a and b hold
__device__ __forceinline__ uint4 shifted(const uint4& a, const uint4& b, unsigned sh) {
  const bool two = sh & 8, one = sh & 4;
  const unsigned bits = (sh & 3) * 8;
  uint32_t w[6] = {two ? a.z : a.x, two ? a.w : a.y, two ? b.x : a.z, two ? b.y : a.w, two ? b.z : b.x, two ? b.w : b.y};
#pragma unroll
  for (int i = 0; i < 5; ++i) w[i] = one ? w[i + 1] : w[i];
  return make_uint4(__funnelshift_r(w[0], w[1], bits), __funnelshift_r(w[1], w[2], bits), __funnelshift_r(w[2], w[3], bits),
                    __funnelshift_r(w[3], w[4], bits));
}

// Only vectors that lie inside [src, src + bytes) are read, the second of the last pair too.
__host__ __device__ __forceinline__ FlPutShifted put_shifted(unsigned long long src, unsigned long long dst, unsigned long long bytes) {
  FlPutShifted p = {((16 - (dst & 15)) & 15) + 16, 0, 0};                      // 16 more: then src + head - shift is not before src
  p.shift = (unsigned)((src + p.head) & 15);
  const long long body = (long long)bytes - (long long)p.head - 16 + (long long)p.shift;   // bytes of src up to the last vector that may be a second one
  if (body >= 16) p.vectors = (unsigned long long)body >> 4;
  return p;
}

// src and dst at different distances from a multiple of 16, by all threads of the CTA: whole vectors of dst from two neighbouring
// vectors of src each (the second of them is in L1).  Byte by byte throughout, an exchange of blocks of an odd number of elements took 33
// times as long as one of a multiple of eight (8 ranks, 8 x 2.6 MB each: 4427 us against 137; now 134 against 117).
__device__ __forceinline__ void copy_shifted(const uint8_t* src, uint8_t* dst, unsigned long long bytes) {
  constexpr int U = 4;
  const FlPutShifted span = put_shifted(reinterpret_cast<uintptr_t>(src), reinterpret_cast<uintptr_t>(dst), bytes);
  const unsigned long long head = span.head, n = span.vectors;
  const unsigned sh = span.shift;
  if (n == 0) { copy_bytes(src, dst, bytes); return; }
  const uint8_t* s = src + head - sh;
  uint8_t* d = dst + head;
  const unsigned tid = threadIdx.x, nt = blockDim.x;
  unsigned long long i = tid;
  for (; i + (U - 1ull) * nt < n; i += (unsigned long long)U * nt) {
    uint4 a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ld_v4(s + 16 * (i + (unsigned long long)u * nt));
      b[u] = ld_v4(s + 16 * (i + (unsigned long long)u * nt) + 16);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) st_v4(d + 16 * (i + (unsigned long long)u * nt), shifted(a[u], b[u], sh));
  }
  for (; i < n; i += nt) st_v4(d + 16 * i, shifted(ld_v4(s + 16 * i), ld_v4(s + 16 * i + 16), sh));
  copy_bytes(src, dst, head);
  copy_bytes(src + head + 16 * n, dst + head + 16 * n, bytes - head - 16 * n);
}

// One thread streams `bytes` (a multiple of 16, as src and dst are) through the ring of shared-memory slots with the bulk-copy engine:
// global -> smem (mbarrier completion) then smem -> global (bulk group).  No multicast anywhere.
__device__ __forceinline__ bool copy_bulk(const uint8_t* src, uint8_t* dst, unsigned long long bytes, uint8_t* ring, int slots, uint64_t* bars,
                                          uint32_t& phase_bits, int* abort_flag, int* status) {
  const int n = (int)((bytes + BULK_SLOT_BYTES - 1) / BULK_SLOT_BYTES);
  auto slot_bytes = [&](int j) {
    unsigned long long off = (unsigned long long)j * BULK_SLOT_BYTES;
    unsigned long long left = bytes - off;
    return (uint32_t)(left < BULK_SLOT_BYTES ? left : BULK_SLOT_BYTES);
  };
  auto issue_load = [&](int j, int s) {
    mbar_arrive_expect_tx(&bars[s], slot_bytes(j));
    bulk_load(ring + s * BULK_SLOT_BYTES, src + (unsigned long long)j * BULK_SLOT_BYTES, slot_bytes(j), &bars[s]);
  };
  for (int j = 0; j < n && j < slots - 1; ++j) issue_load(j, j);
  bool ok = true;
  int s = 0;
  for (int j = 0; j < n; ++j) {
    ok = mbar_wait(&bars[s], (phase_bits >> s) & 1, abort_flag, status, kTimeoutMbarFull, 500 + s);
    if (!ok) break;
    phase_bits ^= 1u << s;
    fence_proxy_async_smem();
    bulk_store(dst + (unsigned long long)j * BULK_SLOT_BYTES, ring + s * BULK_SLOT_BYTES, slot_bytes(j));
    tma_store_commit();
    const int nj = j + slots - 1, ns = s == 0 ? slots - 1 : s - 1;  // reuses the slot read by store j-1
    if (nj < n) {
      tma_store_wait_read<1>();
      issue_load(nj, ns);
    }
    s = s + 1 == slots ? 0 : s + 1;
  }
  tma_store_wait<0>();  // all writes of this piece performed before the flag is published
  if (!ok) let_copies_land();
  return ok;
}

// What the kernel is launched with: FlPutArgs and FlPutSplit in the room of the former.  The host's time per launch moves with the size, us
// of a put of 64 KiB: 688 bytes (both structures as they are) 4.45, 640 and 624 4.35, 608 and 600 4.0, 592 4.27; hence the last field.
struct PutSeg {
  const uint8_t* src;
  uint8_t* dst;
  unsigned long long bytes;
  uint32_t* flags;
  union {
    const uint32_t* wait_flags;                            // chunks in turn
    struct { unsigned first_cta, first_adds; };            // evenly
  };
  unsigned long long* bytes_done;
  int flag_mode;
  unsigned slot_end;
};
struct PutLaunch {
  PutSeg seg[FL_MAX_SEGS];
  int nseg, use_bulk, slots;                               // slots: of a CTA's ring
  unsigned chunk_bytes, seq, even_slots;
  int* status;
  const uint32_t* wait_flag[8];
  unsigned wait_want[8];
  int nwait;
  unsigned long long* done_scratch;
  unsigned long long unused;
};
static_assert(sizeof(PutLaunch) == 600, "see above");

__global__ void __launch_bounds__(1024) put_chunks_kernel(const __grid_constant__ PutLaunch a) {
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  __shared__ uint64_t bars[BULK_MAX_SLOTS];
  __shared__ int abort_flag;
  __shared__ int wait_ok;
  uint32_t phase_bits = 0;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    if (a.use_bulk) {
      for (int s = 0; s < a.slots; ++s) mbar_init(&bars[s], 1);
      mbar_fence_init();
    }
  }
  __syncthreads();
  grid_dep_wait();

  // by all threads; false if the copy was given up
  auto copy = [&](const uint8_t* s, uint8_t* d, unsigned long long len) -> bool {
    if ((reinterpret_cast<uintptr_t>(s) ^ reinterpret_cast<uintptr_t>(d)) & 15) {
      copy_shifted(s, d, len);
    } else if (!a.use_bulk) {
      copy_vec(s, d, len);
    } else {
      const unsigned long long to16 = (16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15, head = to16 < len ? to16 : len, body = (len - head) & ~15ull;
      if (threadIdx.x == 0 && body != 0) {
        if (!copy_bulk(s + head, d + head, body, dyn_smem, a.slots, bars, phase_bits, &abort_flag, a.status)) abort_flag = 1;
        fence_proxy_async_all();
      }
      copy_bytes(s, d, head);
      copy_bytes(s + head + body, d + head + body, len - head - body);
    }
    __syncthreads();
    return abort_flag == 0;
  };
  // The flag update is itself a release at system scope: it orders this thread's bulk stores (complete, see
  // copy_bulk) and, through the barrier above, the other threads' stores before the flag becomes visible.
  bool live = true;
  if (a.even_slots != 0) {
    // a contiguous piece per CTA, whatever the chunks
    const unsigned mine0 = a.even_slots * blockIdx.x / gridDim.x, mine1 = a.even_slots * (blockIdx.x + 1) / gridDim.x;
    for (int si = 0; si < a.nseg && live; ++si) {
      const PutSeg& sg = a.seg[si];
      const unsigned s0 = si == 0 ? 0 : a.seg[si - 1].slot_end, s1 = sg.slot_end;
      const unsigned from = mine0 > s0 ? mine0 : s0, to = mine1 < s1 ? mine1 : s1;
      if (from >= to) continue;
      const unsigned long long off = (unsigned long long)(from - s0) * BULK_SLOT_BYTES, end = (unsigned long long)(to - s0) * BULK_SLOT_BYTES;
      const unsigned long long len = (end < sg.bytes ? end : sg.bytes) - off;
      live = copy(sg.src + off, sg.dst + off, len);
      if (live && threadIdx.x == 0) {
        if (sg.flag_mode == FL_FLAG_COUNT) red_release_sys_add(sg.flags, blockIdx.x == sg.first_cta ? sg.first_adds : 1u);
        if (sg.bytes_done != nullptr) {
          if (a.done_scratch != nullptr) atomicAdd(a.done_scratch + si, len);
          else atomicAdd_system(sg.bytes_done, len);
        }
      }
    }
  } else {
    // CTAs take chunks round-robin over the concatenation of all segments
    unsigned long long chunks_before = 0;
    for (int si = 0; si < a.nseg && live; ++si) {
      const PutSeg& sg = a.seg[si];
      const unsigned long long nch = (sg.bytes + a.chunk_bytes - 1) / a.chunk_bytes;
      unsigned long long done_here = 0;      // thread 0: bytes of this segment this CTA has finished
      unsigned long long first = (blockIdx.x + gridDim.x - (chunks_before % gridDim.x)) % gridDim.x;
      for (unsigned long long c = first; c < nch && live; c += gridDim.x) {
        const unsigned long long off = c * a.chunk_bytes;
        const unsigned long long len = (sg.bytes - off) < a.chunk_bytes ? (sg.bytes - off) : a.chunk_bytes;
        if (sg.wait_flags) {
          if (threadIdx.x == 0) wait_ok = wait_flag_ge(sg.wait_flags + c, a.seq, a.status, 600 + si) ? 1 : 0;
          __syncthreads();
          const int okv = wait_ok;
          __syncthreads();
          if (!okv) { live = false; break; }
        }
        live = copy(sg.src + off, sg.dst + off, len);
        if (!live) break;
        if (threadIdx.x == 0 && sg.flag_mode != FL_FLAG_NONE) {
          if (sg.flag_mode == FL_FLAG_SEQ_PER_CHUNK) st_release_sys(sg.flags + c, a.seq);
          else red_release_sys_add(sg.flags, 1u);
        }
        // device-side completion counter: the host monitor folds it into the path's completed bytes
        if (threadIdx.x == 0 && sg.bytes_done != nullptr) {
          if (a.done_scratch != nullptr) done_here += len;
          else atomicAdd_system(sg.bytes_done, (unsigned long long)len);
        }
      }
      if (threadIdx.x == 0 && done_here != 0) atomicAdd(a.done_scratch + si, done_here);
      chunks_before += nch;
    }
  }
  if (a.nwait == 0) grid_dep_launch();  // a launch that polls lets nobody take a place before it has seen its flags
  if (a.done_scratch != nullptr && threadIdx.x == 0) {
    // every CTA takes a ticket, also one that gave up a wait; the last one forwards the totals and rearms the words
    __threadfence();
    const unsigned long long ticket = atomicAdd(a.done_scratch + FL_MAX_SEGS, 1ull);
    if (ticket == (unsigned long long)gridDim.x - 1) {
      __threadfence();
      for (int si = 0; si < a.nseg; ++si) {
        const unsigned long long total = atomicExch(a.done_scratch + si, 0ull);
        if (total != 0 && a.seg[si].bytes_done != nullptr) atomicAdd_system(a.seg[si].bytes_done, total);
      }
      atomicExch(a.done_scratch + FL_MAX_SEGS, 0ull);
    }
  }
  if (!live) return;
  if (blockIdx.x == 0 && (int)threadIdx.x < a.nwait)
    wait_flag_ge(a.wait_flag[threadIdx.x], a.wait_want[threadIdx.x], a.status, 650 + threadIdx.x);
}

// Neither of these two lets the next kernel start while it may still have to poll: what stands behind one would hold its SMs meanwhile,
// and what a peer waits for before it sets the flags may be a kernel of another stream that then finds no place.
__global__ void wait_flags_kernel(const FlWaitArgs a) {
  const int i = threadIdx.x;
  grid_dep_wait();
  if (i < a.n) wait_flag_ge(a.flag[i], a.want[i], a.status, 700 + i, a.limit_ns ? a.limit_ns : (uint64_t)FL_FLAG_WAIT_NS);
}

__global__ void barrier_kernel(FlSignalPtrs pads, int slot0, int rank, int world, unsigned int seq, int do_signal,
                               int do_wait, int* status) {
  grid_dep_wait();
  const int r = threadIdx.x;
  if (r >= world) return;
  if (do_signal) {
    fence_sys();
    st_release_sys(pads.p[r] + slot0 + rank, seq);
  }
  if (do_wait) wait_flag_ge(pads.p[rank] + slot0 + r, seq, status, 800 + r);
}

}  // namespace fl

// Small puts of one segment, waits and barriers, often several in a row, are launched so that they may be placed while the kernel before
// them drains; they touch nothing, and poll no flag, before that kernel has ended (grid_dep_wait), so what one polls for is never behind it.
template <typename... P, typename... A>
static int launch_after(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

constexpr unsigned PUT_CTAS = 2 * 148;
// Up to so many CTAs a put is launched early, an exchange (several segments) never.  Plainly | early, us: a put and its wait of 4 KiB 6.3 | 5.2,
// 64 KiB 7.6 | 6.4, 512 KiB (8 CTAs) 9.0 | 8.8, 1 MiB (16) 8.8 | 8.8, 2 MiB (32) 9.5 | 8.9, 8 MiB (128) 9.5 | 9.1, 16 MiB (256) 13.5 | 13.9; beyond 32 the
// half microsecond is not worth the room that CTAs take from other streams while they wait their turn.  Eight exchanges of 0.5 MB (8 CTAs)
// 69.8 | 74, of 1 MB (16) 69.5 | 75, of 2 MB (32) 71 | 75, of 4 MB (64) 74 | 74.6, of 21 MB (256) 117 | 140 (on other GPUs of the same model 125 | 103).
constexpr int PUT_EARLY_CTAS = 32;

// The even split of the launch over its G CTAs, where nothing is waited for or flagged chunk by chunk, and no segment is shared by more CTAs
// than it has chunks to count.  Made here, since the kernel's 64-bit divisions stood before its first load: eight exchanges of 1 MB 94 us with
// them, 77 without, of 21 MB 127 and 117, a put of 4 MiB 9.3 and 8.2.  What the kernel multiplies fits 32 bits (up to 237 GB on 296 CTAs).
static void even_split(const FlPutArgs* a, unsigned G, FlPutSplit* sp) {
  sp->slots = 0;
  unsigned long long U = 0;
  for (int i = 0; i < a->nseg; ++i) {
    if (a->seg[i].wait_flags != nullptr || a->seg[i].flag_mode == FL_FLAG_SEQ_PER_CHUNK) return;
    U += (a->seg[i].bytes + fl::BULK_SLOT_BYTES - 1) / fl::BULK_SLOT_BYTES;
    if (U * G > 0xffffffffull) return;
    sp->slot_end[i] = (unsigned)U;
  }
  if (U < G) return;
  const unsigned slots = (unsigned)U;
  for (int i = 0; i < a->nseg; ++i) {
    const unsigned s0 = i == 0 ? 0 : sp->slot_end[i - 1], s1 = sp->slot_end[i];
    if (s0 == s1) continue;
    const unsigned long long chunks = (a->seg[i].bytes + a->chunk_bytes - 1) / a->chunk_bytes;
    const unsigned first = s0 == 0 ? 0 : ((s0 + 1) * G - 1) / slots, others = (s1 == slots ? G - 1 : (s1 * G - 1) / slots) - first;
    if (a->seg[i].flag_mode == FL_FLAG_COUNT && others >= chunks) return;
    sp->first_cta[i] = first;
    sp->first_adds[i] = (unsigned)(chunks - others);
  }
  sp->slots = slots;
}

extern "C" int fl_put_split(const FlPutArgs* args, unsigned int num_ctas, FlPutSplit* out) {
  if (args->nseg < 1 || args->nseg > FL_MAX_SEGS || args->chunk_bytes == 0 || num_ctas == 0) return -1;
  even_split(args, num_ctas, out);
  return 0;
}
extern "C" int fl_put_shifted(unsigned long long src, unsigned long long dst, unsigned long long bytes, FlPutShifted* out) {
  if (((src ^ dst) & 15) == 0) return -1;
  *out = fl::put_shifted(src, dst, bytes);
  return 0;
}

extern "C" int fl_put_chunks(const FlPutArgs* args, int num_ctas, int threads, cudaStream_t stream) {
  if (args->nseg < 1 || args->nseg > FL_MAX_SEGS) return -1;
  if (args->chunk_bytes == 0 || (args->chunk_bytes & 15)) return -2;
  if (threads <= 0 || threads > 1024) threads = 512;
  if (num_ctas <= 0) num_ctas = 1;
  int slots = 0;
  FlPutSplit even;
  if (args->use_bulk) {
    // as many slots as a CTA will fill; threads beyond the one that feeds the engine only where bytes have to be shifted
    for (int i = 0; i < args->nseg; ++i)
      if (((uintptr_t)args->seg[i].src ^ (uintptr_t)args->seg[i].dst) & 15) threads = 512;
    const unsigned G = (unsigned)num_ctas < PUT_CTAS ? (unsigned)num_ctas : PUT_CTAS;
    even_split(args, G, &even);
    unsigned long long per_cta = (args->chunk_bytes + fl::BULK_SLOT_BYTES - 1) / fl::BULK_SLOT_BYTES;
    slots = 4;
    if (even.slots != 0) {
      num_ctas = (int)G;
      per_cta = (even.slots + G - 1) / G;
      slots = fl::BULK_MAX_SLOTS;
    }
    if (per_cta + 1 < (unsigned long long)slots) slots = (int)per_cta + 1;
  } else {
    even_split(args, (unsigned)num_ctas, &even);
  }
  const size_t smem = (size_t)slots * fl::BULK_SLOT_BYTES;
  if (smem > 0) {                           // three slots are 48 KiB, which with the kernel's own few words is more than a launch gets unasked
    static bool set_on[64];                 // per device: a process may drive several GPUs
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return -3;
    if (!set_on[dev]) {
      cudaError_t e = cudaFuncSetAttribute(fl::put_chunks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, fl::BULK_MAX_SLOTS * fl::BULK_SLOT_BYTES);
      // two CTAs per SM are what the split counts on; left to the driver it is the same where launches follow one another (117 us either way)
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fl::put_chunks_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return (int)e;
      set_on[dev] = true;
    }
  }
  fl::PutLaunch k;
  for (int i = 0; i < args->nseg; ++i) {
    const FlSeg& from = args->seg[i];
    k.seg[i].src = reinterpret_cast<const uint8_t*>(from.src);
    k.seg[i].dst = reinterpret_cast<uint8_t*>(from.dst);
    k.seg[i].bytes = from.bytes;
    k.seg[i].flags = from.flags;
    k.seg[i].bytes_done = from.bytes_done;
    k.seg[i].flag_mode = from.flag_mode;
    if (even.slots != 0) {
      k.seg[i].slot_end = even.slot_end[i];
      k.seg[i].first_cta = even.first_cta[i];
      k.seg[i].first_adds = even.first_adds[i];
    } else {
      k.seg[i].wait_flags = from.wait_flags;
    }
  }
  k.nseg = args->nseg; k.use_bulk = args->use_bulk; k.slots = slots;
  k.chunk_bytes = args->chunk_bytes; k.seq = args->seq; k.even_slots = even.slots;
  k.status = args->status;
  k.nwait = args->nwait;
  for (int i = 0; i < args->nwait && i < 8; ++i) { k.wait_flag[i] = args->wait_flag[i]; k.wait_want[i] = args->wait_want[i]; }
  k.done_scratch = args->done_scratch;
  if (num_ctas > PUT_EARLY_CTAS || args->nseg > 1) {
    fl::put_chunks_kernel<<<num_ctas, threads, smem, stream>>>(k);
    return (int)cudaGetLastError();
  }
  return launch_after(fl::put_chunks_kernel, (unsigned)num_ctas, (unsigned)threads, smem, stream, k);
}

extern "C" int fl_all_to_all(const void* send, void* const* recv_peers, unsigned long long bytes_per_peer, int rank,
                             int world, FlSignalPtrs pads, int slot0, unsigned int chunk_bytes, const unsigned int* want,
                             int use_bulk, int num_ctas, int threads, int* status, cudaStream_t stream) {
  if (world < 1 || world > FL_MAX_SEGS) return -1;
  FlPutArgs a;
  memset(&a, 0, sizeof a);
  a.nseg = world;
  for (int k = 0; k < world; ++k) {
    const int p = (rank + k) % world;   // own block first, then walk the ring so peers are hit evenly
    a.seg[k].src = reinterpret_cast<const uint8_t*>(send) + (unsigned long long)p * bytes_per_peer;
    a.seg[k].dst = reinterpret_cast<uint8_t*>(recv_peers[p]) + (unsigned long long)rank * bytes_per_peer;
    a.seg[k].bytes = bytes_per_peer;
    a.seg[k].flags = pads.p[p] + slot0 + rank;
    a.seg[k].flag_mode = FL_FLAG_COUNT;
  }
  a.chunk_bytes = chunk_bytes;
  a.use_bulk = use_bulk;
  a.status = status;
  if (want) {
    a.nwait = world;
    for (int r = 0; r < world; ++r) {
      a.wait_flag[r] = pads.p[rank] + slot0 + r;
      a.wait_want[r] = want[r];
    }
  }
  return fl_put_chunks(&a, num_ctas, threads, stream);
}

extern "C" int fl_wait_flags(const FlWaitArgs* args, cudaStream_t stream) {
  if (args->n < 0 || args->n > 16) return -1;
  if (args->n == 0) return 0;
  return launch_after(fl::wait_flags_kernel, 1, 32, 0, stream, *args);
}

extern "C" int fl_barrier(FlSignalPtrs pads, int slot0, int rank, int world, unsigned int seq, int do_signal,
                          int do_wait, int* status, cudaStream_t stream) {
  if (world < 1 || world > 8) return -1;
  return launch_after(fl::barrier_kernel, 1, 32, 0, stream, pads, slot0, rank, world, seq, do_signal, do_wait, status);
}
