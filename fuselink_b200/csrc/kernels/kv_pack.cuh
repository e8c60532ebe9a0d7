// Prefill -> decode paged KV-cache hand-off: page gather through the block table, optional layout
// change, and the NVLink transfer, in one kernel (see kv_pack.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

enum FlKvLayout : int {
  FL_KV_BLHSD = 0,  // [block][layer][head][slot][dim]   (prefill-side pool, the order the reference's
                    //  element count blocks*layers*heads*block_size*head_dim implies)
  FL_KV_LBSHD = 1,  // [layer][block][slot][head][dim]   (decode-side pool, attention-kernel friendly)
};

struct FlKvSendArgs {
  const void* src_k; const void* src_v;   // local pools (bf16)
  void* dst_k; void* dst_v;               // pools on the decode GPU (peer-mapped addresses)
  int src_layout, dst_layout;
  int src_num_blocks, dst_num_blocks;     // pool sizes in pages (bounds checks)
  int layers, heads, block_size, head_dim;
  int layer_begin, layer_end;             // layers moved by this launch (per-layer pipelining)
  const int* src_block_table;             // [batch, max_blocks] page ids in the source pool
  const int* dst_block_table;             // [batch, max_blocks] page ids in the destination pool
  const int* num_blocks;                  // [batch] pages in use per request
  int batch, max_blocks;
  // control message folded into the transfer: copied by the last CTA before the flag is published
  const void* hdr_src; void* hdr_dst; int hdr_bytes;
  uint32_t* done_flag;                    // word in the decode GPU's signal pad; set to `seq` when done
  unsigned int seq;
  unsigned int* cta_counter;              // local scratch word, zero before first use (self-resetting)
  int* status;
};

// How the CTAs of a launch end: each adds its ticket to cta_counter, with a mark if it gave up waiting for a copy.  The last one resets the
// word and publishes header and flag only where nobody gave up, so that the receiver's own wait tells it of pages that never came.
constexpr unsigned int FL_KV_GAVE_UP = 1u << 16;   // a launch has fewer CTAs
struct FlKvEnd { bool last, publish; };
#ifdef __CUDACC__
__host__ __device__
#endif
inline unsigned int fl_kv_ticket(bool ok) { return ok ? 1u : 1u + FL_KV_GAVE_UP; }
#ifdef __CUDACC__
__host__ __device__
#endif
inline FlKvEnd fl_kv_end(unsigned int before, bool ok, unsigned int ctas) {
  FlKvEnd e;
  e.last = before % FL_KV_GAVE_UP == ctas - 1;
  e.publish = e.last && ok && before < FL_KV_GAVE_UP;
  return e;
}

#ifdef __cplusplus
extern "C" {
#endif
int fl_kv_pack_send(const FlKvSendArgs* a, int num_ctas, cudaStream_t stream);
#ifdef __cplusplus
}
#endif
