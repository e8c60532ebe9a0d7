// The passes of a decoder layer that are not matrix products (see decoder.cu): residual + norm, bias + rotation + page
// write, activation, attention of one new token over its paged cache, greedy choice of the next token.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

enum FlDecDtype : int { FL_DEC_BF16 = 0, FL_DEC_FP16 = 1 };
enum FlDecAct : int { FL_ACT_SILU_GATED = 0, FL_ACT_RELU = 1, FL_ACT_GELU_TANH = 2 };

// What a kernel writes to the status word (device memory or mapped host memory, or null) when an index is outside its table; the
// access is skipped: a row of zeros for the token, no position added, no page written, the page left out of the attention.
// Negative indices count from the end.
enum FlDecStatus : int { FL_DEC_BAD_TOKEN = 1, FL_DEC_BAD_POSITION = 2, FL_DEC_BAD_PAGE = 3,
                        FL_DEC_STALLED = 4 /* a kernel that waited for its operands in vain */ };

// Where the keys and values of a token go.  Layouts are those of kv_pack.cuh.
struct FlPagedKv {
  void* k; void* v;
  const int* block_table; int table_stride;   // [batch][table_stride] page ids
  int layout, layer, layers, num_blocks, block_size, heads;
  int* status;
};

// Tensors of the model's type start at a multiple of 16 bytes (the logits of the greedy choice may start anywhere); otherwise the
// call returns -4 and launches nothing.
#ifdef __cplusplus
extern "C" {
#endif
// x[n] = embed[tokens[n]] (+ pos_embed[pos + offset]); pos: positions, or null for n % seq
int fl_dec_embed(int dtype, const long long* tokens, const long long* pos, const void* embed, const void* pos_embed, void* x,
                 long long rows, int hidden, int seq, int offset, long long vocab, long long pos_rows, int* status, cudaStream_t stream);
// x += y (+ y_bias) where y is given; h = norm(x) * w (+ b): RMS norm without b, layer norm with it
int fl_dec_add_norm(int dtype, void* x, const void* y, const void* y_bias, const void* w, const void* b, void* h, long long rows,
                    int hidden, float eps, cudaStream_t stream);
// qkv [rows, (heads + 2 kv_heads) * dim]: bias added, q and k rotated (rope: [positions][dim / 2] cos then sin), all in place;
// k and v also written to their pages.  pos: positions [rows], or null: row n is token n % seq of request n / seq.
int fl_dec_qkv(int dtype, void* qkv, const void* bias, const float* rope, long long rope_rows, const long long* pos, long long rows,
               int seq, int heads, int dim, const FlPagedKv* kv, cudaStream_t stream);
int fl_dec_act(int dtype, int kind, const void* h, const void* bias, void* out, long long rows, int ffn, cudaStream_t stream);
// out [batch, heads * dim] = attention of q [batch] (row stride q_stride) over positions 0 .. pos of the request's pages
int fl_dec_attention(int dtype, const void* q, long long q_stride, const long long* pos, const FlPagedKv* kv, void* out, int batch,
                     int heads, int dim, cudaStream_t stream);
// out[row] = index of the largest value of logits[row] (the first of equals; NaN counts as largest)
int fl_dec_argmax(int dtype, const void* logits, long long* out, int rows, long long vocab, cudaStream_t stream);
// one decoding step's bookkeeping: history[step][b] = next[b] where the history has such a row; tokens = next; pos += 1; step += 1
int fl_dec_advance(const long long* next, long long* tokens, long long* pos, long long* history, long long* step, int batch, int rows,
                   cudaStream_t stream);
#ifdef __cplusplus
}
#endif
