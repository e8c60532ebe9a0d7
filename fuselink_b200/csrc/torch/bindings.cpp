// Python bindings (pybind11 through the torch extension headers).  Tensors are passed as torch tensors,
// peer buffers as integer device addresses (they live in other ranks' symmetric regions and have no
// tensor in this process).  Every launcher runs on the current CUDA stream.
#include <torch/extension.h>
#include <c10/cuda/CUDAStream.h>
#include <c10/cuda/CUDAGuard.h>

#include "../kernels/grouped_gemm.cuh"
#include "../kernels/shadow_reduce.cuh"
#include "../kernels/comm_kernels.cuh"
#include "../kernels/embbag.cuh"
#include "../kernels/interact.cuh"
#include "../kernels/mlp_bwd.cuh"
#include "../kernels/kv_pack.cuh"
#include "../kernels/decoder.cuh"
#include "../kernels/thin_gemm.cuh"
#include "../kernels/moe_dispatch.cuh"
#include "../kernels/moe_route.cuh"
#include "../kernels/fp8_gemm.cuh"
#include "../mem/vmm.h"
#include "../monitor/monitor.h"
void fl_monitor_bind(pybind11::module& m);

namespace py = pybind11;

static cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

static void check_rc(int rc, const char* what, const char* detail = nullptr) {
  if (rc == 0) return;
  std::string msg = std::string(what) + " failed with code " + std::to_string(rc);
  if (rc > 0) msg += std::string(" (") + cudaGetErrorString((cudaError_t)rc) + ")";
  if (detail && detail[0]) msg += std::string(": ") + detail;
  throw std::runtime_error(msg);
}

static FlPeerPtrs to_peers(const std::vector<int64_t>& v) {
  FlPeerPtrs p;
  memset(&p, 0, sizeof p);
  TORCH_CHECK(v.size() <= FL_MAX_PEERS, "at most 8 peers");
  for (size_t i = 0; i < v.size(); ++i) p.p[i] = reinterpret_cast<void*>(v[i]);
  return p;
}
static void* opt_ptr(const c10::optional<torch::Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }

// ------------------------------------------------------------------------------------------------ GEMM
static void grouped_gemm(int64_t group_mode, int64_t num_groups, int64_t cap, int64_t M, int64_t N, int64_t K,
                         c10::optional<torch::Tensor> counts, torch::Tensor A, bool a_mn, int64_t lda, int64_t gsa,
                         torch::Tensor B, bool b_mn, int64_t ldb, int64_t gsb, int64_t epilogue,
                         c10::optional<torch::Tensor> C, int64_t ldc, int64_t gsc, c10::optional<torch::Tensor> gu,
                         int64_t ldgu, c10::optional<torch::Tensor> dgu, c10::optional<torch::Tensor> row_info,
                         std::vector<int64_t> peers, double sgd_lr, bool zero_tail, int64_t group_m, int64_t max_ctas,
                         c10::optional<torch::Tensor> status, int64_t peer_rows, int64_t expect_rows) {
  TORCH_CHECK(A.is_cuda() && B.is_cuda(), "grouped_gemm needs CUDA tensors");
  TORCH_CHECK(A.scalar_type() == torch::kBFloat16 && B.scalar_type() == torch::kBFloat16, "bf16 operands expected");
  c10::cuda::CUDAGuard guard(A.device());
  FlGemmDesc d;
  memset(&d, 0, sizeof d);
  d.group_mode = (int)group_mode; d.num_groups = (int)num_groups; d.cap = (int)cap;
  d.M = (int)M; d.N = (int)N; d.K = (int)K;
  d.counts = counts.has_value() ? counts->data_ptr<int>() : nullptr;
  d.elem_bytes = 2;
  d.A = A.data_ptr(); d.a_mn_major = a_mn; d.lda = lda; d.gsa = gsa;
  d.B = B.data_ptr(); d.b_mn_major = b_mn; d.ldb = ldb; d.gsb = gsb;
  d.epilogue = (int)epilogue;
  d.C = opt_ptr(C); d.ldc = ldc; d.gsc = gsc;
  d.gu = opt_ptr(gu); d.ldgu = ldgu; d.dgu = opt_ptr(dgu);
  d.row_info = row_info.has_value() ? row_info->data_ptr<int>() : nullptr;
  d.peers = to_peers(peers); d.num_peers = (int)peers.size(); d.peer_rows = peer_rows;
  d.sgd_lr = (float)sgd_lr; d.zero_tail = zero_tail; d.group_m = (int)group_m; d.max_ctas = (int)max_ctas;
  d.status = status.has_value() ? status->data_ptr<int>() : nullptr;
  d.expect_rows = (int)std::min<int64_t>(std::max<int64_t>(expect_rows, 0), INT32_MAX);
  check_rc(fl_grouped_gemm(&d, cur_stream()), "fl_grouped_gemm", fl_gemm_last_error());
}

// Weight-gradient GEMM whose result rows go straight to the ranks that sum them (FlGemmDesc::push_world): a: [G*cap, M],
// b: [G*cap, N] token-major, peers: every rank's staging [G][world][M / world][N].
static void grouped_gemm_wgrad_push(int64_t num_groups, int64_t cap, torch::Tensor counts, torch::Tensor A, torch::Tensor B,
                                    std::vector<int64_t> peers, int64_t rank, int64_t block_log2, int64_t group_m,
                                    int64_t max_ctas, c10::optional<torch::Tensor> status) {
  TORCH_CHECK(A.is_cuda() && B.is_cuda() && counts.is_cuda(), "grouped_gemm_wgrad_push needs CUDA tensors");
  TORCH_CHECK(A.scalar_type() == torch::kBFloat16 && B.scalar_type() == torch::kBFloat16, "bf16 operands expected");
  TORCH_CHECK(A.dim() == 2 && B.dim() == 2 && A.size(0) == num_groups * cap && B.size(0) == num_groups * cap &&
              A.is_contiguous() && B.is_contiguous(), "a: [G*cap, M], b: [G*cap, N] contiguous");
  c10::cuda::CUDAGuard guard(A.device());
  const int64_t M = A.size(1), N = B.size(1);
  FlGemmDesc d;
  memset(&d, 0, sizeof d);
  d.group_mode = 1; d.num_groups = (int)num_groups; d.cap = (int)cap; d.M = (int)M; d.N = (int)N;
  d.counts = counts.data_ptr<int>(); d.elem_bytes = 2;
  d.A = A.data_ptr(); d.a_mn_major = 1; d.lda = M; d.gsa = cap * M;
  d.B = B.data_ptr(); d.b_mn_major = 1; d.ldb = N; d.gsb = cap * N;
  d.epilogue = FL_EPI_WGRAD; d.ldc = N;
  d.peers = to_peers(peers); d.num_peers = (int)peers.size();
  d.push_world = (int)peers.size(); d.push_rank = (int)rank; d.push_block_log2 = (int)block_log2;
  d.group_m = (int)group_m; d.max_ctas = (int)max_ctas;
  d.status = status.has_value() ? status->data_ptr<int>() : nullptr;
  check_rc(fl_grouped_gemm(&d, cur_stream()), "fl_grouped_gemm", fl_gemm_last_error());
}

// Sum of the staged partial rows over the sources, then w - lr * sum (lr != 0) or the sum itself into every rank's `out`.
static void shadow_update(torch::Tensor part, c10::optional<torch::Tensor> w, std::vector<int64_t> out_peers, int64_t groups,
                          int64_t rank, int64_t M, int64_t N, int64_t block_log2, int64_t group_stride, double lr,
                          int64_t max_ctas) {
  TORCH_CHECK(part.is_cuda() && part.scalar_type() == torch::kBFloat16 && part.is_contiguous(), "staging: contiguous bf16 on the GPU");
  TORCH_CHECK(part.numel() >= groups * M * N, "staging smaller than groups x M x N");
  TORCH_CHECK(lr == 0.0 || (w.has_value() && w->is_cuda() && w->scalar_type() == torch::kBFloat16), "weights: bf16 on the GPU");
  c10::cuda::CUDAGuard guard(part.device());
  FlShadowUpdateArgs a;
  memset(&a, 0, sizeof a);
  a.part = part.data_ptr(); a.w = opt_ptr(w); a.out_peers = to_peers(out_peers);
  a.groups = (int)groups; a.world = (int)out_peers.size(); a.rank = (int)rank; a.M = (int)M; a.N = (int)N;
  a.block_log2 = (int)block_log2; a.group_stride = group_stride; a.lr = (float)lr; a.max_ctas = (int)max_ctas;
  check_rc(fl_shadow_update(&a, cur_stream()), "fl_shadow_update", fl_shadow_update_error());
}

// ------------------------------------------------------------------------------------------------ comm
// segs: list of (src_addr, dst_addr, bytes, flags_addr, flag_mode, wait_flags_addr)
static void put_chunks(const std::vector<std::tuple<int64_t, int64_t, int64_t, int64_t, int64_t, int64_t>>& segs,
                       int64_t chunk_bytes, int64_t seq, bool use_bulk, int64_t num_ctas, int64_t threads,
                       int64_t status_addr, const std::vector<int64_t>& counters, int64_t counter_scratch) {
  FlPutArgs a;
  memset(&a, 0, sizeof a);
  TORCH_CHECK(segs.size() >= 1 && segs.size() <= FL_MAX_SEGS, "1..8 segments per launch");
  a.nseg = (int)segs.size();
  for (size_t i = 0; i < segs.size(); ++i) {
    a.seg[i].src = reinterpret_cast<const void*>(std::get<0>(segs[i]));
    a.seg[i].dst = reinterpret_cast<void*>(std::get<1>(segs[i]));
    a.seg[i].bytes = (unsigned long long)std::get<2>(segs[i]);
    a.seg[i].flags = reinterpret_cast<uint32_t*>(std::get<3>(segs[i]));
    a.seg[i].flag_mode = (int)std::get<4>(segs[i]);
    a.seg[i].wait_flags = reinterpret_cast<const uint32_t*>(std::get<5>(segs[i]));
    a.seg[i].bytes_done = i < counters.size() ? reinterpret_cast<unsigned long long*>(counters[i]) : nullptr;
  }
  a.chunk_bytes = (unsigned)chunk_bytes; a.seq = (unsigned)seq; a.use_bulk = use_bulk;
  a.status = reinterpret_cast<int*>(status_addr);
  a.done_scratch = reinterpret_cast<unsigned long long*>(counter_scratch);
  check_rc(fl_put_chunks(&a, (int)num_ctas, (int)threads, cur_stream()), "fl_put_chunks");
}
static void all_to_all(int64_t send_addr, const std::vector<int64_t>& recv_peers, int64_t bytes_per_peer, int64_t rank,
                       const std::vector<int64_t>& pads, int64_t slot0, int64_t chunk_bytes,
                       const std::vector<int64_t>& want, bool use_bulk, int64_t num_ctas, int64_t threads, int64_t status_addr) {
  const int world = (int)recv_peers.size();
  TORCH_CHECK(world >= 1 && world <= 8 && (int)pads.size() == world, "1..8 ranks");
  void* rp[8];
  FlSignalPtrs sp;
  memset(&sp, 0, sizeof sp);
  unsigned int w[8];
  for (int i = 0; i < world; ++i) {
    rp[i] = reinterpret_cast<void*>(recv_peers[i]);
    sp.p[i] = reinterpret_cast<uint32_t*>(pads[i]);
    if (!want.empty()) w[i] = (unsigned)want[i];
  }
  check_rc(fl_all_to_all(reinterpret_cast<const void*>(send_addr), rp, (unsigned long long)bytes_per_peer, (int)rank, world, sp,
                         (int)slot0, (unsigned)chunk_bytes, want.empty() ? nullptr : w, use_bulk, (int)num_ctas, (int)threads,
                         reinterpret_cast<int*>(status_addr), cur_stream()), "fl_all_to_all");
}
static void wait_flags(const std::vector<std::pair<int64_t, int64_t>>& flags, int64_t status_addr, int64_t limit_ms) {
  FlWaitArgs a;
  memset(&a, 0, sizeof a);
  TORCH_CHECK(flags.size() <= 16, "at most 16 flags per wait");
  a.n = (int)flags.size();
  for (size_t i = 0; i < flags.size(); ++i) {
    a.flag[i] = reinterpret_cast<const uint32_t*>(flags[i].first);
    a.want[i] = (unsigned)flags[i].second;
  }
  a.status = reinterpret_cast<int*>(status_addr);
  a.limit_ns = limit_ms > 0 ? (unsigned long long)limit_ms * 1000000ull : 0ull;
  check_rc(fl_wait_flags(&a, cur_stream()), "fl_wait_flags");
}
static void barrier(const std::vector<int64_t>& pads, int64_t slot0, int64_t rank, int64_t world, int64_t seq,
                    bool do_signal, bool do_wait, int64_t status_addr) {
  FlSignalPtrs p;
  memset(&p, 0, sizeof p);
  for (size_t i = 0; i < pads.size() && i < 8; ++i) p.p[i] = reinterpret_cast<uint32_t*>(pads[i]);
  check_rc(fl_barrier(p, (int)slot0, (int)rank, (int)world, (unsigned)seq, do_signal, do_wait,
                      reinterpret_cast<int*>(status_addr), cur_stream()), "fl_barrier");
}

// ------------------------------------------------------------------------------------------------ DLRM
static void embbag(bool backward, torch::Tensor weights, torch::Tensor indices, int64_t t_first, int64_t t_total,
                   int64_t b_local, std::vector<int64_t> peers, double lr, int64_t num_ctas, int64_t status_addr) {
  TORCH_CHECK(weights.is_cuda() && indices.is_cuda(), "CUDA tensors expected");
  TORCH_CHECK(weights.scalar_type() == torch::kFloat32 && weights.dim() == 3 && weights.is_contiguous(), "weights: [T_local, rows, dim] fp32");
  TORCH_CHECK(indices.scalar_type() == torch::kInt64 && indices.dim() == 3 && indices.is_contiguous(), "indices: [T_local, B_global, pooling] int64");
  c10::cuda::CUDAGuard guard(weights.device());
  FlEmbBagArgs a;
  memset(&a, 0, sizeof a);
  a.weights = weights.data_ptr<float>(); a.weights_rw = weights.data_ptr<float>();
  a.indices = reinterpret_cast<const long long*>(indices.data_ptr<int64_t>());
  a.t_local = (int)weights.size(0); a.rows = weights.size(1); a.dim = (int)weights.size(2);
  TORCH_CHECK(indices.size(0) == weights.size(0), "indices/weights table count mismatch");
  a.b_global = (int)indices.size(1); a.pooling = (int)indices.size(2);
  a.t_first = (int)t_first; a.t_total = (int)t_total; a.b_local = (int)b_local;
  a.out_peers = to_peers(peers); a.lr = (float)lr; a.status = reinterpret_cast<int*>(status_addr);
  if (backward) check_rc(fl_embbag_a2a_bwd_sgd(&a, (int)num_ctas, cur_stream()), "fl_embbag_a2a_bwd_sgd");
  else check_rc(fl_embbag_a2a_fwd(&a, (int)num_ctas, cur_stream()), "fl_embbag_a2a_fwd");
}

// Pairwise-dot interaction: out [B, ld] = x | upper triangle of z z^T | zeros, z = x and the pooled vectors of the sample.
static FlInteractArgs interact_args(const torch::Tensor& x, const torch::Tensor& pooled, const torch::Tensor& wide) {
  for (const auto& t : {x, pooled, wide})
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kFloat32 && t.is_contiguous(), "interact: contiguous fp32 CUDA tensors expected");
  TORCH_CHECK(x.dim() == 2 && pooled.dim() == 3 && wide.dim() == 2 && pooled.size(0) == x.size(0) && wide.size(0) == x.size(0) &&
              pooled.size(2) == x.size(1), "x: [B, dim], pooled: [B, vectors - 1, dim], out: [B, ld]");
  FlInteractArgs a;
  memset(&a, 0, sizeof a);
  a.x = x.data_ptr<float>(); a.pooled = pooled.data_ptr<float>();
  a.batch = x.size(0); a.vectors = (int)pooled.size(1) + 1; a.dim = (int)x.size(1); a.ld = wide.size(1);
  return a;
}
static void interact_fwd(torch::Tensor x, torch::Tensor pooled, torch::Tensor out) {
  FlInteractArgs a = interact_args(x, pooled, out);
  c10::cuda::CUDAGuard guard(x.device());
  a.out = out.data_ptr<float>();
  check_rc(fl_interact_fwd(&a, cur_stream()), "fl_interact_fwd");
}
static void interact_bwd(torch::Tensor x, torch::Tensor pooled, torch::Tensor dout, torch::Tensor dx, torch::Tensor dpooled, double scale) {
  FlInteractArgs a = interact_args(x, pooled, dout);
  for (const auto& t : {dx, dpooled})
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kFloat32 && t.is_contiguous(), "interact: contiguous fp32 CUDA tensors expected");
  TORCH_CHECK(dx.numel() == x.numel() && dpooled.numel() == pooled.numel(), "gradients: as large as the vectors");
  c10::cuda::CUDAGuard guard(x.device());
  a.dout = dout.data_ptr<float>(); a.dx = dx.data_ptr<float>(); a.dpooled = dpooled.data_ptr<float>(); a.scale = (float)scale;
  check_rc(fl_interact_bwd(&a, cur_stream()), "fl_interact_bwd");
}

// ------------------------------------------------------------------------------------------------ KV
static void kv_pack_send(torch::Tensor src_k, torch::Tensor src_v, int64_t dst_k, int64_t dst_v, int64_t src_layout,
                         int64_t dst_layout, int64_t src_num_blocks, int64_t dst_num_blocks, int64_t layers,
                         int64_t heads, int64_t block_size, int64_t head_dim, int64_t layer_begin, int64_t layer_end,
                         torch::Tensor src_bt, torch::Tensor dst_bt, torch::Tensor nblocks,
                         c10::optional<torch::Tensor> hdr, int64_t hdr_dst, int64_t done_flag, int64_t seq,
                         torch::Tensor cta_counter, int64_t num_ctas, int64_t status_addr) {
  TORCH_CHECK(src_k.is_cuda() && src_v.is_cuda(), "CUDA tensors expected");
  TORCH_CHECK(src_bt.scalar_type() == torch::kInt32 && dst_bt.scalar_type() == torch::kInt32 && nblocks.scalar_type() == torch::kInt32,
              "block tables are int32");
  c10::cuda::CUDAGuard guard(src_k.device());
  FlKvSendArgs a;
  memset(&a, 0, sizeof a);
  a.src_k = src_k.data_ptr(); a.src_v = src_v.data_ptr();
  a.dst_k = reinterpret_cast<void*>(dst_k); a.dst_v = reinterpret_cast<void*>(dst_v);
  a.src_layout = (int)src_layout; a.dst_layout = (int)dst_layout;
  a.src_num_blocks = (int)src_num_blocks; a.dst_num_blocks = (int)dst_num_blocks;
  a.layers = (int)layers; a.heads = (int)heads; a.block_size = (int)block_size; a.head_dim = (int)head_dim;
  a.layer_begin = (int)layer_begin; a.layer_end = (int)layer_end;
  a.src_block_table = src_bt.data_ptr<int>(); a.dst_block_table = dst_bt.data_ptr<int>();
  a.num_blocks = nblocks.data_ptr<int>();
  a.batch = (int)src_bt.size(0); a.max_blocks = (int)src_bt.size(1);
  if (hdr.has_value()) {
    a.hdr_src = hdr->data_ptr(); a.hdr_bytes = (int)hdr->nbytes();
    a.hdr_dst = reinterpret_cast<void*>(hdr_dst);
  }
  a.done_flag = reinterpret_cast<uint32_t*>(done_flag); a.seq = (unsigned)seq;
  a.cta_counter = reinterpret_cast<unsigned*>(cta_counter.data_ptr());
  a.status = reinterpret_cast<int*>(status_addr);
  check_rc(fl_kv_pack_send(&a, (int)num_ctas, cur_stream()), "fl_kv_pack_send");
}

// ------------------------------------------------------------------------------------------------ decoder
static int dec_dtype(const torch::Tensor& t) {
  TORCH_CHECK(t.is_cuda() && (t.scalar_type() == torch::kBFloat16 || t.scalar_type() == torch::kHalf), "bf16 or fp16 on the GPU expected");
  return t.scalar_type() == torch::kBFloat16 ? FL_DEC_BF16 : FL_DEC_FP16;
}
static void dec_like(const c10::optional<torch::Tensor>& t, const torch::Tensor& as, int64_t numel, const char* what) {
  TORCH_CHECK(!t.has_value() || (t->is_cuda() && t->scalar_type() == as.scalar_type() && t->is_contiguous() && t->numel() == numel), what);
}
static const long long* dec_i64(const c10::optional<torch::Tensor>& t, int64_t numel, const char* what) {
  if (!t.has_value()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == torch::kInt64 && t->is_contiguous() && t->numel() == numel, what);
  return reinterpret_cast<const long long*>(t->data_ptr<int64_t>());
}
// Whether the kernels may read these tensors (None: not given): plain tensors with memory, of `like`'s type and device, contiguous,
// from a multiple of 16 bytes on, and matrices of `shape` where that is given.  Native because a shard asks it about some 200 tensors on every call.
static bool dec_takes(py::list tensors, torch::Tensor like, c10::optional<std::pair<int64_t, int64_t>> shape) {
  const auto dtype = like.scalar_type();
  const auto device = like.device();
  for (py::handle h : tensors) {
    if (h.is_none()) continue;
    if (!THPVariable_CheckTypeExact(Py_TYPE(h.ptr()))) return false;
    const at::Tensor& t = THPVariable_Unpack(h.ptr());
    if (!t.has_storage() || t.scalar_type() != dtype || t.device() != device || !t.is_contiguous() ||
        (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15))
      return false;
    if (shape.has_value() && (t.dim() != 2 || t.size(0) != shape->first || t.size(1) != shape->second)) return false;
  }
  return true;
}
static FlPagedKv dec_kv(torch::Tensor k_pool, torch::Tensor v_pool, torch::Tensor table, int64_t layout, int64_t layer, int64_t layers,
                        int64_t num_blocks, int64_t block_size, int64_t kv_heads, int64_t dim, int64_t status_addr) {
  TORCH_CHECK(k_pool.is_cuda() && v_pool.is_cuda() && k_pool.is_contiguous() && v_pool.is_contiguous(), "pools: contiguous on the GPU");
  TORCH_CHECK(table.is_cuda() && table.scalar_type() == torch::kInt32 && table.is_contiguous() && table.dim() == 2, "block_table: [batch, blocks] int32");
  TORCH_CHECK(layer >= 0 && layer < layers && block_size > 0, "layer out of range");
  const int64_t need = num_blocks * layers * block_size * kv_heads * dim;
  TORCH_CHECK(k_pool.numel() >= need && v_pool.numel() >= need, "pools smaller than num_blocks pages");
  FlPagedKv kv;
  kv.k = k_pool.data_ptr(); kv.v = v_pool.data_ptr();
  kv.block_table = table.data_ptr<int>(); kv.table_stride = (int)table.size(1);
  kv.layout = (int)layout; kv.layer = (int)layer; kv.layers = (int)layers; kv.num_blocks = (int)num_blocks;
  kv.block_size = (int)block_size; kv.heads = (int)kv_heads;
  kv.status = reinterpret_cast<int*>(status_addr);
  return kv;
}
static void dec_embed(torch::Tensor tokens, c10::optional<torch::Tensor> pos, torch::Tensor embed, c10::optional<torch::Tensor> pos_embed,
                      torch::Tensor x, int64_t seq, int64_t offset, int64_t status_addr) {
  const int dt = dec_dtype(x);
  const int64_t rows = tokens.numel(), H = embed.size(1);
  TORCH_CHECK(embed.scalar_type() == x.scalar_type() && embed.is_contiguous() && x.is_contiguous() && x.numel() == rows * H, "x: [rows, hidden] like embed");
  if (pos_embed.has_value()) dec_like(pos_embed, x, pos_embed->size(0) * H, "pos_embed: [positions, hidden]");
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(fl_dec_embed(dt, dec_i64(tokens, rows, "tokens: int64"), dec_i64(pos, rows, "positions: int64"), embed.data_ptr(), opt_ptr(pos_embed),
                        x.data_ptr(), rows, (int)H, (int)seq, (int)offset, embed.size(0), pos_embed.has_value() ? pos_embed->size(0) : 0,
                        reinterpret_cast<int*>(status_addr), cur_stream()), "fl_dec_embed");
}
static void dec_add_norm(torch::Tensor x, c10::optional<torch::Tensor> y, c10::optional<torch::Tensor> y_bias, torch::Tensor w,
                         c10::optional<torch::Tensor> b, torch::Tensor h, double eps) {
  const int dt = dec_dtype(x);
  const int64_t H = w.numel(), rows = x.numel() / H;
  TORCH_CHECK(x.is_contiguous() && x.numel() == rows * H && w.scalar_type() == x.scalar_type() && w.is_contiguous(), "x: [rows, hidden]");
  dec_like(y, x, x.numel(), "y: like x"); dec_like(y_bias, x, H, "y_bias: [hidden]"); dec_like(b, x, H, "b: [hidden]"); dec_like(h, x, x.numel(), "h: like x");
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(fl_dec_add_norm(dt, x.data_ptr(), opt_ptr(y), opt_ptr(y_bias), w.data_ptr(), opt_ptr(b), h.data_ptr(), rows, (int)H, (float)eps,
                           cur_stream()), "fl_dec_add_norm");
}
static void dec_qkv(torch::Tensor qkv, c10::optional<torch::Tensor> bias, c10::optional<torch::Tensor> rope, c10::optional<torch::Tensor> pos,
                    int64_t seq, torch::Tensor k_pool, torch::Tensor v_pool, torch::Tensor table, int64_t layout, int64_t layer,
                    int64_t layers, int64_t num_blocks, int64_t block_size, int64_t heads, int64_t kv_heads, int64_t dim,
                    int64_t status_addr) {
  const int dt = dec_dtype(qkv);
  const int64_t width = (heads + 2 * kv_heads) * dim, rows = qkv.numel() / width;
  TORCH_CHECK(qkv.is_contiguous() && qkv.numel() == rows * width, "qkv: [rows, (heads + 2 kv_heads) * dim]");
  TORCH_CHECK(k_pool.scalar_type() == qkv.scalar_type() && v_pool.scalar_type() == qkv.scalar_type(), "pools of the model's type expected");
  TORCH_CHECK(pos.has_value() ? table.size(0) >= rows : (seq > 0 && table.size(0) * seq >= rows), "block_table: one row per request");
  TORCH_CHECK(!rope.has_value() || (rope->is_cuda() && rope->scalar_type() == torch::kFloat32 && rope->is_contiguous() && rope->size(-1) == dim),
              "rope: [positions, dim] fp32");
  dec_like(bias, qkv, width, "bias: [(heads + 2 kv_heads) * dim]");
  c10::cuda::CUDAGuard guard(qkv.device());
  const FlPagedKv kv = dec_kv(k_pool, v_pool, table, layout, layer, layers, num_blocks, block_size, kv_heads, dim, status_addr);
  check_rc(fl_dec_qkv(dt, qkv.data_ptr(), opt_ptr(bias), rope.has_value() ? rope->data_ptr<float>() : nullptr, rope.has_value() ? rope->size(0) : 0,
                      dec_i64(pos, rows, "positions: int64"), rows, (int)seq, (int)heads, (int)dim, &kv, cur_stream()), "fl_dec_qkv");
}
static void dec_act(torch::Tensor h, c10::optional<torch::Tensor> bias, torch::Tensor out, int64_t kind) {
  const int dt = dec_dtype(h);
  const int64_t F = out.size(-1), rows = out.numel() / F;
  TORCH_CHECK(h.is_contiguous() && out.is_contiguous() && out.scalar_type() == h.scalar_type() &&
              h.numel() == rows * F * (kind == FL_ACT_SILU_GATED ? 2 : 1), "h: [rows, ffn] (gate and up: [rows, 2 ffn])");
  dec_like(bias, h, F, "bias: [ffn]");
  c10::cuda::CUDAGuard guard(h.device());
  check_rc(fl_dec_act(dt, (int)kind, h.data_ptr(), opt_ptr(bias), out.data_ptr(), rows, (int)F, cur_stream()), "fl_dec_act");
}
static void dec_attention(torch::Tensor qkv, torch::Tensor pos, torch::Tensor k_pool, torch::Tensor v_pool, torch::Tensor table, int64_t layer,
                          int64_t layers, int64_t num_blocks, int64_t block_size, int64_t heads, int64_t kv_heads, int64_t dim, torch::Tensor out,
                          int64_t status_addr) {
  const int dt = dec_dtype(qkv);
  const int64_t width = (heads + 2 * kv_heads) * dim, batch = qkv.numel() / width;
  TORCH_CHECK(qkv.is_contiguous() && qkv.numel() == batch * width && table.size(0) >= batch, "qkv: [batch, (heads + 2 kv_heads) * dim]");
  TORCH_CHECK(k_pool.scalar_type() == qkv.scalar_type() && v_pool.scalar_type() == qkv.scalar_type(), "pools of the model's type expected");
  dec_like(out, qkv, batch * heads * dim, "out: [batch, heads * dim]");
  c10::cuda::CUDAGuard guard(qkv.device());
  const FlPagedKv kv = dec_kv(k_pool, v_pool, table, FL_KV_LBSHD, layer, layers, num_blocks, block_size, kv_heads, dim, status_addr);
  check_rc(fl_dec_attention(dt, qkv.data_ptr(), width, dec_i64(pos, batch, "positions: int64"), &kv, out.data_ptr(), (int)batch, (int)heads, (int)dim,
                            cur_stream()), "fl_dec_attention");
}
// x [rows, k] times w [n, k], see thin_gemm.cuh
static torch::Tensor dec_product(torch::Tensor x, torch::Tensor w, c10::optional<torch::Tensor> bias, int64_t epilogue, bool early, int64_t status_addr) {
  const int dt = dec_dtype(x);
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.is_contiguous() && w.is_contiguous() && w.is_cuda() && w.scalar_type() == x.scalar_type() &&
              w.size(1) == x.size(1) && w.device() == x.device(), "product: x [rows, k] and w [n, k], contiguous, of one type and device");
  TORCH_CHECK(epilogue != FL_THIN_SILU_GATED || w.size(0) % 2 == 0, "product: gate and up rows in equal number");
  const int64_t n = epilogue == FL_THIN_SILU_GATED ? w.size(0) / 2 : w.size(0);
  dec_like(bias, x, n, "bias: [n]");
  TORCH_CHECK(x.size(1) <= INT32_MAX && x.size(0) <= FL_THIN_MAX_ROWS, "product: too large");
  c10::cuda::CUDAGuard guard(x.device());
  auto y = torch::empty({x.size(0), n}, x.options());
  check_rc(fl_thin_gemm(dt, x.data_ptr(), (int)x.size(0), w.data_ptr(), n, (int)x.size(1), opt_ptr(bias), (int)epilogue, y.data_ptr(), early,
                        reinterpret_cast<int*>(status_addr), cur_stream()), "fl_thin_gemm");
  return y;
}
// queries of [rows, (heads + 2 kv_heads) * dim] (the rest is unwritten); keys and values to their pages, as dec_qkv
static torch::Tensor dec_qkv_product(torch::Tensor x, torch::Tensor w, c10::optional<torch::Tensor> bias, c10::optional<torch::Tensor> rope,
                                     torch::Tensor pos, torch::Tensor k_pool, torch::Tensor v_pool, torch::Tensor table, int64_t layout, int64_t layer,
                                     int64_t layers, int64_t num_blocks, int64_t block_size, int64_t heads, int64_t kv_heads, int64_t dim, bool early,
                                     int64_t status_addr) {
  const int dt = dec_dtype(x);
  TORCH_CHECK(x.dim() == 2 && w.dim() == 2 && x.is_contiguous() && w.is_contiguous() && w.is_cuda() && w.scalar_type() == x.scalar_type() &&
              w.size(1) == x.size(1) && w.device() == x.device(), "product: x [rows, k] and w [n, k], contiguous, of one type and device");
  const int64_t rows = x.size(0), n = w.size(0);
  TORCH_CHECK(n == (heads + 2 * kv_heads) * dim, "w: [(heads + 2 kv_heads) * dim, hidden]");
  TORCH_CHECK(x.size(1) <= INT32_MAX && rows <= FL_THIN_MAX_ROWS, "product: too large");
  TORCH_CHECK(k_pool.scalar_type() == x.scalar_type() && v_pool.scalar_type() == x.scalar_type(), "pools of the model's type expected");
  TORCH_CHECK(table.size(0) >= rows, "block_table: one row per request");
  TORCH_CHECK(!rope.has_value() || (rope->is_cuda() && rope->scalar_type() == torch::kFloat32 && rope->is_contiguous() && rope->size(-1) == dim),
              "rope: [positions, dim] fp32");
  dec_like(bias, x, n, "bias: [(heads + 2 kv_heads) * dim]");
  c10::cuda::CUDAGuard guard(x.device());
  FlThinQkv q = {};
  q.rope = rope.has_value() ? rope->data_ptr<float>() : nullptr;
  q.rope_rows = rope.has_value() ? rope->size(0) : 0;
  q.pos = dec_i64(pos, rows, "positions: int64");
  q.heads = (int)heads; q.dim = (int)dim;
  q.kv = dec_kv(k_pool, v_pool, table, layout, layer, layers, num_blocks, block_size, kv_heads, dim, status_addr);
  auto y = torch::empty({rows, n}, x.options());
  check_rc(fl_thin_qkv(dt, x.data_ptr(), (int)rows, w.data_ptr(), n, (int)x.size(1), opt_ptr(bias), &q, y.data_ptr(), early,
                       reinterpret_cast<int*>(status_addr), cur_stream()), "fl_thin_qkv");
  return y;
}
static torch::Tensor dec_argmax(torch::Tensor logits) {
  const int dt = dec_dtype(logits);
  TORCH_CHECK(logits.dim() == 2 && logits.is_contiguous(), "logits: [rows, vocab]");
  c10::cuda::CUDAGuard guard(logits.device());
  auto out = torch::empty({logits.size(0)}, logits.options().dtype(torch::kInt64));
  check_rc(fl_dec_argmax(dt, logits.data_ptr(), reinterpret_cast<long long*>(out.data_ptr<int64_t>()), (int)logits.size(0), logits.size(1),
                         cur_stream()), "fl_dec_argmax");
  return out;
}
static void dec_advance(torch::Tensor next, torch::Tensor tokens, torch::Tensor pos, torch::Tensor history, torch::Tensor step) {
  const int64_t B = next.numel();
  TORCH_CHECK(history.dim() == 2 && history.size(1) == B, "history: [rows, batch]");
  c10::cuda::CUDAGuard guard(next.device());
  check_rc(fl_dec_advance(dec_i64(next, B, "next: int64"), const_cast<long long*>(dec_i64(tokens, B, "tokens: int64")),
                          const_cast<long long*>(dec_i64(pos, B, "pos: int64")), const_cast<long long*>(dec_i64(history, history.numel(), "history: int64")),
                          const_cast<long long*>(dec_i64(step, 1, "step: int64")), (int)B, (int)history.size(0), cur_stream()), "fl_dec_advance");
}

// ------------------------------------------------------------------------------------------------ MoE
static void moe_dispatch(torch::Tensor x, torch::Tensor topk_idx, c10::optional<torch::Tensor> row_scale,
                         int64_t num_experts, int64_t experts_per_rank, int64_t cap, int64_t rank, int64_t world,
                         torch::Tensor local_count, torch::Tensor base, torch::Tensor pos, torch::Tensor slot,
                         std::vector<int64_t> count_peers, int64_t parity, std::vector<int64_t> x_peers,
                         std::vector<int64_t> info_peers, bool reuse_slots, int64_t status_addr) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.is_contiguous() && x.dim() == 2, "x: [tokens, hidden] bf16");
  TORCH_CHECK(topk_idx.scalar_type() == torch::kInt32 && topk_idx.is_contiguous() && topk_idx.dim() == 2, "topk_idx: [tokens, topk] int32");
  c10::cuda::CUDAGuard guard(x.device());
  FlMoeDispatchArgs a;
  memset(&a, 0, sizeof a);
  a.x = x.data_ptr(); a.topk_idx = topk_idx.data_ptr<int>();
  a.row_scale = row_scale.has_value() ? row_scale->data_ptr<float>() : nullptr;
  a.tokens = (int)x.size(0); a.topk = (int)topk_idx.size(1); a.hidden = (int)x.size(1);
  a.num_experts = (int)num_experts; a.experts_per_rank = (int)experts_per_rank; a.cap = (int)cap;
  a.rank = (int)rank; a.world = (int)world;
  a.local_count = local_count.data_ptr<int>(); a.base = base.data_ptr<int>();
  // a spare (zero) element behind the per-expert counters is the ticket that lets counting and reservation share a launch
  a.ticket = local_count.numel() > num_experts ? local_count.data_ptr<int>() + num_experts : nullptr;
  a.pos = pos.data_ptr<int>(); a.slot = slot.data_ptr<int>();
  a.count_peers = to_peers(count_peers); a.parity = (int)parity;
  a.x_peers = to_peers(x_peers); a.info_peers = to_peers(info_peers);
  a.reuse_slots = reuse_slots; a.status = reinterpret_cast<int*>(status_addr);
  check_rc(fl_moe_dispatch(&a, cur_stream()), "fl_moe_dispatch");
}
// logits [T, E] bf16, bias [E] -> probs [T, E], weights [T, k], experts [T, k] as int32 and int64, first-choice shares [E], aux []
static std::vector<torch::Tensor> moe_route(torch::Tensor logits, torch::Tensor bias, int64_t topk) {
  TORCH_CHECK(logits.is_cuda() && logits.scalar_type() == torch::kBFloat16 && logits.is_contiguous() && logits.dim() == 2, "logits: [tokens, experts] bf16");
  TORCH_CHECK(bias.device() == logits.device() && bias.scalar_type() == torch::kFloat32 && bias.is_contiguous() && bias.numel() == logits.size(1), "bias: [experts] fp32");
  c10::cuda::CUDAGuard guard(logits.device());
  const int64_t T = logits.size(0), E = logits.size(1);
  const auto f = logits.options().dtype(torch::kFloat32);
  FlMoeRouteArgs a;
  memset(&a, 0, sizeof a);
  a.tokens = (int)T; a.experts = (int)E; a.topk = (int)topk;
  auto probs = torch::empty({T, E}, f), w = torch::empty({T, topk}, f), share = torch::empty({E}, f), aux = torch::empty({}, f);
  auto part = torch::empty({fl_moe_route_blocks(a.tokens), 2, E}, f);
  auto idx = torch::empty({T, topk}, f.dtype(torch::kInt32)), idx64 = torch::empty({T, topk}, f.dtype(torch::kInt64));
  a.logits = logits.data_ptr(); a.bias = bias.data_ptr<float>(); a.probs = probs.data_ptr<float>(); a.w = w.data_ptr<float>();
  a.idx = idx.data_ptr<int>(); a.idx64 = reinterpret_cast<long long*>(idx64.data_ptr<int64_t>());
  a.part = part.data_ptr<float>(); a.share = share.data_ptr<float>(); a.aux = aux.data_ptr<float>();
  check_rc(fl_moe_route(&a, cur_stream()), "fl_moe_route");
  return {probs, w, idx, idx64, share, aux};
}
static torch::Tensor moe_route_bwd(torch::Tensor probs, torch::Tensor w, torch::Tensor idx, torch::Tensor share,
                                   c10::optional<torch::Tensor> dw, c10::optional<torch::Tensor> daux) {
  TORCH_CHECK(probs.is_cuda() && w.size(0) == probs.size(0) && share.numel() == probs.size(1), "what moe_route returned");
  for (const auto& t : {probs, w, share})
    TORCH_CHECK(t.scalar_type() == torch::kFloat32 && t.is_contiguous(), "contiguous fp32 expected");
  TORCH_CHECK(idx.scalar_type() == torch::kInt32 && idx.is_contiguous() && idx.sizes() == w.sizes(), "idx: [tokens, topk] int32");
  for (const auto& t : {dw, daux})
    TORCH_CHECK(!t.has_value() || (t->is_cuda() && t->scalar_type() == torch::kFloat32 && t->is_contiguous()), "gradients: contiguous fp32");
  TORCH_CHECK((!dw.has_value() || dw->numel() == w.numel()) && (!daux.has_value() || daux->numel() == 1), "gradients: as large as the outputs");
  c10::cuda::CUDAGuard guard(probs.device());
  FlMoeRouteArgs a;
  memset(&a, 0, sizeof a);
  a.tokens = (int)probs.size(0); a.experts = (int)probs.size(1); a.topk = (int)w.size(1);
  auto out = torch::empty(probs.sizes(), probs.options().dtype(torch::kBFloat16));
  a.probs = probs.data_ptr<float>(); a.w = w.data_ptr<float>(); a.idx = idx.data_ptr<int>(); a.share = share.data_ptr<float>();
  a.dw = (const float*)opt_ptr(dw); a.daux = (const float*)opt_ptr(daux); a.dlogits = out.data_ptr();
  check_rc(fl_moe_route_bwd(&a, cur_stream()), "fl_moe_route_bwd");
  return out;
}
// gradient of relu(z + bias): (dz, the bias gradient) from dy and the layer's output y, see mlp_bwd.cuh
static std::pair<torch::Tensor, torch::Tensor> relu_bias_bwd(torch::Tensor dy, torch::Tensor y) {
  TORCH_CHECK(dy.is_cuda() && dy.device() == y.device() && dy.scalar_type() == torch::kFloat32 && y.scalar_type() == torch::kFloat32 &&
              dy.dim() == 2 && dy.sizes() == y.sizes() && dy.is_contiguous() && y.is_contiguous() && dy.size(1) <= INT32_MAX, "dy, y: [rows, cols] fp32");
  c10::cuda::CUDAGuard guard(dy.device());
  const int64_t rows = dy.size(0);
  const int cols = (int)dy.size(1);
  auto dz = torch::empty_like(dy), db = torch::empty({cols}, dy.options()), part = torch::empty({fl_relu_bias_parts(rows, cols), cols}, dy.options());
  if (rows == 0 || cols == 0) return {dz, db.zero_()};
  check_rc(fl_relu_bias_bwd(dy.data_ptr<float>(), y.data_ptr<float>(), dz.data_ptr<float>(), part.data_ptr<float>(), db.data_ptr<float>(), rows, cols,
                            cur_stream()), "fl_relu_bias_bwd");
  return {dz, db};
}
// An MLP's layers behind one another, and their gradients (models/dlrm.py, _Mlp).  Native because a small batch takes the GPU less time than
// the host needs for some forty calls.  params: weight, bias of every layer.
static std::vector<torch::Tensor> mlp_forward(torch::Tensor x, bool relu_last, bool padded, const std::vector<torch::Tensor>& params) {
  const size_t n = params.size() / 2;
  TORCH_CHECK(params.size() == 2 * n && n > 0, "params: weight and bias of every layer");
  std::vector<torch::Tensor> acts;
  for (size_t i = 0; i < n; ++i) {
    const torch::Tensor &w = params[2 * i], &b = params[2 * i + 1];
    const torch::Tensor& rows = i == 0 ? x : acts.back();
    auto z = at::addmm(b, padded && i == 0 ? rows.narrow(1, 0, w.size(1)) : rows, w.t());
    if (i + 1 < n || relu_last) z.relu_();
    acts.push_back(z);
  }
  return acts;
}
// dy^T r over slices of `slice` rows, the slices' results added up in fp32
static torch::Tensor sliced_gram(const torch::Tensor& dy, const torch::Tensor& r, int64_t slice) {
  const int64_t B = dy.size(0), n = B / slice, m = n * slice;
  if (n < 2) return at::mm(dy.t(), r);
  auto out = at::bmm(dy.narrow(0, 0, m).view({n, slice, dy.size(1)}).transpose(1, 2), r.narrow(0, 0, m).view({n, slice, r.size(1)})).sum(0);
  return m == B ? out : out.addmm_(dy.narrow(0, m, B - m).t(), r.narrow(0, m, B - m));
}
// inputs: x, then the outputs of the layers that have a ReLU.  want: of x, then of every parameter.  Returns the gradients in that order.
static std::vector<c10::optional<torch::Tensor>> mlp_backward(torch::Tensor dy, const std::vector<torch::Tensor>& inputs, bool relu_last,
                                                              const std::vector<torch::Tensor>& params, const std::vector<bool>& want, int64_t slice) {
  const size_t n = params.size() / 2;
  TORCH_CHECK(inputs.size() == n + relu_last && want.size() == 2 * n + 1, "one input per layer");
  std::vector<c10::optional<torch::Tensor>> grads(2 * n + 1);
  for (size_t i = n; i-- > 0;) {
    const torch::Tensor &w = params[2 * i], &x = inputs[i];
    const int64_t width = x.size(1), cols = w.size(1);
    torch::Tensor db;
    if (i + 1 < n || relu_last) {
      std::tie(dy, db) = relu_bias_bwd(dy.contiguous(), inputs[i + 1]);
    } else if (want[2 * i + 2]) {
      db = dy.sum(0);
    }
    if (want[2 * i + 2]) grads[2 * i + 2] = db;
    if (want[2 * i + 1])
      grads[2 * i + 1] = width != cols ? sliced_gram(dy.contiguous(), x, slice).narrow(1, 0, cols).contiguous() : at::mm(dy.t(), x);
    if (i > 0 || want[0]) dy = at::mm(dy, width == cols ? w : at::constant_pad_nd(w, {0, width - cols}));
  }
  if (want[0]) grads[0] = dy;
  return grads;
}
static void moe_zero_tail(int64_t buf, int64_t counts, int64_t experts_local, int64_t cap, int64_t width) {
  check_rc(fl_moe_zero_tail(reinterpret_cast<void*>(buf), reinterpret_cast<const int*>(counts), (int)experts_local,
                            (int)cap, (int)width, cur_stream()), "fl_moe_zero_tail");
}
static void moe_combine(torch::Tensor slots, c10::optional<torch::Tensor> w, torch::Tensor out, int64_t topk) {
  c10::cuda::CUDAGuard guard(out.device());
  check_rc(fl_moe_combine(slots.data_ptr(), w.has_value() ? w->data_ptr<float>() : nullptr, out.data_ptr(),
                          (int)out.size(0), (int)topk, (int)out.size(1), cur_stream()), "fl_moe_combine");
}
static void moe_combine_dw(torch::Tensor dout, torch::Tensor slots, torch::Tensor dw, int64_t topk) {
  c10::cuda::CUDAGuard guard(dout.device());
  check_rc(fl_moe_combine_dw(dout.data_ptr(), slots.data_ptr(), dw.data_ptr<float>(), (int)dout.size(0), (int)topk,
                             (int)dout.size(1), cur_stream()), "fl_moe_combine_dw");
}

// ------------------------------------------------------------------------------------------------ fp8
static void fp8_quantize_rows(torch::Tensor x, torch::Tensor q, torch::Tensor scale, c10::optional<torch::Tensor> counts,
                              int64_t cap) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.is_contiguous() && x.dim() == 2, "x: [rows, K] bf16");
  c10::cuda::CUDAGuard guard(x.device());
  check_rc(fl_fp8_quantize_rows(x.data_ptr(), q.data_ptr(), scale.data_ptr<float>(), x.size(0), (int)x.size(1),
                                counts.has_value() ? counts->data_ptr<int>() : nullptr, (int)cap, cur_stream()),
           "fl_fp8_quantize_rows");
}
static void fp8_quantize_blocks(torch::Tensor w, torch::Tensor q, torch::Tensor scale) {
  TORCH_CHECK(w.is_cuda() && w.scalar_type() == torch::kBFloat16 && w.is_contiguous() && w.dim() == 3, "w: [G, R, C] bf16");
  c10::cuda::CUDAGuard guard(w.device());
  check_rc(fl_fp8_quantize_blocks(w.data_ptr(), q.data_ptr(), scale.data_ptr<float>(), (int)w.size(0), (int)w.size(1),
                                  (int)w.size(2), cur_stream()), "fl_fp8_quantize_blocks");
}
static void fp8_grouped_gemm(int64_t num_groups, int64_t cap, int64_t N, int64_t K, c10::optional<torch::Tensor> counts,
                             torch::Tensor A, torch::Tensor a_scale, torch::Tensor B, bool b_mn, torch::Tensor b_scale,
                             int64_t epilogue, c10::optional<torch::Tensor> C, int64_t ldc, c10::optional<torch::Tensor> gu,
                             int64_t ldgu, c10::optional<torch::Tensor> dgu, c10::optional<torch::Tensor> row_info,
                             std::vector<int64_t> peers, bool zero_tail, int64_t group_m, int64_t max_ctas,
                             c10::optional<torch::Tensor> status, int64_t peer_rows) {
  TORCH_CHECK(A.is_cuda() && B.is_cuda() && A.element_size() == 1 && B.element_size() == 1, "fp8 operands expected");
  c10::cuda::CUDAGuard guard(A.device());
  FlFp8GemmDesc d;
  memset(&d, 0, sizeof d);
  d.num_groups = (int)num_groups; d.cap = (int)cap; d.N = (int)N; d.K = (int)K;
  d.counts = counts.has_value() ? counts->data_ptr<int>() : nullptr;
  d.A = A.data_ptr(); d.a_scale = a_scale.data_ptr<float>();
  d.B = B.data_ptr(); d.b_mn_major = b_mn; d.b_scale = b_scale.data_ptr<float>();
  d.epilogue = (int)epilogue; d.C = opt_ptr(C); d.ldc = ldc; d.gu = opt_ptr(gu); d.ldgu = ldgu; d.dgu = opt_ptr(dgu);
  d.row_info = row_info.has_value() ? row_info->data_ptr<int>() : nullptr;
  d.peers = to_peers(peers); d.num_peers = (int)peers.size(); d.peer_rows = peer_rows;
  d.zero_tail = zero_tail; d.group_m = (int)group_m; d.max_ctas = (int)max_ctas;
  d.status = status.has_value() ? status->data_ptr<int>() : nullptr;
  check_rc(fl_fp8_grouped_gemm(&d, cur_stream()), "fl_fp8_grouped_gemm", fl_fp8_last_error());
}

// ------------------------------------------------------------------------------------------------ memory
static torch::Tensor tensor_from_ptr(int64_t ptr, std::vector<int64_t> shape, py::object dtype, int64_t device) {
  auto st = torch::python::detail::py_object_to_dtype(dtype);
  auto opts = torch::TensorOptions().dtype(st).device(device < 0 ? torch::Device(torch::kCPU) : torch::Device(torch::kCUDA, (c10::DeviceIndex)device));
  return torch::from_blob(reinterpret_cast<void*>(ptr), shape, [](void*) {}, opts);
}

static int64_t vmm_create(int64_t device, int64_t size, int64_t slab_bytes) {
  FlVmmRegion* r = fl_vmm_create((int)device, (size_t)size, (size_t)slab_bytes);
  if (!r) throw std::runtime_error(std::string("fl_vmm_create: ") + fl_vmm_last_error());
  return reinterpret_cast<int64_t>(r);
}
static int64_t vmm_import(int64_t device, std::vector<int> fds, int64_t slab_bytes) {
  FlVmmRegion* r = fl_vmm_import((int)device, fds.data(), (int)fds.size(), (size_t)slab_bytes);
  if (!r) throw std::runtime_error(std::string("fl_vmm_import: ") + fl_vmm_last_error());
  return reinterpret_cast<int64_t>(r);
}
static int64_t vmm_alias(int64_t region, int64_t device) {
  FlVmmRegion* r = fl_vmm_alias(reinterpret_cast<FlVmmRegion*>(region), (int)device);
  if (!r) throw std::runtime_error(std::string("fl_vmm_alias: ") + fl_vmm_last_error());
  return reinterpret_cast<int64_t>(r);
}
static int64_t vmm_adopt(int64_t ptr, int64_t size, int64_t device) {
  FlVmmRegion* r = fl_vmm_adopt(reinterpret_cast<void*>(ptr), (size_t)size, (int)device);
  if (!r) throw std::runtime_error(std::string("fl_vmm_adopt: ") + fl_vmm_last_error());
  return reinterpret_cast<int64_t>(r);
}
static int vmm_export_fd(int64_t region, int64_t slab) {
  int fd = -1;
  if (fl_vmm_export_fd(reinterpret_cast<FlVmmRegion*>(region), (int)slab, &fd))
    throw std::runtime_error(std::string("fl_vmm_export_fd: ") + fl_vmm_last_error());
  return fd;
}
static int64_t vmm_remap_slab(int64_t region, int64_t slab, int64_t target, bool keep, std::vector<int> access) {
  long usec = 0;
  if (fl_vmm_remap_slab(reinterpret_cast<FlVmmRegion*>(region), (int)slab, (int)target, keep, access.data(),
                        (int)access.size(), &usec))
    throw std::runtime_error(std::string("fl_vmm_remap_slab: ") + fl_vmm_last_error());
  return usec;
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("grouped_gemm", &grouped_gemm, py::arg("group_mode"), py::arg("num_groups"), py::arg("cap"), py::arg("M"), py::arg("N"), py::arg("K"),
        py::arg("counts"), py::arg("A"), py::arg("a_mn"), py::arg("lda"), py::arg("gsa"), py::arg("B"), py::arg("b_mn"), py::arg("ldb"), py::arg("gsb"),
        py::arg("epilogue"), py::arg("C"), py::arg("ldc"), py::arg("gsc"), py::arg("gu"), py::arg("ldgu"), py::arg("dgu"), py::arg("row_info"),
        py::arg("peers"), py::arg("sgd_lr"), py::arg("zero_tail"), py::arg("group_m"), py::arg("max_ctas"), py::arg("status"), py::arg("peer_rows"),
        py::arg("expect_rows") = 0);
  m.def("grouped_gemm_wgrad_push", &grouped_gemm_wgrad_push);
  m.def("shadow_update", &shadow_update);
  m.def("gemm_set_variant", [](int64_t v) { fl_gemm_set_variant((int)v); });
  m.def("gemm_get_variant", []() { return fl_gemm_get_variant(); });
  m.def("fp8_quantize_rows", &fp8_quantize_rows);
  m.def("fp8_quantize_blocks", &fp8_quantize_blocks);
  m.def("fp8_grouped_gemm", &fp8_grouped_gemm);
  m.def("put_chunks", &put_chunks, py::arg("segs"), py::arg("chunk_bytes"), py::arg("seq"), py::arg("use_bulk"), py::arg("num_ctas"),
        py::arg("threads"), py::arg("status_addr"), py::arg("counters") = std::vector<int64_t>(), py::arg("counter_scratch") = 0);
  m.def("wait_flags", &wait_flags, py::arg("flags"), py::arg("status_addr"), py::arg("limit_ms") = 0);
  m.def("all_to_all", &all_to_all);
  m.def("barrier", &barrier);
  m.def("embbag", &embbag);
  m.def("kv_pack_send", &kv_pack_send);
  m.def("dec_takes", &dec_takes, py::arg("tensors"), py::arg("like"), py::arg("shape") = py::none());
  m.def("dec_embed", &dec_embed, py::arg("tokens"), py::arg("pos"), py::arg("embed"), py::arg("pos_embed"), py::arg("x"), py::arg("seq"),
        py::arg("offset"), py::arg("status_addr") = 0);
  m.def("dec_add_norm", &dec_add_norm);
  m.def("dec_qkv", &dec_qkv, py::arg("qkv"), py::arg("bias"), py::arg("rope"), py::arg("pos"), py::arg("seq"), py::arg("k_pool"),
        py::arg("v_pool"), py::arg("table"), py::arg("layout"), py::arg("layer"), py::arg("layers"), py::arg("num_blocks"),
        py::arg("block_size"), py::arg("heads"), py::arg("kv_heads"), py::arg("dim"), py::arg("status_addr") = 0);
  m.def("moe_route", &moe_route);
  m.def("moe_route_bwd", &moe_route_bwd);
  m.def("interact_fwd", &interact_fwd);
  m.def("interact_bwd", &interact_bwd);
  m.def("relu_bias_bwd", &relu_bias_bwd);
  m.def("mlp_forward", &mlp_forward);
  m.def("mlp_backward", &mlp_backward);
  m.def("dec_act", &dec_act);
  m.def("dec_attention", &dec_attention, py::arg("qkv"), py::arg("pos"), py::arg("k_pool"), py::arg("v_pool"), py::arg("table"),
        py::arg("layer"), py::arg("layers"), py::arg("num_blocks"), py::arg("block_size"), py::arg("heads"), py::arg("kv_heads"),
        py::arg("dim"), py::arg("out"), py::arg("status_addr") = 0);
  m.def("dec_product", &dec_product, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("epilogue"), py::arg("early") = false,
        py::arg("status_addr") = 0);
  m.def("dec_qkv_product", &dec_qkv_product);
  m.attr("THIN_MAX_ROWS") = FL_THIN_MAX_ROWS;
  m.def("dec_argmax", &dec_argmax);
  m.def("dec_advance", &dec_advance);
  m.def("moe_dispatch", &moe_dispatch);
  m.def("moe_zero_tail", &moe_zero_tail);
  m.def("moe_combine", &moe_combine);
  m.def("moe_combine_dw", &moe_combine_dw);
  m.def("tensor_from_ptr", &tensor_from_ptr);

  m.def("vmm_init", [](int64_t backend) {
    if (fl_vmm_init((int)backend)) throw std::runtime_error(std::string("fl_vmm_init: ") + fl_vmm_last_error());
  });
  m.def("vmm_backend", []() { return fl_vmm_backend(); });
  m.def("vmm_granularity", [](int64_t dev) {
    size_t g = 0;
    if (fl_vmm_granularity((int)dev, &g)) throw std::runtime_error(std::string("fl_vmm_granularity: ") + fl_vmm_last_error());
    return (int64_t)g;
  });
  m.def("vmm_create", &vmm_create);
  m.def("vmm_import", &vmm_import);
  m.def("vmm_alias", &vmm_alias);
  m.def("vmm_adopt", &vmm_adopt);
  m.def("vmm_destroy", [](int64_t r) { fl_vmm_destroy(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_ptr", [](int64_t r) { return (int64_t)(uintptr_t)fl_vmm_ptr(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_size", [](int64_t r) { return (int64_t)fl_vmm_size(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_slab_bytes", [](int64_t r) { return (int64_t)fl_vmm_slab_bytes(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_num_slabs", [](int64_t r) { return fl_vmm_num_slabs(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_slab_device", [](int64_t r, int64_t s) { return fl_vmm_slab_device(reinterpret_cast<FlVmmRegion*>(r), (int)s); });
  m.def("vmm_export_fd", &vmm_export_fd);
  m.def("vmm_grant", [](int64_t r, int64_t dev) {
    if (fl_vmm_grant(reinterpret_cast<FlVmmRegion*>(r), (int)dev)) throw std::runtime_error(std::string("fl_vmm_grant: ") + fl_vmm_last_error());
  });
  m.def("vmm_remap_slab", &vmm_remap_slab);
  m.def("vmm_dmabuf_fd", [](int64_t p, int64_t size) {
    int fd = -1;
    uint64_t off = 0;
    if (fl_vmm_dmabuf_fd(reinterpret_cast<const void*>(p), (size_t)size, &fd, &off))
      throw std::runtime_error(std::string("fl_vmm_dmabuf_fd: ") + fl_vmm_last_error());
    return std::make_pair(fd, (int64_t)off);
  });
  m.def("vmm_ptr2dev", [](int64_t p) { return fl_vmm_ptr2dev(reinterpret_cast<const void*>(p)); });
  m.def("pool_init", [](int64_t ndev, int64_t slabs, int64_t slab_bytes) {
    if (fl_pool_init((int)ndev, (int)slabs, (size_t)slab_bytes)) throw std::runtime_error(std::string("fl_pool_init: ") + fl_vmm_last_error());
  });
  m.def("pool_shutdown", []() { fl_pool_shutdown(); });
  m.def("pool_free_slabs", [](int64_t dev) { return fl_pool_free_slabs((int)dev); });
  m.def("pool_slab_bytes", []() { return (int64_t)fl_pool_slab_bytes(); });
  m.def("pool_alloc", [](int64_t dev, int64_t size) {
    FlVmmRegion* r = fl_pool_alloc((int)dev, (size_t)size);
    if (!r) throw std::runtime_error(std::string("fl_pool_alloc: ") + fl_vmm_last_error());
    return reinterpret_cast<int64_t>(r);
  });
  m.def("pool_register", [](int64_t ptr, int64_t size, int64_t dev) {
    FlVmmRegion* r = fl_pool_register(reinterpret_cast<void*>(ptr), (size_t)size, (int)dev);
    if (!r) throw std::runtime_error(std::string("fl_pool_register: ") + fl_vmm_last_error());
    return reinterpret_cast<int64_t>(r);
  });
  m.def("pool_remap", [](int64_t r, int64_t slab, int64_t target, bool keep, std::vector<int> access) {
    long usec = 0;
    if (fl_pool_remap(reinterpret_cast<FlVmmRegion*>(r), (int)slab, (int)target, keep, access.data(), (int)access.size(), &usec))
      throw std::runtime_error(std::string("fl_pool_remap: ") + fl_vmm_last_error());
    return (int64_t)usec;
  });
  m.def("pool_release", [](int64_t r) { fl_pool_release(reinterpret_cast<FlVmmRegion*>(r)); });
  m.def("vmm_usage", [](int64_t dev) { return (int64_t)fl_vmm_usage((int)dev); });

  fl_monitor_bind(m);
}
