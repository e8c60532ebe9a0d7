"""Decoder-only transformers used by the disaggregated-serving path (prefill stage and decode stage): the
Llama family (RMSNorm, rotary positions, SwiGLU, no biases, grouped KV heads), the OPT family (pre-LayerNorm,
learned positions with an offset of 2, ReLU, biases, tied output embedding) and GPT-2 (as OPT with tanh-GELU and no
position offset) -- the three model families the reference's serving binary links (experiments/serving/
CMakeLists.txt:116-149: model_llama2, model_opt, model_gpt2).

The reference's serving experiment builds `st::model::Gpt<T>` from an external library with dummy weights
(experiments/serving/model.hh:165-177) and a table of model shapes (common_gpt_hyper_params.h:10-131).
Here the attention over a prompt and the matrix products of more than a handful of rows are library calls, tensor-parallel over a
process group, with random-init bf16 weights; hand-written are the products of a few rows (csrc/kernels/thin_gemm.cu), the KV hand-off between the stages (csrc/kernels/kv_pack.cu), which this model
feeds layer by layer through ``on_layer_done``, and, for bf16 and fp16 on the GPU, every pass between the products and the
attention of a decoding step (csrc/kernels/decoder.cu).  The operation-by-operation formulation below is the same
computation, rounded at the same places; it serves the CPU, fp32 and head sizes the kernels do not take.

Paged KV layouts (block = `block_size` tokens):
  prefill pool  [block][layer][head][slot][dim]   (FL_KV_BLHSD)
  decode pool   [layer][block][slot][head][dim]   (FL_KV_LBSHD)
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Callable, Optional

import torch
import torch.nn.functional as F

from .._ext import require_native

KV_BLHSD, KV_LBSHD = 0, 1
_OPERATIONS = ("_embed", "_norm", "_qkv", "_attn_out", "_mlp", "_logits")      # what the fused route does by itself
_ACT = {"llama": 0, "opt": 1, "gpt2": 2}          # FlDecAct
_STORE = 3                                         # FlThinEpi


@dataclass
class LlamaConfig:
    layers: int = 32
    hidden: int = 4096
    heads: int = 32
    kv_heads: int = 8
    head_dim: int = 128
    ffn: int = 14336
    vocab: int = 128256
    rope_theta: float = 500000.0
    eps: float = 1e-5
    block_size: int = 16
    arch: str = "llama"          # "llama" | "opt" | "gpt2"
    max_pos: int = 4096          # rows of the learned position table (opt, gpt2)

    @property
    def pos_offset(self) -> int:
        return 2 if self.arch == "opt" else 0     # OPT's position table keeps two leading rows for padding ids


# name -> config: the model zoo of the reference's serving scripts plus the Llama-3-8B shape of the build target
MODEL_ZOO = {
    "llama3_8b": LlamaConfig(),
    "llama2_7b": LlamaConfig(layers=32, hidden=4096, heads=32, kv_heads=32, ffn=11008, vocab=32000, rope_theta=10000.0),
    "llama2_13b": LlamaConfig(layers=40, hidden=5120, heads=40, kv_heads=40, ffn=13824, vocab=32000, rope_theta=10000.0),
    "llama2_70b": LlamaConfig(layers=80, hidden=8192, heads=64, kv_heads=8, ffn=28672, vocab=32000, rope_theta=10000.0),
    "opt_125m": LlamaConfig(layers=12, hidden=768, heads=12, kv_heads=12, head_dim=64, ffn=3072, vocab=50272, arch="opt", max_pos=2048),
    "opt_1.3b": LlamaConfig(layers=24, hidden=2048, heads=32, kv_heads=32, head_dim=64, ffn=8192, vocab=50272, arch="opt", max_pos=2048),
    "opt_2.7b": LlamaConfig(layers=32, hidden=2560, heads=32, kv_heads=32, head_dim=80, ffn=10240, vocab=50272, arch="opt", max_pos=2048),
    "opt_6.7b": LlamaConfig(layers=32, hidden=4096, heads=32, kv_heads=32, ffn=16384, vocab=50272, arch="opt", max_pos=2048),
    "opt_13b": LlamaConfig(layers=40, hidden=5120, heads=40, kv_heads=40, ffn=20480, vocab=50272, arch="opt", max_pos=2048),
    "opt_30b": LlamaConfig(layers=48, hidden=7168, heads=56, kv_heads=56, ffn=28672, vocab=50272, arch="opt", max_pos=2048),
    "gpt2": LlamaConfig(layers=12, hidden=768, heads=12, kv_heads=12, head_dim=64, ffn=3072, vocab=50257, arch="gpt2", max_pos=1024),
    "gpt2_xl": LlamaConfig(layers=48, hidden=1600, heads=25, kv_heads=25, head_dim=64, ffn=6400, vocab=50257, arch="gpt2", max_pos=1024),
    "tiny": LlamaConfig(layers=2, hidden=256, heads=4, kv_heads=2, head_dim=64, ffn=512, vocab=1000),
    "tiny_opt": LlamaConfig(layers=2, hidden=256, heads=4, kv_heads=4, head_dim=64, ffn=512, vocab=1000, arch="opt", max_pos=512),
    "tiny_gpt2": LlamaConfig(layers=2, hidden=256, heads=4, kv_heads=4, head_dim=64, ffn=512, vocab=1000, arch="gpt2", max_pos=512),
}


def _rms(x, w, eps):
    xf = x.float()
    return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)).to(x.dtype) * w


def _ln(x, w, b, eps):
    return F.layer_norm(x.float(), (x.shape[-1],), w.float(), b.float(), eps).to(x.dtype)


def _rope(x, pos, theta):
    """x: [..., n, heads, D]; pos: [..., n] absolute positions."""
    D = x.shape[-1]
    inv = 1.0 / (theta ** (torch.arange(0, D, 2, device=x.device, dtype=torch.float32) / D))
    ang = pos.float().unsqueeze(-1) * inv                      # [..., n, D/2]
    cos, sin = ang.cos().unsqueeze(-2), ang.sin().unsqueeze(-2)
    x1, x2 = x.float()[..., : D // 2], x.float()[..., D // 2:]
    return torch.cat([x1 * cos - x2 * sin, x2 * cos + x1 * sin], -1).to(x.dtype)


class _Status:
    """A word in pinned host memory in which the decoder kernels note an index outside its table, so that the host can look at it
    without waiting for them.  A copied or unpickled shard has a word of its own."""
    WHAT = {1: "a token outside the vocabulary", 2: "a position outside the position embedding or the block table",
            3: "a page id outside the pool"}
    STALLED = 4                  # FL_DEC_STALLED

    def __init__(self):
        self.word = torch.zeros(1, dtype=torch.int32, pin_memory=torch.cuda.is_available())

    def __deepcopy__(self, memo):
        return _Status()

    def __reduce__(self):
        return _Status, ()


class LlamaShard(torch.nn.Module):
    """One tensor-parallel shard of the model.  ``tp_group`` is None for TP=1.  Column-parallel tensors (QKV, the first
    MLP matrix and their biases) are split over the shards, row-parallel ones (attention output, second MLP matrix) are
    reduced over the group and their biases added once after the reduction."""

    def __init__(self, cfg: LlamaConfig, tp_rank: int = 0, tp_size: int = 1, tp_group=None, device="cuda", seed: int = 0,
                 dtype=torch.bfloat16, max_positions: Optional[int] = None):
        super().__init__()
        assert cfg.heads % tp_size == 0 and cfg.kv_heads % tp_size == 0 and cfg.ffn % tp_size == 0
        assert cfg.arch in ("llama", "opt", "gpt2"), cfg.arch
        self.cfg, self.tp_rank, self.tp_size, self.tp_group = cfg, tp_rank, tp_size, tp_group
        self.h_local, self.kvh_local, self.f_local = cfg.heads // tp_size, cfg.kv_heads // tp_size, cfg.ffn // tp_size
        self.gated = cfg.arch == "llama"                                        # SwiGLU: gate and up in one matrix
        if torch.device(device).type == "cuda":
            self._status = _Status()
        D, H = cfg.head_dim, cfg.hidden
        g = torch.Generator(device=device).manual_seed(seed * 31 + 7)           # replicated tensors: same on every shard
        gs = torch.Generator(device=device).manual_seed(seed * 31 + 100 + tp_rank)  # sharded tensors

        def w(shape, gen):
            return (torch.randn(*shape, generator=gen, device=device, dtype=torch.float32) * 0.02).to(dtype)

        def ones(n):
            return torch.ones(n, device=device, dtype=dtype)

        L = cfg.layers
        self.embed = w((cfg.vocab, H), g)
        self.lm_head = w((cfg.vocab, H), g) if cfg.arch == "llama" else self.embed    # OPT / GPT-2 tie the output embedding
        self.final_norm = ones(H)
        self.wqkv = [w(((self.h_local + 2 * self.kvh_local) * D, H), gs) for _ in range(L)]
        self.wo = [w((H, self.h_local * D), gs) for _ in range(L)]
        self.w13 = [w(((2 if self.gated else 1) * self.f_local, H), gs) for _ in range(L)]
        self.w2 = [w((H, self.f_local), gs) for _ in range(L)]
        self.n1 = [ones(H) for _ in range(L)]
        self.n2 = [ones(H) for _ in range(L)]
        none = [None] * L
        self.n1b, self.n2b, self.bqkv, self.bo, self.b13, self.b2 = none, none, none, none, none, none
        self.final_norm_b, self.pos_embed = None, None
        if cfg.arch != "llama":
            npos = max(cfg.max_pos, max_positions or 0) + cfg.pos_offset
            self.pos_embed = w((npos, H), g)
            self.final_norm_b = w((H,), g)
            self.n1b = [w((H,), g) for _ in range(L)]
            self.n2b = [w((H,), g) for _ in range(L)]
            self.bqkv = [w(((self.h_local + 2 * self.kvh_local) * D,), gs) for _ in range(L)]
            self.b13 = [w((self.f_local,), gs) for _ in range(L)]
            self.bo = [w((H,), g) for _ in range(L)]
            self.b2 = [w((H,), g) for _ in range(L)]

    # ------------------------------------------------------------------------------------------- building blocks
    def _allreduce(self, x):
        if self.tp_size > 1:
            import torch.distributed as dist
            dist.all_reduce(x, group=self.tp_group)
        return x

    def _norm(self, x, w, b):
        return _rms(x, w, self.cfg.eps) if b is None else _ln(x, w, b, self.cfg.eps)

    def _embed(self, tokens, pos):
        x = self.embed[tokens]
        if self.pos_embed is not None:
            x = x + self.pos_embed[pos + self.cfg.pos_offset]
        return x

    def _qkv(self, l, h, pos):
        """h: [..., n, H], pos: [..., n]  ->  q [..., n, h_local, D], k, v [..., n, kvh_local, D] (rotated for Llama)."""
        D = self.cfg.head_dim
        y = h @ self.wqkv[l].t()
        if self.bqkv[l] is not None:
            y = y + self.bqkv[l]
        qkv = y.view(*h.shape[:-1], self.h_local + 2 * self.kvh_local, D)
        q = qkv[..., : self.h_local, :]
        k = qkv[..., self.h_local: self.h_local + self.kvh_local, :]
        v = qkv[..., self.h_local + self.kvh_local:, :]
        if self.cfg.arch == "llama":
            q, k = _rope(q, pos, self.cfg.rope_theta), _rope(k, pos, self.cfg.rope_theta)
        return q, k, v

    def _attn_out(self, l, o):
        y = self._allreduce(o @ self.wo[l].t())
        return y if self.bo[l] is None else y + self.bo[l]

    def _mlp(self, l, x):
        h = x @ self.w13[l].t()
        if self.gated:
            a = F.silu(h[..., : self.f_local]) * h[..., self.f_local:]
        else:
            h = h + self.b13[l]
            a = F.relu(h) if self.cfg.arch == "opt" else F.gelu(h, approximate="tanh")
        y = self._allreduce(a @ self.w2[l].t())
        return y if self.b2[l] is None else y + self.b2[l]

    def _logits(self, x):
        return (self._norm(x, self.final_norm, self.final_norm_b) @ self.lm_head.t()).float()

    # ------------------------------------------------------------------------------------------- fused passes
    def _fused(self, pool: torch.Tensor) -> bool:
        """Whether csrc/kernels/decoder.cu takes this shard: not under autocast, which changes the types between the operations."""
        return self.embed.is_cuda and not torch.is_autocast_enabled("cuda") and self._fits(pool)

    def _fits(self, pool: torch.Tensor) -> bool:
        """16-bit weights and pools, rows and heads in whole 16-byte vectors (a rotated head in two halves of them), heads of at
        most 128; what the kernels read themselves (everything but the matrices) plain tensors of one type on one device,
        contiguous, from a multiple of 16 bytes on; and the operations of this class, not of a subclass or replaced on the object.
        Asked on every call, since all of that is plain attributes."""
        cfg, w = self.cfg, self.embed
        if not (w.dtype in (torch.bfloat16, torch.float16) and cfg.hidden % 8 == 0 and cfg.hidden <= 32768 and self.f_local % 8 == 0
                and cfg.head_dim % 16 == 0 and cfg.head_dim <= 128):
            return False
        if any(getattr(type(self), op) is not getattr(LlamaShard, op) or op in self.__dict__ for op in _OPERATIONS):
            return False
        return require_native().dec_takes([w, pool, self.pos_embed, self.final_norm, self.final_norm_b, *self.n1, *self.n1b, *self.n2, *self.n2b,
                                           *self.bqkv, *self.bo, *self.b13, *self.b2], w)

    def _indices(self, t: torch.Tensor) -> torch.Tensor:
        """Tokens or positions as the kernels read them: int64, contiguous, on the shard's device."""
        if t.dtype not in (torch.int64, torch.int32):
            raise IndexError(f"tokens and positions are int64 or int32, not {t.dtype}")
        return self._here(t.long())

    def _pages(self, table: torch.Tensor) -> torch.Tensor:
        if table.dtype != torch.int32:              # an id that int32 does not hold must not become one inside the pool
            table = table.long().clamp(-2 ** 31, 2 ** 31 - 1).int()
        return self._here(table)

    def _here(self, t: torch.Tensor) -> torch.Tensor:
        if t.device != self.embed.device:
            if t.is_cuda:
                raise RuntimeError(f"tokens, positions and block table on {self.embed.device} expected, not on {t.device}")
            t = t.to(self.embed.device)
        return t.contiguous()

    @staticmethod
    def _same_kind(t: torch.Tensor, as_: torch.Tensor) -> bool:
        return t.dtype == as_.dtype and t.device == as_.device and t.numel() == as_.numel() and t.is_contiguous() and t.data_ptr() % 16 == 0

    def _rope_table(self, positions: int):
        """fp32 [positions, D]: the cosines, then the sines, of every position's angles; made once per base, head size and device
        for at least 4096 positions, for eight of those; a ninth is made on every call.  Tables that were outgrown are kept, since
        a captured graph may hold their addresses."""
        if self.cfg.arch != "llama":
            return None
        D, theta, dev = self.cfg.head_dim, self.cfg.rope_theta, self.embed.device
        made = self.__dict__.setdefault("_rope_tables", {})
        tables = made.get((theta, D, dev), [])
        if tables and tables[-1].shape[0] >= positions:
            return tables[-1]
        n = max(4096, 1 << (positions - 1).bit_length())
        inv = 1.0 / (theta ** (torch.arange(0, D, 2, device=dev, dtype=torch.float32) / D))
        ang = torch.arange(n, device=dev).float().unsqueeze(-1) * inv
        table = torch.cat([ang.cos(), ang.sin()], -1).contiguous()
        if not torch.cuda.is_current_stream_capturing() and (tables or len(made) < 8):
            torch.cuda.current_stream(dev).synchronize()       # another stream may be the next to use it
            tables.append(table)
            made[theta, D, dev] = tables
        return table

    def _status_addr(self) -> int:
        """Where the kernels note a bad index or a stall.  The constructor makes the word, since host memory cannot be had under capture;
        0 (nowhere) only where a shard made elsewhere and moved here is captured in its first call of all."""
        st = self.__dict__.get("_status")
        if st is None:
            if torch.cuda.is_current_stream_capturing():
                return 0
            st = self.__dict__.setdefault("_status", _Status())
        return st.word.data_ptr()

    def check_status(self) -> None:
        """Raise IndexError if a kernel met a token, position or page id outside its table since the last call.  Does not wait:
        behind a synchronisation it covers everything before it.  Every fused call begins with it."""
        st = self.__dict__.get("_status")
        what = 0 if st is None else int(st.word)
        if what:
            st.word.zero_()
            if what == _Status.STALLED:
                raise RuntimeError("decoder: a kernel waited for its operands in vain")
            raise IndexError(f"decoder: {_Status.WHAT.get(what, what)}")

    def _thin(self, rows: int, like: torch.Tensor, *matrices) -> bool:
        """Whether csrc/kernels/thin_gemm.cu makes the products of so many rows with these (list of matrices, rows, columns): plain
        tensors of the shard's type and device, contiguous, from a multiple of 16 bytes on.  Others stay the library's."""
        if not like.is_cuda:
            return False
        C = require_native()
        return 0 < rows <= C.THIN_MAX_ROWS and all(C.dec_takes(list(ws), like, shape) for ws, *shape in matrices)

    def _layers_fused(self, x, pos, seq, k_pool, v_pool, table, layout, num_blocks, attend, on_layer_done=None):
        """Every layer on x [rows, hidden]; ``attend(l, qkv)`` returns the attention output [rows, h_local * D].  Returns
        (x, y, bias): the residual stream without the last branch, the branch and its bias (final_norm adds them up)."""
        C, cfg = require_native(), self.cfg
        rows, kind, status = x.shape[0], _ACT[cfg.arch], self._status_addr()
        rope = self._rope_table(table.shape[1] * cfg.block_size)
        h = torch.empty_like(x)
        H, q, F2 = cfg.hidden, self.h_local * cfg.head_dim, self.f_local
        thin = self._thin(rows, x, (self.wqkv, q + 2 * self.kvh_local * cfg.head_dim, H), (self.wo, H, q),
                          (self.w13, 2 * F2 if self.gated else F2, H), (self.w2, H, F2))
        act = None if thin else torch.empty(rows, self.f_local, dtype=x.dtype, device=x.device)

        def product(a, w, b=None, epilogue=_STORE):
            # `early`: the layers' weights were there before the step's first kernel started
            return C.dec_product(a, w, b, epilogue, True, status) if thin else a @ w.t()

        # A step's keys and values go to their pages where their sums are, if heads divide a tile's 128 columns.  A prefill's attention
        # reads them beside the queries.
        pages_in_product = thin and pos is not None and 128 % cfg.head_dim == 0
        y = bias = None
        for l in range(cfg.layers):
            C.dec_add_norm(x, y, bias, self.n1[l], self.n1b[l], h, cfg.eps)
            where = (k_pool, v_pool, table, layout, l, cfg.layers, num_blocks, cfg.block_size, self.h_local, self.kvh_local, cfg.head_dim)
            if pages_in_product:
                qkv = C.dec_qkv_product(h, self.wqkv[l], self.bqkv[l], rope, pos, *where, True, status)
            else:
                qkv = product(h, self.wqkv[l])
                C.dec_qkv(qkv, self.bqkv[l], rope, pos, seq, *where, status)
            if on_layer_done is not None:
                on_layer_done(l)                                                # KV of this layer may leave now
            y = self._allreduce(product(attend(l, qkv), self.wo[l]))
            C.dec_add_norm(x, y, self.bo[l], self.n2[l], self.n2b[l], h, cfg.eps)
            if thin:
                act = product(h, self.w13[l], None if self.gated else self.b13[l], kind)
            else:
                C.dec_act(h @ self.w13[l].t(), self.b13[l], act, kind)
            y, bias = self._allreduce(product(act, self.w2[l])), self.b2[l]
        return x, y, bias

    def _choose_fused(self, x, y, bias):
        """The tokens chosen at [..., hidden] positions of the residual stream; ``x`` is overwritten."""
        C = require_native()
        h = torch.empty_like(x)
        C.dec_add_norm(x, y, bias, self.final_norm, self.final_norm_b, h, self.cfg.eps)
        rows = h.flatten(0, -2)
        if self.lm_head.dim() == 2 and self._thin(rows.shape[0], rows, ([self.lm_head], self.lm_head.shape[0], h.shape[-1])):
            logits = C.dec_product(rows, self.lm_head, None, _STORE, True, self._status_addr())
        else:
            logits = rows @ self.lm_head.t()
        return C.dec_argmax(logits).view(h.shape[:-1])

    def _prefill_fused(self, tokens, k_pool, v_pool, block_table, on_layer_done, last_pos):
        self.check_status()
        C, cfg = require_native(), self.cfg
        B, S = tokens.shape
        D, hl, kl = cfg.head_dim, self.h_local, self.kvh_local
        tokens, table = self._indices(tokens), self._pages(block_table[:, : S // cfg.block_size])
        if table.shape != (B, S // cfg.block_size):
            raise RuntimeError(f"block table of {tuple(block_table.shape)} for {B} prompts of {S // cfg.block_size} pages")
        if self.pos_embed is not None and S + cfg.pos_offset > self.pos_embed.shape[0]:
            raise IndexError(f"prompts of {S} tokens, {self.pos_embed.shape[0] - cfg.pos_offset} positions")
        num_blocks = k_pool.view(-1, cfg.layers, kl, cfg.block_size, D).shape[0]
        x = torch.empty(B * S, cfg.hidden, dtype=self.embed.dtype, device=tokens.device)
        C.dec_embed(tokens, None, self.embed, self.pos_embed, x, S, cfg.pos_offset, self._status_addr())

        def attend(l, qkv):
            q, k, v = qkv.view(B, S, hl + 2 * kl, D).split([hl, kl, kl], 2)
            o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True, enable_gqa=hl != kl)
            return o.transpose(1, 2).reshape(B * S, hl * D)

        x, y, bias = self._layers_fused(x, None, S, k_pool, v_pool, table, KV_BLHSD, num_blocks, attend, on_layer_done)
        # indexed per request, so that a position counts from the request's own end or is out of its range
        at = (slice(None), -1) if last_pos is None else (torch.arange(B, device=x.device), last_pos)
        x, y = (t.view(B, S, cfg.hidden)[at] for t in (x, y))
        return self._choose_fused(x.contiguous(), y.contiguous(), bias)

    def _decode_fused(self, tokens, positions, k_pool, v_pool, block_table, num_blocks):
        self.check_status()
        C, cfg, status = require_native(), self.cfg, self._status_addr()
        B, D, hl, kl, dev = tokens.shape[0], cfg.head_dim, self.h_local, self.kvh_local, self.embed.device
        if block_table.shape[0] != B:
            raise RuntimeError(f"block table of {tuple(block_table.shape)} for {B} sequences")
        for pool in (k_pool, v_pool):
            pool.view(cfg.layers, num_blocks, cfg.block_size, kl, D)
        tokens, positions, table = self._indices(tokens), self._indices(positions), self._pages(block_table)
        x = torch.empty(B, cfg.hidden, dtype=self.embed.dtype, device=dev)
        C.dec_embed(tokens, positions, self.embed, self.pos_embed, x, 1, cfg.pos_offset, status)
        out = torch.empty(B, hl * D, dtype=x.dtype, device=dev)

        def attend(l, qkv):
            C.dec_attention(qkv, positions, k_pool, v_pool, table, l, cfg.layers, num_blocks, cfg.block_size, hl, kl, D, out, status)
            return out

        return self._choose_fused(*self._layers_fused(x, positions, 1, k_pool, v_pool, table, KV_LBSHD, num_blocks, attend))

    # ------------------------------------------------------------------------------------------- prefill
    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, block_table: torch.Tensor,
                on_layer_done: Optional[Callable[[int], None]] = None, last_pos: Optional[torch.Tensor] = None) -> torch.Tensor:
        """tokens: [B, S] (S a multiple of block_size); pools: flat bf16 in the BLHSD layout; block_table: [B, >=S/bs]
        int32.  Fills the pools, returns the greedy first token of every sequence [B] (int64)."""
        cfg = self.cfg
        B, S = tokens.shape
        bs, D, L = cfg.block_size, cfg.head_dim, cfg.layers
        assert S % bs == 0
        if self._fused(k_pool) and self._same_kind(v_pool, k_pool):
            return self._prefill_fused(tokens, k_pool, v_pool, block_table, on_layer_done, last_pos)
        nblk = S // bs
        kp = k_pool.view(-1, L, self.kvh_local, bs, D)
        vp = v_pool.view(-1, L, self.kvh_local, bs, D)
        blocks = block_table[:, :nblk].long().reshape(-1)                       # [B*nblk]
        pos = torch.arange(S, device=tokens.device).unsqueeze(0).expand(B, S)
        x = self._embed(tokens, pos)                                            # [B, S, H]
        for l in range(L):
            q, k, v = self._qkv(l, self._norm(x, self.n1[l], self.n1b[l]), pos)
            # page write: [B, S, h, D] -> [B*nblk, h, bs, D]
            kp[blocks, l] = k.reshape(B * nblk, bs, self.kvh_local, D).permute(0, 2, 1, 3)
            vp[blocks, l] = v.reshape(B * nblk, bs, self.kvh_local, D).permute(0, 2, 1, 3)
            if on_layer_done is not None:
                on_layer_done(l)                                                # KV of this layer may leave now
            o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True,
                                               enable_gqa=self.h_local != self.kvh_local)
            x = x + self._attn_out(l, o.transpose(1, 2).reshape(B, S, self.h_local * D))
            x = x + self._mlp(l, self._norm(x, self.n2[l], self.n2b[l]))
        xl = x[:, -1] if last_pos is None else x[torch.arange(B, device=x.device), last_pos]
        return self._logits(xl).argmax(-1)

    # ------------------------------------------------------------------------------------------- decode
    @torch.no_grad()
    def decode_step(self, tokens: torch.Tensor, positions: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor,
                    block_table: torch.Tensor, num_pool_blocks: int) -> torch.Tensor:
        """One greedy step for B sequences.  tokens, positions: [B]; pools: flat bf16 in the LBSHD layout;
        block_table: [B, max_blocks] int32 covering position + 1 tokens.  Returns next tokens [B]."""
        cfg = self.cfg
        B = tokens.shape[0]
        bs, D, L = cfg.block_size, cfg.head_dim, cfg.layers
        if 0 < B <= 65535 and self._fused(k_pool) and self._same_kind(v_pool, k_pool):
            return self._decode_fused(tokens, positions, k_pool, v_pool, block_table, num_pool_blocks)
        kp = k_pool.view(L, num_pool_blocks, bs, self.kvh_local, D)
        vp = v_pool.view(L, num_pool_blocks, bs, self.kvh_local, D)
        bt = block_table.long()
        maxblk = bt.shape[1]
        ar = torch.arange(B, device=tokens.device)
        cur_blk = bt[ar, positions // bs]
        cur_slot = positions % bs
        ctx = maxblk * bs
        mask = (torch.arange(ctx, device=tokens.device).unsqueeze(0) <= positions.unsqueeze(1)).view(B, 1, 1, ctx)
        p1 = positions.unsqueeze(1)
        x = self._embed(tokens, positions)                                       # [B, H]
        for l in range(L):
            q, k, v = self._qkv(l, self._norm(x, self.n1[l], self.n1b[l]).unsqueeze(1), p1)   # [B, 1, heads, D]
            kp[l, cur_blk, cur_slot] = k[:, 0]
            vp[l, cur_blk, cur_slot] = v[:, 0]
            K = kp[l][bt].reshape(B, ctx, self.kvh_local, D)                     # gather this sequence's pages
            V = vp[l][bt].reshape(B, ctx, self.kvh_local, D)
            o = F.scaled_dot_product_attention(q.transpose(1, 2), K.transpose(1, 2), V.transpose(1, 2), attn_mask=mask,
                                               enable_gqa=self.h_local != self.kvh_local)
            x = x + self._attn_out(l, o.transpose(1, 2).reshape(B, self.h_local * D))
            x = x + self._mlp(l, self._norm(x, self.n2[l], self.n2b[l]))
        return self._logits(x).argmax(-1)

    # reference path for tests: full-sequence forward without paging, returns logits of the last position
    @torch.no_grad()
    def forward_dense(self, tokens: torch.Tensor, all_positions: bool = False) -> torch.Tensor:
        cfg = self.cfg
        B, S = tokens.shape
        D = cfg.head_dim
        pos = torch.arange(S, device=tokens.device).unsqueeze(0).expand(B, S)
        x = self._embed(tokens, pos)
        for l in range(cfg.layers):
            q, k, v = self._qkv(l, self._norm(x, self.n1[l], self.n1b[l]), pos)
            o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), is_causal=True,
                                               enable_gqa=self.h_local != self.kvh_local)
            x = x + self._attn_out(l, o.transpose(1, 2).reshape(B, S, self.h_local * D))
            x = x + self._mlp(l, self._norm(x, self.n2[l], self.n2b[l]))
        return self._logits(x if all_positions else x[:, -1])

    # ------------------------------------------------------------------------------------------- checkpoints
    def _hf_names(self, l: int):
        a = self.cfg.arch
        if a == "llama":
            pre = f"model.layers.{l}."
            return dict(q=pre + "self_attn.q_proj", k=pre + "self_attn.k_proj", v=pre + "self_attn.v_proj", o=pre + "self_attn.o_proj",
                        gate=pre + "mlp.gate_proj", up=pre + "mlp.up_proj", down=pre + "mlp.down_proj",
                        n1=pre + "input_layernorm", n2=pre + "post_attention_layernorm")
        if a == "opt":
            pre = f"model.decoder.layers.{l}."
            return dict(q=pre + "self_attn.q_proj", k=pre + "self_attn.k_proj", v=pre + "self_attn.v_proj", o=pre + "self_attn.out_proj",
                        up=pre + "fc1", down=pre + "fc2", n1=pre + "self_attn_layer_norm", n2=pre + "final_layer_norm")
        pre = f"transformer.h.{l}."
        return dict(qkv=pre + "attn.c_attn", o=pre + "attn.c_proj", up=pre + "mlp.c_fc", down=pre + "mlp.c_proj", n1=pre + "ln_1", n2=pre + "ln_2")

    _HF_TOP = {"llama": ("model.embed_tokens", None, "model.norm", "lm_head"),
               "opt": ("model.decoder.embed_tokens", "model.decoder.embed_positions", "model.decoder.final_layer_norm", "lm_head"),
               "gpt2": ("transformer.wte", "transformer.wpe", "transformer.ln_f", "lm_head")}

    @torch.no_grad()
    def load_hf_state_dict(self, sd: dict) -> None:
        """Fill this shard from a Hugging Face ``state_dict`` of the matching family (LlamaForCausalLM, OPTForCausalLM,
        GPT2LMHeadModel).  Column-parallel tensors are cut by head / by MLP column for this shard's ``tp_rank``, so every
        shard reads the same full checkpoint.  GPT-2 stores its projections transposed ([in, out])."""
        cfg, D = self.cfg, self.cfg.head_dim
        r, hl, kl, fl = self.tp_rank, self.h_local, self.kvh_local, self.f_local
        gpt2 = cfg.arch == "gpt2"

        def put(dst, src):
            assert dst.shape == src.shape, (tuple(dst.shape), tuple(src.shape))
            dst.copy_(src.to(device=dst.device, dtype=dst.dtype))

        def W(name):                                       # weight as [out, in]
            w = sd[name + ".weight"]
            return w.t() if gpt2 else w

        emb, pos, fin, head = self._HF_TOP[cfg.arch]
        put(self.embed, sd[emb + ".weight"])
        if cfg.arch == "llama":
            put(self.lm_head, sd.get(head + ".weight", sd[emb + ".weight"]))
        put(self.final_norm, sd[fin + ".weight"])
        if pos is not None:
            n = min(self.pos_embed.shape[0], sd[pos + ".weight"].shape[0])
            self.pos_embed[:n].copy_(sd[pos + ".weight"][:n].to(self.pos_embed.dtype))
            put(self.final_norm_b, sd[fin + ".bias"])
        for l in range(cfg.layers):
            nm = self._hf_names(l)
            if gpt2:
                wq, wk, wv = W(nm["qkv"]).split(cfg.hidden, 0)
                bq, bk, bv = sd[nm["qkv"] + ".bias"].split(cfg.hidden, 0)
            else:
                wq, wk, wv = W(nm["q"]), W(nm["k"]), W(nm["v"])
                if cfg.arch == "opt":
                    bq, bk, bv = (sd[nm[x] + ".bias"] for x in "qkv")
            put(self.wqkv[l], torch.cat([wq[r * hl * D:(r + 1) * hl * D], wk[r * kl * D:(r + 1) * kl * D], wv[r * kl * D:(r + 1) * kl * D]]))
            put(self.wo[l], W(nm["o"])[:, r * hl * D:(r + 1) * hl * D])
            put(self.w2[l], W(nm["down"])[:, r * fl:(r + 1) * fl])
            put(self.n1[l], sd[nm["n1"] + ".weight"])
            put(self.n2[l], sd[nm["n2"] + ".weight"])
            if self.gated:
                put(self.w13[l], torch.cat([W(nm["gate"])[r * fl:(r + 1) * fl], W(nm["up"])[r * fl:(r + 1) * fl]]))
            else:
                put(self.w13[l], W(nm["up"])[r * fl:(r + 1) * fl])
                put(self.b13[l], sd[nm["up"] + ".bias"][r * fl:(r + 1) * fl])
                put(self.bqkv[l], torch.cat([bq[r * hl * D:(r + 1) * hl * D], bk[r * kl * D:(r + 1) * kl * D], bv[r * kl * D:(r + 1) * kl * D]]))
                put(self.bo[l], sd[nm["o"] + ".bias"])
                put(self.b2[l], sd[nm["down"] + ".bias"])
                put(self.n1b[l], sd[nm["n1"] + ".bias"])
                put(self.n2b[l], sd[nm["n2"] + ".bias"])

    @torch.no_grad()
    def export_hf_state_dict(self) -> dict:
        """The inverse of :meth:`load_hf_state_dict` for an unsharded model (TP = 1)."""
        assert self.tp_size == 1, "gather the shards first"
        cfg, D = self.cfg, self.cfg.head_dim
        gpt2 = cfg.arch == "gpt2"
        sd = {}

        def outW(name, w):                                 # w is [out, in]
            sd[name + ".weight"] = (w.t() if gpt2 else w).contiguous().clone()

        emb, pos, fin, head = self._HF_TOP[cfg.arch]
        sd[emb + ".weight"] = self.embed.clone()
        sd[head + ".weight"] = self.lm_head.clone()
        sd[fin + ".weight"] = self.final_norm.clone()
        if pos is not None:
            sd[pos + ".weight"] = self.pos_embed.clone()
            sd[fin + ".bias"] = self.final_norm_b.clone()
        nq, nk = cfg.heads * D, cfg.kv_heads * D
        for l in range(cfg.layers):
            nm = self._hf_names(l)
            wq, wk, wv = self.wqkv[l].split([nq, nk, nk], 0)
            if gpt2:
                outW(nm["qkv"], self.wqkv[l])
                sd[nm["qkv"] + ".bias"] = self.bqkv[l].clone()
            else:
                outW(nm["q"], wq); outW(nm["k"], wk); outW(nm["v"], wv)
                if cfg.arch == "opt":
                    for x, b in zip("qkv", self.bqkv[l].split([nq, nk, nk], 0)):
                        sd[nm[x] + ".bias"] = b.clone()
            outW(nm["o"], self.wo[l])
            outW(nm["down"], self.w2[l])
            sd[nm["n1"] + ".weight"] = self.n1[l].clone()
            sd[nm["n2"] + ".weight"] = self.n2[l].clone()
            if self.gated:
                outW(nm["gate"], self.w13[l][: cfg.ffn]); outW(nm["up"], self.w13[l][cfg.ffn:])
            else:
                outW(nm["up"], self.w13[l])
                sd[nm["up"] + ".bias"] = self.b13[l].clone()
                sd[nm["o"] + ".bias"] = self.bo[l].clone()
                sd[nm["down"] + ".bias"] = self.b2[l].clone()
                sd[nm["n1"] + ".bias"] = self.n1b[l].clone()
                sd[nm["n2"] + ".bias"] = self.n2b[l].clone()
        return sd

    def state_dict_flat(self) -> dict:
        """Every tensor of this shard under a flat name (for ``torch.save``)."""
        out = {"embed": self.embed, "final_norm": self.final_norm}
        if self.lm_head is not self.embed:
            out["lm_head"] = self.lm_head
        for name in ("pos_embed", "final_norm_b"):
            if getattr(self, name) is not None:
                out[name] = getattr(self, name)
        for name in ("wqkv", "wo", "w13", "w2", "n1", "n2", "n1b", "n2b", "bqkv", "bo", "b13", "b2"):
            for l, t in enumerate(getattr(self, name)):
                if t is not None:
                    out[f"{name}.{l}"] = t
        return out

    @torch.no_grad()
    def load_state_dict_flat(self, sd: dict) -> None:
        mine = self.state_dict_flat()
        missing = set(mine) - set(sd)
        assert not missing, f"checkpoint lacks {sorted(missing)[:4]}"
        for k, t in mine.items():
            t.copy_(sd[k].to(device=t.device, dtype=t.dtype))


def load_checkpoint_file(path: str) -> dict:
    """A Hugging Face style ``state_dict`` from ``path``: a ``.pt`` / ``.bin`` file (``torch.load``), a ``.safetensors``
    file, or a directory holding any number of those shards."""
    import os
    if os.path.isdir(path):
        sd = {}
        for f in sorted(os.listdir(path)):
            if f.endswith((".pt", ".bin", ".safetensors")):
                sd.update(load_checkpoint_file(os.path.join(path, f)))
        if not sd:
            raise FileNotFoundError(f"no .pt / .bin / .safetensors file in {path}")
        return sd
    if path.endswith(".safetensors"):
        from safetensors.torch import load_file
        return load_file(path)
    sd = torch.load(path, map_location="cpu", weights_only=True)
    return sd.get("state_dict", sd) if isinstance(sd, dict) else sd


DecoderShard = LlamaShard      # the class serves every family of the zoo; the old name is kept for callers
