"""Performance cases: the work that programs built on this framework have it do, on one GPU, through its public entry points.

  moe        MoELayer: a training step (forward, backward, expert SGD fused or expert gradients handed out) or inference
  dlrm       DLRM.train_step
  prefill    PrefillStage.run: prompt processing with the layer-by-layer KV hand-off to the decode side
  kv         KVLink.send_layers alone: the hand-off of pages that are already there
  decode     DecodeStage.decode: greedy tokens over the paged cache
  put, a2a   Channel.put and all_to_all between the (virtual) ranks of a symmetric heap

Sizes are those of the benchmark configurations, the model zoo and the tests, and generic ones between them.  Peers are
virtual ranks on the same GPU; a wait is always enqueued after the work that satisfies it.
"""
from __future__ import annotations

import copy
import functools
import math
import weakref

import numpy as np
import torch

from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
from fuselink_b200.models.moe import MoELayer, zipf_log_bias
from fuselink_b200.ops.comm import Channel, all_to_all
from fuselink_b200.ops.moe import MoEConfig, MoEWorkspace
from fuselink_b200.parallel.symm import SymmetricHeap
from fuselink_b200.serving.disagg import DecodeStage, KVLink, PrefillStage, ServeParams

DEV = "cuda:0"
MIB = 1 << 20
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # The benchmark's training step: Mixtral-shaped experts, a full batch per GPU, skewed router, SGD fused into the GEMMs.
        dict(name="moe train 8192", kind="moe", tokens=8192, hidden=4096, ffn=14336, experts=8, topk=2, zipf=1.2, mode="train", fp8=False, fused=True),
        # A smaller layer inside a transformer under an ordinary optimizer (expert gradients handed out), ragged token count.
        dict(name="moe train ragged", kind="moe", tokens=1531, hidden=2048, ffn=5632, experts=16, topk=2, zipf=0.0, mode="train", fp8=False, fused=False),
        # The fp8 option of the same training step.
        dict(name="moe train fp8", kind="moe", tokens=4096, hidden=4096, ffn=14336, experts=8, topk=2, zipf=1.2, mode="train", fp8=True, fused=True),
        # A serving batch through the big layer, forward only: a few hundred rows per expert, all the weights.
        dict(name="moe infer 1000", kind="moe", tokens=1000, hidden=4096, ffn=14336, experts=8, topk=2, zipf=0.0, mode="infer", fp8=False, fused=False),
        # The benchmark's recommendation model at its full batch, and a small ragged batch of a smaller one.
        dict(name="dlrm 65536", kind="dlrm", batch=65536, tables=26, rows=1_000_000, pooling=20, zipf=1.05),
        dict(name="dlrm ragged", kind="dlrm", batch=2053, tables=11, rows=120_000, pooling=7, zipf=1.05),
        # Disaggregated serving at the benchmark's shape: 16 prompts of 2048 tokens; the hand-off alone; a few decode steps.
        dict(name="prefill 16x2048", kind="prefill", model="llama3_8b", batch=16, length=2048, dtype="bf16"),
        dict(name="kv hand-off", kind="kv", model="llama3_8b", tp=1, batch=16, length=2048, layers=32),
        dict(name="decode 16x2048", kind="decode", model="llama3_8b", batch=16, length=2048, steps=8, dtype="bf16"),
        # A small model and a small batch, in half precision: every kernel is short, the chain of launches is what a token costs.
        dict(name="decode small", kind="decode", model="opt_1.3b", batch=3, length=389, steps=16, dtype="fp16"),
        # A message where latency is all that counts, and the exchange of medium blocks between eight ranks.
        dict(name="put 64 KiB", kind="put", bytes=65536),
        dict(name="a2a 8 ranks", kind="a2a", world=8, elems=1_310_720),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["moe", "moe", "moe", "dlrm", "dlrm", "prefill", "kv", "decode", "decode", "put", "a2a"])
    if kind == "moe":
        mode = rng.choice(["train", "train", "infer"])
        fp8 = rng.random() < 0.25
        if rng.random() < 0.5:
            H, F, E = 4096, 14336, 8
        else:
            H = rng.choice([512, 1024, 2048])
            F, E = 256 * rng.randint(2 * H // 256, 7 * H // 512), rng.choice([4, 8, 16, 32] if H < 2048 else [4, 8, 16])
        k = rng.choice([1, 2, 2, 4])
        most = min(8192, 8192 * 2 * 4096 * 14336 // (k * H * F))
        T = _log(rng, min(most, max(900, 128 * E // k)), most)
        return dict(kind=kind, tokens=T, hidden=H, ffn=F, experts=E, topk=k, zipf=rng.choice([0.0, 1.2]) if E == 8 else 0.0, mode=mode, fp8=fp8,
                    fused=mode == "train" and rng.random() < 0.5)
    if kind == "dlrm":
        return dict(kind=kind, batch=_log(rng, 128, 65536), tables=rng.randint(2, 26), rows=_log(rng, 10_000, 1_000_000),
                    pooling=rng.randint(1, 20), zipf=1.05)
    if kind in ("prefill", "decode"):
        name = rng.choice(["llama3_8b", "gpt2", "opt_125m", "opt_1.3b"])
        most = 1008 if name == "gpt2" else 2016
        dtype = rng.choice(["bf16", "bf16", "fp16"])
        if kind == "prefill":
            length = 16 * _log(rng, 1, most // 16)
            return dict(kind=kind, model=name, batch=min(_log(rng, 1, 32), max(1, 32768 // length)), length=length, dtype=dtype)
        steps = rng.randint(4, 16)
        return dict(kind=kind, model=name, batch=_log(rng, 1, 32), length=_log(rng, 16, most - 32), steps=steps, dtype=dtype)
    if kind == "kv":
        name, tp = rng.choice([("llama3_8b", 1), ("llama3_8b", 4), ("opt_1.3b", 1), ("opt_1.3b", 2), ("gpt2", 1)])
        return dict(kind=kind, model=name, tp=tp, batch=rng.randint(1, 16), length=16 * rng.randint(1, 128),
                    layers=rng.choice([1, MODEL_ZOO[name].layers]))
    if kind == "put":
        return dict(kind=kind, bytes=2 * _log(rng, 8, 512 * MIB))
    W = rng.choice([2, 4, 8])
    n = _log(rng, 512, 64 * MIB // W)
    return dict(kind=kind, world=W, elems=n if rng.random() < 0.5 else (n + 7) // 8 * 8)


class State:
    """What a program keeps between calls.  The heaps of a state that is gone are given back when the next one is made."""


_open = []


def _keep(heaps):
    s = State()
    s.heaps = heaps
    _open.append((weakref.ref(s), heaps))
    return s


def _close_unused():
    for entry in [e for e in _open if e[0]() is None]:
        _open.remove(entry)
        for h in entry[1]:
            h.close()


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def prepare(case, seed):
    _close_unused()
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(s):
    return s.run(s)


# ---- MoE ------------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _empty_moe(H, F, E, k, fp8, zipf, fused):
    """The layer without memory behind its parameters; a program that loads a checkpoint starts from the same."""
    cfg = MoEConfig(hidden=H, ffn=F, num_experts=E, topk=k, tokens=1, fp8=fp8)
    return MoELayer(cfg, None, 0, 1, device="meta", zipf_s=zipf or None, fused_sgd_lr=0.01 if fused else 0.0)


def _prepare_moe(c, seed):
    T, H, F, E, k = c["tokens"], c["hidden"], c["ffn"], c["experts"], c["topk"]
    layer = copy.deepcopy(_empty_moe(H, F, E, k, c["fp8"], c["zipf"], c["fused"])).to_empty(device=DEV)
    cfg = MoEConfig(hidden=H, ffn=F, num_experts=E, topk=k, tokens=T, fp8=c["fp8"])
    cap = (T + 127) // 128 * 128
    heap = SymmetricHeap.create((2 * E * cap + 2 * T * k) * H * 2 + E * cap * 4 + 4 * MIB, device=0)
    s = _keep([heap])
    g = _gen(seed)
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0, 0.02, generator=g)
        layer.router_bias.copy_(zipf_log_bias(E, c["zipf"]) if c["zipf"] else torch.zeros(E))
    layer.cfg, layer.ws = cfg, MoEWorkspace(heap, cfg, "moe")
    s.layer = layer.train() if c["mode"] == "train" else layer.eval()
    s.x = torch.randn(T, H, generator=g, device=DEV).to(torch.bfloat16)
    # the gradient that reaches the layer's output, and the weight of the load-balancing term of the loss
    s.dout = (torch.randn(T, H, generator=g, device=DEV) * 2e-4).to(torch.bfloat16)
    s.aux = torch.full((), 0.01, device=DEV)
    s.fused = c["fused"]
    s.run = _run_moe_train if c["mode"] == "train" else _run_moe_infer
    return s


def _run_moe_train(s):
    layer = s.layer
    x = s.x.detach().requires_grad_(True)
    out = layer(x)
    torch.autograd.backward([out, layer.l_aux], [s.dout, s.aux])
    res = {"out": out.detach(), "dx": x.grad, "drouter": layer.router.grad}
    if s.fused:
        res.update(w13=layer.w13.detach(), w2=layer.w2.detach())
    else:
        res.update(dw13=layer.w13.grad, dw2=layer.w2.grad)
    layer.zero_grad(set_to_none=True)
    return res


def _run_moe_infer(s):
    with torch.no_grad():
        return s.layer(s.x)


# ---- DLRM -----------------------------------------------------------------------------------------------------------------
def _dlrm_config(c):
    return DLRMConfig(num_tables=c["tables"], rows=c["rows"], pooling=c["pooling"], global_batch=c["batch"], zipf_alpha=c["zipf"])


def _prepare_dlrm(c, seed):
    torch.backends.cuda.matmul.allow_tf32 = True          # as the benchmark's programs set it for the dense MLPs
    cfg = _dlrm_config(c)
    heap = SymmetricHeap.create(2 * cfg.global_batch * cfg.num_tables * cfg.dim * 4 + 16 * MIB, device=0)
    s = _keep([heap])
    s.model = DLRM(cfg, heap, 0, 1, device=DEV, seed=int(seed))
    s.opt = torch.optim.SGD(s.model.dense_parameters(), lr=cfg.lr)
    s.batch = synthetic_batch(cfg, 0, 1, DEV, seed=int(seed) + 1)
    s.views = {"pooled": s.model.pooled.local, "grad_pooled": s.model.gpooled.local, "tables": s.model.tables}
    s.run = _run_dlrm
    return s


def _run_dlrm(s):
    loss = s.model.train_step(*s.batch, s.opt)
    return {"loss": loss, "dense": [p.detach() for p in s.model.dense_parameters()], **s.views}


# ---- transfers ------------------------------------------------------------------------------------------------------------
def _prepare_put(c, seed):
    n = c["bytes"]
    heaps = SymmetricHeap.emulated(2, n + 4 * MIB)
    s = _keep(heaps)
    s.chans = [Channel(h, "put") for h in heaps]
    s.dst = [h.alloc_tensor([n], torch.uint8) for h in heaps]
    s.src = torch.randn(n // 2, generator=_gen(seed), device=DEV).to(torch.bfloat16)
    s.bytes, s.out, s.run = n, s.dst[1].local, _run_put
    return s


def _run_put(s):
    s.chans[0].put(s.src, 1, s.dst[0].offset)
    s.chans[1].expect(0, s.bytes)
    s.chans[1].wait([0])
    return s.out


def _prepare_a2a(c, seed):
    W, n = c["world"], c["elems"]
    heaps = SymmetricHeap.emulated(W, W * n * 2 + 4 * MIB)
    s = _keep(heaps)
    s.chans = [Channel(h, "a2a") for h in heaps]
    s.recv = [h.alloc_tensor([W, n], torch.bfloat16) for h in heaps]
    g = _gen(seed)
    s.send = [torch.randn(W, n, generator=g, device=DEV).to(torch.bfloat16) for _ in range(W)]
    s.out, s.run = [r.local for r in s.recv], _run_a2a
    return s


def _run_a2a(s):
    for c, x, r in zip(s.chans, s.send, s.recv):
        all_to_all(c, x, r, wait=False)
    for c in s.chans:
        c.wait()
    return s.out


# ---- serving --------------------------------------------------------------------------------------------------------------
def _params(c, steps):
    return ServeParams(model=MODEL_ZOO[c["model"]], batch_size=c["batch"], input_len=c["length"], num_decoding_step=steps,
                       dtype=DTYPES[c.get("dtype", "bf16")])


def _pool_bytes(p, kv_heads):
    m = p.model
    return 2 * p.batch_size * p.max_blocks_per_req * m.layers * kv_heads * m.block_size * m.head_dim * 2


def _lm(c, seed):
    """Random weights with the two properties of trained models that greedy decoding depends on: residual branches that add up
    to about the size of the embedding, and next tokens that win by a clear margin (the output head is the embedding in another
    order), so that a token does not hang on the last bit of a logit."""
    cfg = MODEL_ZOO[c["model"]]
    m = LlamaShard(cfg, device=DEV, seed=int(seed), dtype=DTYPES[c["dtype"]])
    for w in m.wo + m.w2:
        w.mul_((2 * cfg.layers) ** -0.5)
    order = torch.randperm(cfg.vocab, generator=_gen(seed), device=DEV)
    m.lm_head = m.embed[order]                 # normal(0, 0.02), as the constructor makes it
    m.embed.mul_(50.0)
    return m


def _prepare_prefill(c, seed):
    p = _params(c, 16)
    heaps = SymmetricHeap.emulated(2, _pool_bytes(p, p.model.kv_heads) + 4 * MIB)
    s = _keep(heaps)
    model = _lm(c, seed)
    s.links = [KVLink(h, p, model.kvh_local) for h in heaps]
    s.stage = PrefillStage(p, model, s.links[0], dst_rank=1)
    s.tokens = torch.randint(0, p.model.vocab, (p.batch_size, p.input_len), generator=_gen(seed + 1), device=DEV)
    link = s.links[1]
    s.out = {"header": link.hdr.local, "k": link.k_pool.local, "v": link.v_pool.local}
    s.run = _run_prefill
    return s


def _run_prefill(s):
    s.stage.run(s.tokens)
    return s.out


def _prepare_decode(c, seed):
    p = _params(c, c["steps"])
    m = p.model
    heaps = SymmetricHeap.emulated(1, _pool_bytes(p, m.kv_heads) + 4 * MIB)
    s = _keep(heaps)
    model, g = _lm(c, seed), _gen(seed + 1)
    link = KVLink(heaps[0], p, model.kvh_local)
    for pool in (link.k_pool.local, link.v_pool.local):
        pool.normal_(0.0, 1.0, generator=g)
    s.stage = DecodeStage(p, model, link)
    s.tokens = torch.randint(0, m.vocab, (p.batch_size,), generator=g, device=DEV)
    # the positions that the pass writes (pages of a request are consecutive in this stage's block table)
    written = slice(p.input_len, p.input_len + p.num_decoding_step)
    s.new = {n: pool.local.view(m.layers, p.batch_size, -1, m.kv_heads, m.head_dim)[:, :, written]
             for n, pool in (("k", link.k_pool), ("v", link.v_pool))}
    s.run = _run_decode
    return s


def _run_decode(s):
    tokens, _ = s.stage.decode(s.tokens)
    return {"tokens": tokens, **s.new}


def _prepare_kv(c, seed):
    p = _params(c, 16)
    m = p.model
    kvh = m.kv_heads // c["tp"]
    heaps = SymmetricHeap.emulated(2, _pool_bytes(p, kvh) + 4 * MIB)
    s = _keep(heaps)
    s.links = [KVLink(h, p, kvh) for h in heaps]
    g, B, nb, mb = _gen(seed), p.batch_size, p.context_blocks_per_req, p.max_blocks_per_req
    n = B * nb * m.layers * s.links[0].page_elems
    s.k, s.v = (torch.empty(n, dtype=p.dtype, device=DEV).normal_(0.0, 1.0, generator=g) for _ in range(2))
    # pages are wherever the allocators of the two sides found room
    s.src_bt = torch.randperm(B * nb, generator=g, device=DEV).view(B, nb).int()
    s.dst_bt = torch.randperm(B * mb, generator=g, device=DEV)[: B * nb].view(B, nb).int()
    s.nblocks = torch.full((B,), nb, dtype=torch.int32, device=DEV)
    s.src_blocks, s.layers = B * nb, c["layers"]
    s.out = [s.links[1].k_pool.local, s.links[1].v_pool.local]
    s.run = _run_kv
    return s


def _run_kv(s):
    link = s.links[0]
    link.seq += 1
    link.send_layers(1, s.k, s.v, s.src_blocks, s.src_bt, s.dst_bt, s.nblocks, 0, s.layers)
    return s.out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------
def _touched_rows(rows, alpha, n):
    """Expected number of different rows among n Zipf(alpha) draws from `rows`."""
    p = np.arange(1, rows + 1, dtype=np.float64) ** -alpha
    return float(-np.expm1(n * np.log1p(-np.minimum(p / p.sum(), 0.999999))).sum())


def _lm_layer(m):
    """(bytes of a layer's matrices and of one token's K and V in the layer, in elements)"""
    q, kv = m.heads * m.head_dim, m.kv_heads * m.head_dim
    return (q + 2 * kv) * m.hidden + q * m.hidden + (3 if m.arch == "llama" else 2) * m.hidden * m.ffn, 2 * kv


def work(case):
    c, kind = case, case["kind"]
    if kind == "moe":
        T, H, F, E, k = c["tokens"], c["hidden"], c["ffn"], c["experts"], c["topk"]
        expert = 3 * H * F
        seen = E * (1.0 - (1.0 - 1.0 / E) ** (T * k)) if not c["zipf"] else min(E, T * k)     # experts that get a row
        fwd = 2.0 * T * k * expert + 2.0 * T * E * H
        if c["mode"] == "infer":
            return {"bytes": 2.0 * seen * expert + 4.0 * T * H, "flops": fwd}
        # weights read once, written once (the update, or the gradients); x, dout in, out, dx out
        return {"bytes": 4.0 * E * expert + 8.0 * T * H, "flops": 3 * fwd}
    if kind == "dlrm":
        cfg = _dlrm_config(c)
        B, t, D = c["batch"], c["tables"], cfg.dim
        sizes = (cfg.dense_features,) + cfg.bottom
        top = (t * (t + 1) // 2 + D,) + cfg.top
        mlp = sum(a * b for s in (sizes, top) for a, b in zip(s, s[1:]))
        rows = t * _touched_rows(c["rows"], c["zipf"], B * c["pooling"])
        # rows read and written back; the pooled vectors and their gradients are buffers that other ranks read and write
        return {"bytes": 2 * rows * D * 4 + 8.0 * B * t * c["pooling"] + 2.0 * B * t * D * 4 + 4.0 * B * (cfg.dense_features + 1),
                "flops": 6.0 * B * (mlp + (t + 1) * t // 2 * D) + 3.0 * B * t * c["pooling"] * D}
    if kind == "put":
        return {"bytes": 2.0 * c["bytes"], "flops": 0}
    if kind == "a2a":
        return {"bytes": 2.0 * c["world"] ** 2 * c["elems"] * 2, "flops": 0}
    m, B, n = MODEL_ZOO[c["model"]], c["batch"], c["length"]
    layer, kv = _lm_layer(m)
    if kind == "kv":
        return {"bytes": 2.0 * 2 * B * n * c["layers"] * kv // c["tp"], "flops": 0}
    attn = 4.0 * m.heads * m.head_dim                      # per query and key
    head = m.vocab * m.hidden
    if kind == "prefill":
        return {"bytes": 2.0 * (m.layers * layer + head) + 2 * 2.0 * B * n * m.layers * kv,
                "flops": 2.0 * B * (n * m.layers * layer + head) + B * attn * m.layers * n * (n + 1) / 2}
    ctx = sum(n + i + 1 for i in range(c["steps"]))
    return {"bytes": 2.0 * c["steps"] * (m.layers * layer + head) + 2.0 * B * ctx * m.layers * kv,
            "flops": 2.0 * B * c["steps"] * (m.layers * layer + head) + B * ctx * m.layers * attn}


def tolerance(case):
    kind = case["kind"]
    if kind in ("put", "a2a", "kv"):
        return "exact"
    if kind == "moe":
        # bf16 results; with fp8 an activation may be quantised to the neighbouring value
        return {"rel": 2e-2 if case["fp8"] else 1e-2}
    if kind == "dlrm":
        # tf32 products; a ReLU whose input is within their error of zero passes its gradient or does not, which changes all of
        # one sample's gradient a little and some of it by as much as its size
        return {"rel": 1e-2, "max": 0.99}
    # The residual stream is rounded twice in every layer, 0.1 % each time in bf16: about 1 % after 32 layers, in either of two
    # implementations.  Tokens win by a margin and have to be the same.
    return {"rel": 2e-2 if case["dtype"] == "bf16" else 3e-3}
