"""The fused route of the decoder (models/llama.py over csrc/kernels/decoder.cu) takes the calls that the operation-by-operation
route takes and answers alike: both on host memory, the kernels as plain PyTorch with the same arguments."""
import ctypes
import math
import os

import pytest
import torch
import torch.nn.functional as F

from fuselink_b200.models import llama
from fuselink_b200.models.llama import KV_BLHSD, MODEL_ZOO, LlamaShard


class Kernels:
    """What the kernels are specified to do (decoder.cuh), values rounded at the same places."""

    @staticmethod
    def _bound(indices, table=None):
        """The types that the bindings take."""
        assert all(t is None or (t.dtype == torch.int64 and t.is_contiguous()) for t in indices)
        assert table is None or (table.dtype == torch.int32 and table.is_contiguous())

    def dec_embed(self, tokens, pos, embed, pos_embed, x, seq, offset, status=0):
        self._bound([tokens, pos])
        tokens = tokens.reshape(-1)
        x.copy_(embed[tokens])
        if pos_embed is not None:
            x += pos_embed[(torch.arange(tokens.numel()) % seq if pos is None else pos) + offset]

    def dec_add_norm(self, x, y, y_bias, w, b, h, eps):
        if y is not None:
            x += y if y_bias is None else y + y_bias
        h.copy_(llama._rms(x, w, eps) if b is None else llama._ln(x, w, b, eps))

    def dec_qkv(self, qkv, bias, rope, pos, seq, k_pool, v_pool, table, layout, layer, layers, num_blocks, bs, heads, kv_heads, dim, status=0):
        self._bound([pos], table)
        rows = torch.arange(qkv.shape[0])
        at, req = (rows % seq, rows // seq) if pos is None else (pos, rows)
        if bias is not None:
            qkv += bias
        y = qkv.view(len(rows), heads + 2 * kv_heads, dim)
        if rope is not None:
            cos, sin = (rope[at].unsqueeze(1)[..., s] for s in (slice(0, dim // 2), slice(dim // 2, None)))
            z = y[:, :heads + kv_heads].float()
            a, b = z[..., :dim // 2], z[..., dim // 2:]
            y[:, :heads + kv_heads] = torch.cat([a * cos - b * sin, b * cos + a * sin], -1).to(qkv.dtype)
        page, slot = table.long()[req, at // bs], at % bs
        for pool, v in ((k_pool, y[:, heads:heads + kv_heads]), (v_pool, y[:, heads + kv_heads:])):
            if layout == KV_BLHSD:
                pool.view(num_blocks, layers, kv_heads, bs, dim)[page, layer, :, slot] = v
            else:
                pool.view(layers, num_blocks, bs, kv_heads, dim)[layer, page, slot] = v

    def dec_act(self, h, bias, out, kind):
        if kind == 0:
            out.copy_(F.silu(h[:, :out.shape[1]]) * h[:, out.shape[1]:])
        else:
            out.copy_(F.relu(h + bias) if kind == 1 else F.gelu(h + bias, approximate="tanh"))

    def dec_attention(self, qkv, pos, k_pool, v_pool, table, layer, layers, num_blocks, bs, heads, kv_heads, dim, out, status=0):
        self._bound([pos], table)
        assert 1 <= qkv.shape[0] <= 65535
        for b in range(qkv.shape[0]):
            n = int(pos[b]) + 1
            k, v = (p.view(layers, num_blocks, bs, kv_heads, dim)[layer][table[b].long()].reshape(-1, kv_heads, dim)[:n].float()
                    .repeat_interleave(heads // kv_heads, 1) for p in (k_pool, v_pool))
            q = qkv[b, :heads * dim].view(heads, dim).float()
            p = (torch.einsum("hd,nhd->hn", q, k) / math.sqrt(dim)).softmax(-1)
            out[b] = torch.einsum("hn,nhd->hd", p, v).reshape(-1).to(out.dtype)

    def dec_argmax(self, logits):
        assert logits.dim() == 2
        return logits.float().argmax(-1)


FUSED, PLAIN = True, False


@pytest.fixture
def route(monkeypatch):
    """route(FUSED) and route(PLAIN) choose the route of the calls that follow."""
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)      # nothing to wait for on host memory
    monkeypatch.setattr(llama, "require_native", Kernels)
    return lambda fused: monkeypatch.setattr(LlamaShard, "_fused", lambda self, pool: fused)


def _net(model, dtype=torch.bfloat16):
    net = LlamaShard(MODEL_ZOO[model], device="cpu", seed=2, dtype=dtype)
    net.lm_head = net.embed.roll(1, 0).clone()         # next tokens that win by a margin
    net.embed.mul_(50)
    return net


def _prefill(net, tokens, table=None, blocks=None, **kw):
    cfg, (B, S) = net.cfg, tokens.shape
    per = S // cfg.block_size
    if table is None:
        table = torch.randperm(B * per, generator=torch.Generator().manual_seed(1)).view(B, per).int()
    pools = [torch.zeros((blocks or B * per) * cfg.layers * cfg.kv_heads * cfg.block_size * cfg.head_dim, dtype=net.embed.dtype) for _ in range(2)]
    return net.prefill(tokens, *pools, table, **kw), *pools


def _tokens(net, B, S):
    return torch.randint(0, net.cfg.vocab, (B, S), generator=torch.Generator().manual_seed(5))


def _alike(a, b, dtype=torch.bfloat16):
    assert torch.equal(a[0], b[0])
    for x, y in zip(a[1:], b[1:]):
        assert (x.float() - y.float()).norm() <= 4 * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * y.float().norm()


@pytest.mark.parametrize("model", ["tiny", "tiny_opt", "tiny_gpt2"])
@pytest.mark.parametrize("last_pos", [None, 3, -1, -20, torch.tensor([0, 31, 7]), torch.tensor([-1, 5, -32]), torch.tensor([4, -2, 9], dtype=torch.int32),
                                      torch.tensor([[1, 2, 3], [4, 5, -6]])])
def test_the_position_that_gives_the_first_token(model, last_pos, route):
    """Positions count from the request's own end where they are negative, in either route."""
    net = _net(model)
    toks = _tokens(net, 3, 32)
    res = []
    for r in (FUSED, PLAIN):
        route(r)
        res.append(_prefill(net, toks, last_pos=last_pos))
    _alike(*res)


@pytest.mark.parametrize("last_pos", [32, -33, torch.tensor([0, 40, 1])])
def test_a_position_outside_the_prompt_is_an_error(last_pos, route):
    net = _net("tiny")
    for r in (FUSED, PLAIN):
        route(r)
        with pytest.raises(IndexError):
            _prefill(net, _tokens(net, 3, 32), last_pos=last_pos)


def _decode(net, tokens, positions, table, nb):
    cfg = net.cfg
    g = torch.Generator().manual_seed(6)
    pools = [torch.randn(cfg.layers * nb * cfg.block_size * cfg.kv_heads * cfg.head_dim, generator=g).to(net.embed.dtype) for _ in range(2)]
    return net.decode_step(tokens, positions, *pools, table, nb), *pools


@pytest.mark.parametrize("model", ["tiny", "tiny_opt", "tiny_gpt2"])
@pytest.mark.parametrize("form", [lambda t: t.int(), lambda t: t.long(), lambda t: torch.stack([t, t], -1)[..., 0], lambda t: t.t().contiguous().t()])
def test_forms_of_tokens_positions_and_tables(model, form, route):
    """int32 and int64, contiguous or not."""
    net = _net(model)
    table = torch.tensor([[3, 0], [1, 5], [4, 2]])
    res = []
    for r in (FUSED, PLAIN):
        route(r)
        first = _prefill(net, form(_tokens(net, 3, 32)), form(table))
        step = _decode(net, form(_tokens(net, 3, 1)[:, 0]), form(torch.tensor([30, 0, 17])), form(table), 6)
        res.append((first[0], *first[1:], *step[1:], step[0].float()))
    _alike(*res)


@pytest.mark.parametrize("batch", [0, 65536])
def test_batches_the_attention_kernel_does_not_take(batch, route):
    """It takes 1 to 65535 requests; other steps keep the general route."""
    import dataclasses
    route(FUSED)
    net = LlamaShard(dataclasses.replace(MODEL_ZOO["tiny"], layers=1, hidden=64, heads=1, kv_heads=1, ffn=64, vocab=16), device="cpu")
    toks = torch.zeros(batch, dtype=torch.long)
    assert _decode(net, toks, toks, torch.zeros(batch, 1, dtype=torch.int32), 1)[0].shape == (batch,)


def test_another_rotation_base_is_followed(route, monkeypatch):
    import dataclasses
    from unittest import mock
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)           # tables are kept
    monkeypatch.setattr(torch.cuda, "current_stream", mock.Mock())
    net = _net("tiny")
    net.cfg = dataclasses.replace(net.cfg)
    for theta in (10000.0, 500000.0, 10000.0):
        net.cfg.rope_theta = theta
        res = []
        for r in (FUSED, PLAIN):
            route(r)
            res.append(_prefill(net, _tokens(net, 2, 48)))
        _alike(*res)
    assert len(net._rope_tables) == 2
    for theta in range(20000, 20010):
        net.cfg.rope_theta = float(theta)
        assert torch.equal(net._rope_table(100), net._rope_table(4096))
    assert len(net._rope_tables) == 8 and all(len(t) == 1 for t in net._rope_tables.values())


def test_indices_of_other_types_are_an_error(route):
    net = _net("tiny")
    table = torch.tensor([[0, 1]])
    for r in (FUSED, PLAIN):
        route(r)
        for dtype in (torch.float32, torch.int16):
            with pytest.raises((IndexError, RuntimeError)):
                _prefill(net, _tokens(net, 1, 32).to(dtype), table)
            with pytest.raises((IndexError, RuntimeError)):
                _decode(net, torch.tensor([1]).to(dtype), torch.tensor([5]), table, 2)
        for bad in (1 << 32, -(1 << 32) + 1):
            with pytest.raises(IndexError):
                _prefill(net, _tokens(net, 1, 32), torch.tensor([[0, bad]]))


@pytest.mark.parametrize("table", [torch.zeros(3, 1, dtype=torch.int32), torch.zeros(2, 2, dtype=torch.int32)])
def test_a_block_table_that_does_not_cover_the_prompts_is_an_error(table, route):
    net = _net("tiny")
    for r in (FUSED, PLAIN):
        route(r)
        with pytest.raises((IndexError, RuntimeError)):
            _prefill(net, _tokens(net, 3, 32), table, blocks=6)


def test_prompts_longer_than_the_position_embedding_are_an_error(route):
    net = _net("tiny_gpt2")
    net.pos_embed = net.pos_embed[:31].clone()
    for r in (FUSED, PLAIN):
        route(r)
        with pytest.raises(IndexError):
            _prefill(net, _tokens(net, 1, 32))


def test_pools_of_another_size_are_an_error(route):
    net = _net("tiny")
    cfg = net.cfg
    page = cfg.layers * cfg.kv_heads * cfg.block_size * cfg.head_dim
    for r in (FUSED, PLAIN):
        route(r)
        for k, v in ((2 * page, 2 * page + 8), (2 * page + 8, 2 * page)):
            pools = torch.zeros(k, dtype=torch.bfloat16), torch.zeros(v, dtype=torch.bfloat16)
            with pytest.raises(RuntimeError):
                net.prefill(_tokens(net, 1, 32), *pools, torch.tensor([[0, 1]]))
            with pytest.raises(RuntimeError):
                net.decode_step(torch.tensor([1]), torch.tensor([3]), *pools, torch.tensor([[0, 1]]), 2)
        with pytest.raises((IndexError, RuntimeError)):
            pools = [torch.zeros(2 * page, dtype=torch.bfloat16) for _ in range(2)]
            net.decode_step(torch.tensor([1, 2]), torch.tensor([3, 3]), *pools, torch.tensor([[0, 1]]), 2)


def test_a_noted_index_is_raised_once(route):
    import copy
    import pickle
    net = _net("tiny")
    net.check_status()
    route(FUSED)
    net._status = llama._Status()
    for call in (net.check_status, lambda: _prefill(net, _tokens(net, 1, 32))):
        net._status.word[0] = 2
        with pytest.raises(IndexError, match="position"):
            call()
        net.check_status()
    net._status.word[0] = 1
    for other in (copy.deepcopy(net), pickle.loads(pickle.dumps(net))):
        other.check_status()                        # a word of its own
        assert other._status.word.data_ptr() != net._status.word.data_ptr()


def _shifted(t):
    """The same values from an address that is a multiple of 2 bytes only."""
    flat = torch.empty(t.numel() + 9, dtype=t.dtype)
    first = next(i for i in range(1, 9) if flat[i:].data_ptr() % 16 == 2)
    flat[first:first + t.numel()] = t.reshape(-1)
    return flat[first:first + t.numel()].view(t.shape)


@pytest.mark.parametrize("name", ["embed", "pos_embed", "final_norm", "final_norm_b", "n1", "n1b", "n2", "n2b", "bqkv", "bo", "b13", "b2", "pool"])
def test_tensors_the_kernels_do_not_take_go_the_general_route(name):
    pool = torch.zeros(64, dtype=torch.bfloat16)
    for change in (_shifted, lambda t: t.float(), lambda t: torch.stack([t, t], -1)[..., 0]):
        net = _net("tiny_opt")
        assert net._fits(pool)
        if name == "pool":
            assert not net._fits(change(pool)) and not net._same_kind(change(pool), pool)
        elif isinstance(getattr(net, name), list):
            getattr(net, name)[1] = change(getattr(net, name)[1])
            assert not net._fits(pool)
        else:
            setattr(net, name, change(getattr(net, name)))
            assert not net._fits(pool)


@pytest.mark.parametrize("op", ["_embed", "_norm", "_qkv", "_attn_out", "_mlp", "_logits"])
def test_replaced_operations_go_the_general_route(op):
    pool = torch.zeros(64, dtype=torch.bfloat16)
    own = getattr(LlamaShard, op)
    net = type("Other", (LlamaShard,), {op: lambda self, *a: own(self, *a)})(MODEL_ZOO["tiny"], device="cpu")
    assert not net._fits(pool)
    net = type("Same", (LlamaShard,), {"more": 1})(MODEL_ZOO["tiny"], device="cpu")
    assert net._fits(pool)
    setattr(net, op, lambda *a: own(net, *a))
    assert not net._fits(pool)


def test_tensor_subclasses_and_autocast_go_the_general_route(monkeypatch):
    from unittest import mock
    pool = torch.zeros(64, dtype=torch.bfloat16)
    net = _net("tiny")
    monkeypatch.setattr(net, "embed", mock.Mock(is_cuda=True))
    monkeypatch.setattr(LlamaShard, "_fits", lambda self, pool: True)
    assert net._fused(pool)
    monkeypatch.setattr(torch, "is_autocast_enabled", lambda device: device == "cuda")
    assert not net._fused(pool)
    monkeypatch.undo()
    net = _net("tiny")
    net.n1[0] = net.n1[0].as_subclass(type("Wrapped", (torch.Tensor,), {}))
    assert not net._fits(pool)


def test_c_entries_refuse_addresses_they_cannot_read():
    """Every pointer in turn off its 16 bytes; nothing is launched for zero rows, so the addresses are never used."""
    from fuselink_b200 import build
    lib = ctypes.CDLL(os.path.join(build.LIB, "libfuselink.so"))
    P, I, LL, F32 = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float

    class Kv(ctypes.Structure):
        _fields_ = [("k", P), ("v", P), ("block_table", P)] + [(n, I) for n in ("table_stride", "layout", "layer", "layers", "num_blocks", "block_size", "heads")] + [("status", P)]

    def kv(k, v):
        return ctypes.byref(Kv(k, v, 0x1000, 4, 1, 0, 1, 8, 16, 2))

    calls = [
        (3, lambda p: lib.fl_dec_embed(I(0), P(8), P(8), P(p[0]), P(p[1]), P(p[2]), LL(0), I(64), I(1), I(0), LL(10), LL(10), P(), P())),
        (6, lambda p: lib.fl_dec_add_norm(I(0), *map(P, p), LL(0), I(64), F32(1e-5), P())),
        (4, lambda p: lib.fl_dec_qkv(I(0), P(p[0]), P(p[1]), P(), LL(0), P(8), LL(0), I(1), I(2), I(64), kv(p[2], p[3]), P())),
        (3, lambda p: lib.fl_dec_act(I(0), I(1), *map(P, p), LL(0), I(64), P())),
    ]
    for n, call in calls:
        assert call([0x100000] * n) == 0
        for i in range(n):
            for off in (2, 4, 8):
                assert call([0x100000 + (off if k == i else 0) for k in range(n)]) == -4
    attention = lambda q, k, v: lib.fl_dec_attention(I(0), P(q), LL(384), P(8), kv(k, v), P(0x100000), I(1), I(2), I(64), P())
    for bad in ((2, 0, 0), (0, 4, 0), (0, 0, 8)):
        assert attention(*(0x100000 + b for b in bad)) == -4
