"""The fused decoder passes (csrc/kernels/decoder.cu) against the same operations in fp32 / PyTorch."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DT = [torch.bfloat16, torch.float16]


def _eps(dt):
    return 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11          # half a unit in the last place, relative


def _rand(*shape, dt, seed):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("batch,heads,kv_heads,dim,bs,lens", [
    (1, 1, 1, 64, 16, [1]), (3, 4, 2, 64, 16, [15, 16, 17]), (2, 32, 8, 128, 16, [2049, 700]), (2, 12, 12, 80, 8, [129, 1]),
    (2, 24, 2, 128, 5, [333, 1000]), (17, 8, 8, 96, 16, [7 * i + 1 for i in range(17)]),
    (1, 8, 8, 128, 32, [5000]), (150, 4, 4, 64, 16, [40 + i for i in range(150)]),
])
def test_paged_attention_of_one_token(dt, batch, heads, kv_heads, dim, bs, lens):
    from fuselink_b200 import C
    L, layer, maxblk = 2, 1, max(lens) // bs + 3
    nb = batch * maxblk
    kp, vp = (_rand(L, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    qkv = _rand(batch, (heads + 2 * kv_heads) * dim, dt=dt, seed=4)
    pos = torch.tensor(lens, device="cuda") - 1
    out = torch.full((batch, heads * dim), float("nan"), dtype=dt, device="cuda")
    C.dec_attention(qkv, pos, kp, vp, bt, layer, L, nb, bs, heads, kv_heads, dim, out)
    for b, n in enumerate(lens):
        k, v = (p[layer][bt[b].long()].reshape(-1, kv_heads, dim)[:n].float().repeat_interleave(heads // kv_heads, 1) for p in (kp, vp))
        q = qkv[b, : heads * dim].view(heads, dim).float()
        want = torch.einsum("hn,nhd->hd", (torch.einsum("hd,nhd->hn", q, k) / math.sqrt(dim)).softmax(-1), v).reshape(-1)
        # the probabilities are rounded to the type before the second product (a sum of at most max|v| x eps), and the result
        assert (out[b].float() - want).abs().max() <= 2 * _eps(dt) * v.abs().max() + 1e-5


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("kv_heads,dim,bs,lens", [(2, 64, 16, [40, 5]), (8, 128, 16, [2049, 1500]), (2, 80, 8, [300, 90]), (4, 64, 32, [1000] * 160)])
@pytest.mark.parametrize("value,where", [(float("nan"), "first"), (float("nan"), "last"), (float("nan"), "all"), (float("inf"), "first"), (float("-inf"), "first"),
                                         (float("-inf"), "last"), (float("-inf"), "all")])
def test_paged_attention_passes_on_what_is_not_finite(dt, kv_heads, dim, bs, lens, value, where):
    """A NaN or infinite score makes the head NaN, as a softmax does; one of -inf (here a whole step of 16 tokens, before or behind
    finite ones) weighs nothing, and nothing but such scores is NaN.  Other heads and requests are as without."""
    from fuselink_b200 import C
    heads, batch, maxblk = 2 * kv_heads, len(lens), max(lens) // bs + 1
    nb = batch * maxblk
    kp, vp = (_rand(1, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    qkv = _rand(batch, (heads + 2 * kv_heads) * dim, dt=dt, seed=4)
    qkv[:, 0:heads * dim:dim] = 1                                   # every query's first column: the score gets the key's infinity
    n = lens[0]
    for tok in dict(first=range(min(16, n - 1)), last=range((n - 1) // 16 * 16, n), all=range(n))[where]:
        kp[0, bt[0, tok // bs].long(), tok % bs, 1, 0] = value
    pos = torch.tensor(lens, device="cuda") - 1
    out = torch.empty(batch, heads * dim, dtype=dt, device="cuda")
    C.dec_attention(qkv, pos, kp, vp, bt, 0, 1, nb, bs, heads, kv_heads, dim, out)
    for b in (0, batch - 1):
        k, v = (p[0][bt[b].long()].reshape(-1, kv_heads, dim)[:lens[b]].float().repeat_interleave(2, 1) for p in (kp, vp))
        q = qkv[b, : heads * dim].view(heads, dim).float()
        want = torch.einsum("hn,nhd->hd", ((q.unsqueeze(0) * k).sum(-1).t() / math.sqrt(dim)).softmax(-1), v).reshape(-1)
        got = out[b].float()
        if b == 0:
            assert want.view(heads, dim)[2:4].isnan().all() == (value != float("-inf") or where == "all")
        assert torch.equal(got.isnan(), want.isnan())
        # as above: the probabilities' rounding to the type and the result's
        assert ((got - want).abs()[~want.isnan()] <= 2 * _eps(dt) * v.abs().max() + 1e-5).all()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("rows,hidden", [(1, 64), (5, 768), (200, 2048), (3, 8192), (2, 20480), (150, 1032)])
@pytest.mark.parametrize("ln", [False, True])
def test_add_norm(dt, rows, hidden, ln):
    from fuselink_b200 import C
    from fuselink_b200.models.llama import _ln, _rms
    x, y = _rand(rows, hidden, dt=dt, seed=1), _rand(rows, hidden, dt=dt, seed=2)
    yb, w, b = (_rand(hidden, dt=dt, seed=s) for s in (3, 4, 5))
    for yy, bias in ((None, None), (y, None), (y, yb)):
        xs, h = x.clone(), torch.empty_like(x)
        C.dec_add_norm(xs, yy, bias, w, b if ln else None, h, 1e-5)
        want_x = x if yy is None else x + (yy if bias is None else yy + bias)
        assert torch.equal(xs, want_x)
        want = _ln(want_x, w, b, 1e-5) if ln else _rms(want_x, w, 1e-5)
        # The sums are taken in another order, so a value next to the middle between two neighbours may be rounded to the other
        # one, 2 eps away relatively: the result, and with the RMS norm also the normalised value before it meets its weight.
        # The layer norm adds its bias to a product that may cancel it: the absolute term.
        assert ((h - want).float().abs() <= (2.02 if ln else 4.05) * _eps(dt) * want.float().abs() + (2e-6 if ln else 0)).all()


@pytest.mark.parametrize("model,dt", [("tiny", torch.bfloat16), ("tiny_opt", torch.float16), ("tiny_gpt2", torch.bfloat16)])
@pytest.mark.parametrize("batch,length", [(1, 16), (3, 48)])
def test_fused_layers_match_the_operations(model, dt, batch, length, monkeypatch):
    """Prefill and two decoding steps with the kernels and without them: pages and tokens."""
    from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
    cfg = MODEL_ZOO[model]
    net = LlamaShard(cfg, device="cuda", seed=2, dtype=dt)
    net.lm_head = net.embed.roll(1, 0).clone()         # next tokens that win by a margin
    net.embed.mul_(50)
    bs, D, kl, L = cfg.block_size, cfg.head_dim, cfg.kv_heads, cfg.layers
    per = length // bs + 1
    nb = batch * per
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(1)).view(batch, per).int().cuda()
    toks = torch.randint(0, cfg.vocab, (batch, length), generator=torch.Generator().manual_seed(2)).cuda()
    res = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(LlamaShard, "_fused", lambda self, pool: False)
        kp, vp = (torch.zeros(nb * L * kl * bs * D, dtype=dt, device="cuda") for _ in range(2))
        first = net.prefill(toks, kp, vp, bt)
        kd, vd = (p.view(nb, L, kl, bs, D).permute(1, 0, 3, 2, 4).contiguous().view(-1) for p in (kp, vp))
        t, out = first, [first]
        for s in range(2):
            t = net.decode_step(t, torch.full((batch,), length + s, device="cuda"), kd, vd, bt, nb)
            out.append(t)
        res.append((torch.stack(out), kp, vp, kd, vd))
    assert torch.equal(res[0][0], res[1][0])
    for a, b in zip(res[0][1:], res[1][1:]):
        # two layers of a handful of roundings each
        assert (a.float() - b.float()).norm() <= 4 * _eps(dt) * b.float().norm()


@pytest.mark.parametrize("rows,vocab", [(1, 1), (3, 1000), (16, 50257), (2, 128256)])
def test_argmax(rows, vocab):
    from fuselink_b200 import C
    x = _rand(rows, vocab, dt=torch.bfloat16, seed=3)
    got = C.dec_argmax(x)
    best = x.float().max(1, keepdim=True).values
    first = (x.float() == best).int().argmax(1)
    assert torch.equal(got, first)


@pytest.mark.parametrize("rows,vocab", [(3, 32767), (3, 32768), (37, 32775), (38, 32775), (2, 128256)])
@pytest.mark.parametrize("dt", DT)
def test_argmax_over_the_ctas_of_a_row(rows, vocab, dt):
    """The line to a cluster per row (32768 entries, 37 rows) and what its CTAs compare: equal values, NaN, nothing but -inf."""
    from fuselink_b200 import C
    x = torch.zeros(rows, vocab, dtype=dt, device="cuda")
    for at in (vocab - 1, vocab // 2, 4097, 4096):
        x[0, at] = 1
        assert C.dec_argmax(x)[0] == at
    x[1, vocab - 2], x[1, 7], x[1, vocab - 9] = float("inf"), float("inf"), float("nan")
    assert C.dec_argmax(x)[1] == vocab - 9                  # NaN is the largest, as in torch.argmax
    x[1, vocab // 3] = float("nan")
    x[-1] = float("-inf")
    want = torch.zeros(rows, dtype=torch.int64, device="cuda")
    want[0], want[1] = 4096, vocab // 3
    if rows == 2:
        want[1] = 0
    assert torch.equal(C.dec_argmax(x), want)


@pytest.mark.parametrize("kind,ffn", [(0, 512), (1, 24), (2, 3072)])
def test_activation(kind, ffn):
    from fuselink_b200 import C
    h, b = _rand(7, ffn * (2 if kind == 0 else 1), dt=torch.bfloat16, seed=1), _rand(ffn, dt=torch.bfloat16, seed=2)
    out = torch.empty(7, ffn, dtype=torch.bfloat16, device="cuda")
    C.dec_act(h, None if kind == 0 else b, out, kind)
    want = F.silu(h[:, :ffn]) * h[:, ffn:] if kind == 0 else F.relu(h + b) if kind == 1 else F.gelu(h + b, approximate="tanh")
    assert ((out - want).float().abs() <= 2.02 * 2.0 ** -8 * want.float().abs() + 1e-6).all()


@pytest.mark.parametrize("dt", DT)
def test_silu_of_every_value(dt):
    """Of every 16-bit value, against 64 bits: rounded once, as is the product with 1.  4e-37 and 6e-8: the largest result that e^-x = inf
    (x < -88.7) loses, and fp16's smallest step."""
    from fuselink_b200 import C
    x = torch.arange(-32768, 32768, device="cuda").to(torch.int16).view(dt).view(16, 4096)
    out = torch.empty_like(x)
    C.dec_act(torch.cat([x, torch.ones_like(x)], 1), None, out, 0)
    want = F.silu(x.double())
    want[x == float("-inf")] = float("nan")                          # -inf / inf, as before
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    fin = want.isfinite()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[~fin & ~want.isnan()].double(), want[~fin & ~want.isnan()])
    assert ((out.double() - want)[fin].abs() <= 1.01 * eps * want[fin].abs() + (4e-37 if dt == torch.bfloat16 else 6e-8)).all()


def test_silu_of_bf16_gates_is_that_of_full_precision():
    """The hardware's exponential and quotient stand before a rounding to bf16: of every gate the bits that expf and an IEEE division give,
    which are also the decoding products' (thin_gemm.cu)."""
    from fuselink_b200 import C
    x = torch.arange(-32768, 32768, device="cuda").to(torch.int16).view(torch.bfloat16).view(512, 128)
    out = torch.empty_like(x)
    C.dec_act(torch.cat([x, torch.ones_like(x)], 1), None, out, 0)
    want = (x.float() / (1 + torch.exp(-x.float()))).to(torch.bfloat16)
    assert torch.equal(out.isnan(), want.isnan())
    assert torch.equal(out.view(torch.int16)[~out.isnan()], want.view(torch.int16)[~out.isnan()])


def _shard(model):
    from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
    net = LlamaShard(MODEL_ZOO[model], device="cuda", seed=2)
    cfg = net.cfg
    pools = lambda blocks: [torch.zeros(blocks * cfg.layers * cfg.kv_heads * cfg.block_size * cfg.head_dim, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    return net, pools


@pytest.mark.parametrize("model", ["tiny", "tiny_gpt2"])
@pytest.mark.parametrize("token,table,pos,message", [
    (1000, [0, 1], 20, "token"), (-1001, [0, 1], 20, "token"), (3, [0, 1], 32, "position"), (3, [0, 1], 1 << 40, "position"), (3, [0, 1], -33, "position"),
    (3, [0, 2], 20, "page"), (3, [-3, 1], 20, "page"), (3, [1 << 30, 1], 20, "page"),
])
def test_an_index_outside_its_table_is_an_error(model, token, table, pos, message):
    """Skipped and noted by the kernels; raised by the next call or by check_status behind a synchronisation."""
    net, pools = _shard(model)
    k, v = pools(2)
    bt = torch.tensor([table], dtype=torch.int32, device="cuda")
    tok, at = torch.tensor([token], device="cuda"), torch.tensor([pos], device="cuda")
    ok = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda"), torch.tensor([5], device="cuda")
    assert net._fused(k)
    for look in (net.check_status, lambda: net.decode_step(ok[1], ok[1], k, v, ok[0], 2)):
        net.decode_step(tok, at, k, v, bt, 2)
        torch.cuda.synchronize()
        with pytest.raises(IndexError, match=message):
            look()
        net.decode_step(ok[1], ok[1], k, v, ok[0], 2)
        torch.cuda.synchronize()
        net.check_status()
    if message != "position":
        toks = torch.full((1, 32), 7, device="cuda")
        toks[0, 9] = token
        net.prefill(toks, k, v, bt)
        torch.cuda.synchronize()
        with pytest.raises(IndexError, match=message):
            net.check_status()


@pytest.mark.parametrize("model", ["tiny", "tiny_gpt2"])
def test_negative_indices_count_from_the_end(model, monkeypatch):
    """As in the general route: tokens, pages and positions; the pages written are the same."""
    from fuselink_b200.models.llama import LlamaShard
    net, pools = _shard(model)
    res = []
    for fused in (True, False):
        if not fused:
            monkeypatch.setattr(LlamaShard, "_fused", lambda self, pool: False)
        k, v = pools(6)
        toks = torch.arange(-48, 48, device="cuda").view(2, 48)
        net.prefill(toks, k, v, torch.tensor([[0, -1, 2], [-3, 1, 4]], device="cuda"))
        kd, vd = pools(6)
        net.decode_step(torch.tensor([-1, 2, 3], device="cuda"), torch.tensor([-1, -20, 7], device="cuda"), kd, vd,
                        torch.tensor([[0, 1], [2, 3], [-2, -1]], dtype=torch.int32, device="cuda"), 6)
        torch.cuda.synchronize()
        net.check_status()
        n = kd.numel() // net.cfg.layers                                      # the first layer: not yet behind an attention over nothing
        res.append((k, v, kd[:n], vd[:n]))
    for a, b in zip(*res):
        assert torch.equal(a != 0, b != 0)
        assert (a.float() - b.float()).norm() <= 4 * _eps(torch.bfloat16) * b.float().norm()


@pytest.mark.parametrize("bs", [16, 8])
def test_attention_leaves_out_a_page_outside_the_pool(bs):
    from fuselink_b200 import C
    heads, kv_heads, dim, n, maxblk = 4, 2, 64, 300, 300 // bs + 1
    kp, vp = (_rand(1, maxblk, bs, kv_heads, dim, dt=torch.bfloat16, seed=s) for s in (1, 2))
    bt = torch.randperm(maxblk, generator=torch.Generator().manual_seed(3)).view(1, maxblk).int().cuda()
    bad = bt.clone()
    bad[0, 3], bad[0, 7] = maxblk, -maxblk - 1
    qkv = _rand(1, (heads + 2 * kv_heads) * dim, dt=torch.bfloat16, seed=4)
    out, status = torch.empty(1, heads * dim, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    C.dec_attention(qkv, torch.tensor([n - 1], device="cuda"), kp, vp, bad, 0, 1, maxblk, bs, heads, kv_heads, dim, out, status.data_ptr())
    assert status.item() == 3
    keep = torch.arange(n, device="cuda")
    keep = keep[(keep // bs != 3) & (keep // bs != 7)]
    k, v = (p[0][bt[0].long()].reshape(-1, kv_heads, dim)[keep].float().repeat_interleave(2, 1) for p in (kp, vp))
    q = qkv[0, : heads * dim].view(heads, dim).float()
    want = torch.einsum("hn,nhd->hd", (torch.einsum("hd,nhd->hn", q, k) / math.sqrt(dim)).softmax(-1), v).reshape(-1)
    # the probabilities' rounding to the type and the result's
    assert (out[0].float() - want).abs().max() <= 2 * _eps(torch.bfloat16) * v.abs().max() + 1e-5


def test_a_first_call_under_capture_notes_what_it_meets():
    net, pools = _shard("tiny")
    k, v = pools(2)
    tok, at = torch.tensor([3], device="cuda"), torch.tensor([5], device="cuda")
    bt = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        net.decode_step(tok, at, k, v, bt, 2)
    for t, bad in ((3, False), (1000, True), (4, False)):
        tok.fill_(t)
        g.replay()
        torch.cuda.synchronize()
        if bad:
            with pytest.raises(IndexError, match="token"):
                net.check_status()
        else:
            net.check_status()


@pytest.mark.parametrize("batch", [1, 16, 17])
def test_a_gated_layer_knows_no_bias(batch):
    """A llama shard's b13 is looked at by no route: neither refused nor added."""
    net, pools = _shard("tiny")
    bt = torch.arange(2 * batch, dtype=torch.int32, device="cuda").view(batch, 2)
    tok, at = torch.arange(batch, device="cuda"), torch.full((batch,), 5, device="cuda")
    res = []
    for bias in (None, torch.ones(net.f_local, dtype=torch.bfloat16, device="cuda")):
        net.b13 = [bias] * net.cfg.layers
        k, v = pools(2 * batch)
        assert net._fused(k)
        res.append((net.decode_step(tok, at, k, v, bt, 2 * batch), k, v))
    for a, b in zip(*res):
        assert torch.equal(a, b)


def _ring(batch, heads, kv_heads, dim, bs, maxblk):
    """(CTAs per context, warps per CTA) of the attention through the ring, None where the pages go through registers: the rule of
    fl_dec_attention, so that the cases below reach what they are for."""
    units, cap = batch * kv_heads * -(-(heads // kv_heads) // 8), maxblk * bs
    if dim not in (64, 128) or bs % 16 or units * (cap // 16) < 3 * 8 * 148:
        return None
    splits = max(1, min(2 * 148 // units, -(-cap // 128), 8))
    return splits, 8 if units * splits <= 148 and cap >= splits * 8 * 32 else 4


def _check(out, q, k, v, dt):
    """out against the attention of q [heads, dim] over k, v [n, kv_heads, dim], both in fp32 from here on.  Scores are summed up product
    by product: in a library's matrix product an infinite key may become NaN by inf - inf."""
    (n, kv_heads, dim), heads = k.shape, q.shape[0]
    q, k, v = q.float().view(kv_heads, heads // kv_heads, dim), k.float(), v.float()
    s = torch.stack([(q[:, i].unsqueeze(0) * k).sum(-1).t() for i in range(q.shape[1])], 1)            # [kv_heads, group, n]
    p = (s / math.sqrt(dim)).softmax(-1)
    want, size = (torch.einsum("kgn,nkd->kgd", p, t).reshape(-1) for t in (v, v.abs()))
    got, fine = out.float(), ~want.isnan()
    assert torch.equal(got.isnan(), want.isnan())
    # The probabilities are rounded to the type before the second product, and so is the result; 1e-4: scores up to about 30 summed in
    # fp32 in another order, and the exponentials; in fp16 a probability below 2^-14 loses up to half a step of 2^-24.
    bound = (1.01 * _eps(dt) + 1e-4) * size + _eps(dt) * want.abs() + (n * 2.0 ** -25 * v.abs().mean() if dt == torch.float16 else 0) + 1e-6
    assert ((got - want).abs() <= bound)[fine].all(), ((got - want).abs() / bound)[fine].max()
    return want


def _of(pool, pages, n, bad=()):
    """The first n tokens of `pages` of a pool [blocks, bs, kv_heads, dim], without those of the pages in `bad`."""
    keep = torch.arange(n, device="cuda")
    for p in bad:
        keep = keep[keep // pool.shape[1] != p]
    return pool[pages.long() % pool.shape[0]].flatten(0, 1)[keep]


def _queries(batch, heads, kv_heads, dim, dt):
    """(qkv, keys [batch, kv_heads, dim]): queries of three times the usual size, so that a head looks at a few tokens and not at the mean
    of all; and for each KV head a key that its queries give about the weight of the best of some thousand others."""
    qkv = _rand(batch, (heads + 2 * kv_heads) * dim, dt=dt, seed=4)
    q = qkv[:, : heads * dim].view(batch, kv_heads, heads // kv_heads, dim)
    key = (0.33 * q.float().sum(2)).to(dt)
    q *= 3
    return qkv, key


RING = [  # batch, heads, kv_heads, dim, bs, lens (the first one fills the table), what the rule says
    (16, 32, 8, 128, 16, [2064 - 67 * i for i in range(16)], (2, 4)),           # the context cut over two CTAs, an early launch
    (17, 8, 8, 128, 16, [512, 1, 15, 16, 17, 33] + [300 + i for i in range(11)], (2, 4)),      # no early launch
    (40, 16, 8, 128, 16, [400 - 3 * i for i in range(40)], (1, 4)),
    (1, 32, 8, 128, 16, [7312], (8, 8)), (1, 8, 8, 128, 32, [7297], (8, 8)),
    (16, 24, 2, 128, 48, [960 - 50 * i for i in range(16)], (4, 4)),            # twelve heads per KV head: two parts; three steps per page
    (4, 32, 32, 64, 16, [1008, 17, 500, 999], (2, 4)), (2, 16, 8, 64, 64, [3648, 3], (8, 8)), (30, 8, 8, 64, 16, [256] * 30, (1, 4)),
    (1, 4, 1, 64, 16, [57000], (8, 8)), (1, 2, 1, 128, 16, [56900], (8, 8)),    # more than 32 steps per warp: its page ids a second time
    (16, 32, 8, 128, 16, [448 - 13 * i for i in range(16)], (2, 4)), (16, 32, 8, 128, 16, [432 - 13 * i for i in range(16)], None),      # the line
]


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("batch,heads,kv_heads,dim,bs,lens,how", RING)
def test_attention_through_the_ring(dt, batch, heads, kv_heads, dim, bs, lens, how):
    """Against the same in fp32.  What the pages hold behind a context may be anything: here NaN."""
    from fuselink_b200 import C
    L, layer, maxblk = 2, 1, -(-lens[0] // bs)
    nb = batch * maxblk
    assert _ring(batch, heads, kv_heads, dim, bs, maxblk) == how
    kp, vp = (_rand(L, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    qkv, key = _queries(batch, heads, kv_heads, dim, dt)
    for b, n in enumerate(lens):
        for tok in (0, n // 2, n - 1):
            kp[layer, bt[b, tok // bs].long(), tok % bs] = key[b]
        behind = torch.arange(n, maxblk * bs, device="cuda")
        for p in (kp, vp):
            p[layer, bt[b, behind // bs].long(), behind % bs] = float("nan")
    bt[:, ::3] -= nb                                                # negative ids count from the end
    pos = torch.tensor(lens, device="cuda") - 1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.full((batch, heads * dim), float("nan"), dtype=dt, device="cuda")
    C.dec_attention(qkv, pos, kp, vp, bt, layer, L, nb, bs, heads, kv_heads, dim, out, status.data_ptr())
    assert status.item() == 0
    for b, n in enumerate(lens):
        _check(out[b], qkv[b, : heads * dim].view(heads, dim), _of(kp[layer], bt[b], n), _of(vp[layer], bt[b], n), dt)


@pytest.mark.parametrize("batch,kv_heads,dim,n,how", [(16, 8, 128, 2064, (2, 4)), (1, 8, 128, 7312, (8, 8)), (4, 32, 64, 1008, (2, 4)), (30, 8, 64, 256, (1, 4))])
def test_the_ring_leaves_out_a_page_outside_the_pool(batch, kv_heads, dim, n, how):
    from fuselink_b200 import C
    bs, heads, dt, maxblk = 16, 2 * kv_heads, torch.bfloat16, n // 16
    nb = batch * maxblk
    assert _ring(batch, heads, kv_heads, dim, bs, maxblk) == how
    kp, vp = (_rand(1, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    outside = {0: nb, 5: -nb - 1, 6: 2 ** 31 - 1, maxblk - 1: -2 ** 31}
    for p, value in outside.items():
        bt[batch - 1, p] = value
    (qkv, _), pos = _queries(batch, heads, kv_heads, dim, dt), torch.full((batch,), n - 1, device="cuda")
    out, status = torch.empty(batch, heads * dim, dtype=dt, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    C.dec_attention(qkv, pos, kp, vp, bt, 0, 1, nb, bs, heads, kv_heads, dim, out, status.data_ptr())
    assert status.item() == 3
    for b in {0, batch - 1}:
        k, v = (_of(p[0], bt[b], n, outside if b == batch - 1 else ()) for p in (kp, vp))
        _check(out[b], qkv[b, : heads * dim].view(heads, dim), k, v, dt)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("batch,kv_heads,dim,n,how", [(16, 8, 128, 2049, (2, 4)), (1, 8, 128, 7300, (8, 8)), (4, 32, 64, 1000, (2, 4))])
@pytest.mark.parametrize("value,where", [(float("nan"), "first"), (float("nan"), "last"), (float("inf"), "middle"), (float("-inf"), "first"), (float("-inf"), "last"),
                                         (float("-inf"), "all")])
def test_the_ring_passes_on_what_is_not_finite(dt, batch, kv_heads, dim, n, how, value, where):
    """As through registers: NaN and infinite scores make the head NaN, those of -inf weigh nothing; other heads and requests as without."""
    from fuselink_b200 import C
    bs, heads, maxblk = 16, 2 * kv_heads, -(-n // 16)
    nb = batch * maxblk
    assert _ring(batch, heads, kv_heads, dim, bs, maxblk) == how
    kp, vp = (_rand(1, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    qkv = _rand(batch, (heads + 2 * kv_heads) * dim, dt=dt, seed=4)
    qkv[:, 0:heads * dim:dim] = 1                                   # every query's first column: the score gets the key's infinity
    at = {"first": torch.arange(16), "middle": torch.tensor([n // 2]), "last": torch.arange((n - 1) // 16 * 16, n), "all": torch.arange(n)}[where].cuda()
    kp[0, bt[0, at // bs].long(), at % bs, 1, 0] = value
    out = torch.empty(batch, heads * dim, dtype=dt, device="cuda")
    C.dec_attention(qkv, torch.full((batch,), n - 1, device="cuda"), kp, vp, bt, 0, 1, nb, bs, heads, kv_heads, dim, out)
    for b in {0, batch - 1}:
        want = _check(out[b], qkv[b, : heads * dim].view(heads, dim), _of(kp[0], bt[b], n), _of(vp[0], bt[b], n), dt)
        if b == 0:
            assert want.view(heads, dim)[2:4].isnan().all() == (value != float("-inf") or where == "all")


@pytest.mark.parametrize("batch,heads,kv_heads,dim,n", [(16, 32, 8, 128, 2047), (1, 8, 8, 128, 7311), (4, 32, 32, 64, 1007), (3, 4, 4, 64, 389), (17, 8, 8, 128, 511)])
def test_the_chain_attends_to_the_token_that_was_just_written(batch, heads, kv_heads, dim, n):
    """Page write and attention, launched one behind the other as a step does, through several layers and steps without a wait in
    between: every attention sees its own step's keys and values, which weigh more than all others together."""
    from fuselink_b200 import C
    L, bs, steps, dt = 6, 16, 2, torch.bfloat16
    maxblk = (n + steps) // bs + 1
    nb = batch * maxblk
    kp, vp = (_rand(L, nb, bs, kv_heads, dim, dt=dt, seed=s) for s in (1, 2))
    k0, v0 = kp.clone(), vp.clone()
    bt = torch.randperm(nb, generator=torch.Generator().manual_seed(3)).view(batch, maxblk).int().cuda()
    qkv = [[_rand(batch, (heads + 2 * kv_heads) * dim, dt=dt, seed=100 * s + l) for l in range(L)] for s in range(steps)]
    for x in sum(qkv, []):
        x = x.view(batch, heads + 2 * kv_heads, dim)
        x[:, heads:heads + kv_heads] = x[:, :heads].float().view(batch, kv_heads, -1, dim).sum(2).to(dt)
    outs = [[torch.empty(batch, heads * dim, dtype=dt, device="cuda") for _ in range(L)] for _ in range(steps)]
    pos = [torch.full((batch,), n + s, device="cuda") for s in range(steps)]
    torch.cuda.synchronize()
    for s in range(steps):
        for l in range(L):
            C.dec_qkv(qkv[s][l], None, None, pos[s], 1, kp, vp, bt, 1, l, L, nb, bs, heads, kv_heads, dim)
            C.dec_attention(qkv[s][l], pos[s], kp, vp, bt, l, L, nb, bs, heads, kv_heads, dim, outs[s][l])
    for s in range(steps):
        for l in range(L):
            new = qkv[s][l].view(batch, -1, dim)
            for b in range(batch):
                page, slot = bt[b, (n + s) // bs].long(), (n + s) % bs
                k0[l, page, slot], v0[l, page, slot] = new[b, heads:heads + kv_heads], new[b, heads + kv_heads:]
            for b in {0, batch - 1}:
                _check(outs[s][l][b], new[b, :heads], _of(k0[l], bt[b], n + s + 1), _of(v0[l], bt[b], n + s + 1), dt)
    assert torch.equal(kp, k0) and torch.equal(vp, v0)
