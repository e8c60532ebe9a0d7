"""KV pack+send kernel and the disaggregated prefill -> decode path, both stages as virtual ranks on one GPU."""
import queue

import pytest
import torch

pytestmark = pytest.mark.gpu


def _setup(batch=3, input_len=64, steps=8, model="tiny"):
    from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
    from fuselink_b200.parallel.symm import SymmetricHeap
    from fuselink_b200.serving.disagg import KVLink, ServeParams
    p = ServeParams(model=MODEL_ZOO[model], batch_size=batch, input_len=input_len, num_decoding_step=steps)
    heaps = SymmetricHeap.emulated(2, 64 << 20)
    net = LlamaShard(p.model, device="cuda", seed=1)
    links = [KVLink(h, p, net.kvh_local) for h in heaps]
    return p, heaps, net, links


@pytest.mark.parametrize("same_layout", [False, True])
def test_kv_pack_send_matches_page_gather(same_layout):
    from fuselink_b200 import C
    from fuselink_b200.ops import ref
    L, H, S, D, B, maxb = 3, 2, 16, 64, 4, 5
    src_blocks, dst_blocks = 32, 40
    g = torch.Generator(device="cuda").manual_seed(0)
    page = H * S * D
    src_k = torch.randn(src_blocks * L * page, generator=g, device="cuda").to(torch.bfloat16)
    src_v = torch.randn(src_blocks * L * page, generator=g, device="cuda").to(torch.bfloat16)
    dst_k = torch.zeros(dst_blocks * L * page, dtype=torch.bfloat16, device="cuda")
    dst_v = torch.zeros_like(dst_k)
    nb = torch.tensor([5, 1, 0, 3], dtype=torch.int32, device="cuda")
    src_bt = torch.randperm(src_blocks, generator=torch.Generator().manual_seed(1))[:B * maxb].view(B, maxb).int().cuda()
    dst_bt = torch.randperm(dst_blocks, generator=torch.Generator().manual_seed(2))[:B * maxb].view(B, maxb).int().cuda()
    flag = torch.zeros(4, dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    hdr = torch.arange(10, dtype=torch.int64, device="cuda")
    hdr_dst = torch.zeros(10, dtype=torch.int64, device="cuda")
    dl = 0 if same_layout else 1
    for l0, l1, seq in [(0, 2, 1), (2, 3, 2)]:          # two launches: layers [0,2) then [2,3)
        C.kv_pack_send(src_k, src_v, dst_k.data_ptr(), dst_v.data_ptr(), 0, dl, src_blocks, dst_blocks, L, H, S, D, l0, l1,
                       src_bt, dst_bt, nb, hdr, hdr_dst.data_ptr(), flag.data_ptr(), seq, counter, 7, status.data_ptr())
    torch.cuda.synchronize()
    assert status[0].item() == 0 and flag[0].item() == 2 and counter.item() == 0
    assert torch.equal(hdr, hdr_dst)
    for src, dst in ((src_k, dst_k), (src_v, dst_v)):
        want = ref.kv_gather_pages(src, 0, src_bt.cpu(), nb.cpu(), L, H, S, D)
        got = ref.kv_gather_pages(dst, dl, dst_bt.cpu(), nb.cpu(), L, H, S, D)
        for w, g_ in zip(want, got):
            assert torch.equal(w, g_)
    # pages that were not addressed stay untouched
    used = set(int(dst_bt[b, j]) for b in range(B) for j in range(int(nb[b])))
    view = dst_k.view(L, dst_blocks, -1) if dl == 1 else dst_k.view(dst_blocks, L, -1).transpose(0, 1)
    for blk in range(dst_blocks):
        if blk not in used:
            assert (view[:, blk] == 0).all()


def test_kv_bad_block_id_is_reported_and_skipped():
    from fuselink_b200 import C
    L, H, S, D = 1, 1, 16, 64
    src = torch.ones(4 * L * H * S * D, dtype=torch.bfloat16, device="cuda")
    dst = torch.zeros(4 * L * H * S * D, dtype=torch.bfloat16, device="cuda")
    bt = torch.tensor([[0, 9]], dtype=torch.int32, device="cuda")           # 9 is outside the 4-page pools
    nb = torch.tensor([2], dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    counter = torch.zeros(1, dtype=torch.int32, device="cuda")
    C.kv_pack_send(src, src, dst.data_ptr(), dst.data_ptr(), 0, 0, 4, 4, L, H, S, D, 0, 1, bt, bt, nb, None, 0, 0, 1, counter, 2,
                   status.data_ptr())
    torch.cuda.synchronize()
    assert status[0].item() == 6                                              # kBadIndex: recorded, access skipped
    assert (dst.view(4, -1)[0] == 1).all() and (dst.view(4, -1)[1:] == 0).all()


@pytest.mark.parametrize("pipeline", [True, False])
def test_offline_prefill_to_decode_matches_dense_model(pipeline):
    from fuselink_b200.serving.disagg import DecodeStage, PrefillStage, make_prompts
    p, heaps, net, links = _setup()
    try:
        pre = PrefillStage(p, net, links[0], dst_rank=1, pipeline_layers=pipeline)
        dec = DecodeStage(p, net, links[1])
        prompts = make_prompts(p, "cuda", seed=3)
        rp = pre.run(prompts)
        rd = dec.run()
        for h in heaps:
            h.check_status()
        gen = rd.extra["generated"]                                           # [B, 1 + steps]
        assert gen.shape == (p.batch_size, 1 + p.num_decoding_step)
        # oracle: greedy decoding with the un-paged model, recomputing the full sequence each step
        seq = prompts.clone()
        for t in range(1 + p.num_decoding_step):
            nxt = net.forward_dense(seq).argmax(-1)
            agree = (nxt == gen[:, t]).float().mean().item()
            assert agree == 1.0, f"token {t}: paged path disagrees with the dense model ({agree:.2f})"
            seq = torch.cat([seq, gen[:, t:t + 1]], 1)
        assert rp.kv_bytes == 2 * p.batch_size * p.context_blocks_per_req * p.model.layers * links[0].page_elems * 2
        assert rp.kv_ms > 0 and rd.tokens == p.batch_size * p.num_decoding_step
    finally:
        for h in heaps:
            h.close()


def test_online_trace_batches_with_pool_credits():
    from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
    from fuselink_b200.parallel.symm import SymmetricHeap
    from fuselink_b200.serving.disagg import KVLink, ServeParams
    from fuselink_b200.serving.online import OnlineDecode, OnlinePrefill, TraceReader, next_batch, parse_trace
    p = ServeParams(model=MODEL_ZOO["tiny"], batch_size=20, input_len=96, num_decoding_step=4)
    heaps = SymmetricHeap.emulated(2, 96 << 20)
    try:
        net = LlamaShard(p.model, device="cuda", seed=1)
        links = [[KVLink(h, p, net.kvh_local, name=f"kv{i}") for i in range(2)] for h in heaps]
        pre = OnlinePrefill(p, net, links[0], dst_rank=1)
        dec = OnlineDecode(p, net, links[1], src_rank=0)
        trace = [f"ts: {0.001 * i:.3f} prompt: {40 + 7 * (i % 9)} shared: {3 * (i % 4)} out: {5 + i % 3}" for i in range(30)]
        trace.append("ts: 0.030 prompt: 5000 shared: 0 out: 4")               # longer than input_len: must be dropped, not spin
        reqs = parse_trace(trace)
        assert len(reqs) == 31 and reqs[1].active_prompt_len == 47 - 3
        q = queue.Queue()
        TraceReader(reqs, q, time_scale=1.0).start()
        warnings, served, finished = [], 0, False
        while not finished:
            batch, finished = next_batch(q, 20, p.input_len, warnings.append)
            if not batch:
                continue
            st = pre.serve_batch(batch)
            out = dec.serve_batch(max_steps=3)
            assert out["batch"] == len(batch) == st.batch
            assert out["generated"].shape == (len(batch), 4)
            bs = p.model.block_size
            want_pages = sum((r.active_prompt_len + bs - 1) // bs for r in batch)
            assert st.kv_bytes == want_pages * p.model.layers * links[0][0].page_elems * 4   # padding is never sent
            served += len(batch)
        assert served == 30 and len(warnings) == 1
        assert pre.batches >= 2                                               # pools were reused through the credit word
        for h in heaps:
            h.check_status()
    finally:
        for h in heaps:
            h.close()


@pytest.mark.parametrize("H,S,D,layout", [(1, 1, 8, 1), (3, 5, 24, 1), (12, 16, 64, 1), (64, 64, 128, 1), (7, 16, 128, 0)])
@pytest.mark.parametrize("batch", [1, 37, 1500])                       # the last: more requests than the table of totals holds
def test_kv_pack_send_over_page_shapes(H, S, D, layout, batch):
    """Odd head counts and page sizes, pages of 2^16 vectors and more, empty requests; every page lands, nothing else moves."""
    from fuselink_b200 import C
    L, maxb = 2, 3
    if H * S * D * batch > 1 << 24:
        batch = 5
    g = torch.Generator().manual_seed(batch)
    nb = torch.randint(0, maxb + 1, (batch,), generator=g).int()
    nb[0] = maxb
    n = batch * maxb
    src = [torch.randn(n, L, H, S, D, generator=g).to(torch.bfloat16).cuda() for _ in range(2)]
    shape = (n, L, H, S, D) if layout == 0 else (L, n, S, H, D)
    dst = [torch.full(shape, -7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    sbt, dbt = (torch.randperm(n, generator=g).view(batch, maxb).int().cuda() for _ in range(2))
    status, counter = torch.zeros(8, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    C.kv_pack_send(src[0], src[1], dst[0].data_ptr(), dst[1].data_ptr(), 0, layout, n, n, L, H, S, D, 1, 2, sbt, dbt, nb.cuda(),
                   None, 0, 0, 1, counter, 0, status.data_ptr())
    mask = torch.arange(maxb).unsqueeze(0) < nb.unsqueeze(1)
    si, di = sbt.cpu()[mask].long().cuda(), dbt.cpu()[mask].long().cuda()
    for s, d in zip(src, dst):
        want = torch.full_like(d, -7.0)
        if layout == 0:
            want[di, 1] = s[si, 1]
        else:
            want[1, di] = s[si, 1].transpose(1, 2)
        assert torch.equal(d, want)
    assert not status.any()


@pytest.mark.parametrize("input_len,steps", [(64, 8), (64, 3), (64, 0), (32, 8), (32, 20), (71, 9)])
def test_decode_stage_follows_its_parameters_after_the_capture(input_len, steps):
    """Shorter, longer and empty runs from other positions on a stage whose step has been captured: tokens as of an eager stage."""
    from fuselink_b200.models.llama import MODEL_ZOO, LlamaShard
    from fuselink_b200.parallel.symm import SymmetricHeap
    from fuselink_b200.serving.disagg import DecodeStage, KVLink, ServeParams
    p = ServeParams(model=MODEL_ZOO["tiny"], batch_size=3, input_len=64, num_decoding_step=8)
    heap, = SymmetricHeap.emulated(1, 32 << 20)
    try:
        net = LlamaShard(p.model, device="cuda", seed=1)
        net.lm_head = net.embed.roll(1, 0).clone()                      # next tokens that win by a margin
        net.embed.mul_(50)
        link = KVLink(heap, p, net.kvh_local)
        for pool in (link.k_pool.local, link.v_pool.local):
            pool.normal_(generator=torch.Generator(device="cuda").manual_seed(1))
        stages = [DecodeStage(p, net, link, use_graph=g) for g in (True, False)]
        first = torch.tensor([5, 900, 31], device="cuda")
        stages[0].decode(first)
        assert stages[0].graph is not None
        p.input_len, p.num_decoding_step = input_len, steps
        got, want = (s.decode(first + 1)[0] for s in stages)
        assert got.shape == (3, 1 + steps) and torch.equal(got, want)
    finally:
        heap.close()


# (9, 16, 128) ends in one head of a unit of eight, (32, 32, 256) are units of two heads, (16, 16, 32) is the smallest unit and (15, 16, 32) one
# of the other kernel's, (1, 64, 128) is one head, (300, 1, 32) a box of 256 heads; on both sides of 16 MiB of pages
@pytest.mark.parametrize("H,S,D,layout", [(9, 16, 128, 1), (32, 32, 256, 1), (16, 16, 32, 1), (15, 16, 32, 1), (1, 64, 128, 1), (300, 1, 32, 1), (9, 16, 128, 0)])
@pytest.mark.parametrize("more", [-1, 1, 20])
def test_kv_pack_send_through_the_copy_engine(H, S, D, layout, more):
    least = -(-(16 << 20) // (2 * 3 * H * S * D * 2))               # requests of three pages, keys and values
    test_kv_pack_send_over_page_shapes(H, S, D, layout, least + more)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("ctas", [3, 0])
@pytest.mark.parametrize("hdr_bytes,shift", [(8192 + 8, 0), (8192, 8), (8, 0)])     # whole vectors and a rest; not at 16 bytes; less than a vector
def test_kv_hand_off_through_the_copy_engine(layout, ctas, hdr_bytes, shift):
    """What test_kv_pack_send_matches_page_gather checks and ids outside their pools, above 16 MiB: two launches on one counter with header
    and flag, by a few CTAs (many units each) and by all; only the valid pages move, the others are reported."""
    from fuselink_b200 import C
    L, H, S, D, B, maxb = 4, 8, 16, 128, 40, 5                           # a unit is a page of 32 KiB; two layers hold 25 MiB
    n = B * maxb
    g = torch.Generator().manual_seed(ctas)
    src = [torch.randint(-32768, 32768, (n, L, H, S, D), generator=g, dtype=torch.int16).cuda().view(torch.bfloat16) for _ in range(2)]
    shape = (n, L, H, S, D) if layout == 0 else (L, n, S, H, D)
    dst = [torch.full(shape, -7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    nb = torch.randint(0, maxb + 1, (B,), generator=g).int()
    nb[0], nb[7], nb[B - 1] = maxb, 0, maxb
    sbt, dbt = (torch.randperm(n, generator=g).view(B, maxb).int() for _ in range(2))
    valid = torch.arange(maxb).unsqueeze(0) < nb.unsqueeze(1)
    for table, b, j, bad in ((sbt, 0, 1, n), (sbt, B - 1, 4, -1), (dbt, 0, 0, n + 5), (dbt, B - 1, 2, -2 ** 31), (dbt, 0, 4, 2 ** 31 - 1)):
        table[b, j] = bad
        valid[b, j] = False
    status, counter, flag = torch.zeros(8, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    hdr = torch.randint(0, 256, (hdr_bytes + shift,), generator=g, dtype=torch.uint8).cuda()[shift:]
    hdr_dst = torch.zeros(hdr_bytes + 32, dtype=torch.uint8, device="cuda")
    tables = sbt.cuda(), dbt.cuda(), nb.cuda()
    for l0, l1, seq in [(0, 2, 1), (2, 4, 2)]:
        C.kv_pack_send(src[0], src[1], dst[0].data_ptr(), dst[1].data_ptr(), 0, layout, n, n, L, H, S, D, l0, l1, *tables,
                       hdr if seq == 2 else None, hdr_dst.data_ptr() if seq == 2 else 0, flag.data_ptr(), seq, counter, ctas, status.data_ptr())
        assert flag[0].item() == seq and counter.item() == 0
    assert status[0].item() == 6                                         # kBadIndex: recorded, access skipped
    assert torch.equal(hdr_dst[:hdr_bytes], hdr) and (hdr_dst[hdr_bytes:] == 0).all() and (flag[1:] == 0).all()
    si, di = sbt[valid].long().cuda(), dbt[valid].long().cuda()
    for s, d in zip(src, dst):
        want = torch.full_like(d, -7.0)
        if layout == 0:
            want[di] = s[si]
        else:
            want[:, di] = s[si].permute(1, 0, 3, 2, 4)
        assert torch.equal(d.view(torch.int16), want.view(torch.int16))
