"""Block-scaled fp8 grouped GEMM: quantisers against their PyTorch restatement, and the GEMM against an fp32 matmul of
the DEQUANTISED operands (so the check isolates the kernel from the quantisation error)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mk(shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _close(got, ref, tol=1.5e-2):
    if ref.numel() == 0:
        return
    err = (got.float() - ref).abs().max().item()
    den = ref.abs().max().item() + 1e-6
    assert err / den < tol, f"max abs err {err} vs ref max {den}"


def test_quantizers_match_reference():
    from fuselink_b200.ops import fp8
    x = _mk([300, 512], 3.0, seed=1)
    x[7] = 0
    q, s = fp8.quantize_rows(x)
    rq, rs = fp8.ref_quantize_rows(x)
    torch.testing.assert_close(s, rs, rtol=1e-6, atol=0)
    assert (q.float() - rq.float()).abs().max() <= 32            # at most one e4m3 step at the top of the range
    back = fp8.dequantize_rows(q, s)
    assert (back - x.float()).abs().max() <= 0.07 * x.float().abs().max()
    w = _mk([2, 256, 384], 0.05, seed=2)
    wq, ws = fp8.quantize_blocks(w)
    assert ws.shape == (2, 2, 3)
    wb = fp8.dequantize_blocks(wq, ws)
    assert (wb - w.float()).abs().max() <= 0.07 * w.float().abs().max()
    amax = w.float().view(2, 2, 128, 3, 128).abs().amax((2, 4))
    torch.testing.assert_close(ws, amax / 448.0, rtol=1e-6, atol=0)


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("K", [128, 512])
def test_fp8_rows_store(K, b_mn):
    from fuselink_b200.ops import fp8
    G, cap, N = 3, 256, 512
    counts_l = [200, 0, 129]
    counts = torch.tensor(counts_l, dtype=torch.int32, device="cuda")
    a = _mk([G * cap, K], 2.0, seed=3)
    w = _mk([G, N, K], 0.1, seed=4)
    aq, asc = fp8.quantize_rows(a)
    if b_mn:
        wq, wsc = fp8.quantize_blocks(w.transpose(1, 2).contiguous())       # stored [G, K, N]
        wd = fp8.dequantize_blocks(wq, wsc).transpose(1, 2)
    else:
        wq, wsc = fp8.quantize_blocks(w)
        wd = fp8.dequantize_blocks(wq, wsc)
    ad = fp8.dequantize_rows(aq, asc)
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    out = torch.full((G * cap, N), 7.0, dtype=torch.bfloat16, device="cuda")
    fp8.grouped_gemm_rows_fp8(aq, asc, wq, wsc, counts, cap, b_mn_major=b_mn, out=out, zero_tail=True, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0, st.tolist()
    for g, c in enumerate(counts_l):
        _close(out[g * cap:g * cap + c], ad[g * cap:g * cap + c] @ wd[g].t())
        end = min((c + 127) // 128 * 128, cap)
        assert (out[g * cap + c:g * cap + end] == 0).all()
        assert (out[g * cap + end:(g + 1) * cap] == 7.0).all()


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("blocks", [7, 8, 9, 16, 17])
def test_fp8_scales_through_their_ring(blocks, b_mn):
    """The scales travel eight blocks of contraction at a time, in two stages: one block less, as many, one more, over several tiles
    per CTA (two CTAs), rows that end inside a tile and an expert without rows.  Scales differ by powers of two from block to block, so that
    one taken from the wrong block or row shows."""
    from fuselink_b200.ops import fp8
    G, cap, N, K = 3, 384, 768, 128 * blocks
    counts_l = [383, 0, 130]
    counts = torch.tensor(counts_l, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(blocks)
    aq = torch.randint(-8, 9, (G * cap, K), generator=g, device="cuda").float().to(fp8.FP8)
    wq = torch.randint(-8, 9, (G, K, N) if b_mn else (G, N, K), generator=g, device="cuda").float().to(fp8.FP8)
    asc = 2.0 ** torch.randint(-3, 4, (G * cap, blocks), generator=g, device="cuda").float()
    wsc = 2.0 ** torch.randint(-3, 4, (G, wq.shape[1] // 128, wq.shape[2] // 128), generator=g, device="cuda").float()
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    out = fp8.grouped_gemm_rows_fp8(aq, asc, wq, wsc, counts, cap, b_mn_major=b_mn, max_ctas=2, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0, st.tolist()
    ad, wd = fp8.dequantize_rows(aq, asc).double(), fp8.dequantize_blocks(wq, wsc).double()
    for i, c in enumerate(counts_l):
        ref = ad[i * cap:i * cap + c] @ (wd[i] if b_mn else wd[i].t())
        # products of small integers and powers of two: sums exact in fp32, the results rounded to bf16 once (2^-9)
        assert ((out[i * cap:i * cap + c].double() - ref).abs() <= ref.abs() * 2.0 ** -8).all()


def test_fp8_swiglu_scatter_and_dswiglu():
    import torch.nn.functional as F
    from fuselink_b200.ops import fp8, gemm
    G, cap, H, Fd = 2, 256, 256, 512
    counts_l = [256, 77]
    counts = torch.tensor(counts_l, dtype=torch.int32, device="cuda")
    x = _mk([G * cap, H], seed=5)
    w13 = gemm.interleave_gate_up(_mk([G, Fd, H], 0.1, seed=6), _mk([G, Fd, H], 0.1, seed=7))
    xq, xs = fp8.quantize_rows(x)
    wq, ws = fp8.quantize_blocks(w13)
    xd, wd = fp8.dequantize_rows(xq, xs), fp8.dequantize_blocks(wq, ws)
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    gu = torch.empty(G * cap, 2 * Fd, dtype=torch.bfloat16, device="cuda")
    act = fp8.grouped_gemm_rows_fp8(xq, xs, wq, ws, counts, cap, epilogue=fp8.EPI_SWIGLU, gu=gu, zero_tail=True, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0
    for g, c in enumerate(counts_l):
        h = xd[g * cap:g * cap + c] @ wd[g].t()
        gate, up = gemm.deinterleave_gate_up(h.t().contiguous().unsqueeze(0))
        gate, up = gate[0].t(), up[0].t()
        _close(act[g * cap:g * cap + c], F.silu(gate) * up)
        gg, uu = gemm.deinterleave_gate_up(gu[g * cap:g * cap + c].t().contiguous().unsqueeze(0))
        _close(gg[0].t(), gate)
        _close(uu[0].t(), up)
    # second GEMM with the scatter epilogue
    w2 = _mk([G, H, Fd], 0.1, seed=8)
    aq, asc = fp8.quantize_rows(act)
    w2q, w2s = fp8.quantize_blocks(w2)
    dst = torch.zeros(G * cap, H, dtype=torch.bfloat16, device="cuda")
    info = torch.randperm(G * cap, device="cuda").int()
    fp8.grouped_gemm_rows_fp8(aq, asc, w2q, w2s, counts, cap, epilogue=fp8.EPI_SCATTER, row_info=info, peers=[dst.data_ptr()],
                              ldc=H, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0
    ad, w2d = fp8.dequantize_rows(aq, asc), fp8.dequantize_blocks(w2q, w2s)
    for g, c in enumerate(counts_l):
        ref = ad[g * cap:g * cap + c] @ w2d[g].t()
        _close(dst[info[g * cap:g * cap + c].long()], ref)
    # backward of the activation: dAct = dY @ W2 (B MN-major), DSWIGLU epilogue
    dy = _mk([G * cap, H], seed=9)
    dyq, dys = fp8.quantize_rows(dy)
    dgu = torch.zeros_like(gu)
    fp8.grouped_gemm_rows_fp8(dyq, dys, w2q, w2s, counts, cap, b_mn_major=True, epilogue=fp8.EPI_DSWIGLU, gu=gu, dgu=dgu,
                              zero_tail=True, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0
    dyd = fp8.dequantize_rows(dyq, dys)
    for g, c in enumerate(counts_l):
        da = dyd[g * cap:g * cap + c] @ w2d[g]
        gate, up = gemm.deinterleave_gate_up(gu[g * cap:g * cap + c].float().t().contiguous().unsqueeze(0))
        gate, up = gate[0].t(), up[0].t()
        sg = torch.sigmoid(gate)
        dg, du = gemm.deinterleave_gate_up(dgu[g * cap:g * cap + c].t().contiguous().unsqueeze(0))
        _close(dg[0].t(), da * up * (sg * (1 + gate * (1 - sg))), 2e-2)
        _close(du[0].t(), da * gate * sg, 2e-2)


def test_fp8_throughput_smoke():
    from fuselink_b200.ops import fp8
    cap, N, K = 8192, 4096, 4096
    aq, asc = fp8.quantize_rows(_mk([cap, K], seed=10))
    wq, wsc = fp8.quantize_blocks(_mk([1, N, K], 0.02, seed=11))
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    out = fp8.grouped_gemm_rows_fp8(aq, asc, wq, wsc, None, cap, status=st)
    torch.cuda.synchronize()
    assert st[0].item() == 0
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(10):
        fp8.grouped_gemm_rows_fp8(aq, asc, wq, wsc, None, cap, out=out, status=st)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / 10
    print(f"\n[fp8 gemm smoke] 8192x4096x4096 e4m3 1x128: {ms:.3f} ms  {2.0 * cap * N * K / ms / 1e9:.0f} TFLOP/s")


@pytest.mark.parametrize("K", [128, 384, 1024, 1152, 3072])            # one block, an odd number, whole and partial groups of eight
@pytest.mark.parametrize("cap,counts", [(0, None), (256, [0, 130, 256, 1]), (200, [7, 0, 200, 129]), (128, [0, 0, 0])])
@pytest.mark.parametrize("offset", [0, 4])                              # 4: addresses that are multiples of 8 bytes only
def test_row_quantizer_over_groups(K, cap, counts, offset):
    """Rows that hold tokens, up to a whole tile, and no others."""
    from fuselink_b200 import C
    from fuselink_b200.ops import fp8
    rows = cap * len(counts) if counts else 77
    x = _mk([rows * K + offset], 3.0, seed=K)[offset:].view(rows, K)
    x[0] = 0
    cnt = torch.tensor(counts, dtype=torch.int32, device="cuda") if counts else None
    q = torch.full((rows * K + offset,), 5, dtype=torch.uint8, device="cuda")[offset:].view(rows, K).view(fp8.FP8)
    s = torch.full((rows, K // 128), -1.0, device="cuda")
    C.fp8_quantize_rows(x, q, s, cnt, cap)
    used = torch.ones(rows, dtype=torch.bool, device="cuda")
    for g, n in enumerate(counts or []):
        used[g * cap + min((n + 127) // 128 * 128, cap):(g + 1) * cap] = False
    rq, rs = fp8.ref_quantize_rows(x)
    torch.testing.assert_close(s[used], rs[used], rtol=1e-6, atol=0)
    assert (q[used].float() - rq[used].float()).abs().max() <= 32 if used.any() else True
    assert (s[~used] == -1).all() and (q[~used].view(torch.uint8) == 5).all()


def test_block_quantizer_at_8_byte_addresses():
    from fuselink_b200.ops import fp8
    w = _mk([2 * 256 * 384 + 4], 0.05, seed=2)[4:].view(2, 256, 384)
    q, s = fp8.quantize_blocks(w)
    q0, s0 = fp8.quantize_blocks(w.clone())
    assert torch.equal(q.view(torch.uint8), q0.view(torch.uint8)) and torch.equal(s, s0)


def test_fp8_epilogues_at_gates_whose_sigmoid_is_subnormal():
    """1 + e^-g is beyond 2^126 below g = -87.3, where the hardware's fast quotient gives 0.  One product per sum, so gate, up and dAct are
    exact; what is left is the exponential (CUDA's bound for __expf at 88.6: 105 ulp, below 2^-16) and the rounding to bf16 (2^-8: eight bits)."""
    from fuselink_b200.ops import fp8, gemm
    cap, H, Fd = 256, 128, 256
    tol = 1.02 * 2.0 ** -8
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    first, second = (torch.zeros(1, Fd, H, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    first[:, :, 0], second[:, :, 1] = 1, 1                              # gate: the row's first value, up: its second
    w = gemm.interleave_gate_up(first, second).float().to(fp8.FP8)
    x = torch.zeros(cap, H, device="cuda")
    x[:, 0], x[:, 1] = -1, 4
    scale = torch.linspace(80, 88.6, cap, device="cuda").view(cap, 1)
    act = fp8.grouped_gemm_rows_fp8(x.to(fp8.FP8), scale, w, torch.ones(1, 2 * Fd // 128, 1, device="cuda"), None, cap, epilogue=fp8.EPI_SWIGLU,
                                    gu=torch.empty(cap, 2 * Fd, dtype=torch.bfloat16, device="cuda"), status=st)
    g, u = -scale.double(), 4 * scale.double()
    want = (g * torch.sigmoid(g) * u).expand(cap, Fd)
    assert ((act.double() - want).abs() <= tol * want.abs()).all()

    gate, up = scale.neg().to(torch.bfloat16).expand(cap, Fd), torch.full((cap, Fd), 4., dtype=torch.bfloat16, device="cuda")
    gu = gemm.interleave_gate_up(gate.t().unsqueeze(0), up.t().unsqueeze(0))[0].t().contiguous()
    dgu = torch.empty_like(gu)
    w2 = torch.zeros(1, H, Fd, device="cuda")
    w2[:, 0] = -1
    fp8.grouped_gemm_rows_fp8(x.to(fp8.FP8), torch.ones(cap, 1, device="cuda"), w2.to(fp8.FP8), torch.ones(1, 1, Fd // 128, device="cuda"), None, cap,
                              b_mn_major=True, epilogue=fp8.EPI_DSWIGLU, gu=gu, dgu=dgu, status=st)
    dg, du = (t[0].t().double() for t in gemm.deinterleave_gate_up(dgu.t().contiguous().unsqueeze(0)))
    g = gate.double()                                                   # dAct = 1
    sg = torch.sigmoid(g)
    assert (g >= -88.5).all()                                           # what -88.6 rounds to; e^89 is inf
    for got, want in ((du, g * sg), (dg, 4 * sg * (1 + g * (1 - sg)))):
        assert ((got - want).abs() <= tol * want.abs()).all()
    assert st[0].item() == 0
