"""Tiles chosen by the rows that a group is expected to have (FlGemmDesc::expect_rows): the choice changes no result, whatever the rows
that the groups then have."""
import pytest
import torch

pytestmark = pytest.mark.gpu

G, CAP = 3, 1280
EXPECT = [0, 1, 125, 250, 447, 448, 1023, 1024, 2 ** 31 - 1]       # both sides of every line of the rule


@pytest.fixture(autouse=True)
def _automatic():
    from fuselink_b200 import C
    before = C.gemm_get_variant()
    yield
    C.gemm_set_variant(before)


def _mk(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _outcomes(launch):
    """launch(expect_rows) under every expectation and under each of the three variants by itself."""
    from fuselink_b200 import C
    C.gemm_set_variant(3)
    res = {("rows", e): launch(e) for e in EXPECT}
    for v in (0, 1, 2):
        C.gemm_set_variant(v)
        res["variant", v] = launch(250)
    return res


def _same(launch):
    """...are the same bits; returns them."""
    res = _outcomes(launch)
    first = res["rows", 0]
    for how, outs in res.items():
        for a, b in zip(first, outs):
            assert torch.equal(a, b), how
    return first


def _close(got, want, tol=2e-2):
    assert (got.float() - want).abs().max() <= tol * want.abs().max()


# the fullest and the emptiest that a group may be, edges of the tiles of 128 and 256 rows
@pytest.mark.parametrize("counts_l", [[1280, 0, 1], [128, 129, 256], [257, 1000, 447]])
@pytest.mark.parametrize("max_ctas", [0, 10])
def test_no_result_depends_on_the_expected_rows(counts_l, max_ctas):
    from fuselink_b200.ops import gemm
    H, F = 256, 768                                                 # N: 256 (one tile of any kind), 768, 1536
    counts = torch.tensor(counts_l, dtype=torch.int32, device="cuda")
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    x, w13, w2 = _mk(G * CAP, H, seed=1), _mk(G, 2 * F, H, scale=0.1, seed=2), _mk(G, H, F, scale=0.1, seed=3)
    act, dy = _mk(G * CAP, F, seed=4), _mk(G * CAP, H, seed=5)
    for g, c in enumerate(counts_l):                                # a contraction over rows takes whole tiles of them
        for t in (x, act, dy):
            t[g * CAP + c:(g + 1) * CAP] = 0
    fill = lambda *s: torch.full(s, 7.0, dtype=torch.bfloat16, device="cuda")
    kw = dict(status=st, max_ctas=max_ctas)
    rows = [slice(g * CAP, g * CAP + c) for g, c in enumerate(counts_l)]

    def swiglu(e):
        out, gu = fill(G * CAP, F), fill(G * CAP, 2 * F)
        gemm.grouped_gemm_rows(x, w13, counts, CAP, epilogue=gemm.EPI_SWIGLU, out=out, gu=gu, zero_tail=True, expect_rows=e, **kw)
        return out, gu
    out, gu = _same(swiglu)
    for g, r in enumerate(rows):
        gate, up = gemm.deinterleave_gate_up(w13[g:g + 1])
        if counts_l[g]:
            z = x[r].float()
            _close(out[r], torch.nn.functional.silu(z @ gate[0].float().t()) * (z @ up[0].float().t()))

    def dswiglu(e):
        dgu = fill(G * CAP, 2 * F)
        gemm.grouped_gemm_rows(dy, w2, counts, CAP, b_mn_major=True, epilogue=gemm.EPI_DSWIGLU, gu=gu, dgu=dgu, zero_tail=True, expect_rows=e, **kw)
        return dgu,
    _same(dswiglu)

    perm = torch.randperm(G * CAP, generator=torch.Generator().manual_seed(6)).int().cuda()

    def scatter(a, w, n, mn):
        def launch(e):
            buf = fill(G * CAP, n)
            gemm.grouped_gemm_rows(a, w, counts, CAP, b_mn_major=mn, epilogue=gemm.EPI_SCATTER, row_info=perm, peers=[buf.data_ptr()], ldc=n,
                                   peer_rows=G * CAP, expect_rows=e, **kw)
            return buf,
        return launch
    buf, = _same(scatter(act, w2, H, False))                        # narrower than a wide tile
    for g, r in enumerate(rows):
        if counts_l[g]:
            _close(buf[perm[r].long()], act[r].float() @ w2[g].float().t())
    _same(scatter(gu, _mk(G, 2 * F, 1024, scale=0.1, seed=7), 1024, True))

    def store(e):
        c = fill(G * CAP, 2 * F)
        gemm.grouped_gemm_rows(x, w13, counts, CAP, out=c, zero_tail=True, expect_rows=e, **kw)
        return c,
    _same(store)

    def wgrad(e):
        w = _mk(G, F, H, seed=8)
        gemm.grouped_gemm_wgrad(act, x, counts, CAP, G, out=w, sgd_lr=0.5, expect_rows=e, **kw)
        return gemm.grouped_gemm_wgrad(act, x, counts, CAP, G, expect_rows=e, **kw), w
    dw, _ = _same(wgrad)
    for g, r in enumerate(rows):
        if counts_l[g]:
            _close(dw[g], act[r].float().t() @ x[r].float())
    assert st[0] == 0


@pytest.mark.parametrize("M,N", [(8, 32), (40, 96), (264, 288), (512, 544), (1000, 64), (256, 1056)])
@pytest.mark.parametrize("rows", [[3, 0, 190], [64, 65, 384]])
@pytest.mark.parametrize("lr", [0.0, 0.25, 0.01])                       # 0.01: a product that is not exact, so that one rounding more or less shows
def test_weight_gradients_through_the_pair_kernel(M, N, rows, lr):
    """Bit by bit what one CTA per tile stores from registers: matrices that end inside a block of 32 rows x 64 columns or inside a tile, an
    expert without rows, a contraction that ends inside a k-block, several tiles per pair, and nothing written behind the matrices."""
    from fuselink_b200 import C
    from fuselink_b200.ops.gemm import grouped_gemm_wgrad
    G, cap = len(rows), 384
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a, b = (torch.randn(G * cap, n, generator=g, device="cuda").to(torch.bfloat16) for n in (M, N))
    for i, n in enumerate(rows):                       # the rows behind an expert's last are zeros, as the kernels before leave them
        a[i * cap + n:(i + 1) * cap], b[i * cap + n:(i + 1) * cap] = 0, 0
    counts = torch.tensor(rows, dtype=torch.int32, device="cuda")
    w = torch.randn(G * M * N + 4096, generator=g, device="cuda").to(torch.bfloat16)
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    got, before = {}, C.gemm_get_variant()
    try:
        for v in (0, 1):
            C.gemm_set_variant(v)
            got[v] = w.clone()
            for _ in range(2):
                grouped_gemm_wgrad(a, b, counts, cap, G, out=got[v][: G * M * N].view(G, M, N), sgd_lr=lr, max_ctas=4, status=st)
            torch.cuda.synchronize()
            assert st[0].item() == 0, st.tolist()
    finally:
        C.gemm_set_variant(before)
    assert torch.equal(got[0], got[1]) and torch.equal(got[1][G * M * N:], w[G * M * N:])
    if lr == 0.0:
        want = torch.stack([a[i * cap:i * cap + n].double().t() @ b[i * cap:i * cap + n].double() for i, n in enumerate(rows)])
        # rounded to bf16 once; sums of up to 384 products in fp32
        assert ((got[1][: G * M * N].view(G, M, N).double() - want).abs() <= 2.0 ** -8 * want.abs() + 384 * 2.0 ** -23 * 16).all()


@pytest.mark.parametrize("N,K", [(128, 64), (384, 200), (512, 1024)])
@pytest.mark.parametrize("rows", [[1, 0, 128], [129, 31, 256], [257, 300, 384]])
@pytest.mark.parametrize("mn", [False, True])
def test_activation_gradients_through_the_pair_kernel(N, K, rows, mn):
    """Bit by bit what one CTA per tile stores from registers: columns that end in the middle of a tile, rows that end inside a block of 32,
    a CTA of the pair without rows, an expert without any; zeros up to a whole 128 rows and nothing behind them."""
    from fuselink_b200 import C
    from fuselink_b200.ops.gemm import EPI_DSWIGLU, grouped_gemm_rows
    G, cap = len(rows), 384
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    a, b, gu = rnd(G * cap, K), rnd(G, K, N) if mn else rnd(G, N, K), rnd(G * cap, 2 * N) * 3
    counts = torch.tensor(rows, dtype=torch.int32, device="cuda")
    st = torch.zeros(8, dtype=torch.int32, device="cuda")
    got, before = {}, C.gemm_get_variant()
    try:
        for v in (0, 1):
            C.gemm_set_variant(v)
            got[v] = torch.full((G * cap + 40, 2 * N), 7.0, dtype=torch.bfloat16, device="cuda")
            for _ in range(2):
                grouped_gemm_rows(a, b, counts, cap, b_mn_major=mn, epilogue=EPI_DSWIGLU, gu=gu, dgu=got[v], zero_tail=True, max_ctas=4, status=st)
            torch.cuda.synchronize()
            assert st[0].item() == 0, st.tolist()
    finally:
        C.gemm_set_variant(before)
    assert torch.equal(got[0], got[1])
    for i, n in enumerate(rows):
        end = (n + 127) // 128 * 128
        assert (got[1][i * cap + n:i * cap + end] == 0).all() and (got[1][i * cap + end:(i + 1) * cap] == 7).all()
        assert n == 0 or got[1][i * cap:i * cap + n].float().abs().amax(1).min() > 0
