"""Products of a few rows with a large matrix (csrc/kernels/thin_gemm.cu) against PyTorch."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DT = [torch.bfloat16, torch.float16]


def _eighths(*shape, dt, seed):
    """Multiples of 1/8 in [-1/2, 1/2]: every sum of their products below 2^18 is exact in fp32, in any order."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randint(-4, 5, shape, generator=g, device="cuda") / 8).to(dt)


# edges of the tiles (128 rows of w, 64 columns, 16 rows of x) and of the cuts along k (8, 4, 2, 1 CTAs per tile)
@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("rows,n,k", [(1, 1, 8), (3, 127, 72), (15, 128, 64), (16, 129, 1024), (9, 2048, 2048), (16, 6144, 520),
                                      (7, 1000, 8200), (5, 12288, 768), (13, 640, 264), (16, 38000, 128), (2, 50257, 768), (4, 128, 65536)])
@pytest.mark.parametrize("early", [False, True])
def test_sums_are_exact(dt, rows, n, k, early):
    from fuselink_b200 import C
    x, w, b = _eighths(rows, k, dt=dt, seed=1), _eighths(n, k, dt=dt, seed=2), _eighths(n, dt=dt, seed=3)
    sums = (x.double() @ w.double().t()).to(dt)
    for _ in range(2):
        assert torch.equal(C.dec_product(x, w, None, 3, early), sums)
    assert torch.equal(C.dec_product(x, w, b, 3, early), sums + b)
    assert torch.equal(C.dec_product(x, w, b, 1, early), F.relu(sums + b))
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    want = F.gelu(sums + b, approximate="tanh")                     # as for the separate activation kernel
    assert ((C.dec_product(x, w, b, 2, early) - want).float().abs() <= 2.02 * eps * want.float().abs() + 1e-6).all()


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("rows,n,k", [(1, 8, 64), (16, 64, 2048), (5, 72, 136), (11, 14336, 512), (16, 1000, 264), (2, 20000, 128)])
def test_gated(dt, rows, n, k):
    from fuselink_b200 import C
    x, w = _eighths(rows, k, dt=dt, seed=1), _eighths(2 * n, k, dt=dt, seed=2)
    h = (x.double() @ w.double().t()).to(dt)
    want = F.silu(h[:, :n]) * h[:, n:]
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    # the gate may be rounded to its neighbour (2 eps), the product is rounded once more; 6e-8: fp16's smallest step
    assert ((C.dec_product(x, w, None, 0) - want).float().abs() <= 4.05 * eps * want.float().abs() + 6e-8).all()


@pytest.mark.parametrize("rows,n,k", [(16, 6144, 4096), (3, 2048, 8192)])
def test_error_of_ordinary_values(rows, n, k):
    from fuselink_b200 import C
    g = torch.Generator(device="cuda").manual_seed(5)
    x, w = (torch.randn(a, k, generator=g, device="cuda").to(torch.bfloat16) for a in (rows, n))
    want = x.double() @ w.double().t()
    # rounding to bf16, and one rounding of the running sum (at most the sum of the magnitudes) per 16 products
    bound = 2.0 ** -8 * want.abs() + (k // 16 + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())
    assert ((C.dec_product(x, w, None, 3).double() - want).abs() <= bound).all()


def test_not_finite_values_stay_in_their_row_and_column():
    from fuselink_b200 import C
    x, w = _eighths(4, 256, dt=torch.bfloat16, seed=1), _eighths(300, 256, dt=torch.bfloat16, seed=2)
    x[1, 3], w[7, 9] = float("nan"), float("inf")
    got = C.dec_product(x, w, None, 1)
    want = F.relu((x.double() @ w.double().t()).to(torch.bfloat16))
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num(nan=-1), want.nan_to_num(nan=-1))


def test_arguments():
    from fuselink_b200 import C
    x, w = torch.zeros(2, 64, dtype=torch.half, device="cuda"), torch.zeros(8, 64, dtype=torch.half, device="cuda")
    for bad in ((x, w[:, :32].contiguous(), None, 3), (x.repeat(9, 1), w, None, 3), (x, w.bfloat16(), None, 3), (x, w, x[0, :7], 3),
                (x[:, :63].contiguous(), w[:, :63].contiguous(), None, 3), (x, w[:7], None, 0), (x.view(-1)[1:65].view(1, 64), w, None, 3)):
        with pytest.raises(RuntimeError):
            C.dec_product(*bad)


def test_the_kernel_before_may_take_longer_than_a_wait():
    """An early product waits as long as the kernel before it runs, here one that polls a flag for longer than the 2 s of a wait inside
    a kernel; only then does its own limit count."""
    from fuselink_b200 import C
    x, w = _eighths(5, 512, dt=torch.bfloat16, seed=1), _eighths(300, 512, dt=torch.bfloat16, seed=2)
    flag, timed_out = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(8, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = C.dec_product(x, w, None, 3)
    torch.cuda.synchronize()
    C.wait_flags([(flag.data_ptr(), 1)], timed_out.data_ptr(), 2600)          # a flag that nothing sets
    got = C.dec_product(x, w, None, 3, True, status.data_ptr())
    torch.cuda.synchronize()
    assert timed_out[0] != 0 and status[0] == 0
    assert torch.equal(got, want)


@pytest.mark.parametrize("dt", DT)
@pytest.mark.parametrize("rows,k,heads,kv_heads,dim", [(1, 64, 1, 1, 16), (3, 2048, 32, 32, 64), (16, 512, 5, 1, 128), (9, 264, 3, 2, 32), (13, 4096, 32, 8, 128)])
@pytest.mark.parametrize("rope,bias", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("layout", [0, 1])
def test_qkv_with_rotation_and_pages(dt, rows, k, heads, kv_heads, dim, rope, bias, layout):
    """Against the product and the pass behind it, bit by bit: negative positions and pages, positions beyond the table of angles, a
    page outside the pool and one outside the block table among them."""
    from fuselink_b200 import C
    n, L, nblk, bs, layer = (heads + 2 * kv_heads) * dim, 2, 40, 16, 1
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, w = _eighths(rows, k, dt=dt, seed=1), _eighths(n, k, dt=dt, seed=2)
    b = _eighths(n, dt=dt, seed=3) if bias else None
    ang = torch.rand(30, dim // 2, generator=g, device="cuda") * 6
    table = torch.cat([ang.cos(), ang.sin()], 1).contiguous() if rope else None
    bt = torch.randperm(nblk, generator=g, device="cuda")[:16 * 2].int().view(16, 2).contiguous()
    pos = torch.randint(0, 32, (rows,), generator=g, device="cuda")
    if rows > 4:
        pos[1], pos[2], bt[3], pos[4] = -3, 1000, nblk, 2 ** 33
        bt[0] -= nblk
    pools = [[torch.zeros(nblk * L * bs * kv_heads * dim, dtype=dt, device="cuda") for _ in range(2)] for _ in range(2)]
    st = torch.zeros(2, dtype=torch.int32, device="cuda")
    qkv = C.dec_product(x, w, None, 3)
    C.dec_qkv(qkv, b, table, pos, 1, *pools[0], bt, layout, layer, L, nblk, bs, heads, kv_heads, dim, st.data_ptr())
    got = C.dec_qkv_product(x, w, b, table, pos, *pools[1], bt, layout, layer, L, nblk, bs, heads, kv_heads, dim, True, st.data_ptr() + 4)
    assert torch.equal(got[:, :heads * dim], qkv[:, :heads * dim])
    for p, q in zip(*pools):
        assert torch.equal(p, q) and p.any()
    assert (st[0] != 0) == (st[1] != 0) == (rows > 4)


def test_arguments_of_qkv():
    from fuselink_b200 import C
    cuda = dict(dtype=torch.half, device="cuda")
    x, w = torch.zeros(2, 64, **cuda), torch.zeros(96, 64, **cuda)
    pos, bt, pool = torch.zeros(2, dtype=torch.long, device="cuda"), torch.zeros(2, 1, dtype=torch.int32, device="cuda"), torch.zeros(4 * 16 * 48, **cuda)

    def call(x=x, w=w, bias=None, rope=None, pos=pos, k=pool, v=pool, bt=bt, layer=0, blocks=4, heads=1, kv_heads=1, dim=32):
        return C.dec_qkv_product(x, w, bias, rope, pos, k, v, bt, 1, layer, 1, blocks, 16, heads, kv_heads, dim, True, 0)

    call()
    rope = torch.zeros(4, 32, device="cuda")
    for bad in (dict(dim=16), dict(w=torch.zeros(144, 64, **cuda), dim=48), dict(pos=pos[:1]), dict(bt=bt[:1]), dict(layer=1), dict(blocks=64), dict(bias=x[0]),
                dict(rope=rope[:, :16]), dict(rope=rope.half()), dict(k=pool.bfloat16()), dict(x=x.repeat(9, 1)), dict(w=w.bfloat16()),
                dict(rope=torch.zeros(130, device="cuda")[1:129].view(4, 32)), dict(x=torch.zeros(200, **cuda)[1:129].view(2, 64))):
        with pytest.raises(RuntimeError):
            call(**bad)
