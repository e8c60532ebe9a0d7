"""The fused feature interaction (csrc/kernels/interact.cu) against the same products in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vectors", [2, 3, 4, 5, 8, 9, 12, 13, 17, 21, 25, 27, 28])      # edges of the groups of four rows
@pytest.mark.parametrize("batch,dim,pad", [(1, 128, 0), (5, 256, 4), (7105, 128, 1)])
def test_interaction(vectors, batch, dim, pad):
    from fuselink_b200 import C
    g = torch.Generator(device="cuda").manual_seed(vectors)
    pairs = vectors * (vectors - 1) // 2
    ld = (dim + pairs + pad + 3) // 4 * 4
    x, pooled = torch.randn(batch, dim, generator=g, device="cuda"), torch.randn(batch, vectors - 1, dim, generator=g, device="cuda")
    out, dout = torch.full((batch, ld), float("nan"), device="cuda"), torch.randn(batch, ld, generator=g, device="cuda")
    C.interact_fwd(x, pooled, out)
    z = torch.cat([x.unsqueeze(1), pooled], 1).double()
    i, j = torch.triu_indices(vectors, vectors, 1, device="cuda")
    want = torch.bmm(z, z.transpose(1, 2))[:, i, j]
    assert torch.equal(out[:, :dim], x)
    assert not out[:, dim + pairs:].any()
    # tf32 keeps 11 bits of every factor; the sums on the tensor cores may round each addition towards zero
    size = torch.bmm(z.abs(), z.abs().transpose(1, 2))[:, i, j]
    assert ((out[:, dim:dim + pairs] - want).abs() <= (2 * 2.0 ** -11 * 1.001 + dim * 2.0 ** -23) * size).all()
    dx, dp = torch.empty_like(x), torch.empty_like(pooled)
    C.interact_bwd(x, pooled, dout, dx, dp, 0.5)
    s = torch.zeros(batch, vectors, vectors, dtype=torch.float64, device="cuda")
    s[:, i, j] = dout[:, dim:dim + pairs].double()
    s = s + s.transpose(1, 2)
    dz, size = torch.bmm(s, z), torch.bmm(s.abs(), z.abs())
    dz[:, 0] += dout[:, :dim]
    size[:, 0] += dout[:, :dim].abs()
    bound = (vectors + 2) * 2.0 ** -24 * size
    assert ((dx - dz[:, 0]).abs() <= bound[:, 0]).all()
    assert ((dp - 0.5 * dz[:, 1:]).abs() <= 0.5 * bound[:, 1:]).all()


@pytest.mark.parametrize("vectors", [4, 8, 12, *range(16, 29)])                     # the counts that a step gives to the kernel
def test_forward_products_are_the_librarys_bits(vectors, monkeypatch):
    """What the choice between kernel and library in models/dlrm.py rests on, with the library of CUDA 12.8."""
    from fuselink_b200 import C
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", True)
    i, j = torch.triu_indices(vectors, vectors, 1, device="cuda")
    for batch in (1, 2, 7, 64, 128, 300, 1000, 2053, 4096, 20011, 65536):
        g = torch.Generator(device="cuda").manual_seed(batch)
        x, pooled = torch.randn(batch, 128, generator=g, device="cuda"), torch.randn(batch, vectors - 1, 128, generator=g, device="cuda")
        out = torch.empty(batch, (128 + len(i) + 7) // 8 * 8, device="cuda")
        C.interact_fwd(x, pooled, out)
        z = torch.cat([x.unsqueeze(1), pooled], 1)
        assert torch.equal(out[:, 128:128 + len(i)], torch.bmm(z, z.transpose(1, 2))[:, i, j]), batch


@pytest.mark.parametrize("tables,tf32", [(6, True), (7, True), (26, True), (26, False)])       # 7 and 27 vectors, and the two kinds of 8
def test_train_step_takes_the_general_path_where_the_kernel_does_not_apply(tables, tf32, monkeypatch):
    """Same step through the kernel, with a hook on the top MLP (general path) and with frozen bottom layers."""
    from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
    from fuselink_b200.parallel.symm import SymmetricHeap
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", tf32)
    cfg = DLRMConfig(num_tables=tables, rows=3000, pooling=4, global_batch=300, lr=0.05)
    heap = SymmetricHeap.create(64 << 20, device=0)
    try:
        models = [DLRM(cfg, heap, 0, 1, device="cuda", seed=3, name=f"d{k}") for k in range(3)]
        models[1].top[0].register_forward_hook(lambda m, i, o: None)
        for p in models[2].bottom.parameters():
            p.requires_grad_(False)
        batch = synthetic_batch(cfg, 0, 1, "cuda", seed=1)
        assert [m._fused_dense(batch[0]) for m in models] == [True, False, True]
        for m in models:
            m.train_step(*batch, torch.optim.SGD([p for p in m.dense_parameters() if p.requires_grad], lr=cfg.lr))
        torch.cuda.synchronize()
        heap.check_status()
        a, b, c = models
        assert (a.gpooled.local != 0).any()
        for u, v in zip([a.gpooled.local, *a.dense_parameters()], [b.gpooled.local, *b.dense_parameters()]):
            torch.testing.assert_close(u, v, rtol=2e-3, atol=2e-7)        # tf32 or not, one rounding of 2^-11 per factor
        torch.testing.assert_close(a.gpooled.local, c.gpooled.local)
    finally:
        heap.close()


@pytest.mark.parametrize("columns", [131, 183, 479])
@pytest.mark.parametrize("batch", [300, 2053, 8192, 20011, 65536])           # one slice, slices and a remainder, slices only
def test_weight_gradient_over_the_padded_width_is_as_exact_as_over_its_own(columns, batch, monkeypatch):
    from fuselink_b200.models.dlrm import _PaddedLinear
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", True)
    g = torch.Generator(device="cuda").manual_seed(columns)
    r = torch.zeros(batch, (columns + 7) // 8 * 8, device="cuda")
    r[:, :columns] = torch.randn(batch, columns, generator=g, device="cuda")
    dy = torch.randn(batch, 1024, generator=g, device="cuda").relu_()
    w, b = (torch.randn(*s, generator=g, device="cuda").requires_grad_(True) for s in ((1024, columns), (1024,)))
    _PaddedLinear.apply(r, w, b).backward(dy)
    x = r[:, :columns].contiguous()
    want = dy.double().t() @ x.double()
    err, lib = ((t.double() - want).norm() / want.norm() for t in (w.grad, dy.t() @ x))
    # both are mostly the rounding of the factors to tf32, equal in the two; 1 % covers the order of the sums
    assert err <= 1.01 * lib
