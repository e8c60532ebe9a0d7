"""The embedding-bag kernels at the edges of their batches of rows and of the rows summed in shared memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pooling", [1, 9, 10, 11, 20, 21, 32])
@pytest.mark.parametrize("dim,rows,batch", [(128, 3, 1), (128, 40, 33), (256, 25, 1000), (512, 5000, 70)])
def test_embbag(pooling, dim, rows, batch):
    from fuselink_b200.models.dlrm import DLRM, DLRMConfig
    from fuselink_b200.parallel.symm import SymmetricHeap
    cfg = DLRMConfig(num_tables=3, rows=rows, dim=dim, pooling=pooling, global_batch=batch, lr=0.05, bottom=(64, dim))
    heap = SymmetricHeap.create(32 << 20, device=0)
    try:
        m = DLRM(cfg, heap, 0, 1, device="cuda", seed=1)
        g = torch.Generator(device="cuda").manual_seed(pooling)
        idx = torch.randint(0, rows, (3, batch, pooling), generator=g, device="cuda")
        idx[0] = idx[0] % 2                                                 # nearly every update on two rows
        before = m.tables.double()
        m.sparse_forward_launch(idx)
        want = torch.stack([before[t][idx[t]].sum(1) for t in range(3)], 1)
        size = torch.stack([before[t][idx[t]].abs().sum(1) for t in range(3)], 1)
        assert ((m.sparse_forward_wait() - want).abs() <= pooling * 2.0 ** -24 * size).all()
        grad = torch.randn(batch, 3, dim, generator=g, device="cuda")
        m.sparse_backward_launch(grad)
        m.sparse_backward_apply(idx)
        step = grad.double().mul(-cfg.lr).transpose(0, 1).unsqueeze(2).expand(3, batch, pooling, dim).reshape(3, -1, dim)
        flat = idx.reshape(3, -1, 1).expand(-1, -1, dim)
        want, size = before.scatter_add(1, flat, step), before.abs().scatter_add(1, flat, step.abs())
        # a row's value is a sum in any order of at most batch * pooling terms, one rounding each, and the product with lr
        # (whose own value is rounded to fp32 as well)
        assert ((m.tables - want).abs() <= (batch * pooling + 3) * 2.0 ** -24 * size).all()
        torch.cuda.synchronize()
        heap.check_status()
    finally:
        heap.close()
