"""The gradient of bias + ReLU (csrc/kernels/mlp_bwd.cu), and the recommendation model's step with its MLPs as one node each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# remainders of the four rows of a warp, of the 32 of a CTA and of the 128 columns (32 where rows are not whole 16 bytes)
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 4), (31, 128), (33, 132), (257, 33), (2053, 1024), (40000, 7)])
@pytest.mark.parametrize("shift", [0, 1])
def test_relu_bias_bwd(rows, cols, shift):
    from fuselink_b200 import C
    g = torch.Generator(device="cuda").manual_seed(rows)
    dy, y = (torch.randn(rows * cols + shift, generator=g, device="cuda")[shift:].view(rows, cols) for _ in range(2))     # shift: not at 16 bytes
    y[0, 0], y[rows // 2, cols // 2] = float("nan"), 0.0
    dz, db = C.relu_bias_bwd(dy, y)
    want = torch.where(y <= 0, 0.0, dy)
    assert torch.equal(dz, want)
    # a sum in any order, one rounding per term
    assert ((db - want.double().sum(0)).abs() <= rows * 2.0 ** -24 * want.double().abs().sum(0)).all()


def test_no_rows():
    from fuselink_b200 import C
    dz, db = C.relu_bias_bwd(torch.empty(0, 8, device="cuda"), torch.empty(0, 8, device="cuda"))
    assert dz.shape == (0, 8) and torch.equal(db, torch.zeros(8, device="cuda"))


@pytest.mark.parametrize("tables,batch", [(2, 7), (11, 300), (26, 2500)])
@pytest.mark.parametrize("tf32", [False, True])
def test_mlp_nodes_match_the_layers(tables, batch, tf32, monkeypatch):
    """One step through the nodes and one through the layers' own calls, which a hook asks for: the same bits, the bias gradients but
    for the order of their sums."""
    from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
    from fuselink_b200.parallel.symm import SymmetricHeap
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", tf32)
    cfg = DLRMConfig(num_tables=tables, rows=500, pooling=3, global_batch=batch)
    res = []
    for hooked in (False, True):
        heap = SymmetricHeap.create(64 << 20, device=0)
        try:
            m = DLRM(cfg, heap, 0, 1, device="cuda", seed=3)
            called = []
            if hooked:
                m.bottom[1].register_forward_hook(lambda *a: called.append(1))
            assert m._plain_mlps() == (not hooked)
            opt = torch.optim.SGD(m.dense_parameters(), lr=0.0)
            grads = {}
            for i, p in enumerate(m.dense_parameters()):
                p.register_post_accumulate_grad_hook(lambda p, i=i: grads.__setitem__(i, p.grad.clone()))
            loss = m.train_step(*synthetic_batch(cfg, 0, 1, "cuda", seed=4), opt)
            torch.cuda.synchronize()
            assert bool(called) == hooked and len(grads) == len(m.dense_parameters())
            res.append((loss, m.gpooled.local.clone(), grads))
        finally:
            heap.close()
    (la, ga, pa), (lb, gb, pb) = res
    assert torch.equal(la, lb) and torch.equal(ga, gb)
    for i in pa:
        if pa[i].dim() == 2:
            assert torch.equal(pa[i], pb[i])
        else:
            # each of the two is within batch roundings of the terms' magnitudes; 1 / batch bounds a sample's gradient of its logit, and
            # the layers' weights, below 1 / sqrt(width) each, do not let it grow
            assert (pa[i] - pb[i]).abs().max() <= 2 * batch * 2.0 ** -24


def test_rows_of_another_width_are_refused():
    """The width of the dense features is the first layer's: neither cut nor filled up."""
    from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
    from fuselink_b200.parallel.symm import SymmetricHeap
    cfg = DLRMConfig(num_tables=2, rows=50, pooling=3, global_batch=8)
    heap = SymmetricHeap.create(16 << 20, device=0)
    try:
        m = DLRM(cfg, heap, 0, 1, device="cuda", seed=3)
        dense, idx, labels = synthetic_batch(cfg, 0, 1, "cuda", seed=4)
        opt = torch.optim.SGD(m.dense_parameters(), lr=0.1)
        for wrong in (torch.cat([dense, dense], 1), dense[:, :5].contiguous()):
            with pytest.raises(RuntimeError):
                m.train_step(wrong, idx, labels, opt)
        m.bottom[4] = m.bottom[2] = torch.nn.Linear(256, 256, device="cuda")       # one layer in two places
        m.bottom[0] = torch.nn.Linear(13, 256, device="cuda")
        m.bottom.extend([torch.nn.Linear(256, 128, device="cuda"), torch.nn.ReLU()])
        m.train_step(dense, idx, labels, torch.optim.SGD(m.dense_parameters(), lr=0.1))
        torch.cuda.synchronize()
        heap.check_status()
    finally:
        heap.close()


@pytest.mark.parametrize("batch", [7, 2053, 65536])
@pytest.mark.parametrize("where", ["feature", "weight", "top weight"])
@pytest.mark.parametrize("tf32", [False, True])
def test_nan_goes_through_as_through_the_layers(batch, where, tf32, monkeypatch):
    """A NaN feature or weight makes the loss NaN and the gradients that the layers' own calls make NaN; the rest is the same bits."""
    from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
    from fuselink_b200.parallel.symm import SymmetricHeap
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", tf32)
    cfg = DLRMConfig(num_tables=3, rows=50, pooling=3, global_batch=batch)
    res = []
    for hooked in (False, True):
        heap = SymmetricHeap.create(2 * batch * 3 * cfg.dim * 4 + (16 << 20), device=0)
        try:
            m = DLRM(cfg, heap, 0, 1, device="cuda", seed=3)
            dense, idx, labels = synthetic_batch(cfg, 0, 1, "cuda", seed=4)
            if hooked:
                m.bottom[1].register_forward_hook(lambda *a: None)
            assert m._plain_mlps() == (not hooked)
            if where == "feature":
                dense[batch // 2, 3] = float("nan")
            else:
                (m.bottom if where == "weight" else m.top)[0].weight.data[5, 2] = float("nan")
            grads = {}
            for i, p in enumerate(m.dense_parameters()):
                p.register_post_accumulate_grad_hook(lambda p, i=i: grads.__setitem__(i, p.grad.clone()))
            loss = m.train_step(dense, idx, labels, torch.optim.SGD(m.dense_parameters(), lr=0.0))
            torch.cuda.synchronize()
            res.append((loss, m.gpooled.local.clone(), grads))
        finally:
            heap.close()
    (la, ga, pa), (lb, gb, pb) = res
    assert la.isnan() and lb.isnan()
    assert gb.isnan().any() and torch.equal(ga.isnan(), gb.isnan()) and torch.equal(ga.nan_to_num(), gb.nan_to_num())
    for i in pa:
        assert torch.equal(pa[i].isnan(), pb[i].isnan())
        if pa[i].dim() == 2:
            assert torch.equal(pa[i].nan_to_num(), pb[i].nan_to_num())
