"""DLRM with table-wise sharded embeddings (the workload the reference runs through an external DLRM
checkout, .gitmodules:5-7).

Sparse side: 26 tables x rows x 128 fp32, sum pooling with a fixed pooling factor, tables spread over the
ranks.  The table owner pools the bags of the GLOBAL batch and its kernel stores each pooled vector
straight into the sample owner's ``[B_local, 26, 128]`` buffer (forward) / reads the gradient from there and
applies SGD to the rows (backward): csrc/kernels/embbag.cu.  Dense side (data parallel): bottom MLP
13-512-256-128, pairwise-dot interaction, top MLP 1024-1024-512-256-1, BCE-with-logits loss, SGD; dense
gradients are averaged with an NCCL all-reduce (not a named hot path).

On CPU tensors the same model runs as plain PyTorch (oracle and gloo tests).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import List, Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from .._ext import require_native
from ..ops import ref
from ..ops.comm import barrier
from ..parallel.symm import SymmetricHeap


@dataclass
class DLRMConfig:
    num_tables: int = 26
    rows: int = 1_000_000
    dim: int = 128
    pooling: int = 20
    dense_features: int = 13
    bottom: tuple = (512, 256, 128)
    top: tuple = (1024, 1024, 512, 256, 1)
    global_batch: int = 65536
    lr: float = 0.01
    zipf_alpha: float = 1.05


def table_split(num_tables: int, world: int) -> List[tuple]:
    """(first, count) of the tables each rank owns: 26 over 8 -> 4,4,3,3,3,3,3,3."""
    out, first = [], 0
    for r in range(world):
        n = num_tables // world + (1 if r < num_tables % world else 0)
        out.append((first, n))
        first += n
    return out


def zipf_indices(shape, rows: int, alpha: float, generator: torch.Generator, device) -> torch.Tensor:
    """Row ids with P(rank k) ~ k^-alpha over `rows` rows (inverse-CDF sampling of the continuous envelope)."""
    u = torch.rand(shape, generator=generator, device=device, dtype=torch.float64)
    if abs(alpha - 1.0) < 1e-9:
        k = torch.exp(u * torch.log(torch.tensor(float(rows) + 1.0, dtype=torch.float64, device=device)))
    else:
        a = 1.0 - alpha
        k = ((u * ((rows + 1.0) ** a - 1.0)) + 1.0) ** (1.0 / a)
    return (k.floor().long() - 1).clamp_(0, rows - 1)


def _mlp(sizes, last_act: bool) -> nn.Sequential:
    layers = []
    for i in range(len(sizes) - 1):
        layers.append(nn.Linear(sizes[i], sizes[i + 1]))
        if i < len(sizes) - 2 or last_act:
            layers.append(nn.ReLU())
    return nn.Sequential(*layers)


def _parameters(mlp) -> list:
    """list(mlp.parameters()), without the general walk for what _mlp makes: a step asks for them several times."""
    if type(mlp) is not nn.Sequential or mlp._parameters or any(type(m) not in (nn.Linear, nn.ReLU) or m._modules for m in mlp._modules.values()):
        return list(mlp.parameters())
    found = {id(p): p for m in mlp._modules.values() for p in m._parameters.values() if p is not None}
    return list(found.values())


def _tf32_allowed() -> bool:
    """Whether the program lets fp32 products run in tf32.  `fp32_precision` answers for both of the framework's settings; the
    older flag raises once the newer setting has been used."""
    matmul = torch.backends.cuda.matmul
    try:
        return matmul.fp32_precision == "tf32"
    except AttributeError:                     # versions that have the flag alone
        return matmul.allow_tf32


class _Interaction(torch.autograd.Function):
    """[B, width] from the bottom MLP's vectors x and the pooled vectors: x, the dot products of all pairs, zeros up to
    ``width``.  The pooled vectors' gradient, times ``scale``, goes straight into ``gpooled``; ``anchor`` (a leaf that wants a
    gradient and gets none) has the backward run whether or not x wants one."""

    @staticmethod
    def forward(ctx, x, pooled, gpooled, scale, width, iu, anchor):
        # The kernel's products are tf32, so it needs the caller's leave.  Where it is taken its results are the library's bits.
        # Below 16 vectors, unless they come in fours, the library answers in fp32 at some batch sizes although it has that leave
        # (5 vectors: at 1000 and from 4096 on, not at 2053); those products stay the library's.
        n = pooled.shape[1] + 1
        if _tf32_allowed() and (n >= 16 or n % 4 == 0):
            out = torch.empty(x.shape[0], width, dtype=x.dtype, device=x.device)
            require_native().interact_fwd(x, pooled, out)
        else:
            z = torch.cat([x.unsqueeze(1), pooled], dim=1)
            inter = torch.bmm(z, z.transpose(1, 2))[:, iu[0], iu[1]]
            out = F.pad(torch.cat([x, inter], dim=1), (0, width - x.shape[1] - inter.shape[1]))
        ctx.save_for_backward(x)
        ctx.pooled, ctx.gpooled, ctx.scale = pooled, gpooled, scale
        return out

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dout):
        x, = ctx.saved_tensors
        dx = torch.empty_like(x)
        require_native().interact_bwd(x, ctx.pooled, dout.contiguous(), dx, ctx.gpooled, ctx.scale)
        return dx, None, None, None, None, None, None


_GRAM_ROWS = 1024


def _gram(dy: torch.Tensor, r: torch.Tensor) -> torch.Tensor:
    """dy^T r over slices of _GRAM_ROWS rows, the slices' results added up in fp32.  The library's aligned tf32 kernels keep one
    running sum over all rows, and its rounding shows: against fp64 the relative error is 2.94e-4 below 8192 rows, 3.31e-4 at
    65536.  In slices it is 2.94e-4 at any number of rows, which is also what the kernels for odd widths give."""
    B = dy.shape[0]
    n = B // _GRAM_ROWS
    if n < 2:
        return dy.t() @ r
    m = n * _GRAM_ROWS
    out = torch.bmm(dy[:m].view(n, _GRAM_ROWS, -1).transpose(1, 2), r[:m].view(n, _GRAM_ROWS, -1)).sum(0)
    return out if m == B else out.addmm_(dy[m:].t(), r[m:])


class _Mlp(torch.autograd.Function):
    """Linear layers with a ReLU behind each (``relu_last``: behind the last one as well) as one node, params = weight, bias, weight,
    bias, ..., of every layer: the ReLU's gradient and the bias gradient are one pass (csrc/kernels/mlp_bwd.cu).  The ReLU itself is a pass
    of its own: as the library products' epilogue it turns NaN into 0 at some sizes.  The rows x may be ``padded`` with zeros to an aligned
    width for the gradients' products: at 479 columns (26 tables) they miss the library's aligned kernels.  The forward product stays at
    the width of the weight, whose bits decide which ReLUs pass a gradient."""

    @staticmethod
    def forward(ctx, x, relu_last, padded, *params):
        acts = require_native().mlp_forward(x, relu_last, padded, params)
        ctx.save_for_backward(x, *(acts if relu_last else acts[:-1]), *params)
        ctx.relu_last = relu_last
        return acts[-1]

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dy):
        saved, want = ctx.saved_tensors, ctx.needs_input_grad
        n = (len(saved) - ctx.relu_last) // 3 + ctx.relu_last
        dx, *grads = require_native().mlp_backward(dy, saved[:n], ctx.relu_last, saved[n:], [want[0], *want[3:]], _GRAM_ROWS)
        return dx, None, None, *grads

    @staticmethod
    def of(mlp, x, relu_last, padded):
        return _Mlp.apply(x, relu_last, padded, *(p for m in list(mlp)[::2] for p in (m.weight, m.bias)))


class _PaddedLinear(torch.autograd.Function):
    """F.linear(r[:, :in], weight, bias) for rows r that are padded with zeros to an aligned width: the gradients' products
    run over the padded width.  At an odd number of columns (479 for 26 tables) they miss the library's aligned kernels."""

    @staticmethod
    def forward(ctx, r, weight, bias):
        ctx.save_for_backward(r, weight)
        return F.linear(r[:, : weight.shape[1]], weight, bias)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dy):
        r, weight = ctx.saved_tensors
        n = weight.shape[1]
        dr = dy @ F.pad(weight, (0, r.shape[1] - n)) if ctx.needs_input_grad[0] else None
        dw = _gram(dy.contiguous(), r)[:, :n].contiguous() if ctx.needs_input_grad[1] else None
        return dr, dw, dy.sum(0) if ctx.needs_input_grad[2] else None


class DLRM(nn.Module):
    def __init__(self, cfg: DLRMConfig, heap: Optional[SymmetricHeap] = None, rank: int = 0, world: int = 1,
                 device="cuda", seed: int = 0, name: str = "dlrm"):
        super().__init__()
        self.cfg, self.rank, self.world, self.heap, self.name = cfg, rank, world, heap, name
        assert cfg.global_batch % world == 0
        self.b_local = cfg.global_batch // world
        self.t_first, self.t_local = table_split(cfg.num_tables, world)[rank]
        bound = cfg.rows ** -0.5
        g = torch.Generator(device="cpu").manual_seed(seed + 1)
        # tables: fp32 U(-1/sqrt(rows), 1/sqrt(rows)); each table's init depends only on its global index
        tabs = []
        for t in range(self.t_first, self.t_first + self.t_local):
            gt = torch.Generator(device=device if str(device) != "cpu" else "cpu").manual_seed(seed * 977 + t)
            tabs.append((torch.rand(cfg.rows, cfg.dim, generator=gt, device=device) * 2 - 1) * bound)
        # a buffer, not a Parameter: the backward kernel applies SGD to it in place; it is part of state_dict() for checkpoints
        self.register_buffer("tables", torch.stack(tabs) if tabs else torch.zeros(0, cfg.rows, cfg.dim, device=device))
        torch.manual_seed(seed)
        self.bottom = _mlp((cfg.dense_features,) + tuple(cfg.bottom), last_act=True).to(device)
        n_vec = cfg.num_tables + 1
        self.n_inter = n_vec * (n_vec - 1) // 2
        self.top = _mlp((self.n_inter + cfg.dim,) + tuple(cfg.top), last_act=False).to(device)
        iu = torch.triu_indices(n_vec, n_vec, offset=1)
        self.register_buffer("iu0", iu[0].to(device))
        self.register_buffer("iu1", iu[1].to(device))
        del g
        self.launches = 0
        if heap is not None:
            shape = [self.b_local, cfg.num_tables, cfg.dim]
            self.pooled = heap.alloc_tensor(shape, torch.float32)    # peers write pooled vectors here
            self.gpooled = heap.alloc_tensor(shape, torch.float32)   # peers read gradients from here

    # ---- sparse --------------------------------------------------------------------------------------------
    def sparse_forward_launch(self, indices: torch.Tensor):
        """indices: [t_local, B_global, pooling] int64 on this rank's device."""
        C = require_native()
        if self.t_local:
            C.embbag(False, self.tables, indices, self.t_first, self.cfg.num_tables, self.b_local, self.pooled.peers(), 0.0, 0,
                     self.heap.status_addr)
            self.launches += 1
        barrier(self.heap, self.name + ":f", signal=True, wait=False)
        self.launches += 1

    def sparse_forward_wait(self) -> torch.Tensor:
        barrier(self.heap, self.name + ":f", signal=False, wait=True)
        self.launches += 1
        return self.pooled.local

    def sparse_backward_launch(self, grad_pooled: torch.Tensor):
        self.gpooled.local.copy_(grad_pooled)
        self._grad_ready()

    def _grad_ready(self):
        barrier(self.heap, self.name + ":b", signal=True, wait=False)
        self.launches += 1

    def sparse_backward_apply(self, indices: torch.Tensor):
        C = require_native()
        barrier(self.heap, self.name + ":b", signal=False, wait=True)
        if self.t_local:
            C.embbag(True, self.tables, indices, self.t_first, self.cfg.num_tables, self.b_local, self.gpooled.peers(),
                     self.cfg.lr, 0, self.heap.status_addr)
            self.launches += 1
        # No trailing barrier is needed: a peer writes this rank's `pooled` for step s+1 only after its own wait on
        # ":b" of step s (which this rank signals after its dense backward), and this rank rewrites `gpooled` only
        # after its wait on ":f" of step s+1 (which peers signal after their step-s backward kernel).

    # ---- dense ---------------------------------------------------------------------------------------------
    def dense_forward(self, dense: torch.Tensor, pooled: torch.Tensor) -> torch.Tensor:
        x = self.bottom(dense)                                            # [B, dim]
        z = torch.cat([x.unsqueeze(1), pooled], dim=1)                    # [B, 27, dim]
        zz = torch.bmm(z, z.transpose(1, 2))                              # [B, 27, 27]
        inter = zz[:, self.iu0, self.iu1]
        return self.top(torch.cat([x, inter], dim=1)).squeeze(-1)

    def _fused_dense(self, dense: torch.Tensor) -> bool:
        """Whether csrc/kernels/interact.cu takes the interaction: fp32 on the GPU, at most 28 vectors of whole 128 columns, no
        autocast, and a dense side that is what __init__ made, since the first layer of the top MLP is then called through its
        weight and the pooled vectors' gradient does not pass through sparse_backward_launch: no hooks, no replaced or converted
        layers or methods."""
        return (dense.is_cuda and dense.dtype == torch.float32 and self.cfg.dim % 128 == 0 and self.cfg.num_tables <= 27
                and not torch.is_autocast_enabled("cuda") and self._plain_dense() and all(p.is_cuda for p in self.dense_parameters()))

    def _plain_dense(self) -> bool:
        if any(getattr(type(self), f) is not getattr(DLRM, f) or f in self.__dict__ for f in ("dense_forward", "sparse_backward_launch")):
            return False
        if torch.nn.modules.module._has_any_global_hook() or not all(type(m) is nn.Sequential for m in (self.bottom, self.top)):
            return False
        first = self.top[0]
        skipped = (self.top, first)                # modules whose __call__ the fused route does not go through
        return (all(type(m) in (nn.Linear, nn.ReLU) for m in self.bottom) and type(first) is nn.Linear
                and not any("forward" in m.__dict__ or m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                            for m in skipped)
                and all(type(p) is nn.Parameter and p.dtype == torch.float32 for p in self.dense_parameters()))

    def _plain_mlps(self) -> bool:
        """Whether the MLPs may be called through their parameters: layers as __init__ made them, no hooks on any."""
        for mlp, relu_last in ((self.bottom, True), (self.top, False)):
            layers = list(mlp)
            linear, relu = layers[::2], layers[1::2]
            if len(linear) != len(relu) + (not relu_last) or not (all(type(m) is nn.Linear and m.bias is not None for m in linear) and
                                                                  all(type(m) is nn.ReLU for m in relu)):
                return False
            if any("forward" in m.__dict__ or m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                   for m in (mlp, *layers)):
                return False
        return True

    def _dense_forward_fused(self, dense: torch.Tensor, pooled: torch.Tensor) -> torch.Tensor:
        """dense_forward with the gradient of ``pooled`` (over the ranks' mean) written to the buffer the tables' owners read."""
        plain = self._plain_mlps()
        x = (_Mlp.of(self.bottom, dense, True, False) if plain else self.bottom(dense)).contiguous()
        if x.data_ptr() % 16:                              # a hook may have put a view of something larger in its place
            x = x.clone()
        n = self.n_inter + self.cfg.dim
        width = (n + 7) // 8 * 8
        anchor = torch.empty(0, device=x.device, requires_grad=True)
        r = _Interaction.apply(x, pooled, self.gpooled.local, 1.0 / self.world, width, (self.iu0, self.iu1), anchor)
        if plain:
            return _Mlp.of(self.top, r, False, True).squeeze(-1)
        first = self.top[0]
        y = _PaddedLinear.apply(r, first.weight, first.bias)
        return self.top[1:](y).squeeze(-1)

    def dense_parameters(self):
        return _parameters(self.bottom) + _parameters(self.top)

    # ---- one training step (public API) --------------------------------------------------------------------
    def train_step(self, dense: torch.Tensor, indices: torch.Tensor, labels: torch.Tensor, opt: torch.optim.Optimizer):
        """Forward + backward + SGD on dense and sparse parameters.  Returns the (detached) loss."""
        fused = self.heap is not None          # a heap was given: the fused kernels (on host memory only in tests that model them)
        direct = fused and self._fused_dense(dense)      # the pooled vectors' gradient is written where the owners read it
        if fused:
            self.sparse_forward_launch(indices)
            pooled = self.sparse_forward_wait().detach().requires_grad_(not direct)
        else:
            pooled = self._pooled_reference(indices).requires_grad_(True)
        logits = (self._dense_forward_fused if direct else self.dense_forward)(dense, pooled)
        loss = F.binary_cross_entropy_with_logits(logits, labels)
        loss.backward()
        work = flat = grads = None
        if self.world > 1:
            # data-parallel part: one bucket for every dense gradient, reduced while the sparse backward runs
            import torch.distributed as dist
            from torch._utils import _flatten_dense_tensors, _unflatten_dense_tensors
            grads = [p.grad for p in self.dense_parameters()]
            flat = _flatten_dense_tensors(grads)
            work = dist.all_reduce(flat, async_op=True)
        # the loss is a mean over the local batch; the global objective is the mean over ranks
        if direct:
            self._grad_ready()
        else:
            gp = pooled.grad / self.world if self.world > 1 else pooled.grad
            if fused:
                self.sparse_backward_launch(gp)
            else:
                self._sparse_backward_reference(indices, gp)
        if fused:
            self.sparse_backward_apply(indices)
        if work is not None:
            work.wait()
            flat /= self.world
            for g, r in zip(grads, _unflatten_dense_tensors(flat, grads)):
                g.copy_(r)
        opt.step()
        opt.zero_grad(set_to_none=True)
        return loss.detach()

    # ---- CPU / gloo path -----------------------------------------------------------------------------------
    def _pooled_reference(self, indices):
        part = ref.embedding_bag_sum(self.tables, indices)                # [B_global, t_local, dim]
        if self.world == 1:
            return part
        import torch.distributed as dist
        full = torch.zeros(self.cfg.global_batch, self.cfg.num_tables, self.cfg.dim)
        full[:, self.t_first:self.t_first + self.t_local] = part
        dist.all_reduce(full)
        return full[self.rank * self.b_local:(self.rank + 1) * self.b_local].clone()

    def _sparse_backward_reference(self, indices, gp):
        if self.world == 1:
            g = gp
        else:
            import torch.distributed as dist
            full = torch.zeros(self.cfg.global_batch, self.cfg.num_tables, self.cfg.dim)
            full[self.rank * self.b_local:(self.rank + 1) * self.b_local] = gp
            dist.all_reduce(full)
            g = full
        ref.embedding_bag_sgd(self.tables, indices, g[:, self.t_first:self.t_first + self.t_local].contiguous(), self.cfg.lr)


def synthetic_batch(cfg: DLRMConfig, rank: int, world: int, device, seed: int):
    """(dense [B_local, 13], indices [t_local, B_global, pooling], labels [B_local]) for one step."""
    t_first, t_local = table_split(cfg.num_tables, world)[rank]
    b_local = cfg.global_batch // world
    g = torch.Generator(device=device).manual_seed(seed * 131 + rank)
    dense = torch.randn(b_local, cfg.dense_features, generator=g, device=device)
    labels = (torch.rand(b_local, generator=g, device=device) < 0.5).float()
    gi = torch.Generator(device=device).manual_seed(seed * 7919 + 13)
    # every rank derives the same global index tensor for a table from (seed, table), then keeps its tables
    idx = []
    for t in range(t_first, t_first + t_local):
        gt = torch.Generator(device=device).manual_seed(seed * 7919 + 13 + t)
        idx.append(zipf_indices((cfg.global_batch, cfg.pooling), cfg.rows, cfg.zipf_alpha, gt, device))
    del gi
    indices = torch.stack(idx) if idx else torch.zeros(0, cfg.global_batch, cfg.pooling, dtype=torch.long, device=device)
    return dense, indices, labels
