#!/usr/bin/env python
"""Single-GPU cases of the data-movement kernels, for timing and for ncu captures (each ends in seconds).

    python bench/kernel_case.py --case copy-ldst|copy-bulk|embbag-fwd|embbag-bwd|kvpack|dispatch|combine [--iters 3]
    python bench/kernel_case.py --case dec-attention|dec-norm|dec-qkv|dec-act|interact-fwd|interact-bwd|route|quant-rows|quant-blocks

All "peer" buffers are regions of the same GPU (emulated symmetric heap), so the numbers are HBM-bound versions
of the kernels: bytes moved / time is compared with the measured device-copy bandwidth.  The second line's cases have no peers:
the decoder's passes at the sizes of llama3_8b (16 requests of 2048 tokens; prefill passes over 16384 rows), the interaction of
65536 samples of 27 vectors, the routing of 8192 tokens to 8 experts, the fp8 quantisers on 8 experts (1024 of 4096 rows in use;
weights of 4096 x 14336)."""
import argparse
import json
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import torch


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--case", default="copy-ldst")
    ap.add_argument("--iters", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=1)
    args = ap.parse_args()
    from fuselink_b200 import C
    from fuselink_b200.parallel.symm import SymmetricHeap
    from fuselink_b200.utils import roofline
    from fuselink_b200.utils.timing import time_kernel
    dev = "cuda"
    case = args.case
    if case.startswith("copy"):
        from fuselink_b200.ops.comm import Channel
        heaps = SymmetricHeap.emulated(2, (512 << 20) + (64 << 20))
        n = 256 << 20
        dst = [h.alloc_tensor([n], torch.uint8) for h in heaps]
        ch = Channel(heaps[0], "c", engine=case.split("-")[1])
        src = torch.randint(0, 255, (n,), dtype=torch.uint8, device=dev)
        fn = lambda: ch.put(src, 1, dst[0].offset)
        nbytes = 2 * n
    elif case.startswith("embbag"):
        from fuselink_b200.models.dlrm import DLRM, DLRMConfig, synthetic_batch
        cfg = DLRMConfig(num_tables=4, rows=1_000_000, global_batch=16384)
        heaps = SymmetricHeap.emulated(1, 2 * 16384 * 4 * 128 * 4 + (64 << 20))
        m = DLRM(cfg, heaps[0], 0, 1, device=dev)
        _, idx, _ = synthetic_batch(cfg, 0, 1, dev, seed=0)
        g = torch.randn(16384, 4, 128, device=dev)
        m.gpooled.local.copy_(g)
        if case == "embbag-fwd":
            fn = lambda: C.embbag(False, m.tables, idx, 0, 4, 16384, m.pooled.peers(), 0.0, 0, heaps[0].status_addr)
            nbytes = idx.numel() * 512 + idx.numel() * 8 + 16384 * 4 * 512
        else:
            fn = lambda: C.embbag(True, m.tables, idx, 0, 4, 16384, m.gpooled.peers(), 0.01, 0, heaps[0].status_addr)
            nbytes = 2 * idx.numel() * 512 + idx.numel() * 8 + 16384 * 4 * 512
    elif case == "kvpack":
        from fuselink_b200.models.llama import MODEL_ZOO
        from fuselink_b200.serving.disagg import KVLink, ServeParams
        cfg = MODEL_ZOO["llama3_8b"]
        p = ServeParams(cfg, batch_size=4, input_len=2048, num_decoding_step=0)
        heaps = SymmetricHeap.emulated(2, 2 * 4 * 128 * 32 * 8 * 16 * 128 * 2 + (64 << 20))
        links = [KVLink(h, p, 8) for h in heaps]
        nb = 4 * 128
        k = torch.randn(nb * 32 * 8 * 16 * 128, device=dev).to(torch.bfloat16)
        v = torch.randn_like(k)
        bt = torch.arange(nb, dtype=torch.int32, device=dev).view(4, 128)
        cnt = torch.full((4,), 128, dtype=torch.int32, device=dev)
        links[0].seq = 1
        fn = lambda: links[0].send_layers(1, k, v, nb, bt, bt.contiguous(), cnt, 0, 32)
        nbytes = 2 * 2 * k.numel() * 2
    elif case in ("dispatch", "combine"):
        from fuselink_b200.ops import moe as M
        cfg = M.MoEConfig()
        heaps = SymmetricHeap.emulated(1, 3 << 30)
        ws = M.MoEWorkspace(heaps[0], cfg)
        x = torch.randn(cfg.tokens, cfg.hidden, device=dev).to(torch.bfloat16)
        idx = torch.stack([torch.randperm(8, device=dev)[:2] for _ in range(cfg.tokens)]).int().contiguous()
        w = torch.rand(cfg.tokens, 2, device=dev)
        if case == "dispatch":
            def fn():
                ws.counts.local.zero_()
                M._dispatch(ws, x, idx, None, ws.xd, reuse=False)
            nbytes = cfg.tokens * cfg.hidden * 2 * 3
        else:
            out = torch.empty_like(x)
            fn = lambda: C.moe_combine(ws.comb.local, w, out, 2)
            nbytes = cfg.tokens * cfg.hidden * 2 * 3
    elif case.startswith("dec-"):
        H, heads, kvh, D, F, bs, B, S = 4096, 32, 8, 128, 14336, 16, 16, 2048
        heaps, rows, eps = [], 16384, 1e-5

        def rnd(*shape):
            return torch.randn(*shape, device=dev).to(torch.bfloat16)

        if case == "dec-attention":
            nb = B * (S // bs)
            kp, vp = (rnd(2, nb, bs, kvh, D) for _ in range(2))
            bt = torch.randperm(nb, device=dev).view(B, -1).int()
            qkv, pos, out = rnd(B, (heads + 2 * kvh) * D), torch.full((B,), S - 1, device=dev), torch.empty(B, heads * D, dtype=torch.bfloat16, device=dev)
            fn = lambda: C.dec_attention(qkv, pos, kp, vp, bt, 1, 2, nb, bs, heads, kvh, D, out)
            nbytes = 2 * B * S * kvh * D * 2
        elif case == "dec-norm":
            x, y, h, w = rnd(rows, H), rnd(rows, H), rnd(rows, H), rnd(H)
            fn = lambda: C.dec_add_norm(x, y, None, w, None, h, eps)
            nbytes = 4 * x.numel() * 2
        elif case == "dec-qkv":
            qkv, nb = rnd(rows, (heads + 2 * kvh) * D), rows // bs
            kp, vp = (torch.empty(nb * kvh * bs * D, dtype=torch.bfloat16, device=dev) for _ in range(2))
            bt = torch.randperm(nb, device=dev).view(rows // S, -1).int()
            rope = torch.rand(S, D, device=dev)
            fn = lambda: C.dec_qkv(qkv, None, rope, None, S, kp, vp, bt, 0, 0, 1, nb, bs, heads, kvh, D)
            nbytes = rows * ((heads + kvh) * 2 + kvh + 2 * kvh) * D * 2         # q and k read and written, v read, k and v to their pages
        else:
            h, out = rnd(rows, 2 * F), rnd(rows, F)
            fn = lambda: C.dec_act(h, None, out, 0)
            nbytes = (h.numel() + out.numel()) * 2
    elif case.startswith("interact"):
        B, n, D, ld = 65536, 27, 128, 480
        heaps = []
        x, pooled, out, dx, dp = (torch.randn(*s, device=dev) for s in ((B, D), (B, n - 1, D), (B, ld), (B, D), (B, n - 1, D)))
        fn = (lambda: C.interact_fwd(x, pooled, out)) if case == "interact-fwd" else (lambda: C.interact_bwd(x, pooled, out, dx, dp, 1.0))
        nbytes = (B * n * D * (1 if case == "interact-fwd" else 2) + B * ld) * 4
    elif case == "route":
        heaps = []
        logits, bias = torch.randn(8192, 8, device=dev).to(torch.bfloat16), torch.zeros(8, device=dev)
        fn = lambda: C.moe_route(logits, bias, 2)
        nbytes = 8192 * (8 * 2 + 8 * 4 + 2 * (4 + 4 + 8))
    elif case.startswith("quant-"):
        from fuselink_b200.ops import fp8
        heaps = []
        if case == "quant-rows":
            x, counts = torch.randn(8 * 4096, 4096, device=dev).to(torch.bfloat16), torch.full((8,), 1024, dtype=torch.int32, device=dev)
            q, s = torch.empty(x.shape, dtype=fp8.FP8, device=dev), torch.empty(8 * 4096, 32, device=dev)
            fn = lambda: C.fp8_quantize_rows(x, q, s, counts, 4096)
            nbytes = 8 * 1024 * 4096 * 3
        else:
            w = torch.randn(8, 4096, 14336, device=dev).to(torch.bfloat16)
            q, s = torch.empty(w.shape, dtype=fp8.FP8, device=dev), torch.empty(8, 32, 112, device=dev)
            fn = lambda: C.fp8_quantize_blocks(w, q, s)
            nbytes = w.numel() * 3
    else:
        raise SystemExit("unknown case")
    ms = time_kernel(fn, warmup=args.warmup, iters=args.iters)
    for h in heaps:
        h.check_status(case)
    print(json.dumps({"case": case, "ms": ms, "bytes": nbytes, "GBs": nbytes / ms / 1e6, "frac_of_measured_copy": roofline.hbm_fraction(nbytes, ms)}))


if __name__ == "__main__":
    main()
