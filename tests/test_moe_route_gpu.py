"""The routing kernels (csrc/kernels/moe_route.cu) against the same operations in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(logits, bias, k):
    probs = torch.softmax(logits + bias.double(), -1)
    E = probs.shape[1]
    idx = torch.sort(probs.detach(), dim=-1, descending=True, stable=True)[1][:, :k]
    w = probs.gather(1, idx)
    share = torch.nn.functional.one_hot(idx[:, 0], E).double().mean(0)
    return w / w.sum(-1, keepdim=True), idx, (probs.mean(0) * share).sum() * E


@pytest.mark.parametrize("experts,topk", [(1, 1), (2, 2), (7, 3), (8, 2), (9, 1), (16, 8), (17, 4), (32, 2), (33, 8), (64, 6)])
@pytest.mark.parametrize("tokens", [1, 63, 64, 65, 1531, 8193])
def test_route(experts, topk, tokens):
    from fuselink_b200.models.moe import _Route
    g = torch.Generator(device="cuda").manual_seed(tokens + experts)
    logits = (torch.randn(tokens, experts, generator=g, device="cuda") * 2).round().div(4).to(torch.bfloat16)      # many ties
    bias = torch.randint(-2, 3, (experts,), generator=g, device="cuda").float()
    dw, daux = torch.randn(tokens, topk, generator=g, device="cuda"), torch.full((), 0.3, device="cuda")
    got_in = logits.clone().requires_grad_(True)
    w, idx, idx64, aux = _Route.apply(got_in, bias, topk)
    want_in = logits.double().requires_grad_(True)
    want_w, want_idx, want_aux = _oracle(want_in, bias, topk)
    assert torch.equal(idx64, want_idx) and torch.equal(idx.long(), want_idx) and idx.dtype == torch.int32
    # the exponential is within 2 units in the last place, sums add experts or tokens / 32 roundings of half a unit
    eps = (experts + 8) * 2.0 ** -23
    torch.testing.assert_close(w.double(), want_w, rtol=eps, atol=0)
    torch.testing.assert_close(aux.double(), want_aux, rtol=eps + (tokens // 1024 + 16) * 2.0 ** -23, atol=0)
    torch.autograd.backward([w, aux], [dw, daux])
    torch.autograd.backward([want_w, want_aux], [dw.double(), daux.double()])
    scale = dw.abs().max().double() + 0.3 * experts / tokens
    # rounded to bf16 once; the differences before that cancel to an error of the size of their terms
    assert ((got_in.grad.double() - want_in.grad).abs() <= 2.0 ** -8 * want_in.grad.abs() + 8 * eps * topk * scale).all()


def test_gradients_of_one_output_and_of_the_gradient():
    from fuselink_b200.models.moe import _Route
    logits = torch.randn(70, 8, device="cuda").to(torch.bfloat16).requires_grad_(True)
    bias = torch.zeros(8, device="cuda")
    w, _, _, aux = _Route.apply(logits, bias, 2)
    once, = torch.autograd.grad(aux, logits, retain_graph=True)
    twice, = torch.autograd.grad(aux, logits, create_graph=True)
    torch.testing.assert_close(once, twice.detach(), rtol=2.0 ** -7, atol=1e-7)
    second, = torch.autograd.grad(twice.float().square().sum(), logits)
    assert torch.isfinite(second.float()).all() and second.abs().max() > 0
    assert torch.autograd.grad(w[:, 0].sum(), logits)[0].abs().max() > 0


def test_route_under_transforms(monkeypatch):
    """vmap, jvp and forward mode through MoELayer.route give what the general route gives; so does an ordinary call, through the kernel."""
    from torch.autograd import forward_ad

    from fuselink_b200.models.moe import MoELayer
    from fuselink_b200.ops.moe import MoEConfig
    layer = MoELayer(MoEConfig(hidden=64, ffn=128, num_experts=8, topk=2, tokens=70), None, 0, 1, device="cuda")
    layer.requires_grad_(False)
    g = torch.Generator(device="cuda").manual_seed(1)
    x, d = ((torch.randn(2, 70, 64, generator=g, device="cuda")).to(torch.bfloat16) for _ in range(2))
    weights = lambda t: layer.route(t)[0]

    def forward_mode():
        with forward_ad.dual_level():
            return forward_ad.unpack_dual(weights(forward_ad.make_dual(x[0], d[0])))

    res = []
    for general in (False, True):
        if general:
            monkeypatch.setattr(MoELayer, "_fused_route", lambda self, y: False)
        res.append((torch.vmap(weights)(x), *torch.func.jvp(weights, (x[0],), (d[0],)), *forward_mode(), weights(x[0])))
    for a, b in zip(*res):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-6)


def test_a_batch_of_gradients():
    from fuselink_b200.models.moe import _Route
    logits = torch.randn(70, 8, device="cuda").to(torch.bfloat16).requires_grad_(True)
    w, _, _, aux = _Route.apply(logits, torch.zeros(8, device="cuda"), 2)
    dw, daux = torch.randn(5, 70, 2, device="cuda"), torch.randn(5, device="cuda")
    for outs, grads in (((w,), (dw,)), ((aux,), (daux,)), ((w, aux), (dw, daux))):
        got, = torch.autograd.grad(outs, logits, grads, retain_graph=True, is_grads_batched=True)
        want = torch.stack([torch.autograd.grad(outs, logits, [g[i] for g in grads], retain_graph=True)[0] for i in range(5)])
        # one rounding to bf16 in either, of sums in another order
        torch.testing.assert_close(got, want, rtol=2.0 ** -7, atol=1e-6)
