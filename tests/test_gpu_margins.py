"""Margins and hinge loss as kernels against the torch operators they stand for: values, both gradients, ties and values that are
not finite, second derivatives, and what goes to the operators as before."""
import math

import pytest
import torch

import l_inf_dist_net_v2_b200 as ldn
from l_inf_dist_net_v2_b200 import losses, norm_dist_cuda as _C

pytestmark = pytest.mark.gpu


def _margins(dist, targets, eps):
    lower, upper, col = dist - eps, dist + eps, targets.view(-1, 1)
    margin = ((-lower) - torch.gather(-upper, 1, col)).scatter(1, col, 0)
    return -dist, margin / (2 * eps)


def _hinge(worst, mix):
    pos = worst.clamp(min=0)
    return (1 - mix) * pos.max(dim=1)[0].mean() + mix * pos.mean()


def _inputs(B, classes, kind="normal"):
    g = torch.Generator(device="cuda").manual_seed(B)
    dist = 3 + torch.randn(B, classes, device="cuda", generator=g)
    if kind == "ties":
        dist = dist.round()
    if kind == "not finite":
        dist[0, 0], dist[-1, -1] = float("inf"), float("nan")
    return dist.requires_grad_(), torch.randint(0, classes, (B,), device="cuda", generator=g)


# one row, one class, fewer and more classes than a warp, more rows than the loss's block has warps
@pytest.mark.parametrize("B, classes", [(1, 1), (1, 10), (7, 31), (33, 32), (256, 10), (300, 100), (3, 1000)])
@pytest.mark.parametrize("kind", ["normal", "ties", "not finite"])
def test_values_and_gradients(B, classes, kind):
    dist, targets = _inputs(B, classes, kind)
    logits, margin = _C.native().margins(dist, targets, 8 / 255)
    loss = _C.native().hinge(margin, 0.25)
    want_logits, want_margin = _margins(dist, targets, 8 / 255)
    want_loss = _hinge(want_margin, 0.25)
    assert torch.allclose(logits, want_logits, rtol=0, atol=0, equal_nan=True)
    assert torch.allclose(margin, want_margin, rtol=2.0 ** -22, atol=0, equal_nan=True)  # (a product with 1 / (2 eps) or a quotient)
    # the same terms in another order: n 32-bit additions of positive terms
    assert torch.allclose(loss, want_loss, rtol=(B * classes + 4) * 2.0 ** -24, atol=0, equal_nan=True)
    seed = torch.randn_like(dist)
    for outputs, wanted in [((loss,), (want_loss,)), ((logits, margin), (want_logits, want_margin)), ((margin,), (want_margin,)),
                            ((logits,), (want_logits,))]:
        up = [seed[:1, 0].reshape(()) if t.dim() == 0 else seed for t in outputs]
        got, = torch.autograd.grad(outputs, dist, up, retain_graph=True)
        want, = torch.autograd.grad(wanted, dist, up, retain_graph=True)
        # the target's entry sums up to `classes` terms of the row's size
        bound = (classes + 4) * 2.0 ** -23 * want.abs().sum(1, keepdim=True).clamp_min(1e-30)
        assert ((got - want).abs() <= bound).logical_or(got.isnan() & want.isnan()).all()


def test_second_derivatives_are_those_of_the_operators():
    dist, targets = _inputs(16, 10)
    weight = torch.randn(16, 10, device="cuda", requires_grad=True)

    def through(margins, hinge):
        logits, margin = margins(dist, targets, 0.1)
        scale = weight.sum()
        g, = torch.autograd.grad(((logits * weight).sum(), (margin * weight).sum(), hinge(margin, 0.25) * scale), dist,
                                 [scale, scale, scale], create_graph=True)
        return torch.autograd.grad(g.square().sum(), weight)[0]

    here, there = through(_C.native().margins, _C.native().hinge), through(_margins, _hinge)
    assert torch.allclose(here, there, rtol=1e-4, atol=1e-4 * there.abs().max().item())


def test_other_calls_take_the_operators():
    ext, (dist, targets) = _C.native(), _inputs(8, 10)
    for args in [(dist.double(), targets, 0.1), (dist.t(), targets, 0.1), (dist[:0], targets[:0], 0.1), (dist, targets.int(), 0.1),
                 (dist, targets[:4], 0.1), (dist, targets, 0.0), (dist, targets.cpu(), 0.1)]:
        assert ext.margins(*args) is None
    assert ext.hinge(dist.half(), 0.25) is None and ext.hinge(dist[:, ::2], 0.25) is None
    batched = torch.vmap(lambda m: losses.hinge()(m, m, None))(torch.randn(3, 8, 10, device="cuda"))
    assert batched.shape == (3,)


@pytest.mark.parametrize("scalar", [False, True])
def test_model(scalar):
    net = ldn.MLPModel(3, 64, [1, 4, 4], num_classes=10, scalar=scalar).cuda().train()
    ldn.set_p_norm(net, math.inf)
    x, targets = torch.rand(32, 1, 4, 4, device="cuda"), torch.arange(32, device="cuda") % 10
    loss, params = losses.hinge(0.25), [p for n, p in net.named_parameters() if n != "scalar"]
    logits, worst = net(x, targets=targets, eps=0.1)
    grads = torch.autograd.grad(loss(logits, worst, targets), params, retain_graph=True)
    dist = net.fc_dist((x.flatten(1), None, None))[0]
    want_logits, want_worst = _margins(dist, targets, 0.1)
    assert torch.equal(logits, want_logits * net.scalar) and torch.allclose(worst, want_worst, rtol=2.0 ** -22, atol=1e-6)
    for a, b in zip(grads, torch.autograd.grad(_hinge(want_worst, 0.25), params)):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-6 * max(1.0, b.abs().max().item()))
    if scalar:
        assert torch.allclose(torch.autograd.grad(logits.sum(), net.scalar)[0], -dist.sum().reshape(1), rtol=1e-5)
