"""The compiled autograd functions against the Python ones they stand in for: the same bits, and the same refusals."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def both(monkeypatch):
    """Runs a callable through the compiled functions and through the Python ones."""
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    assert C.native() is not None

    def run(fn):
        first = fn()
        with monkeypatch.context() as m:
            m.setattr(C, "native", lambda: None)
            return first, fn()
    return run


def _grads(out, inputs, g):
    return torch.autograd.grad(out, [t for t in inputs if t.requires_grad], g)


@pytest.mark.parametrize("p", [8.0, 3, 2.5, 37.5, math.inf])
@pytest.mark.parametrize("need", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("shape", [(5, 8, 6, 2, 3), (70, 33, 20, 1, 1)])
def test_norm_dist(both, p, need, shape):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, G, HW = shape
    torch.manual_seed(0)
    x = torch.rand(B, CI, HW, device="cuda", requires_grad=need[0])
    w = torch.randn(CO, CI // G, device="cuda", requires_grad=need[1])
    g = torch.randn(B, HW, CO, device="cuda").transpose(1, 2)  # an upstream gradient that is not contiguous

    def fn():
        y = ldn.norm_dist(x, w, p, G)
        assert y.requires_grad == any(need)
        return [y.detach(), *(_grads(y, (x, w), g) if any(need) else ())]
    for a, b in zip(*both(fn)):
        if math.isinf(p):
            # (gradients are atomic sums of a few terms, in any order)
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)
        else:
            assert torch.equal(a, b)


@pytest.mark.parametrize("need", [(True, True, True), (True, True, False), (True, False, False), (False, False, True),
                                  (False, False, False)])
def test_bound_inf_dist(both, need):
    import l_inf_dist_net_v2_b200 as ldn
    torch.manual_seed(0)
    lo = torch.rand(7, 12, 5, device="cuda")
    up = (lo + 0.1).requires_grad_(need[1])
    lo.requires_grad_(need[0])
    w = torch.randn(10, 6, device="cuda", requires_grad=need[2])
    g = torch.randn(7, 10, 5, device="cuda")

    def fn():
        yl, yu = ldn.bound_inf_dist(lo, up, w, 2)
        return [yl.detach(), yu.detach(), *(_grads([yl, yu], (lo, up, w), [g, 2 * g]) if any(need) else ())]
    for a, b in zip(*both(fn)):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)


def test_one_output_unused_and_saved_tensor_hooks(both):
    import l_inf_dist_net_v2_b200 as ldn
    torch.manual_seed(0)
    lo = torch.rand(4, 9, 1, device="cuda", requires_grad=True)
    up = (lo.detach() + 0.2).requires_grad_()
    w = torch.randn(5, 9, device="cuda", requires_grad=True)

    def fn():
        packed = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
            yl, _ = ldn.bound_inf_dist(lo, up, w)
        assert len(packed) == 5
        return torch.autograd.grad(yl.sum(), (lo, up, w))
    for a, b in zip(*both(fn)):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)


def test_layers(both):
    import l_inf_dist_net_v2_b200 as ldn
    torch.manual_seed(0)
    fc = ldn.NormDist(20, 12, bias=True).cuda()
    conv = ldn.NormDistConv(3, 8, 3, padding=1, bias=False).cuda()
    x, img = torch.rand(9, 20, device="cuda", requires_grad=True), torch.rand(2, 3, 6, 6, device="cuda", requires_grad=True)

    def fn():
        fc.mean_shift.running_mean.zero_()
        conv.mean_shift.running_mean.zero_()
        a, b = fc(x)[0], conv(img)[0]
        grads = torch.autograd.grad(a.square().sum() + b.square().sum(), [x, img, fc.weight, conv.weight])
        with torch.no_grad():
            fc.eval()
            ev = fc(x, x - 0.1, x + 0.1)
            fc.train()
        return [a.detach(), b.detach(), fc.mean_shift.running_mean.clone(), *grads, *ev]
    for a, b in zip(*both(fn)):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)


def test_what_was_refused_stays_refused():
    import l_inf_dist_net_v2_b200 as ldn
    x, w = torch.rand(4, 6, 1, device="cuda"), torch.randn(5, 6, device="cuda")
    with pytest.raises(NotImplementedError):
        ldn.norm_dist(x, w, -1.0)
    with pytest.raises(NotImplementedError):
        ldn.norm_dist(x, w, 0)
    with pytest.raises(NotImplementedError):
        ldn.norm_dist(x, w, float("nan"))
    with pytest.raises(AssertionError):
        ldn.norm_dist(x, w, 8.0, groups=2)
    with pytest.raises(AssertionError):
        ldn.bound_inf_dist(x, x[:2], w)
    with pytest.raises(RuntimeError):
        ldn.norm_dist(x.double(), w, 8.0)
    with pytest.raises(RuntimeError):
        ldn.norm_dist(x.expand(4, 6, 2), w, 8.0)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: ldn.norm_dist(t, w, 8.0))(x.unsqueeze(0))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: ldn.norm_dist(t, w, 8.0).sum())(x)
    with torch.autograd.forward_ad.dual_level():
        with pytest.raises((RuntimeError, NotImplementedError)):
            ldn.norm_dist(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)), w, 8.0)
    xr = x.clone().requires_grad_()
    grad, = torch.autograd.grad(ldn.norm_dist(xr, w, 8.0).sum(), xr, create_graph=True)
    assert not grad.requires_grad


def _twice(fn, x, c):
    """The gradient of a cubic of fn(x), and the gradient of that gradient's square."""
    g, = torch.autograd.grad((fn(x) ** 3 * c).sum(), x, create_graph=True)
    assert g.requires_grad
    return g.detach(), torch.autograd.grad(g.square().sum(), x)[0]


@pytest.mark.parametrize("shape", [(9, 6, 1), (5, 6, 4), (5, 6, 7)])
def test_mean_shift_differentiates_twice(both, shape):
    import l_inf_dist_net_v2_b200 as ldn
    torch.manual_seed(0)
    layer = ldn.MeanShift(shape[1], affine=False).cuda()
    x = torch.randn(shape, device="cuda", requires_grad=True)
    c = torch.randn(shape, device="cuda")
    got = both(lambda: _twice(lambda t: layer(t)[0], x, c))
    layer.fused = False
    want = _twice(lambda t: layer(t)[0], x, c)
    for result in got:
        for a, b in zip(result, want):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5 * b.abs().max().item())


@pytest.mark.parametrize("geometry", [((3, 3), 1, 1, 1), ((3, 2), 1, 0, 2), ((2, 2), 2, 1, 1)])
def test_unfold_differentiates_twice(both, geometry):
    from l_inf_dist_net_v2_b200.modules import _unfold
    torch.manual_seed(0)
    x = torch.randn(3, 4, 8, 8, device="cuda", requires_grad=True)
    c = torch.randn_like(torch.nn.functional.unfold(x, *geometry))
    want = _twice(lambda t: torch.nn.functional.unfold(t, *geometry), x, c)
    for result in both(lambda: _twice(lambda t: _unfold(t, *geometry), x, c)):
        for a, b in zip(result, want):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5 * b.abs().max().item())


def test_what_sees_operators_sees_them(both):
    """Forward-mode tangents and traced graphs of what torch operators computed before there was a kernel for it."""
    import l_inf_dist_net_v2_b200 as ldn
    from l_inf_dist_net_v2_b200.modules import _unfold
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode
    torch.manual_seed(0)
    layer = ldn.MeanShift(6, affine=False).cuda()
    plain = ldn.MeanShift(6, affine=False).cuda()
    plain.fused = False
    cases = [(lambda t: layer(t)[0], lambda t: plain(t)[0], (5, 6, 4)),
             (lambda t: _unfold(t, (3, 3), 1, 1, 1), lambda t: torch.nn.functional.unfold(t, (3, 3), 1, 1, 1), (2, 3, 6, 6))]

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(func.name())
            return func(*args, **(kwargs or {}))

    def check():
        for fn, reference, shape in cases:
            x, v = torch.randn(shape, device="cuda"), torch.randn(shape, device="cuda")
            with torch.autograd.forward_ad.dual_level():
                got, want = (torch.autograd.forward_ad.unpack_dual(f(torch.autograd.forward_ad.make_dual(x, v)))
                             for f in (fn, reference))
            assert torch.allclose(got.tangent, want.tangent, rtol=1e-5, atol=1e-5)
            names = []
            for f in (fn, reference):
                with Seen() as mode:
                    mode.names = []
                    f(x)
                names.append(mode.names)
            assert names[0] == names[1]
            # gradients in batches, which vmap the backward step
            x.requires_grad_()
            ups = torch.randn(3, *reference(x).shape, device="cuda")
            got, want = (torch.autograd.grad(f(x), x, ups, is_grads_batched=True)[0] for f in (fn, reference))
            assert torch.allclose(got, want, rtol=1e-5, atol=1e-5)
    both(check)
    graph = make_fx(cases[1][0])(torch.randn(2, 3, 6, 6, device="cuda"))
    x = torch.randn(2, 3, 6, 6, device="cuda")
    assert torch.equal(graph(x), cases[1][1](x))
