"""Tiles shared between CTAs, at CTA counts that cut them differently (whole tiles, two or three CTAs per tile, many, a tile per
several CTAs), and the weight-gradient reduction that shares the fold's launch (whole and ragged vectors, one and many row
tiles): every split gives the values of the unlimited one."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def limit():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib.ldn_set_max_ctas
    lib.ldn_set_max_ctas(0)


@pytest.mark.parametrize("shape", [(40, 300, 130, 1, 1), (130, 640, 264, 1, 1), (300, 96, 520, 2, 1), (3, 70, 33, 1, 100),
                                   (64, 1000, 10, 1, 1), (1200, 37, 41, 1, 1)])
@pytest.mark.parametrize("ctas", [1, 2, 5, 24, 60])
@pytest.mark.parametrize("p", [8.0, 3.0, 37.5, math.inf])
def test_splits_agree(limit, shape, ctas, p):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, G, HW = shape
    torch.manual_seed(0)
    x = torch.rand(B, CI, HW, device="cuda", requires_grad=True)
    w = torch.randn(CO, CI // G, device="cuda", requires_grad=True)
    g = torch.randn(B, CO, HW, device="cuda")

    def run():
        y = ldn.norm_dist(x, w, p, G)
        return (y.detach(), *torch.autograd.grad(y, (x, w), g))
    want = run()
    limit(ctas)
    got = run()
    limit(0)
    if math.isinf(p):
        assert torch.equal(got[0], want[0])
    for a, b in zip(got, want):
        # fp32 sums of up to 1200 terms in two orders: 2 sqrt(n) roundings of the sum's magnitude is ample
        assert float((a - b).abs().max()) <= 2 * math.sqrt(1200) * 2.0 ** -24 * float(b.abs().max())


@pytest.mark.parametrize("shape", [(20, 200, 150, 1, 1), (20, 201, 150, 1, 1)])
def test_bounds_splits_agree(limit, shape):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, G, HW = shape
    torch.manual_seed(0)
    lo = torch.rand(B, CI, HW, device="cuda", requires_grad=True)
    up = (lo.detach() + 0.1).requires_grad_()
    w = torch.randn(CO, CI // G, device="cuda", requires_grad=True)

    def run():
        y = ldn.bound_inf_dist(lo, up, w, G)
        return [t.detach() for t in y] + [t for t in torch.autograd.grad(sum(t.sum() for t in y), (lo, up, w))]
    want = run()
    for ctas in (1, 3, 7, 40):
        limit(ctas)
        got = run()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        for a, b in zip(got[2:], want[2:]):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)
