"""The kernels around a convolution layer's distances: batch mean over samples and positions, coefficients of
convolution-shaped outputs, the weight-gradient reduction over many row tiles."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 2), (3, 5, 7), (2, 3, 64), (9, 40, 49), (130, 4, 100), (40, 2, 2500), (33, 3, 2501)])
def test_mean_shift_of_planes(shape):
    import l_inf_dist_net_v2_b200 as ldn
    B, C, HW = shape
    torch.manual_seed(0)
    x = torch.randn(B, C, HW) + 3
    g = torch.randn(B, C, HW)
    ms = ldn.MeanShift(C, affine=False).cuda().train()
    ms.running_mean.fill_(0.5)
    xc = x.cuda().requires_grad_()
    out, _, _ = ms(xc)
    grad, = torch.autograd.grad(out, xc, g.cuda())
    x64, g64 = x.double(), g.double()
    mean = x64.mean(dim=[0, 2])
    # sums of n fp32 terms added as a tree of at most n / 2048 + 24 levels, one rounding of the largest magnitude per level
    tol = (B * HW / 2048 + 24) * 2.0 ** -24
    assert float((out.detach().cpu() - (x64 - mean.view(1, -1, 1))).abs().max()) <= tol * float(x64.abs().max())
    assert float((ms.running_mean.cpu() - (0.45 + 0.1 * mean)).abs().max()) <= tol * float(x64.abs().max())
    want = g64 - g64.mean(dim=[0, 2]).view(1, -1, 1)
    assert float((grad.cpu() - want).abs().max()) <= tol * float(g64.abs().max())


@pytest.mark.parametrize("shape", [(3, 8, 33, 1, 33), (2, 36, 40, 2, 64), (70, 20, 12, 1, 100), (40, 16, 24, 1, 130)])
@pytest.mark.parametrize("p", [8.0, 3.0, 37.5])
def test_convolution_shaped_backward(shape, p):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, G, HW = shape
    torch.manual_seed(0)
    x = torch.rand(B, CI, HW)
    w = torch.randn(CO, CI // G)
    g = torch.randn(B, CO, HW)
    xc, wc = x.cuda().requires_grad_(), w.cuda().requires_grad_()
    gx, gw = torch.autograd.grad(ldn.norm_dist(xc, wc, p, G), (xc, wc), g.cuda())
    x64 = x.double().view(B, G, 1, CI // G, HW).requires_grad_()
    w64 = w.double().view(1, G, CO // G, CI // G, 1).requires_grad_()
    y64 = (x64 - w64).abs().pow(p).sum(3).pow(1 / p).view(B, CO, HW)
    ex, ew = torch.autograd.grad(y64, (x64, w64), g.double())
    # fp32 terms of relative error 2^-24 (2 p + 4) (integer p) or 1e-5 (general p), summed over up to B HW = 7000
    tol = 1e-5 if p == int(p) else 1e-4
    for got, want in ((gx, ex), (gw, ew)):
        assert float((got.cpu().double().view(-1) - want.reshape(-1)).abs().max()) <= tol * float(want.abs().max())


@pytest.mark.parametrize("shape", [(32, 128, 1024), (40, 2, 2500), (33, 3, 2501), (700, 2, 2304)])
def test_mean_of_planes_is_rounded_once(shape):
    """The sum of n < 2^29 equal fp32 terms is exact in 64 bits, so a constant channel's mean is the constant."""
    import l_inf_dist_net_v2_b200 as ldn
    ms = ldn.MeanShift(shape[1], affine=False).cuda().train()
    for value in (0.1, 7.3, -1 / 3):
        x = torch.full(shape, value, device="cuda", requires_grad=True)
        out, _, _ = ms(x)
        grad, = torch.autograd.grad(out, x, torch.full_like(x, value))
        assert not out.any() and not grad.any()
