"""The unfold / fold kernels of NormDistConv against torch's on the CPU: copies are exact, sums agree to rounding."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,k,stride,pad,dil", [
    ((1, 1, 1, 1), (1, 1), 1, 0, 1),
    ((2, 3, 7, 5), (3, 3), 1, 1, 1),     # 35 positions: single stores
    ((3, 2, 8, 8), (3, 3), 1, 1, 1),     # 64 positions: stores of four, rows that wrap inside one
    ((2, 5, 14, 14), (3, 3), 2, 1, 1),   # 7 x 7 positions
    ((2, 3, 9, 11), (2, 5), 3, 2, 2),    # rectangular kernel, dilation, pixels that no patch covers
    ((2, 4, 6, 10), (5, 5), 1, 4, 1),    # padding beyond the kernel's reach
    ((5, 7, 32, 32), (3, 3), 1, 1, 1),
    ((4, 3, 5, 6), (5, 6), 1, 0, 1),     # one position
])
def test_unfold_and_fold(shape, k, stride, pad, dil):
    from l_inf_dist_net_v2_b200 import modules
    from l_inf_dist_net_v2_b200._lib import lib
    torch.manual_seed(0)
    x = torch.randn(shape)
    xc = x.cuda().requires_grad_()
    before = lib.ldn_kernel_launches()
    cols = modules._unfold(xc, k, dil, pad, stride)
    assert lib.ldn_kernel_launches() == before + 1
    want = F.unfold(x, k, dil, pad, stride)
    assert torch.equal(cols.detach().cpu(), want)
    g = torch.randn_like(want)
    grad, = torch.autograd.grad(cols, xc, g.cuda())
    exact = F.fold(g.double(), shape[2:], k, dil, pad, stride)
    # a sum of at most kh kw terms in fp32: (kh kw - 1) roundings of partial sums that the terms' magnitudes bound
    bound = F.fold(g.double().abs(), shape[2:], k, dil, pad, stride) * (k[0] * k[1] * 2.0 ** -24)
    assert bool(((grad.cpu().double() - exact).abs() <= bound).all())


def test_other_inputs_take_torch():
    from l_inf_dist_net_v2_b200 import modules
    x = torch.randn(2, 4, 6, 6, device="cuda")
    for t in (x.to(memory_format=torch.channels_last), x.double(), x.permute(0, 1, 3, 2)):
        assert torch.equal(modules._unfold(t, (3, 3), 1, 1, 1), F.unfold(t, (3, 3), 1, 1, 1))
    with pytest.raises(RuntimeError):
        modules._unfold(x, (9, 9), 1, 0, 1)
    with pytest.raises(RuntimeError):
        modules._unfold(x, (3, 3), 1, 1, 0)
