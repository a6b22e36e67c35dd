"""What the library says about its last call at an even or a general p: whether the matrix products or the lists gave the result,
and no earlier call's duration."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_enable_kernel_timing(0)


def _outcome(lib):
    value = ctypes.c_int(-1)
    status = lib.ldn_last_power_outcome(torch.cuda.current_stream().cuda_stream, ctypes.byref(value))
    return value.value if status == 0 else None


@pytest.mark.parametrize("p", [4.0, 8.0, 37.5, 100.0])
def test_forward(lib, p):
    import l_inf_dist_net_v2_b200 as ldn
    x, w = torch.rand(512, 2048, 1, device="cuda"), torch.randn(2560, 2048, device="cuda")
    ldn.norm_dist(x, w, p)
    assert _outcome(lib) == 0
    x[3, 5] = float("nan")  # the general kernels'
    ldn.norm_dist(x, w, p)
    assert _outcome(lib) == 1
    ldn.norm_dist(x[:8], w[:32], p)  # too small for either
    assert _outcome(lib) is None
    ldn.norm_dist(x, w, p)
    ldn.norm_dist(x, w, float("inf"))
    assert _outcome(lib) is None


def test_backward(lib):
    import l_inf_dist_net_v2_b200 as ldn
    x = torch.rand(512, 2048, 1, device="cuda", requires_grad=True)
    w = torch.randn(2560, 2048, device="cuda", requires_grad=True)
    y, g = ldn.norm_dist(x, w, 8.0), torch.randn(512, 2560, 1, device="cuda")
    torch.autograd.grad(y, (x, w), g, retain_graph=True)
    assert _outcome(lib) == 0
    torch.autograd.grad(y, (x, w), g * 1e38, retain_graph=True)  # coefficients out of range, or not finite
    assert _outcome(lib) in (0, 1)
    g[5, 7] = float("inf")
    torch.autograd.grad(y, (x, w), g, retain_graph=True)
    assert _outcome(lib) == 1


def test_no_earlier_duration_behind_the_lists(lib):
    import l_inf_dist_net_v2_b200 as ldn
    x, w = torch.rand(512, 2048, 1, device="cuda"), torch.randn(2560, 2048, device="cuda")
    lib.ldn_enable_kernel_timing(1)
    ldn.norm_dist(x, w, 5.0)
    assert lib.ldn_last_tile_kernel_ms() > 0
    ldn.norm_dist(x, w, 37.5)
    assert lib.ldn_last_tile_kernel_ms() == -1
