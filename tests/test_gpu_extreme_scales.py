"""The choice of the p = inf path for rows of different scales, as layers have them after training: lists of the rows' own
extreme channels give the result, and the device chooses the dense kernels before anything is listed or walked."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(515, 2050, 6144), (512, 4200, 3076)]
SCALES = [(0.05, 0.0), (0.1, 0.0), (0.2, 0.0), (0.4, 0.0), (0.0, 0.2), (0.0, 0.4), (0.2, 0.2)]


def _outcome():
    from l_inf_dist_net_v2_b200._lib import check, lib
    out = (ctypes.c_int * 2)()
    check(lib.ldn_last_extreme_outcome(torch.cuda.current_stream().cuda_stream, out), "last_extreme_outcome")
    return out[0], out[1]


def _calls(x, w):
    """Values with index, values, bounds: results of this call and its outcome."""
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    y, yu = (torch.empty(x.size(0), w.size(0), 1, device="cuda") for _ in range(2))
    pos = torch.empty_like(y, dtype=torch.int32)
    for call, out in ((lambda: C.inf_dist_forward(x, w, y, pos, 1), (y, pos)),
                      (lambda: C.inf_dist_forward_nograd(x, w, y, 1), (y,)),
                      (lambda: C.bound_inf_dist_forward_nograd(x - 8 / 255, x + 8 / 255, w, y, yu, 1), (y, yu))):
        call()
        yield [t.clone() for t in out]


def _compare(x, w, check):
    from l_inf_dist_net_v2_b200._lib import lib
    got = []
    for out in _calls(x, w):
        check(*_outcome())
        got += out
    lib.ldn_set_max_ctas(torch.cuda.get_device_properties(0).multi_processor_count - 1)
    try:
        want = [t for out in _calls(x, w) for t in out]
    finally:
        lib.ldn_set_max_ctas(0)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("scales", SCALES)
@pytest.mark.parametrize("hidden", [False, True])
def test_rows_of_different_scales(shape, scales, hidden):
    B, CO, CI = shape
    g = torch.Generator(device="cuda").manual_seed(5)
    f = dict(device="cuda", generator=g)
    x = torch.randn(B, CI, **f) * 0.5 if hidden else torch.rand(B, CI, **f)
    w = torch.randn(CO, CI, **f) * torch.exp(scales[0] * torch.randn(CO, 1, **f))
    x = (x * torch.exp(scales[1] * torch.randn(B, 1, **f))).unsqueeze(-1).contiguous()

    def check(dense, searched):
        assert not dense and searched <= B * CO // 32
    _compare(x, w, check)


@pytest.mark.parametrize("kind", ["signs", "one class", "sparse", "outliers", "few values", "nan", "rows of zeros"])
def test_dense_kernels_are_chosen_before_the_walks(kind):
    """Whatever the data does to the lists, outputs are put down for a full search only where the lists' result is kept."""
    B, CO, CI = SHAPES[0]
    g = torch.Generator(device="cuda").manual_seed(6)
    f = dict(device="cuda", generator=g)
    x, w = torch.randn(B, CI, **f) * 0.5, torch.randn(CO, CI, **f)
    if kind == "signs":
        x, w = x.sign(), w.sign()
    if kind == "one class":  # the extreme channels of every row are a quarter of a list's
        w[:, torch.arange(CI, device="cuda") % 4 != 1] *= 0.1
    if kind == "sparse":
        x = x * (torch.rand(B, CI, **f) < 0.05)
        w[:, 256:] *= 1e-3
    if kind == "outliers":
        w[torch.rand(CO, CI, **f) < 1e-3] *= 100
    if kind == "few values":
        w, x = (w * 2).round() / 2, (x * 2).round() / 2
    if kind == "nan":
        x[3, 7] = float("nan")
    if kind == "rows of zeros":
        w[::3], x[::2] = 0, 0

    def check(dense, searched):
        assert not (dense and searched)
    _compare(x.unsqueeze(-1).contiguous(), w, check)
