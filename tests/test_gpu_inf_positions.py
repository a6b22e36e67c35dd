"""p = inf forward over many positions: the one-launch kernel against the tile kernels, bit for bit, and against the largest
32-bit difference and the first channel that has it."""
import pytest
import torch

from l_inf_dist_net_v2_b200 import norm_dist_cuda as _C

pytestmark = pytest.mark.gpu


@pytest.fixture
def tile_kernels():
    from l_inf_dist_net_v2_b200._lib import lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    yield lambda on: lib.ldn_set_max_ctas(sms - 1 if on else 0)
    lib.ldn_set_max_ctas(0)


# (B, CI, CO, G, HW): one channel; a stage of 16 and one more; rows of no whole 16-byte piece; the longest rows (704, bounds
# 352) and one more; 1, 8, 9, 65 and 130 outputs; tiles of 64 positions with remainders and across samples; few tiles, whose
# outputs are split; positions that are and are not whole pieces
SHAPES = [(3, 1, 1, 1, 2), (5, 16, 9, 1, 49), (70, 17, 8, 1, 3), (4, 704, 65, 1, 100), (4, 705, 16, 1, 100), (2, 352, 24, 1, 81),
          (2, 353, 24, 1, 81), (9, 30, 130, 2, 121), (128, 144, 36, 4, 64), (1, 100, 300, 1, 36), (33, 63, 40, 1, 64),
          (40, 260, 128, 1, 196)]
KINDS = ["normal", "ties", "equal", "not finite"]


def _inputs(kind, shape):
    B, CI, CO, G, HW = shape
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(CI + HW))
    x, w = torch.randn(B, CI, HW, **f), torch.randn(CO, CI // G, **f)
    if kind == "ties":
        x, w = x.round(), w.round()
    if kind == "equal":
        x, w = torch.full_like(x, 0.5), torch.full_like(w, 0.5)
    if kind == "not finite":
        x[0, 0, 0], w[0, 0] = float("nan"), float("inf")
        x[-1, -1, -1], w[-1, -1] = float("-inf"), float("nan")
    return x, w


def _run(x, w, G):
    shape = x.size(0), w.size(0), x.size(2)
    y, value, lower, upper, shifted = (torch.full(shape, -7.0, device="cuda") for _ in range(5))
    pos = torch.full(shape, -7, device="cuda", dtype=torch.int32)
    lo, up = x - 0.1, x + 0.1
    lo[::2, ::3], up[::2, ::3] = up[::2, ::3].clone(), lo[::2, ::3].clone()  # crossed bounds meet in the middle
    sub, add = torch.linspace(0, 1, w.size(0), device="cuda"), torch.linspace(2, 3, w.size(0), device="cuda")
    _C.inf_dist_forward(x, w, y, pos, G)
    _C.inf_dist_forward_nograd(x, w, value, G)
    _C.bound_inf_dist_forward_nograd(lo, up, w, lower, upper, G)
    _C.inf_dist_forward_nograd_shifted(x, w, shifted, sub, add, G)
    return y, pos, value, lower, upper, shifted


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_same_as_tile_kernels(shape, kind, tile_kernels):
    G = shape[3]
    x, w = _inputs(kind, shape)
    here = _run(x, w, G)
    tile_kernels(True)
    there = _run(x, w, G)
    tile_kernels(False)
    for a, b in zip(here, there):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    if kind != "not finite":
        B, CI, CO, _, HW = shape
        d = x.view(B, G, 1, CI // G, HW) - w.view(1, G, CO // G, CI // G, 1)
        top = d.abs().amax(3)
        assert torch.equal(here[0].view_as(top), top.clamp_min(1e-10))
        first = (d.abs() == top.unsqueeze(3)).int().argmax(3)
        negative = torch.gather(d, 3, first.unsqueeze(3)).squeeze(3) < 0
        expect = torch.where(top > 1e-10, first - (1 << 31) * negative.long(), torch.zeros_like(first)).to(torch.int32)
        assert torch.equal(here[1].view_as(expect), expect)


def test_input_that_starts_off_a_16_byte_boundary():
    store = torch.randn(4 * 36 * 64 + 1, device="cuda")
    x, w = store[1:].view(4, 36, 64), torch.randn(20, 36, device="cuda")
    for a, b in zip(_run(x, w, 1), _run(x.clone(), w, 1)):
        assert torch.equal(a, b)
