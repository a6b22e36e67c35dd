"""The hinge loss of many rows: one launch that several blocks share, against the torch operators, and never much slower than they
are."""
import pytest
import torch

from l_inf_dist_net_v2_b200 import norm_dist_cuda as _C

pytestmark = pytest.mark.gpu


def _operators(worst, mix):
    pos = worst.clamp(min=0)
    return (1 - mix) * pos.max(dim=1)[0].mean() + mix * pos.mean()


# groups of 2, 4, 8, 16 and 32 lanes, one block, several and all of them, rows that fill no pass of a block
SIZES = [(255, 2), (257, 3), (2049, 8), (513, 9), (4097, 10), (8191, 16), (1025, 17), (32768, 10), (32767, 2), (32768, 1), (1024, 1024),
         (5000, 100)]


@pytest.mark.parametrize("rows, classes", SIZES)
@pytest.mark.parametrize("kind", ["normal", "ties", "not finite"])
def test_values_and_gradients(rows, classes, kind):
    g = torch.Generator(device="cuda").manual_seed(rows)
    margin = torch.randn(rows, classes, device="cuda", generator=g)
    if kind == "ties":
        margin = margin.round()
    if kind == "not finite":
        margin[rows // 2, 0], margin[-1, -1] = float("inf"), float("-inf")
    margin.requires_grad_()
    loss = _C.native().hinge(margin, 0.25)
    again = _C.native().hinge(margin, 0.25)
    assert torch.equal(loss, again)  # (sums in a fixed order)
    want = _operators(margin.double(), 0.25)
    assert torch.allclose(loss.double(), want, rtol=2.0 ** -23, atol=0)  # (64-bit sums, rounded once)
    got, = torch.autograd.grad(loss, margin)
    wanted, = torch.autograd.grad(_operators(margin, 0.25), margin)
    assert torch.allclose(got, wanted, rtol=2.0 ** -21, atol=0)  # (three roundings each)


@pytest.mark.parametrize("rows, classes", SIZES)
def test_not_slower_than_the_operators(rows, classes):
    margin = torch.randn(rows, classes, device="cuda", requires_grad=True)

    def elapsed(loss):
        best = float("inf")
        for _ in range(4):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            start.record()
            for _ in range(10):
                torch.autograd.grad(loss(margin, 0.25), margin)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        return best
    assert elapsed(_C.native().hinge) < 1.5 * elapsed(_operators)


@pytest.mark.parametrize("rows, classes", [(8, 1025), (32769, 2)])
def test_beyond_are_the_operators(rows, classes):
    assert _C.native().hinge(torch.randn(rows, classes, device="cuda"), 0.25) is None
