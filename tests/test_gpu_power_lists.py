"""General exponents from lists of the channels whose terms count, against 64-bit sums: ragged sizes, 16 and 8 rows per tile, and
data for which lists do not help, or cannot be proven to be enough, or do not apply at all.

Bound: the value is a root of a sum whose terms have the exponential's 2.7e-6 and the logarithm's 2e-7 p, divided by p, and
fp32's last bit: 1e-6 of the value."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(512, 1024, 4000), (203, 3333, 3001), (130, 3500, 4501), (517, 3501, 1201), (77, 5121, 5200), (1700, 512, 2500)]
KINDS = ["images", "hidden", "wide", "one large channel", "ties", "flat", "row scales", "far", "equal", "tiny"]


def _operands(kind, shape):
    B, CI, CO = shape
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(B))
    w = torch.randn(CO, CI, **f)
    x = torch.rand(B, CI, **f) if kind == "images" else torch.randn(B, CI, **f) * (3.0 if kind == "wide" else 0.5)
    if kind == "one large channel":  # of every seventh sample, which makes the range wide and its outputs depend on it
        x[::7, 11] = 9.0
    if kind == "ties":
        x, w = (x * 4).round() / 4, (w * 4).round() / 4
    if kind == "flat":
        x, w = x.sign(), w.sign()
    if kind == "row scales":
        x, w = x * torch.exp(torch.randn(B, 1, **f)), w * torch.exp(torch.randn(CO, 1, **f))
    if kind == "far":
        x, w = x + 50, w * 0.1 + 50
    if kind == "equal":
        x, w = torch.full_like(x, 0.25), torch.full_like(w, 0.25)
    if kind == "tiny":
        x, w = x * 1e-12, w * 1e-12
    return x.unsqueeze(-1).contiguous(), w


def _exact(x, w, p):
    x, w = x[:, :, 0].double(), w.double()
    ys = []
    for i in range(0, x.shape[0], max(1, (1 << 27) // w.numel())):
        d = (x[i:i + max(1, (1 << 27) // w.numel())].unsqueeze(1) - w).abs_()
        top = d.amax(-1).clamp_min(1e-10)
        s = d.div_(top.unsqueeze(-1)).pow_(p).sum(-1) + (1e-10 / top).pow(p)
        ys.append(top * s.pow(1 / p))
    return torch.cat(ys).unsqueeze(-1)


def _forward(x, w, p):
    import l_inf_dist_net_v2_b200 as ldn
    from l_inf_dist_net_v2_b200._lib import lib
    before = lib.ldn_kernel_launches()
    with torch.no_grad():
        y = ldn.norm_dist(x, w, p, 1)
    return y, lib.ldn_kernel_launches() - before


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_values(shape, kind):
    x, w = _operands(kind, shape)
    for p in (37.5, 99.0):
        y, launches = _forward(x, w, p)
        assert launches > 8  # (this path's, and the gated ones behind it)
        want = _exact(x, w, p)
        assert ((y.double() - want).abs() <= 1e-6 * want).all(), p


@pytest.mark.parametrize("where", ["x", "w"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_that_are_not_finite(where, value):
    x, w = _operands("hidden", SHAPES[0])
    {"x": x[:, :, 0], "w": w}[where][3, 5] = value
    y, _ = _forward(x, w, 37.5)
    few, _ = _forward(x[:15].contiguous(), w, 37.5)  # (too few samples for this path)
    y = y[:15]
    assert torch.equal(y.isfinite(), few.isfinite())
    ok = few.isfinite()
    assert ((y - few).abs() <= 1e-6 * few)[ok].all()


def test_replay_with_other_data():
    x, w = _operands("images", SHAPES[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _forward(x, w, 37.5)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y, _ = _forward(x, w, 37.5)
    for kind in ("hidden", "flat", "images"):
        x2, w2 = _operands(kind, SHAPES[0])
        x.copy_(x2)
        w.copy_(w2)
        graph.replay()
        torch.cuda.synchronize()
        want = _exact(x, w, 37.5)
        assert ((y.double() - want).abs() <= 1e-6 * want).all(), kind
    del graph
