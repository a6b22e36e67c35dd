"""Even exponents as products on the tensor cores, against 64-bit sums: ragged sizes (rows, channels and outputs that fill no tile,
no stage, no vector), groups, convolution shapes, one gradient alone, batches in chunks, and data that the expansion does not
suit (cancelling outputs, rows of different scales, a common offset, values that are not finite), for which other kernels give
the result.

Bounds: a value is a rounded root of a sum whose terms carry 2^-23 each, so 2-norms of 1e-7 are what fp32 gives; a gradient adds
(p - 1) times the output's error and its coefficient's, 1e-6."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B, CI, CO, G, HW
SHAPES = [(512, 1024, 1024, 1, 1), (300, 1001, 2050, 1, 1), (257, 2049, 1301, 1, 1), (8, 576, 128, 1, 900), (9, 576, 129, 1, 841),
          (40, 1000, 600, 2, 49), (1100, 640, 700, 1, 1)]


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_set_max_ctas(0)
    lib.ldn_set_fused_scratch_limit(0)


def _operands(shape, kind="hidden"):
    B, CI, CO, G, HW = shape
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(CI + CO))
    x = torch.rand(B, CI, HW, **f) if kind == "images" else torch.randn(B, CI, HW, **f) * 0.5
    w, g = torch.randn(CO, CI // G, **f), torch.randn(B, CO, HW, **f)
    if kind == "equal rows":  # outputs that are (almost) 0
        x[::50, :, 0] = w[:len(x[::50])].repeat(1, G) + 1e-3 * torch.randn(x[::50, :, 0].shape, **f)
    if kind == "row scales":
        x *= torch.exp(2 * torch.randn(B, 1, 1, **f))
        w *= torch.exp(2 * torch.randn(CO, 1, **f))
    if kind == "offset":
        x, w = x * 0.1 + 30, w * 0.1 + 30
    if kind == "one channel":  # its values lie close together, far from zero
        x[:, 3], w[:, 3] = x[:, 3] * 0.01 + 2, w[:, 3] * 0.01 + 2
    if kind == "tiny":
        x, w = x * 1e-6, w * 1e-6
    return x.contiguous().requires_grad_(), w.contiguous().requires_grad_(), g


def _exact(x, w, g, p, G):
    B, CI, HW = x.shape
    CO = w.shape[0]

    def rows(t):
        return t.double().view(B, G, -1, HW).permute(1, 0, 3, 2).reshape(G, B * HW, -1)

    def back(t):
        return torch.stack(t).reshape(G, B, HW, -1).permute(1, 0, 3, 2).reshape(B, -1, HW)
    xr, gr, wr = rows(x.detach()), rows(g), w.detach().double().view(G, CO // G, -1)
    ys, gxs, gws = [], [], []
    for k in range(G):
        y, gx, gw = [], [], torch.zeros_like(wr[k])
        for i in range(0, B * HW, max(1, (1 << 27) // wr[k].numel())):
            part = slice(i, i + max(1, (1 << 27) // wr[k].numel()))
            d = xr[k, part].unsqueeze(1) - wr[k]
            v = d.abs().pow(p).sum(-1).pow(1 / p)
            t = (d / v.unsqueeze(-1)).pow(p - 1) * gr[k, part].unsqueeze(-1)
            y.append(v)
            gx.append(t.sum(1))
            gw -= t.sum(0)
        ys.append(torch.cat(y))
        gxs.append(torch.cat(gx))
        gws.append(gw)
    return back(ys), back(gxs), torch.cat(gws)


def _error(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _run(x, w, g, p, G):
    import l_inf_dist_net_v2_b200 as ldn
    from l_inf_dist_net_v2_b200._lib import lib
    before = lib.ldn_kernel_launches()
    y = ldn.norm_dist(x, w, p, G)
    middle = lib.ldn_kernel_launches()
    grads = torch.autograd.grad(y, (x, w), g)
    return (y.detach(), *grads), middle - before, lib.ldn_kernel_launches() - middle


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("p", [8.0, 6.0, 4.0, 2.0])
def test_values_and_gradients(lib, shape, p):
    for kind in ("images", "hidden"):
        x, w, g = _operands(shape, kind)
        got, forward, backward = _run(x, w, g, p, shape[3])
        if p == 8.0 and shape in SHAPES[:3]:
            assert forward > 4 and backward > 8  # (more launches than the direct kernels make)
        for a, b, bound in zip(got, _exact(x, w, g, p, shape[3]), (1e-7, 1e-6, 1e-6)):
            assert _error(a, b) < bound


@pytest.mark.parametrize("shape", [SHAPES[1], SHAPES[4]])
def test_one_gradient_alone(lib, shape):
    import l_inf_dist_net_v2_b200 as ldn
    x, w, g = _operands(shape)
    both, _, _ = _run(x, w, g, 8.0, shape[3])
    y = ldn.norm_dist(x, w, 8.0, shape[3])
    for i, t in enumerate((x, w)):
        got, = torch.autograd.grad(y, t, g, retain_graph=True)
        assert _error(got, both[1 + i].double()) < 1e-6


@pytest.mark.parametrize("ctas", [2, 3, 37, 140])
def test_fewer_ctas(lib, ctas):
    x, w, g = _operands(SHAPES[2])
    want, _, _ = _run(x, w, g, 8.0, 1)
    lib.ldn_set_max_ctas(ctas)
    got, _, _ = _run(x, w, g, 8.0, 1)
    for a, b in zip(got, want):
        assert _error(a, b.double()) < 2e-6  # (either within 1e-6)


def test_chunks_of_a_batch_add_up(lib):
    x, w, g = _operands(SHAPES[6])
    want, _, _ = _run(x, w, g, 8.0, 1)
    lib.ldn_set_fused_scratch_limit(4 * 4 * 700 * 640)  # four row tiles: chunks of 512 samples
    got, _, _ = _run(x, w, g, 8.0, 1)
    for a, b in zip(got, want):
        assert _error(a, b.double()) < 1e-6


@pytest.mark.parametrize("kind", ["equal rows", "row scales", "offset", "one channel", "tiny"])
def test_data_that_the_expansion_does_not_suit(lib, kind):
    x, w, g = _operands(SHAPES[0], kind)
    got, _, _ = _run(x, w, g, 8.0, 1)
    lib.ldn_set_max_ctas(1)  # the direct kernels
    direct, _, _ = _run(x, w, g, 8.0, 1)
    y, gx, gw = _exact(x, w, g, 8.0, 1)
    # (gradients take the output as it is, so they have its error too; elementwise for the values, which differ in size)
    assert ((got[0].double() - y) / y).abs().max() < 2 * ((direct[0].double() - y) / y).abs().max() + 1e-6
    for a, d, b in ((got[1], direct[1], gx), (got[2], direct[2], gw)):
        assert _error(a, b) < 2 * _error(d, b) + 1e-7
    if kind == "one channel":
        assert _error(got[1][:, 3], gx[:, 3]) < 2 * _error(direct[1][:, 3], gx[:, 3]) + 1e-7


@pytest.mark.parametrize("where", ["x", "w", "g"])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_that_are_not_finite(lib, where, value):
    x, w, g = _operands(SHAPES[0])
    with torch.no_grad():
        {"x": x, "w": w, "g": g}[where][5, 7] = value
    got, _, _ = _run(x, w, g, 8.0, 1)
    lib.ldn_set_max_ctas(1)
    want, _, _ = _run(x, w, g, 8.0, 1)
    for a, b in zip(got, want):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        ok = b.isfinite()
        assert _error(a[ok], b[ok].double()) < 1e-6


def test_replay_of_a_captured_step(lib):
    import l_inf_dist_net_v2_b200 as ldn
    x, w, g = _operands(SHAPES[1])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(2):
            torch.autograd.grad(ldn.norm_dist(x, w, 8.0, 1), (x, w), g)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = ldn.norm_dist(x, w, 8.0, 1)
        gx, gw = torch.autograd.grad(y, (x, w), g)
    for kind in ("images", "offset", "hidden"):  # the second one makes the direct kernels run
        x2, w2, _ = _operands(SHAPES[1], kind)
        with torch.no_grad():
            x.copy_(x2)
            w.copy_(w2)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip((y.detach(), gx, gw), _exact(x, w, g, 8.0, 1)):
            assert _error(a, b) < (1e-6 if kind != "offset" else 1e-5)
    del graph
