"""Even exponents where the matrix products run under a limit: few and odd numbers of CTAs, batches whose gradients add up chunk
by chunk, and tiles that both CTAs of a pair have (few rows).  Every case makes sure by the launches that the products ran; the
references are 64-bit sums with the call's own outputs, the bounds those of one rounding per term (1e-7 for values, (p - 1) of
them for gradients)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_set_max_ctas(0)
    lib.ldn_set_fused_scratch_limit(0)


def _operands(B, CI, CO, HW=1, images=False):
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(B + CI))
    x = torch.rand(B, CI, HW, **f) if images else 0.5 * torch.randn(B, CI, HW, **f)
    return x.requires_grad_(), torch.randn(CO, CI, **f).requires_grad_(), torch.randn(B, CO, HW, **f)


def _exact(x, w, g, y, p):
    """Values, and gradients that follow from the values given."""
    B, CI, HW = x.shape
    CO = w.shape[0]

    def rows(t):
        return t.detach().double().permute(0, 2, 1).reshape(B * HW, -1)
    xr, a, wd = rows(x), rows(g) / rows(y).pow(p - 1), w.detach().double()
    vs, gx, gw = [], [], torch.zeros_like(wd)
    step = max(1, (1 << 26) // w.numel())
    for i in range(0, B * HW, step):
        t = xr[i:i + step].unsqueeze(1) - wd
        q = t.pow(int(p) - 1)
        vs.append((q * t).sum(-1).pow(1 / p))
        q *= a[i:i + step].unsqueeze(-1)
        gx.append(q.sum(1))
        gw -= q.sum(0)

    def back(t):
        return torch.cat(t).view(B, HW, -1).permute(0, 2, 1)
    return back(vs), back(gx), gw


def _error(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


def _run(lib, x, w, g, p, y=None):
    import l_inf_dist_net_v2_b200 as ldn
    before = lib.ldn_kernel_launches()
    y = ldn.norm_dist(x, w, p) if y is None else y
    middle = lib.ldn_kernel_launches()
    grads = torch.autograd.grad(y, (x, w), g, retain_graph=True)
    return y, grads, middle - before, lib.ldn_kernel_launches() - middle


def _check(x, w, g, p, y, grads):
    want = _exact(x, w, g, y, p)
    assert _error(y.detach(), want[0]) < 1e-7
    for a, b in zip(grads, want[1:]):
        assert _error(a, b) < 1e-6


@pytest.mark.parametrize("ctas", [2, 3, 5, 37, 140])
@pytest.mark.parametrize("size", [(512, 1536, 2048), (257, 2049, 1301)])
def test_fewer_ctas(lib, ctas, size):
    x, w, g = _operands(*size)
    lib.ldn_set_max_ctas(ctas)
    y, grads, forward, backward = _run(lib, x, w, g, 8.0)
    assert forward > 4 and backward > 8
    _check(x, w, g, 8.0, y, grads)


# chunks of whole samples, each large enough for the products; rows that are no multiple of 16 bytes (stored one by one)
@pytest.mark.parametrize("size", [(2200, 1024, 1300), (2200, 1001, 1300)])
@pytest.mark.parametrize("unsuited", [False, True])
def test_chunks_add_up(lib, size, unsuited):
    x, w, g = _operands(*size)
    if unsuited:  # the second chunk's gradients come from few samples: the direct kernels add them
        g[1024:2048] *= torch.nn.functional.one_hot(torch.randint(1024, (size[2],), device="cuda"), 1024).T.unsqueeze(-1)
    y, _, _, whole = _run(lib, x, w, g, 8.0)
    lib.ldn_set_fused_scratch_limit(8 * 4 * size[1] * size[2])  # eight row tiles: chunks of 1024, 1024 and 152 samples
    _, grads, _, chunked = _run(lib, x, w, g, 8.0, y)
    assert whole > 8 and chunked > 16
    _check(x, w, g, 8.0, y, grads)


@pytest.mark.parametrize("p", [8.0, 6.0, 4.0, 2.0])
@pytest.mark.parametrize("images", [False, True])
def test_few_rows(lib, p, images):
    x, w, g = _operands(32, 576, 128, 1024, images)
    y, grads, forward, backward = _run(lib, x, w, g, p)
    assert forward > 4 and backward > 8
    _check(x, w, g, p, y, grads)
