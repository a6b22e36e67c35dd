"""Gradients of even exponents, entry by entry: data whose channels lie away from zero, hardly differ, or are constant but for one
sample, and data on either side of the guards.  The yardstick is the direct kernels' error against 64 bits on the same inputs and
outputs: what the products give may be at most twice as far off, as a whole, in the worst channel, and at the 99th percentile
of the entries' relative errors.  (Each is a rounding error's size times a constant: the margin of 1e-7 is that of a result
rounded once to 32 bits, its seven powers 1e-6 for a single entry.)"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

B, CI, CO = 512, 1536, 2048


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_set_max_ctas(0)


def _operands(kind, p):
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))

    def uniform(rows, a=0.0, b=1.0):
        return a + (b - a) * torch.rand(rows, CI, **f)

    def normal(rows, mean=0.0, deviation=1.0):
        return mean + deviation * torch.randn(rows, CI, **f)
    x, w, g = uniform(B), normal(CO), torch.randn(B, CO, **f)
    if kind == "both uniform":
        w = uniform(CO)
    elif kind == "narrow weights":
        w = uniform(CO, 0.25, 0.75)
    elif kind == "common offset":
        x, w = uniform(B, 1, 2), normal(CO, 1.5, 0.5)
    elif kind == "both in 1 to 2":
        x, w = uniform(B, 1, 2), uniform(CO, 1, 2)
    elif kind == "both in 1.25 to 2.25":
        x, w = uniform(B, 1.25, 2.25), uniform(CO, 1.25, 2.25)
    elif kind == "some channels far off":
        x[:, :64], w[:, :64] = uniform(B, 2.5, 3.4)[:, :64], uniform(CO, 2.5, 3.4)[:, :64]
    elif kind == "pixels that hardly differ":
        x = normal(B, 0.5, 0.02)
    elif kind == "bright pixels":
        x = normal(B, 0.8, 0.1)
    elif kind == "constant pixels":  # all the same, or one sample with the smallest step of 8 bits
        x[:, :32], x[:, 32:64] = 0.3, 0.0
        x[3, 40:64] = 1 / 255
    elif kind == "activations":
        x = normal(B, 0, 0.5)
    elif kind == "wide clusters":  # as wide as they are apart
        centers = torch.randn(2, CI, **f)
        x = centers[torch.arange(B, device="cuda") % 2] + normal(B)
        w = centers[torch.arange(CO, device="cuda") % 2] + normal(CO)
    elif kind == "clusters":  # small differences between rows of one cluster: the largest coefficients
        centers = torch.randn(2, CI, **f)
        x = centers[torch.arange(B, device="cuda") % 2] + normal(B, 0, 0.3)
        w = centers[torch.arange(CO, device="cuda") % 2] + normal(CO, 0, 0.3)
    elif kind == "row scales":
        x *= torch.exp(torch.randn(B, 1, **f))
    elif kind == "one gradient per sample":
        g *= torch.nn.functional.one_hot(torch.randint(CO, (B,), **f), CO)
    elif kind == "one gradient per output":
        g *= torch.nn.functional.one_hot(torch.randint(B, (CO,), **f), B).T
    elif kind == "some samples without gradient":
        g[::3] = 0
    return x.unsqueeze(-1).requires_grad_(), w.requires_grad_(), g.unsqueeze(-1)


def _exact(x, w, g, y, p):
    a = (g.double() / y.double().pow(p - 1)).squeeze(-1)
    gx, gw = [], torch.zeros(CO, CI, dtype=torch.float64, device="cuda")
    xd, wd = x.detach().double().squeeze(-1), w.detach().double()
    for i in range(0, B, 32):
        t = xd[i:i + 32].unsqueeze(1) - wd
        q = t * a[i:i + 32].unsqueeze(-1)
        t *= t
        for _ in range(int(p) // 2 - 1):
            q *= t
        gx.append(q.sum(1))
        gw -= q.sum(0)
    return torch.cat(gx).unsqueeze(-1), gw


def _errors(got, want):
    d = got.double() - want
    channels = d.norm(dim=0) / want.norm(dim=0).clamp(min=1e-300)
    entries = (d / want).abs()[want != 0].flatten()
    return d.norm() / want.norm(), channels.max(), entries.kthvalue(int(0.99 * len(entries))).values


# whether the products are the ones to give the result
SUITED = ["images", "both uniform", "narrow weights", "common offset", "both in 1 to 2", "both in 1.25 to 2.25", "some channels far off",
          "pixels that hardly differ", "bright pixels", "constant pixels", "activations", "some samples without gradient"]
UNSUITED = ["clusters", "wide clusters", "row scales", "one gradient per sample", "one gradient per output"]


@pytest.mark.parametrize("p", [8.0, 6.0, 4.0, 2.0])
@pytest.mark.parametrize("kind", SUITED + UNSUITED)
def test_entries_of_both_gradients(lib, kind, p):
    import l_inf_dist_net_v2_b200 as ldn
    x, w, g = _operands(kind, p)
    y = ldn.norm_dist(x, w, p)
    before = lib.ldn_kernel_launches()
    got = torch.autograd.grad(y, (x, w), g, retain_graph=True)
    assert lib.ldn_kernel_launches() - before > 8  # (more than the direct kernels make)
    direct_ran = ctypes.c_int(-1)
    assert lib.ldn_last_power_outcome(torch.cuda.current_stream().cuda_stream, ctypes.byref(direct_ran)) == 0
    if kind in SUITED or p == 8.0:
        assert direct_ran.value == (kind in UNSUITED)
    lib.ldn_set_max_ctas(1)  # the direct kernels
    direct = torch.autograd.grad(y, (x, w), g, retain_graph=True)
    want = _exact(x, w, g, y.detach(), p)
    for a, d, b in zip(got, direct, want):
        for mine, theirs, margin in zip(_errors(a, b), _errors(d, b), (1e-7, 1e-7, 1e-6)):
            assert mine < 2 * theirs + margin


@pytest.mark.parametrize("kind", ["images", "both in 1 to 2", "one gradient per output", "one gradient per sample"])
@pytest.mark.parametrize("which", [0, 1])
def test_one_gradient_alone(lib, kind, which):
    import l_inf_dist_net_v2_b200 as ldn
    x, w, g = _operands(kind, 8.0)
    y = ldn.norm_dist(x, w, 8.0)
    got, = torch.autograd.grad(y, (x, w)[which], g, retain_graph=True)
    lib.ldn_set_max_ctas(1)
    direct, = torch.autograd.grad(y, (x, w)[which], g, retain_graph=True)
    want = _exact(x, w, g, y.detach(), 8.0)[which]
    for mine, theirs, margin in zip(_errors(got, want), _errors(direct, want), (1e-7, 1e-7, 1e-6)):
        assert mine < 2 * theirs + margin
