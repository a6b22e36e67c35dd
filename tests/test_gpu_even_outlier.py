"""Even exponents, forward, with one value far beyond the others: almost every output is small on the common scale, and the direct
kernels have to give it.  That may cost the preparation, not the products as well."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_set_max_ctas(0)


def _elapsed(f):
    best = float("inf")
    for _ in range(5):
        start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        start.record()
        for _ in range(5):
            f()
        end.record()
        torch.cuda.synchronize()
        best = min(best, start.elapsed_time(end) / 5)
    return best


# (an outlier among the samples, among the weights; the operand that is written out as powers is the smaller or the larger one)
@pytest.mark.parametrize("B, CI, CO", [(512, 3072, 5120), (5120, 3072, 512)])
@pytest.mark.parametrize("operand", [0, 1])
@pytest.mark.parametrize("p", [4.0, 8.0])
def test_one_large_value(lib, B, CI, CO, operand, p):
    import l_inf_dist_net_v2_b200 as ldn
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    x, w = torch.rand(B, CI, 1, **f), torch.randn(CO, CI, **f)
    (x, w)[operand][7, 5] = 300.0
    got = ldn.norm_dist(x, w, p)
    with_outlier = _elapsed(lambda: ldn.norm_dist(x, w, p))
    lib.ldn_set_max_ctas(1)  # the direct kernels, for a part of the batch
    part = slice(0, 16)
    want = ldn.norm_dist(x[part], w, p)
    assert ((got[part] - want) / want).abs().max() < 1e-5
    lib.ldn_set_max_ctas(0)
    (x, w)[operand][7, 5] = float("inf")  # what goes to the direct kernels from the preparation
    direct = _elapsed(lambda: ldn.norm_dist(x, w, p))
    assert with_outlier < 1.07 * direct


@pytest.mark.parametrize("size", [0.5, 3.0, 10.0])
def test_values_that_are_not_far_off(lib, size):
    """Rows of different norms on one scale: nothing is given up that the list can hold, and what is given up is right."""
    import l_inf_dist_net_v2_b200 as ldn
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    x, w = torch.randn(512, 1024, 1, **f), torch.randn(2048, 1024, **f)
    x[::3] *= 0.1
    w[::2] *= 0.1
    w[5, 7] = size
    got = ldn.norm_dist(x, w, 8.0).squeeze(-1)
    want = torch.cat([(x[i:i + 32].double().squeeze(-1).unsqueeze(1) - w.double()).abs().pow(8).sum(-1).pow(1 / 8) for i in range(0, 512, 32)])
    assert ((got.double() - want) / want).abs().max() < 3e-6
