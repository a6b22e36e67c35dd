"""Values of even exponents for operands with a common offset, from none to one that the matrix products refuse: never more than twice
as far from 64 bits as the direct kernels', on average and at the worst output.  (Margins: half a unit in the last place on
average, two units for one output.)  Refused data costs the direct kernels' time and a little."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    from l_inf_dist_net_v2_b200._lib import lib
    yield lib
    lib.ldn_set_max_ctas(0)


def _exact(x, w, p):
    B, CI, HW = x.shape
    xr, wd = x.double().permute(0, 2, 1).reshape(B * HW, CI), w.double()
    out, step = [], max(1, (1 << 27) // w.numel())
    for i in range(0, len(xr), step):
        t = (xr[i:i + step].unsqueeze(1) - wd).square()
        q = t.clone()
        for _ in range(p // 2 - 1):
            q *= t
        out.append(q.sum(-1).pow(1 / p))
    return torch.cat(out).view(B, HW, -1).permute(0, 2, 1)


@pytest.mark.parametrize("size", [(512, 1536, 2048, 1), (512, 256, 8192, 1), (32, 576, 128, 1024)])
@pytest.mark.parametrize("kind", ["normal", "uniform"])
@pytest.mark.parametrize("p", [2, 4, 6, 8])
def test_offsets(lib, size, kind, p):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, HW = size
    f = dict(device="cuda", generator=torch.Generator(device="cuda").manual_seed(CI))
    draw = torch.rand if kind == "uniform" else (lambda *a, **k: 0.7 * torch.randn(*a, **k))
    x0, w0 = draw(B, CI, HW, **f), draw(CO, CI, **f)
    for offset in (0.0, 0.25, 0.5, 0.75, 1.0, 1.5, 2.0, 3.0):
        x, w = x0 + offset, w0 + offset
        want = _exact(x, w, p)
        errors = []
        for ctas in (0, 1):  # (one: the direct kernels)
            lib.ldn_set_max_ctas(ctas)
            e = (ldn.norm_dist(x, w, float(p)).double() - want) / want
            errors.append((e.square().mean().sqrt().item(), e.abs().max().item()))
        (mean, worst), (direct_mean, direct_worst) = errors
        assert mean < 2 * direct_mean + 3e-8, offset
        assert worst < 2 * direct_worst + 1.2e-7, offset


@pytest.mark.parametrize("size", [(512, 3072, 5120, 1), (32, 576, 128, 1024)])
@pytest.mark.parametrize("p", [4.0, 8.0])
def test_refused_data_is_known_before_the_products(lib, size, p):
    import l_inf_dist_net_v2_b200 as ldn
    B, CI, CO, HW = size
    x, w = 2 + torch.rand(B, CI, HW, device="cuda"), 2 + torch.rand(CO, CI, device="cuda")

    def elapsed():
        best = float("inf")
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            start.record()
            for _ in range(5):
                ldn.norm_dist(x, w, p)
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end) / 5)
        return best
    refused = elapsed()
    value = ctypes.c_int(-1)
    assert lib.ldn_last_power_outcome(torch.cuda.current_stream().cuda_stream, ctypes.byref(value)) == 0 and value.value == 1
    x[1, 2, 0] = float("inf")  # what goes to the direct kernels from the preparation
    assert refused < 1.07 * elapsed()
