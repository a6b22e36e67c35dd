"""p = inf forward from the extreme channels of both operands against the dense kernels: the same bits, values and indices, whatever
the data does to the proof (ties, hard outputs, a sample that fails, values that are not finite)."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def dense():
    """Switches the path off: it needs the whole chip."""
    from l_inf_dist_net_v2_b200._lib import lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    yield lambda on: lib.ldn_set_max_ctas(sms - 1 if on else 0)
    lib.ldn_set_max_ctas(0)


def _operands(kind, B, CO, CI):
    g = torch.Generator(device="cuda").manual_seed(3)
    f = dict(device="cuda", generator=g)
    w = torch.randn(CO, CI, **f)
    x = torch.rand(B, CI, **f) if kind == "images" else torch.randn(B, CI, **f) * 0.5
    if kind == "ties":  # multiples of 1/4: many channels reach the maximum of an output
        x, w = (x * 4).round() / 4, (w * 4).round() / 4
    if kind == "hard rows":  # a few samples with one huge value: their outputs cannot be proven unless it is in the list
        x[::97] = torch.where(torch.rand(x[::97].shape, **f) < 0.5, 3.0, -3.0)
    if kind == "flat":  # nothing can be proven
        w = torch.where(torch.rand(CO, CI, **f) < 0.5, 1.0, -1.0)
        x = x.sign()
    if kind == "identity":  # weights as the layers initialise them with identity_val
        rows = torch.arange(CO, device="cuda")
        w[rows, rows % CI] = -10.0
    if kind == "equal":
        x, w = torch.zeros_like(x), torch.zeros_like(w)
    if kind == "nan":
        x[1, 5] = float("nan")
    if kind == "inf":
        w[7, 9] = -float("inf")
    if kind == "tiny":
        x, w = x * 1e-38, w * 1e-38
    return x.unsqueeze(-1).contiguous(), w


KINDS = ["images", "hidden", "ties", "hard rows", "flat", "identity", "equal", "nan", "inf", "tiny"]
SHAPES = [(640, 5000, 2048), (197, 12001, 2730), (515, 2050, 6144), (1500, 1401, 3072)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_value_and_index(dense, shape, kind):
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    from l_inf_dist_net_v2_b200._lib import lib
    B, CO, CI = shape
    x, w = _operands(kind, B, CO, CI)

    def run():
        y = torch.full((B, CO, 1), -1.0, device="cuda")
        pos = torch.full((B, CO, 1), 12345, device="cuda", dtype=torch.int32)
        v, s = torch.empty_like(y), torch.empty_like(y)
        sub, add = torch.arange(CO, device="cuda") * 0.25, torch.full((CO,), 0.3, device="cuda")
        before = lib.ldn_kernel_launches()
        C.inf_dist_forward(x, w, y, pos, 1)
        launches = lib.ldn_kernel_launches() - before
        C.inf_dist_forward_nograd(x, w, v, 1)
        C.inf_dist_forward_nograd_shifted(x, w, s, sub, add, 1)
        return launches, y, pos, v, s
    many, *got = run()
    dense(True)
    few, *want = run()
    assert many > few, "the path was not taken"
    for a, b in zip(got, want):
        assert torch.equal(a, b) or torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_bounds(dense, shape, kind):
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    B, CO, CI = shape
    x, w = _operands(kind, B, CO, CI)
    lo, up = x - 8 / 255, x + 8 / 255
    lo[0], up[0] = up[0].clone(), lo[0].clone()  # crossed bounds become their midpoint
    sub = torch.arange(CO, device="cuda") * 0.25

    def run():
        out = [torch.full((B, CO, 1), -1.0, device="cuda") for _ in range(4)]
        C.bound_inf_dist_forward_nograd(lo, up, w, out[0], out[1], 1)
        C.bound_inf_dist_forward_nograd_shifted(lo, up, w, out[2], out[3], sub, None, 1)
        return out
    got = run()
    dense(True)
    for a, b in zip(got, run()):
        assert torch.equal(a, b) or torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_unaligned_rows_streams_and_capture(dense):
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    B, CO, CI = 500, 5200, 2501
    x, w = _operands("hidden", B, CO, CI)
    out = [torch.empty(B, CO, 1, device="cuda") for _ in range(4)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for k, st in enumerate(streams):
        with torch.cuda.stream(st):
            C.inf_dist_forward_nograd(x, w, out[k], 1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        C.inf_dist_forward_nograd(x, w, out[2], 1)
    x2 = x.flip(0).contiguous()
    x.copy_(x2)
    out[2].fill_(0)
    graph.replay()
    torch.cuda.synchronize()
    dense(True)
    C.inf_dist_forward_nograd(x2, w, out[3], 1)
    assert torch.equal(out[2], out[3])
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[3].flip(0))


def _outcome():
    """(whether the device chose the dense kernels, outputs searched in full) of the last call on the current stream."""
    import ctypes

    from l_inf_dist_net_v2_b200._lib import check, lib
    out = (ctypes.c_int * 2)()
    check(lib.ldn_last_extreme_outcome(torch.cuda.current_stream().cuda_stream, out), "last_extreme_outcome")
    return out[0], out[1]


# what each kind of data is there to reach; the others may go either way
CHOICE = {"images": 0, "hidden": 0, "hard rows": 0, "identity": 0, "flat": 1, "nan": 1, "inf": 1}


@pytest.mark.parametrize("shape", SHAPES)
def test_which_kernels_gave_the_result(shape):
    """The bits above are the dense kernels' whichever ran: here, that the lists gave them where they should, and that some
    outputs were left to the full search."""
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    B, CO, CI = shape
    y, pos, yu = torch.empty(B, CO, 1, device="cuda"), torch.empty(B, CO, 1, device="cuda", dtype=torch.int32), \
        torch.empty(B, CO, 1, device="cuda")
    searched = 0
    for kind, dense in CHOICE.items():
        x, w = _operands(kind, B, CO, CI)
        for call in (lambda: C.inf_dist_forward(x, w, y, pos, 1), lambda: C.inf_dist_forward_nograd(x, w, y, 1),
                     lambda: C.bound_inf_dist_forward_nograd(x - 8 / 255, x + 8 / 255, w, y, yu, 1)):
            call()
            chosen, hard = _outcome()
            assert chosen == dense, kind
            if not dense:
                searched += hard
    assert searched > 0


def test_no_outcome_of_another_call():
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    B, CO, CI = SHAPES[0]
    x, w = _operands("images", B, CO, CI)
    y = torch.empty(B, CO, 1, device="cuda")
    C.inf_dist_forward_nograd(x, w, y, 1)
    assert _outcome()[0] == 0
    C.norm_dist_forward(x[:8].contiguous(), w[:64].contiguous(), y.view(-1)[:512].view(8, 64, 1), 1, 8.0)
    with pytest.raises(RuntimeError, match="status 1"):
        _outcome()
