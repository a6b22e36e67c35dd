"""Scratch that a large p = inf call can do without: it is taken where it is there for the asking, never at the expense of the
block that the call's general path has."""
import pytest
import torch

pytestmark = pytest.mark.gpu

B, CI, CO = 512, 2560, 5200
DENSE_BYTES = 24 << 20  # the general path's partial results: 148 CTAs x 2 x 64 KB, and some


@pytest.fixture()
def setup():
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    from l_inf_dist_net_v2_b200._lib import lib
    torch.manual_seed(0)
    x, w = torch.rand(B, CI, 1, device="cuda"), torch.randn(CO, CI, device="cuda")
    y, want = torch.empty(B, CO, 1, device="cuda"), torch.empty(B, CO, 1, device="cuda")
    C.inf_dist_forward_nograd(x, w, want, 1)  # (all kernels of both paths are loaded)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def call():
        y.zero_()
        torch.cuda.synchronize()
        before = lib.ldn_kernel_launches()
        with torch.cuda.stream(stream):
            C.inf_dist_forward_nograd(x, w, y, 1)
        torch.cuda.synchronize()
        assert torch.equal(y, want)
        return lib.ldn_kernel_launches() - before
    yield call, stream, lib
    torch.cuda.synchronize()
    lib.ldn_release_scratch()


def _free():
    return torch.cuda.mem_get_info()[0]


def test_a_reservation_is_not_enlarged_for_it(setup):
    call, stream, lib = setup
    assert lib.ldn_reserve_scratch(stream.cuda_stream, DENSE_BYTES) == 0
    call()
    before = _free()
    few = call()
    assert _free() == before
    assert lib.ldn_reserve_scratch(stream.cuda_stream, 4 * DENSE_BYTES) == 0
    assert call() > few


def test_a_full_device_leaves_the_block_that_is_there(setup):
    from l_inf_dist_net_v2_b200 import norm_dist_cuda as C
    call, stream, lib = setup
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    small = torch.zeros(8, 8, 1, device="cuda"), torch.zeros(8, 8, device="cuda"), torch.zeros(8, 8, 1, device="cuda")
    lib.ldn_set_max_ctas(sms - 1)  # the general path alone; a graph on the stream keeps earlier blocks alive
    try:
        few = call()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            C.inf_dist_forward_nograd(*small, 1)
    finally:
        lib.ldn_set_max_ctas(0)
    torch.cuda.empty_cache()
    fill = torch.empty((_free() - (20 << 20)) >> 21 << 21, dtype=torch.uint8, device="cuda")
    assert _free() < DENSE_BYTES
    try:
        left = []
        for _ in range(3):
            assert call() == few
            left.append(_free())
        assert left[1] == left[2]
    finally:
        del fill
        torch.cuda.empty_cache()
    graph.replay()
    torch.cuda.synchronize()
    del graph
    assert lib.ldn_release_scratch() == 0
    assert call() > few  # asked for again once the scratch has been given back
