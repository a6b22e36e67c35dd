"""Gradients of the p = inf distance over many positions: the scatter by shared-memory columns and its edges."""
import pytest
import torch

from l_inf_dist_net_v2_b200 import norm_dist_cuda as _C

pytestmark = pytest.mark.gpu


# one channel; rows of 224 channels (the longest by columns) and 225 (atomics); blocks of positions with remainders; one
# output, and numbers around the 8 outputs in flight; 16384 outputs in all (the fewest by columns) and 16383; groups
@pytest.mark.parametrize("B, CI, CO, G, HW", [
    (300, 1, 7, 1, 49), (33, 224, 9, 1, 121), (33, 225, 9, 1, 121), (64, 448, 16, 2, 31), (128, 3, 1, 1, 128),
    (8, 12, 64, 4, 32), (43, 5, 1, 1, 381), (700, 30, 24, 3, 2), (2, 144, 8, 1, 1024), (129, 16, 8, 8, 33),
])
@pytest.mark.parametrize("need", ["both", "input", "weight"])
def test_gradients_by_columns(B, CI, CO, G, HW, need):
    gen = torch.Generator(device="cuda").manual_seed(B + HW)
    n = CI // G
    go = torch.randn(B, CO, HW, device="cuda", generator=gen)
    idx = torch.randint(0, n, (B, CO, HW), device="cuda", generator=gen)
    idx[:, :, ::3] = n // 2  # many outputs of a position, and many positions, share a channel
    neg = torch.rand(B, CO, HW, device="cuda", generator=gen) < 0.5
    pos = torch.where(neg, idx - (1 << 31), idx).to(torch.int32)
    gx = torch.full((B, CI, HW), float("nan"), device="cuda")
    gw = torch.full((CO, n), float("nan"), device="cuda")
    if need == "input":
        _C.inf_dist_backward_input(go, pos, gx, G)
    else:
        _C.inf_dist_backward_input_weight(go, pos, gx if need == "both" else None, gw, G)

    def reference(v):
        rows, i = v.double().view(B, G, CO // G, HW), idx.view(B, G, CO // G, HW)
        x = torch.zeros(B, G, n, HW, device="cuda", dtype=torch.float64).scatter_add_(2, i, rows).view(B, CI, HW)
        w = torch.zeros(CO, n, device="cuda", dtype=torch.float64)
        return x, w.scatter_add_(1, idx.permute(1, 0, 2).reshape(CO, -1), v.double().permute(1, 0, 2).reshape(CO, -1))

    signed = torch.where(neg, -go, go)
    (x, w), (x_abs, w_abs) = reference(signed), reference(go.abs())
    # a sum of k 32-bit terms in any order is within (k - 1) 2^-24 of the sum of magnitudes (k >= 1 terms; an untouched entry is 0)
    if need != "weight":
        assert ((gx - x).abs() <= (CO // G) * 2.0 ** -24 * x_abs).all()
    if need != "input":
        assert ((gw + w).abs() <= B * HW * 2.0 ** -24 * w_abs).all()
