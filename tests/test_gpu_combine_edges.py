"""Combination of the cameras' rows at the edges of its work split: rows shorter and longer than a warp's two vectors a
lane, odd widths, fewer and more cameras than lanes, queries that many, one or no cameras see."""
import pytest
import torch

from dfa3d_b200.rebatch import CombineCamerasFunction, GatherQueriesFunction, RebatchPlan

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("cams", [1, 6, 32, 33, 70])
@pytest.mark.parametrize("W", [1, 7, 64, 128, 255, 256, 260, 1024])
def test_combine_matches_a_loop_over_cameras(lib_built, cams, W):
    bs, Q = 2, 13
    g = torch.Generator().manual_seed(cams * 1000 + W)
    mask = torch.rand(cams, bs, Q, 3, generator=g) < 0.2
    mask[:, :, 0] = True
    mask[:, :, 1] = False
    plan = RebatchPlan(mask.to(DEV))
    rows = torch.randn(bs * plan.rows, W, generator=g).to(DEV).requires_grad_(True)
    want = torch.zeros(bs, Q, W, device=DEV, dtype=torch.float64)
    for j in range(bs):
        for p, q in enumerate(plan.packed_query.tolist()):
            want[j, q] += rows[j * plan.rows + p].detach().double()
    got = CombineCamerasFunction.apply(rows, plan)
    assert (got.double() - want * plan.inv_count[..., None].double()).abs().max() <= 1e-5
    # the gather's backward is the same kernel without the division by the number of cameras
    src = torch.randn(bs, Q, W, generator=g).to(DEV).requires_grad_(True)
    grad, = torch.autograd.grad(GatherQueriesFunction.apply(src, plan), src, rows.detach())
    assert (grad.double() - want).abs().max() <= 1e-5
