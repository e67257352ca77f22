"""Spatial cross-attention without gradients projects a query once for all cameras that see it: same results as one row
per camera, for items that share a warp and items that have one, with cameras that see no query or all of them, and where
the separate operations take over."""
import pytest
import torch

from dfa3d_b200 import modules

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("levels,P", [(1, 4), (1, 8), (2, 5 * 4), (4, 8)])
@pytest.mark.parametrize("seen", ["some", "none", "all"])
@pytest.mark.parametrize("bs,empty", [(1, False), (2, False), (1, True)])
def test_one_row_per_query_equals_one_row_per_camera(lib_built, levels, P, seen, bs, empty):
    torch.manual_seed(levels * 10 + P)
    E, H, D, cams, Q, Z = 64, 4, 6, 3, 35, 4
    hw = [(7, 9), (5, 4), (3, 3), (2, 1)][:levels]
    N = sum(h * w for h, w in hw)
    shapes = torch.tensor(hw, device=DEV)
    lsi = torch.cat([shapes.new_zeros(1), shapes.prod(1).cumsum(0)[:-1]])
    net = modules.SpatialCrossAttention_DFA3D(
        E, cams, 0.0, modules.MSDeformableAttention3D_DFA3D(E, H, levels, P), bev_h=5, bev_w=7, num_head=H,
        use_empty=empty).to(DEV)
    with torch.no_grad():
        for p in net.parameters():
            p.copy_(torch.randn_like(p) * 0.1)
    mask = {"some": torch.rand(cams, bs, Q, Z) < 0.3, "none": torch.zeros(cams, bs, Q, Z, dtype=torch.bool),
            "all": torch.ones(cams, bs, Q, Z, dtype=torch.bool)}[seen]
    mask[1] = seen == "all"                                  # a camera that sees nothing
    kw = dict(value=torch.randn(cams, N, bs, E, device=DEV), value_dpt_dist=torch.rand(cams, N, bs, D, device=DEV),
              reference_points_cam=torch.rand(cams, bs, Q, Z, 3, device=DEV), bev_mask=mask.to(DEV),
              spatial_shapes=shapes, level_start_index=lsi)
    query = torch.randn(bs, Q, E, device=DEV)
    want = net(query, **kw).detach()
    with torch.no_grad():
        got = net(query, **kw)
    assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
