"""Depth-distribution producer at the edges of its tiles: map widths around 32 pixels, bin counts around a multiple of
four and at the limit, levels that read each map pixel several times or skip most of them; gradients arriving as
fp32, bf16 and fp16.  Checked against softmax / sigmoid + nearest interpolation and its autograd."""
import pytest
import torch

from helpers import assert_close
from test_gpu_dist_producer import level_tensors, reference_dist

pytestmark = pytest.mark.gpu
DEV = "cuda"


# bins: one, two and four a word, up to 64, 128 and 256 of them
@pytest.mark.parametrize("map_w,D", [(1, 1), (31, 4), (32, 64), (33, 65), (64, 3), (100, 256), (7, 255), (50, 66), (33, 128),
                                     (9, 130), (40, 127)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_tile_edges_match_softmax_and_nearest_resize(lib_built, map_w, D, dtype):
    from dfa3d_b200.dist_producer import depth_distribution
    g = torch.Generator().manual_seed(map_w + D)
    levels = ((9, 2 * map_w + 1), (5, map_w), (2, max(1, map_w // 3)), (1, 1))
    logits = (torch.randn(2, D, 5, map_w, generator=g) * 2).to(DEV).requires_grad_(True)
    shapes, lsi, N = level_tensors(levels)
    ref = logits.detach().clone().requires_grad_(True)
    activation = "sigmoid" if map_w == 33 else "softmax"
    want = reference_dist(ref, levels, activation)
    got = depth_distribution(logits, shapes, lsi, N, activation=activation, dtype=dtype)
    step = {torch.float32: 2e-6, torch.bfloat16: 2 ** -7, torch.float16: 2 ** -10}[dtype]
    assert ((got.float() - want.detach()).abs() <= want.detach().abs() * step + 2 ** -24).all()
    gd = torch.randn(2, N, D, generator=g).to(DEV, dtype)
    got.backward(gd)
    want.backward(gd.float())
    assert_close("grad_logits", logits.grad, ref.grad, rtol=1e-4, atol_frac=2e-6)


@pytest.mark.parametrize("map_h,map_w", [(70, 1), (33, 3), (9, 11), (2, 47), (3, 64)])
def test_tiles_that_run_over_map_rows(lib_built, map_h, map_w):
    """A tile is 32 consecutive map pixels: of one row, the end of one and the start of the next, or of up to 32 rows."""
    from dfa3d_b200.dist_producer import depth_distribution
    g = torch.Generator().manual_seed(map_h)
    levels = ((2 * map_h + 1, 2 * map_w), (map_h, map_w), (map_h // 3 + 1, map_w // 2 + 1))
    logits = torch.randn(2, 20, map_h, map_w, generator=g).to(DEV).requires_grad_(True)
    shapes, lsi, N = level_tensors(levels)
    ref = logits.detach().clone().requires_grad_(True)
    want = reference_dist(ref, levels, "softmax")
    got = depth_distribution(logits, shapes, lsi, N)
    assert ((got - want.detach()).abs() <= want.detach().abs() * 2e-6 + 2 ** -24).all()
    gd = torch.randn(2, N, 20, generator=g).to(DEV)
    got.backward(gd)
    want.backward(gd)
    assert_close("grad_logits", logits.grad, ref.grad, rtol=1e-4, atol_frac=2e-6)
